// tlq_gravity.cu -- self-gravity: the reference's MultiGrid
// (source/sources.f90:99-485) and its multipole boundary values (:531-787)
// on the GPU, run before each stage like Godunov's (HLLC.f90:15-24):
// MultiGrid on the density of the step's U, PHIT = PHIP + PHI, and the
// stage's source term from PHIT.
//
// The mesh is a cube of N = 2^L cells (the reference's lvlm = size); level l
// holds n = N/2^l cells and three arrays (the error E, the residue R and the
// scratch T of the reference's Error/Residue/ret), each (n+2)^3 doubles with
// one ghost layer, index i + (n+2) (j + (n+2) k), i in 0..n+1 -- the layout
// of the reference's level arrays and of phi(0:nx+1, ...).
//
// The smoother is the reference's, in its order.  Its two half-sweeps split
// the cells by k parity and s(i, j) = [i even and j odd] (the reference's
// parity test states that one condition twice), so within a half-sweep a
// cell with s = 0 reads the new value of its x neighbour in rows of even j
// and of its y neighbour in columns of odd i: a Gauss-Seidel order along i
// and j.  A block walks a plane's anti-diagonals i + j = d in order, and
// every other neighbour (east, north, the k planes, the source) still holds
// its value from before the half-sweep.  A relax's ten half-sweeps run in one
// cooperative launch, skewed by a few diagonals per half-sweep
// (k_mg_relax_plane, up to 128 cells: the plane in shared memory, values
// tagged with their half-sweep exchanged between planes; k_mg_relax_pipe,
// above: from the level arrays, each plane's block checking its neighbour
// planes' progress; k_mg_half, one launch per half-sweep, where the planes
// cannot all be resident).  With the order kept and FP64 without contraction, every
// level is bit-identical to a sequential restatement; only the stopping
// test's sum |dphi| is summed in another order (it decides only whether the
// next V-cycle runs).
//
// The reference's loop test (Dif > 10 and fewer than 31 cycles) runs on the
// device, so the solve needs no host round trip: in a CUDA graph the
// V-cycles are the body of a while node whose condition that test sets; run
// directly, up to 31 cycle slots whose launches return once the test failed.  Levels of at most 8 cells run inside one block (one
// launch per cycle).
//
// Built with -fmad=false (FP64 as the restatement evaluates it).
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <string>

#include "tlq_convert.cuh"
#include "tlq_ctx.h"
#include "tlq_mg_wait.cuh"

namespace tlq {
namespace {

constexpr int MG_MAXL = 11;         // levels 0..10: meshes up to 1024^3
constexpr int MG_COARSE_N = 8;      // levels of at most this many cells run in the one-block kernel
constexpr int MG_CYCLES = 31;       // the reference's V-cycle cap (sources.f90:140)
constexpr int MG_PF = 4;            // diagonal steps the smoother's loads run ahead
constexpr int MG_MOM_THREADS = 256;
constexpr int MG_MOM_BLOCKS = 152 * 2;
constexpr int MG_SOLVE_LIMIT = 100000;  // coarsest-level Gauss-Seidel passes before giving up
struct MgLevel {
  int n;
  double* E;
  double* R;
  double* T;   // source(i,j,k)*dxl**2 of the smoother, formed once with R
  void* X;     // the shared-memory relax's exchange between planes (Tagged; null: level too large)
  const void* sched;  // and its schedule (MgSched)
  double dxl;  // (xr - xl) / n (sources.f90:232; x extent for every axis, as there)
};

struct MgCtl {
  int run;     // this MultiGrid call runs (the step runs: t < tfin)
  int active;  // the current V-cycle runs
  int iter;    // V-cycles started
  int status;  // MG_ST_* bits
  double dif;  // the last smoother pass's summed |change| (the reference's Dif)
  double c0[5], cm[5][5], sm[5][5];  // multipole moments (sources.f90:599-681)
  double part[2 * 1024];             // per-plane partial sums of the last pass's |change|
  int abort;                         // a pipelined relax gave up waiting (sticky for the call)
  unsigned call;                     // MultiGrid calls begun (tags of the exchange arrays)
  int prog[1026];                    // pipelined relax: plane k's last finished diagonal, hs*(2n+2) + d
  long long wait_limit;              // polls of a neighbour's progress before giving up (set at allocation)
};

__host__ __device__ __forceinline__ long long mgi(int n, int i, int j, int k) {
  return (long long)i + (long long)(n + 2) * ((long long)j + (long long)(n + 2) * (long long)k);
}

// Where the density of the step's state is read (U(1, 0:nx+1, ...)).
struct DensSoA {
  const double* U;
  Layout L;
  __device__ double operator()(int i, int j, int k) const { return U[L.at(i, j, k)]; }
};
struct DensAoS {
  const double* U;
  Aos A;
  __device__ double operator()(int i, int j, int k) const { return U[A.at(i, j, k)]; }
};

// ---------------------------------------------------------------------------
// Multipole boundary values (sources.f90:9-96, 558-787)
// ---------------------------------------------------------------------------
__device__ double legendre(double x, int l) {
  const double x2 = x * x;
  switch (l) {
    case 0: return 1.0;
    case 1: return x;
    case 2: return 0.5 * (3.0 * x2 - 1.0);
    case 3: return 0.5 * (5.0 * (x2 * x) - 3.0 * x);
    default: return (1.0 / 8.0) * ((35.0 * (x2 * x2) - 30.0 * x2) + 3.0);
  }
}

// aLegendre with its (1 - x^2)^(1/2) and ^(3/2) as square roots (the
// reference raises to the real powers 1/2 and 3/2; equal up to rounding).
// |x| <= 1 here (x = z/r with r >= |z| in rounded arithmetic), so 1 - x^2 >= 0.
__device__ double alegendre(double x, int l, int m) {
  const double x2 = x * x, s = 1.0 - x2, q = sf::sqrt_rn(s);
  switch (l) {
    case 0: return 1.0;
    case 1: return m == 0 ? x : -q;
    case 2:
      if (m == 0) return 0.50 * (3.0 * x2 - 1.0);
      if (m == 1) return -(3.0 * x * q);
      return 3.0 * s;
    case 3:
      if (m == 0) return 0.50 * (5.0 * (x2 * x) - 3.0 * x);
      if (m == 1) return 1.5 * (1.0 - 5.0 * x2) * q;
      if (m == 2) return 15.0 * x * s;
      return -(15.0 * (s * q));
    default:
      if (m == 0) return (1.0 / 8.0) * ((35.0 * (x2 * x2) - 30.0 * x2) + 3.0);
      if (m == 1) return -(2.5 * (7.0 * (x2 * x) - 3.0 * x) * q);
      if (m == 2) return 7.5 * (7.0 * x2 - 1.0) * s;
      if (m == 3) return -(105.0 * x * (s * q));
      return 105.0 * (s * s);
  }
}

// The spherical quantities of the multipole terms at the centre of cell
// (i, j, k) (pangle, aangle, distance; one rank), by algebra instead of the
// reference's transcendental round trips: cos(theta) = z/r (it forms
// cos(acos(z/r))), and cos(m phi), sin(m phi) from cos phi = x/rho, sin phi
// = y/rho, rho = |(x, y)|, by the Chebyshev recurrence (it takes cos and sin
// of m atan2(y, x)).  Equal up to rounding; on the FP64 pipe these are a few
// operations instead of eleven transcendental functions per cell, the roots
// and divisions on the integer pipe beside them.
struct Sph {
  double coth, r, c[5], s[5];
};
__device__ Sph sph_terms(const Params& p, int i, int j, int k) {
  const double x = (p.xl + p.dx * (double)i) - p.dx / 2.0;
  const double y = (p.yl + p.dy * (double)j) - p.dy / 2.0;
  const double z = (p.zl + p.dz * (double)k) - p.dz / 2.0;
  Sph o;
  const double rho2 = x * x + y * y;
  o.r = sf::sqrt_rn(rho2 + z * z);
  o.coth = sf::div(z, o.r);
  const double rho = sf::sqrt_rn(rho2);
  const double c1 = rho > 0.0 ? sf::div(x, rho) : 1.0, s1 = rho > 0.0 ? sf::div(y, rho) : 0.0;
  o.c[0] = 1.0;
  o.s[0] = 0.0;
  o.c[1] = c1;
  o.s[1] = s1;
#pragma unroll
  for (int m = 2; m <= 4; ++m) {
    o.c[m] = 2.0 * c1 * o.c[m - 1] - o.c[m - 2];
    o.s[m] = 2.0 * c1 * o.s[m - 1] - o.s[m - 2];
  }
  return o;
}

// 25 sums per block: c0 l = 0..4, then cm and sm for l = 1..4, m = 1..l.
// FP64 pipe (128^3: 765 us with the roots and divisions on it, 586 without).
template <class Dens>
__global__ void __launch_bounds__(MG_MOM_THREADS) k_mg_moments(const MgCtl* c, const Clock* clk, Params p, Dens rho,
                                                             double* part) {
  __shared__ double red[MG_MOM_THREADS / 32][25];
  if (!c->run || clk->it % 10 != 0) return;
  const int n = p.nx;
  const double vol = p.dx, vy = p.dy, vz = p.dz;
  double acc[25];
#pragma unroll
  for (int q = 0; q < 25; ++q) acc[q] = 0.0;
  const long long cells = (long long)n * n * n;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < cells;
       q += (long long)gridDim.x * blockDim.x) {
    const int i = 1 + (int)(q % n), j = 1 + (int)((q / n) % n), k = 1 + (int)(q / ((long long)n * n));
    const Sph sp = sph_terms(p, i, j, k);
    const double coth = sp.coth, r = sp.r;
    // the cell's mass once (the reference multiplies rho dx dy dz into every
    // term; the order of the products only changes the rounding)
    const double dm = rho(i, j, k) * vol * vy * vz;
    acc[0] += dm;  // Legendre(.,0) r**0 = 1
    int slot = 5;
    double rl = 1.0;
#pragma unroll
    for (int l = 1; l <= 4; ++l) {
      rl = rl * r;
      const double w = rl * dm;
      acc[l] += legendre(coth, l) * w;
#pragma unroll
      for (int m = 1; m <= l; ++m, ++slot) {
        const double t = alegendre(coth, l, m) * w;
        acc[slot] += t * sp.c[m];
        acc[slot + 10] += t * sp.s[m];
      }
    }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 25; ++q) {
    double v = acc[q];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[w][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < 25) {
    double v = 0.0;
    for (int q = 0; q < MG_MOM_THREADS / 32; ++q) v += red[q][threadIdx.x];
    part[blockIdx.x * 25 + threadIdx.x] = v;
  }
}

// The moments from the blocks' sums, a warp per moment.
__global__ void __launch_bounds__(25 * 32) k_mg_moments_final(MgCtl* c, const Clock* clk, const double* part,
                                                            int nblocks) {
  // slots 5..14 (cm) and 15..24 (sm): (l, m) = (1,1) (2,1) (2,2) (3,1) .. (4,4)
  constexpr int LS[10] = {1, 2, 2, 3, 3, 3, 4, 4, 4, 4}, MS[10] = {1, 1, 2, 1, 2, 3, 1, 2, 3, 4};
  if (!c->run || clk->it % 10 != 0) return;
  const int q = threadIdx.x / 32;
  double v = 0.0;
  for (int b = threadIdx.x % 32; b < nblocks; b += 32) v += part[b * 25 + q];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (threadIdx.x % 32) return;
  if (q < 5) {
    c->c0[q] = v;
    return;
  }
  const int r = q < 15 ? q - 5 : q - 15, l = LS[r], m = MS[r];
  double cf = 2.0;  // 2 (l - m)! / (l + m)!
  for (int f = l - m + 1; f <= l + m; ++f) cf = cf / (double)f;
  if (q < 15)
    c->cm[l][m] = cf * v;
  else
    c->sm[l][m] = cf * v;
}

// phi_x/y/zboundaries: the six faces' ghost cells (edges untouched).
__global__ void k_mg_faces(const MgCtl* c, const Clock* clk, Params p, double* phi) {
  if (!c->run || clk->it % 10 != 0) return;
  const int n = p.nx;
  const long long per = (long long)n * n;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < 6 * per;
       q += (long long)gridDim.x * blockDim.x) {
    const int f = (int)(q / per);
    const int a = 1 + (int)((q % per) / n), b = 1 + (int)(q % n);
    const int bnd = (f & 1) ? n + 1 : 0;
    int i, j, k;
    if (f < 2) { i = bnd; j = a; k = b; }
    else if (f < 4) { i = a; j = bnd; k = b; }
    else { i = a; j = b; k = bnd; }
    const Sph sp = sph_terms(p, i, j, k);
    const double coth = sp.coth, rb = sp.r;
    double v = sf::div(-c->c0[0], rb), rp = rb;
#pragma unroll
    for (int l = 1; l <= 4; ++l) {  // (degree l's terms over r**(l+1) at once)
      rp = rp * rb;
      double t = c->c0[l] * legendre(coth, l);
#pragma unroll
      for (int m = 1; m <= l; ++m)
        t = t + 2.0 * (c->cm[l][m] * sp.c[m] + c->sm[l][m] * sp.s[m]) * alegendre(coth, l, m);
      v = v - sf::div(t, rp);
    }
    phi[mgi(n, i, j, k)] = 6.67430e-8 * v;
  }
}

// ---------------------------------------------------------------------------
// Cycle control
// ---------------------------------------------------------------------------
// The loop test of the V-cycles (sources.f90:140): another cycle while
// Dif > 10 and fewer than 31 ran.  As the condition of a graph's loop node
// where the V-cycles are the body of one (loop), so that cycles after
// convergence are not launched at all.
__device__ void mg_loop_test(MgCtl* c, bool loop, cudaGraphConditionalHandle h) {
  const int go = c->run && c->dif > 10.0 && c->iter < MG_CYCLES;
  c->active = go;
  if (go) c->iter = c->iter + 1;
  if (loop) cudaGraphSetConditional(h, go ? 1u : 0u);
}

__global__ void k_mg_begin(MgCtl* c, const Clock* clk, bool loop, cudaGraphConditionalHandle h) {
  c->run = clk->t < clk->tfin;  // the loop test of mainHD.f90:61 (the step's)
  c->iter = 0;
  c->dif = 1.e28;
  c->abort = 0;
  c->call = c->call + 1u;
  mg_loop_test(c, loop, h);
}

// One warp: Dif from the planes' sums (256 of them on 128 cells: 19 us as
// one thread's chain of FP64 additions), and the next loop test.
__global__ void k_mg_cycle_end(MgCtl* c, int nparts, bool loop, cudaGraphConditionalHandle h) {
  if (!c->active) return;
  double v = 0.0;
  for (int q = threadIdx.x; q < nparts; q += 32) v += c->part[q];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (threadIdx.x) return;
  c->dif = v;
  mg_loop_test(c, loop, h);
}

// Residue(0) = 4 pi G dens, Error(0) = phi (sources.f90:136-137).
template <class Dens>
__global__ void k_mg_init(const MgCtl* c, Dens rho, int n, const double* phi, double* E0, double* R0, double* T0,
                          double dxl) {
  if (!c->run) return;
  const long long cells = (long long)(n + 2) * (n + 2) * (n + 2);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < cells;
       q += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(q % (n + 2)), j = (int)((q / (n + 2)) % (n + 2)), k = (int)(q / ((long long)(n + 2) * (n + 2)));
    const double r = 4.0 * 3.14159265358979 * 6.67430e-8 * rho(i, j, k);
    R0[q] = r;
    T0[q] = r * (dxl * dxl);
    E0[q] = phi[q];
  }
}

// phi = Error(0) (sources.f90:189); PHIT = PHIP + PHI into the stage's
// potential plane (HLLC.f90:22).
// A solve that gave up (a bounded wait or the coarsest solve) marks the
// step's status as timed out.
__global__ void k_mg_end(const MgCtl* c, Clock* clk, int n, const double* E0, double* phig, const double* phip,
                         double* phit, float* phitf, Layout L) {
  if (!c->run) return;
  if (blockIdx.x == 0 && threadIdx.x == 0 && c->status) atomicOr(&clk->status, ST_TIMEOUT);
  const long long cells = (long long)(n + 2) * (n + 2) * (n + 2);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < cells;
       q += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(q % (n + 2)), j = (int)((q / (n + 2)) % (n + 2)), k = (int)(q / ((long long)(n + 2) * (n + 2)));
    const double v = E0[q];
    phig[q] = v;
    if (phit) {
      const long long o = L.at(i, j, k);
      const double pt = phip[o] + v;
      phit[o] = pt;
      if (phitf) phitf[o] = d2f(pt);  // the mixed form's stages read it in FP32
    }
  }
}

// ---------------------------------------------------------------------------
// Level operators
// ---------------------------------------------------------------------------
// One smoother update (sources.f90:378-379, 447-449), sdx = source*dxl**2.
// The reference's tail ((1/6) a) w + (1-w) old with w = 1 equals (1/6) a
// bit for bit unless that is a signed zero or old is not finite (then the
// 0*old term can change the sign or give a NaN): those take the literal
// expression, every other update saves its three FP64 operations (the FP64
// pipe bounds the smoother).  SOFT: the product on the integer pipe, where
// the FP64 pipe is the limit (64 and 128 cells: 1 and 3 % of a step).
// (mg_tail is a call: inlined, its three operations ran for every update and
// their result was dropped, 10 warp instructions of the FP64 pipe for 7.)
__device__ __noinline__ double mg_tail(double v, double old) {
  const double w = 1.0;
  return v * w + (1.0 - w) * old;
}
template <bool SOFT = false>
__device__ __forceinline__ double mg_new(double east, double west, double north, double south, double up, double down,
                                         double sdx, double old) {
  double a = east + west;
  a = a + north;
  a = a + south;
  a = a + up;
  a = a + down;
  a = a - sdx;
  double v = SOFT ? sf::mul(1.0 / 6.0, a) : (1.0 / 6.0) * a;
  const long long vb = __double_as_longlong(v), ob = __double_as_longlong(old);
  if ((vb & 0x7fffffffffffffffLL) == 0 || ((ob >> 52) & 0x7ff) == 0x7ff) v = mg_tail(v, old);
  return v;
}

// Cells (i even, j odd) of plane k: none of them shares a face with another,
// so they update in any order (threads t of nt share them).
template <bool TRACK>
__device__ double mg_parallel_plane(const MgLevel& lv, int k, int t, int nt) {
  const int n = lv.n, h = n / 2;
  double acc = 0.0;
  for (int q = t; q < h * h; q += nt) {
    const int i = 2 * (q % h + 1), j = 2 * (q / h) + 1;
    const long long o = mgi(n, i, j, k), s1 = n + 2, s2 = (long long)(n + 2) * (n + 2);
    const double old = lv.E[o];
    const double v = mg_new(lv.E[o + 1], lv.E[o - 1], lv.E[o + s1], lv.E[o - s1], lv.E[o + s2], lv.E[o - s2], lv.T[o],
                            old);
    lv.E[o] = v;
    if (TRACK) acc += fabs(v - old);
  }
  return acc;
}

// The other cells of plane k (s = 0) in the reference's order: anti-diagonal
// d = i + j after anti-diagonal, thread i of the plane's group.  West (i-1,
// j) and south (i, j-1) lie on diagonal d-1: south is this thread's own last
// value, west its neighbour's (pub, double-buffered by diagonal parity).
// The loads of the other neighbours run MG_PF diagonals ahead.  Every thread
// of the block calls this with the same n (uniform barriers); i > n idles.
template <bool TRACK>
__device__ double mg_wave_plane(const MgLevel& lv, int k, int i, double* pub) {
  const int n = lv.n;
  const long long s1 = n + 2, s2 = (long long)(n + 2) * (n + 2);
  double* __restrict__ E = lv.E;
  const double* __restrict__ R = lv.T;
  double rc[MG_PF], re[MG_PF], rn[MG_PF], ru[MG_PF], rd[MG_PF], rs[MG_PF];
  const bool col = i >= 1 && i <= n;
#pragma unroll
  for (int q = 0; q < MG_PF; ++q) {
    const int j = 2 + q - i;
    if (col && j >= 1 && j <= n) {
      const long long o = mgi(n, i, j, k);
      rc[q] = E[o]; re[q] = E[o + 1]; rn[q] = E[o + s1]; ru[q] = E[o + s2]; rd[q] = E[o - s2]; rs[q] = R[o];
    }
  }
  double prev = 0.0, acc = 0.0;
  for (int d0 = 2; d0 <= 2 * n; d0 += MG_PF) {
#pragma unroll
    for (int q = 0; q < MG_PF; ++q) {
      const int d = d0 + q;
      if (d <= 2 * n) {
        const int j = d - i;
        if (col && j >= 1 && j <= n) {
          const long long o = mgi(n, i, j, k);
          const double west = i == 1 ? E[o - 1] : pub[((d - 1) & 1) * (n + 1) + i - 1];
          const double south = j == 1 ? E[o - s1] : prev;
          const double old = rc[q];
          double cur = old;
          if ((i & 1) || !(j & 1)) {  // s = 0: this half-sweep's cell
            cur = mg_new(re[q], west, rn[q], south, ru[q], rd[q], rs[q], old);
            E[o] = cur;
            if (TRACK) acc += fabs(cur - old);
          }
          pub[(d & 1) * (n + 1) + i] = cur;
          prev = cur;
        }
        const int jn = d + MG_PF - i;  // this slot's next diagonal
        if (col && jn >= 1 && jn <= n) {
          const long long o = mgi(n, i, jn, k);
          rc[q] = E[o]; re[q] = E[o + 1]; rn[q] = E[o + s1]; ru[q] = E[o + s2]; rd[q] = E[o - s2]; rs[q] = R[o];
        }
        __syncthreads();
      }
    }
  }
  return acc;
}

// Sum over the block (blockDim.x a multiple of 32), in a fixed order; the
// result in thread 0.
__device__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += red[q];
  return s;
}

// One half-sweep of a level above MG_COARSE_N cells: block b = plane k = b+1
// (n threads).  half 0: cells with k parity = s; half 1: the others
// (sources.f90:438-452 and :456-468).  part: where the plane's summed
// |change| goes (null: not needed).
template <int NT, bool TRACK>
__global__ void __launch_bounds__(NT) k_mg_half(const MgCtl* c, MgLevel lv, int half, double* part) {
  __shared__ double pub[2 * 1025];
  __shared__ double red[32];
  if (!c->active) return;
  const int k = blockIdx.x + 1;
  const int sk = (k & 1) ^ half;  // the s of this half-sweep's cells in plane k
  double acc;
  if (sk)
    acc = mg_parallel_plane<TRACK>(lv, k, threadIdx.x, blockDim.x);
  else
    acc = mg_wave_plane<TRACK>(lv, k, threadIdx.x + 1, pub);
  if (TRACK) {
    const double s = block_sum(acc, red);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
  }
}

// ---------------------------------------------------------------------------
// A whole relax (5 passes of 2 half-sweeps) in one cooperative launch: block
// b owns plane k = b+1 through all ten half-sweeps, so the half-sweeps of
// neighbouring planes overlap instead of running one after another.  Plane
// k may start diagonals d0..d1 of half-sweep hs once planes k-1 and k+1 have
// finished diagonal d1+1 of half-sweep hs-1: every value it reads from them
// (the cells (i, j, k+-1), i + j <= d1) then holds its hs-1 value, and every
// cell of theirs that reads one of plane k's cells it is about to change
// (the same (i, j)) has read it.  The waits are bounded; a block that gives
// up sets the status and the abort flag and every block leaves.  Values of
// other planes are loaded around L1 (ld.global.cg: L1 is not coherent
// between the SMs of one launch).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double ldcg(const double* p) { return __ldcg(p); }

// Thread 0 waits until planes k-1, k+1 (those in 1..n) reach `need`; false
// when it gave up (the block then leaves the relax).
__device__ bool mg_wait(MgCtl* c, int k, int n, int need, int* s_ok) {
  if (threadIdx.x == 0) {
    int ok = 1;
    volatile int* prog = c->prog;
    for (int nb = k - 1; nb <= k + 1 && ok; nb += 2) {
      if (nb < 1 || nb > n) continue;
      MgWait wait;
      while (prog[nb] < need) {
        if (wait.out(c)) {
          ok = 0;
          break;
        }
        __nanosleep(64);
      }
    }
    if (!ok) {
      atomicOr(&c->status, MG_ST_TIMEOUT);
      atomicExch(&c->abort, 1);
    }
    __threadfence();
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

__device__ __forceinline__ void mg_publish(MgCtl* c, int k, int value) {
  __syncthreads();  // every thread's stores of the chunk are issued
  if (threadIdx.x == 0) {
    __threadfence();
    atomicExch(&c->prog[k], value);
  }
}

// Time step t of a block processes diagonal d = t - SKEW hs of every
// half-sweep hs at once: a cell of half-sweep hs reads its own plane's
// cells of half-sweep hs-1 on diagonals d-1..d+1 (processed SKEW-1 steps or
// more earlier) and its neighbour planes' cells of hs-1 on diagonal d
// (their step t + 1 - SKEW), so the ten half-sweeps of a relax take
// 2n + 9 SKEW steps instead of 20n.  A plane checks its neighbours once per
// CH steps, which SKEW = CH + 1 allows.

size_t pipe_smem(int n) { return (size_t)10 * 2 * (n + 1) * sizeof(double); }

// NT threads at most, MINB blocks per SM at least, neighbour checks every
// CH steps; the block is n x HG threads: thread t works on one column for the
// K = 10/HG half-sweeps g K .. g K + K-1 of group g = t / n (more warps per
// plane to hide the FP64 latency), loading G of them at a time.  Columns by
// parity: the first n/2 threads of a group take the odd columns, the others
// the even ones.  A step's cells that do not change (the other colour's, or
// on an odd diagonal the wave cells of even columns) then fill whole warps
// (n >= 64), which skip the update: the FP64 pipe charges a warp instruction
// the same with 16 active lanes as with 32 (measured on GB300), so this
// saves a third of the smoother's FP64 issue.  The diagonal's values in
// shared memory are laid out by thread, odd columns first (pslot).
template <int NT, int MINB, int HG, int G, int CH, bool TRACK>
__global__ void __launch_bounds__(NT, MINB) k_mg_relax_pipe(MgCtl* c, MgLevel lv, double* part) {
  constexpr int K = 10 / HG;
  constexpr int SKEW = CH + 1;  // steps between consecutive half-sweeps: a neighbour check per CH steps
  static_assert(K * HG == 10, "HG divides the ten half-sweeps");
  extern __shared__ double pub[];  // per half-sweep, per diagonal parity: the diagonal's values by pslot
  __shared__ double red[32];
  __shared__ int s_ok;
  if (!c->active) return;
  const int n = lv.n, k = blockIdx.x + 1;
  // threads past n x HG (whole warps) only take part in the barriers
  const bool live = (int)threadIdx.x < n * HG;
  const int col = (int)(threadIdx.x % n), hn = n >> 1;
  const int i = col < hn ? 2 * col + 1 : 2 * (col - hn) + 2;
  const int h0 = live ? (int)(threadIdx.x / n) * K : 0;
  // slot of column ii in a diagonal's shared-memory values
  auto pslot = [hn](int ii) { return (ii & 1) ? (ii >> 1) : hn + (ii >> 1) - 1; };
  const long long s1 = n + 2, s2 = (long long)(n + 2) * (n + 2);
  double* __restrict__ E = lv.E;
  const double* __restrict__ Sd = lv.T;
  const int tmax = 2 * n + 9 * SKEW;
  double prev[K];
#pragma unroll
  for (int q = 0; q < K; ++q) prev[q] = 0.0;
  double acc8 = 0.0, acc9 = 0.0;
  for (int t0 = 2; t0 <= tmax; t0 += CH) {
    const int t1 = min(t0 + CH - 1, tmax);
    const int need = t1 + 1 - SKEW;  // the neighbours' last step this chunk reads
    if (need >= 2 && !mg_wait(c, k, n, need, &s_ok)) return;
    for (int t = t0; t <= t1; ++t) {
      // The loads of G half-sweeps before their stores: the cells a step
      // reads and the cells it writes lie SKEW diagonals or more apart,
      // so these loads need not wait behind those stores.
#pragma unroll
      for (int g = 0; g < K; g += G) {
      double rc[K], re[K], rn[K], ru[K], rd[K], rs[K], rw[K], rv[K];
#pragma unroll
      for (int q = g; q < (g + G < K ? g + G : K); ++q) {
        const int hs = h0 + q;
        const int d = t - SKEW * hs, j = d - i;
        if (live && d >= 2 && d <= 2 * n && j >= 1 && j <= n) {
          const long long o = mgi(n, i, j, k);
          const bool par = ((k & 1) ^ (hs & 1)) != 0;
          // whether the cell changes in this half-sweep (the wave cells that
          // do not still pass their value on through shared memory)
          const bool upd = par ? (!(i & 1) && (j & 1)) : ((i & 1) || !(j & 1));
          if (upd || !par) rc[q] = E[o];
          if (upd) {
            re[q] = E[o + 1]; rn[q] = E[o + s1];
            ru[q] = ldcg(E + o + s2); rd[q] = ldcg(E + o - s2); rs[q] = Sd[o];
            // west and south from memory: the parallel cells' (other colour,
            // this plane, hs-1) and the ghosts; the wave cells' others come
            // from this half-sweep's previous diagonal
            rw[q] = (par || i == 1) ? E[o - 1] : 0.0;
            rv[q] = (par || j == 1) ? E[o - s1] : 0.0;
          }
        }
      }
#pragma unroll
      for (int q = g; q < (g + G < K ? g + G : K); ++q) {
        const int hs = h0 + q;
        const int d = t - SKEW * hs;
        if (!live || d < 2 || d > 2 * n) continue;  // (uniform within the group)
        const int j = d - i;
        if (j < 1 || j > n) continue;
        const long long o = mgi(n, i, j, k);
        const bool par = ((k & 1) ^ (hs & 1)) != 0;  // cells (i even, j odd) of this plane
        const double old = rc[q];
        if (par) {
          if (!(i & 1) && (j & 1)) {
            const double v = mg_new(re[q], rw[q], rn[q], rv[q], ru[q], rd[q], rs[q], old);
            E[o] = v;
            if (TRACK && hs == 8) acc8 += fabs(v - old);
            if (TRACK && hs == 9) acc9 += fabs(v - old);
          }
        } else {
          double* pb = pub + hs * 2 * (n + 1);
          const double west = i == 1 ? rw[q] : pb[((d - 1) & 1) * (n + 1) + pslot(i - 1)];
          const double south = j == 1 ? rv[q] : prev[q];
          double cur = old;
          if ((i & 1) || !(j & 1)) {
            cur = mg_new(re[q], west, rn[q], south, ru[q], rd[q], rs[q], old);
            E[o] = cur;
            if (TRACK && hs == 8) acc8 += fabs(cur - old);
            if (TRACK && hs == 9) acc9 += fabs(cur - old);
          }
          pb[(d & 1) * (n + 1) + pslot(i)] = cur;
          prev[q] = cur;
        }
      }
      }
      __syncthreads();
    }
    mg_publish(c, k, t1);
  }
  if (TRACK) {
    const double a = block_sum(acc8, red);
    if (threadIdx.x == 0) part[blockIdx.x] = a;
    const double b = block_sum(acc9, red);
    if (threadIdx.x == 0) part[n + blockIdx.x] = b;
  }
}

// ---------------------------------------------------------------------------
// The skewed relax with the block's plane in shared memory (levels of 16 to
// 128 cells: (N+2)^2 doubles, 135 KB at 128).  Only plane k's block writes
// plane k during a relax, so its copy in shared memory is the current one: an
// update reads its old value and its four in-plane neighbours there.  The
// ghost rows and columns do not change during a relax; the level array takes
// the plane back at the end.  Layout: column parity, row, column / 2, so that
// a warp's cells of one diagonal (consecutive columns of one parity) fall on
// distinct banks.
//
// Time step t processes diagonal t - S hs of half-sweep hs, S = MG_SKEW.  In
// half-sweeps 2g and 2g+1 (group g) plane k changes the cells s = 0 (the
// wave) in one and the cells i even, j odd in the other.  S is even, so both
// lie on rows of one parity at any step: an odd column has a wave cell every
// step, an even column a wave cell and one of the other kind in turn.  The
// step's cells of all five groups are dealt to the block's first threads: the
// FP64 pipe charges a warp instruction the same whatever its active lanes
// (a thread per column and group keeps 20 warps of a 128-cell plane busy with
// 9 warps' worth of cells on average).  Which cell a thread has at a step, and
// its offsets, come from a schedule formed once per context (MgSched): worked
// out in the kernel it was most of a step's instructions.
//
// The planes above and below exchange values through X, 16 bytes a cell: the
// value and a tag that names this relax and the half-sweep which formed it
// (the values from before the relax, the ghost planes' among them, have the
// tag MG_INITIAL), written and read in one 128-bit access.  A reader uses a
// value when its tag is the one it needs, else loads again (a bounded number
// of times): no fence, no flag, no block-wide poll.  The value cannot be overwritten early: the neighbour's
// next update of that cell needs this plane's.  X is laid out by diagonal, so
// a warp's cells are contiguous.
//
// Half as many helper threads as there are cells run ahead of the workers:
// during step t they check the values that step t + 1 needs (loaded during
// step t - 1), leave them in shared memory with the source, and issue the
// loads of step t + 2.  The workers only read shared memory: with loads, tag
// checks and address arithmetic in their path a step took 1,600 cycles,
// of which the update's seven dependent FP64 operations are 570.
//
// What bounds a step: those operations and the barrier; on 128 cells the
// FP64 pipe.  Measured per launch on the 128^3 cloud (ncu), against a thread
// per column and group with loads one step ahead and a fence and a poll by
// the whole block every few steps: 128 cells 743 -> 380 us, 64: 260 -> 130,
// 32: 143 -> 65, 16: 98 -> 43; with mg_tail's operations out of every update
// 316, 115, 62 and 41.
// ---------------------------------------------------------------------------
constexpr int MG_SKEW = 4;  // (6: 4 % slower, 2 more steps per half-sweep; 2 leaves a value no time to arrive)
constexpr unsigned MG_INITIAL = 15;

template <int N>
struct PlaneGeo {
  static constexpr int NT = (5 * N + 31) / 32 * 32;       // workers: the most cells of a step, whole warps
  static constexpr int NH = (NT / 2 + 31) / 32 * 32;      // helpers, two cells each
  static constexpr int R = N / 2 + 1, PS = (N + 2) * R;
  static constexpr int STEPS = (2 * N + 9 * MG_SKEW) / 2 * 2;  // t = 2 .. 2N + 9 S (an even number of steps)
  static constexpr int ROWS = STEPS + 4;                       // and those the helpers look ahead to
  // the plane, and two steps' values from above, below and the source per worker
  static constexpr size_t smem = ((size_t)(N + 2) * (N + 2) + 2 * 3 * (size_t)NT) * sizeof(double);
};
// Cells of a level's exchange array: planes 0..N+1 of diagonals 0..2N+1 by column.
bool exch_level(int n) { return n > MG_COARSE_N && n <= 128; }
long long exch_cells(int n) { return (long long)(n + 2) * (2 * n + 2) * n; }

using Tagged = unsigned __int128;  // the double's bits, the tag above them
__device__ __forceinline__ double tagged_value(Tagged r) { return __longlong_as_double((long long)r); }
__device__ __forceinline__ unsigned long long tagged_tag(Tagged r) { return (unsigned long long)(r >> 64); }
// Loaded where `take`; asynchronous: nothing here waits for the value.
__device__ __forceinline__ void ld_tagged(Tagged& r, const Tagged* p, bool take) {
  asm volatile(
      "{\n\t.reg .pred t;\n\tsetp.ne.b32 t, %2, 0;\n\t@t ld.relaxed.gpu.global.b128 %0, [%1];\n\t}"
      : "+q"(r)
      : "l"(p), "r"((int)take)
      : "memory");
}
__device__ __forceinline__ void st_tagged(Tagged* p, double v, unsigned long long tag) {
  const Tagged r = (Tagged)tag << 64 | (unsigned long long)__double_as_longlong(v);
  asm volatile("st.relaxed.gpu.global.b128 [%0], %1;" ::"l"(p), "q"(r) : "memory");
}
__device__ __forceinline__ void ld_pred(double& r, const double* p, bool take) {
  asm volatile("{\n\t.reg .pred t;\n\tsetp.ne.b32 t, %2, 0;\n\t@t ld.global.f64 %0, [%1];\n\t}"
               : "+d"(r)
               : "l"(p), "r"((int)take));
}

// One entry of a level's schedule, [plane parity][step - 2][thread]: the
// cell's offset in the shared plane and its half-sweep, its offsets in a
// plane of X and of the level arrays; og = 0: no cell.
struct alignas(8) MgSched {
  unsigned short o, hs, x, og;
};
long long sched_entries(int n) {  // per plane parity
  const long long rows = (2 * n + 9 * MG_SKEW) / 2 * 2 + 4, nt = (5 * n + 31) / 32 * 32;  // PlaneGeo's
  return rows * nt;
}
__host__ __device__ __forceinline__ int mg_xcol(int n, int i) { return (i & 1) ? i >> 1 : n / 2 + (i >> 1) - 1; }

// The schedule of an n-cell level: one thread per entry.  Group g's own time
// is t - 2 S g; its wave's diagonal there holds the odd columns lo..hi, and
// the even columns' turn (the wave's on even steps) the even ones.
__global__ void k_mg_sched(int n, MgSched* out, int rows, int nt) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (q >= 2LL * rows * nt) return;
  const int f0 = (int)(q % nt), t = 2 + (int)((q / nt) % rows), kp = (int)(q / ((long long)rows * nt));
  MgSched e = {0, 0, 0, 0};
  int f = f0;
  for (int g = 0; g < 5; ++g) {
    const int tau = t - 2 * MG_SKEW * g;
    const int dw = tau - MG_SKEW * kp, d = (tau & 1) ? tau - MG_SKEW * (1 - kp) : dw;
    const int lo = max(1, dw - n) | 1, hi = min(n, dw - 1), le = (max(2, d - n) + 1) & ~1, he = min(n, d - 1);
    const int no = hi >= lo ? (hi - lo) / 2 + 1 : 0, ne = he >= le ? (he - le) / 2 + 1 : 0;
    if (f < no + ne) {
      const bool odd = f < no;
      const int i = odd ? lo + 2 * f : le + 2 * (f - no);
      const int hs = 2 * g + ((odd || !(t & 1)) ? kp : 1 - kp), j = t - MG_SKEW * hs - i;
      e.o = (unsigned short)(((i & 1) * (n + 2) + j) * (n / 2 + 1) + (i >> 1));
      e.hs = (unsigned short)hs;
      e.x = (unsigned short)((i + j) * n + mg_xcol(n, i));
      e.og = (unsigned short)(i + (n + 2) * j);
      break;
    }
    f -= no + ne;
  }
  out[q] = e;
}

// The last pass's |change|.  (A call or an expression: the tracked relax of
// 128 cells takes 345 us both ways, the untracked one 316.)
__device__ __noinline__ double mg_change(double acc, double v, double old) { return acc + fabs(v - old); }

template <int N, bool TRACK>
__global__ void __launch_bounds__(PlaneGeo<N>::NT + PlaneGeo<N>::NH, 1)
    k_mg_relax_plane(MgCtl* c, MgLevel lv, int leg, double* part) {
  using G = PlaneGeo<N>;
  constexpr int R = G::R, PS = G::PS, NT = G::NT, NH = G::NH;
  constexpr int s1 = N + 2, s2 = (N + 2) * (N + 2);
  constexpr int XP = (2 * N + 2) * N;  // X: plane stride
  static_assert(MG_SKEW % 2 == 0, "rows of one parity per step");
  static_assert(XP <= 65536 && s2 <= 65536, "schedule entries of 16 bits");
  extern __shared__ double P[];
  __shared__ double red[32];
  __shared__ int s_gave_up[2];  // by parity of a pair of steps: set in the pair, read after it
  if (!c->active) return;
  double* const B = P + s2;  // [step parity][above, below, source][worker]
  const int k = blockIdx.x + 1, tid = threadIdx.x;
  double* __restrict__ E = lv.E + (long long)s2 * k;
  Tagged* X = static_cast<Tagged*>(lv.X) + (long long)XP * k;
  const uint2* __restrict__ sched =
      reinterpret_cast<const uint2*>(static_cast<const MgSched*>(lv.sched)) + (long long)(k & 1) * G::ROWS * NT;
  const unsigned long long seq = (unsigned long long)(c->call * 64u + 2u * (unsigned)c->iter + (unsigned)leg) << 4;
  // the plane into shared memory and, tagged, into X; the ghost planes by
  // their neighbours' blocks
  for (int j = tid / 32; j < N + 2; j += (NT + NH) / 32)
    for (int i = tid % 32; i < N + 2; i += 32) {
      const int o = i + s1 * j;
      const double v = E[o];
      P[((i & 1) * (N + 2) + j) * R + (i >> 1)] = v;
      if (i >= 1 && i <= N && j >= 1 && j <= N) {
        const int x = (i + j) * N + mg_xcol(N, i);
        st_tagged(X + x, v, seq | MG_INITIAL);
        if (k == 1) st_tagged(X - XP + x, E[o - s2], seq | MG_INITIAL);
        if (k == N) st_tagged(X + XP + x, E[o + s2], seq | MG_INITIAL);
      }
    }
  if (tid < 2) s_gave_up[tid] = 0;
  double acc = 0.0;
  if (tid < NT) {
    // ---- workers: one cell a step ------------------------------------------
    sched += tid;
    uint2 m = __ldg(sched), next = __ldg(sched + NT);  // (x: o | hs << 16, y: x | og << 16)
    sched += 2 * NT;
    __syncthreads();
    __syncthreads();  // step 2's values
    for (int t0 = 2; t0 < 2 + G::STEPS; t0 += 2) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {  // step t0 + q
        if (m.y != 0u) {
          const int o = (int)(m.x & 0xffffu);
          double* pc = P + o;
          // east and west lie in the other parity's half
          const double* pe = pc + (o >= PS ? 1 - PS : PS);
          const double* b = B + q * 3 * NT + tid;
          const double old = pc[0];
          const double v = mg_new<(N >= 64)>(pe[0], pe[-1], pc[R], pc[-R], b[0], b[NT], b[2 * NT], old);
          pc[0] = v;
          st_tagged(X + (m.y & 0xffffu), v, seq | (m.x >> 16));
          if (TRACK) {
            if ((m.x >> 16) >= 8u) acc = mg_change(acc, v, old);  // the last pass
          }
        }
        m = next;
        next = __ldg(sched);
        sched += NT;
        __syncthreads();
      }
      if (*(volatile int*)&s_gave_up[(t0 >> 1) & 1]) return;
    }
  } else {
    // ---- helpers: two cells each -------------------------------------------
    const double* __restrict__ Sd = lv.T + (long long)s2 * k;
    const int h = tid - NT;
    const bool two = h + NH < NT, top = k == N, bottom = k == 1;
    sched += h;
    uint2 cell[2], ahead[2];  // the entries of the step whose loads are in flight, and of the one after
    Tagged ru[2] = {0, 0}, rd[2] = {0, 0};
    double rs[2] = {0.0, 0.0};
    auto entries = [&](uint2* e) {
      e[0] = __ldg(sched);
      e[1] = two ? __ldg(sched + NH) : make_uint2(0u, 0u);
      sched += NT;
    };
    auto fetch = [&]() {
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const Tagged* x = X + (cell[w].y & 0xffffu);
        ld_tagged(ru[w], x + XP, cell[w].y != 0u);
        ld_tagged(rd[w], x - XP, cell[w].y != 0u);
        ld_pred(rs[w], Sd + (cell[w].y >> 16), cell[w].y != 0u);
      }
    };
    // the values in flight, checked, into slot s of B
    auto deliver = [&](int s, int* gave_up) {
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        if (cell[w].y == 0u) continue;
        const unsigned hs = cell[w].x >> 16, prev = hs == 0u ? MG_INITIAL : hs - 1u;
        const unsigned long long wu = seq | (top ? MG_INITIAL : prev), wd = seq | (bottom ? MG_INITIAL : prev);
        const Tagged* x = X + (cell[w].y & 0xffffu);
        MgWait wait;
        while (tagged_tag(ru[w]) != wu || tagged_tag(rd[w]) != wd) {
          if (wait.out(c)) {
            *gave_up = 1;
            atomicOr(&c->status, MG_ST_TIMEOUT);
            atomicExch(&c->abort, 1);
            break;
          }
          ld_tagged(ru[w], x + XP, true);
          ld_tagged(rd[w], x - XP, true);
        }
        double* b = B + s * 3 * NT + h + w * NH;
        b[0] = tagged_value(ru[w]);
        b[NT] = tagged_value(rd[w]);
        b[2 * NT] = rs[w];
      }
    };
    entries(cell);
    entries(ahead);
    __syncthreads();
    fetch();
    deliver(0, &s_gave_up[1]);  // step 2's (t0 = 2: pair parity 1)
    cell[0] = ahead[0];
    cell[1] = ahead[1];
    entries(ahead);
    fetch();
    __syncthreads();
    for (int t0 = 2; t0 < 2 + G::STEPS; t0 += 2) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {  // during step t0 + q
        deliver(q ^ 1, &s_gave_up[(t0 >> 1) & 1]);
        cell[0] = ahead[0];
        cell[1] = ahead[1];
        entries(ahead);
        fetch();
        __syncthreads();
      }
      if (*(volatile int*)&s_gave_up[(t0 >> 1) & 1]) return;
    }
  }
  for (int j = 1 + tid / 32; j <= N; j += (NT + NH) / 32)
    for (int i = 1 + tid % 32; i <= N; i += 32) E[i + s1 * j] = P[((i & 1) * (N + 2) + j) * R + (i >> 1)];
  if (TRACK) {
    const double a = block_sum(acc, red);
    if (tid == 0) {
      part[blockIdx.x] = a;
      part[N + blockIdx.x] = 0.0;  // (where other paths sum the second half-sweep)
    }
  }
}

// Progress of every plane (and its two ghost planes) to "nothing done".
__global__ void k_mg_prog_reset(MgCtl* c, int n) {
  if (!c->active) return;
  for (int q = threadIdx.x; q <= n + 1; q += blockDim.x) c->prog[q] = -1;
}

// A coarse level's error at cell (i, j, k) and, where the cell lies at the
// level's edge, in its ghosts.  The reference sets each face's ghosts to
// -(first interior layer) over the whole face, face after face (sources.f90:
// 262-283, 285-290): whatever the order of the faces, a ghost then holds the
// nearest interior cell's value, negated once per coordinate out of range.
__device__ __forceinline__ void mg_put(double* E, int n, int i, int j, int k, double v) {
  double* p = E + mgi(n, i, j, k);
  if (n == 1) {
    for (int q = 0; q < 27; ++q) E[q] = (q == 13 || ((q % 3 != 1) + (q / 3 % 3 != 1) + (q / 9 != 1)) == 2) ? v : -v;
    return;
  }
  const int s1 = n + 2, s2 = s1 * s1;
  const int x = i == 1 ? -1 : i == n ? 1 : 0, y = j == 1 ? -s1 : j == n ? s1 : 0, z = k == 1 ? -s2 : k == n ? s2 : 0;
  p[0] = v;
  if (x) p[x] = -v;
  if (y) p[y] = -v;
  if (z) p[z] = -v;
  if (x && y) p[x + y] = v;
  if (x && z) p[x + z] = v;
  if (y && z) p[y + z] = v;
  if (x && y && z) p[x + y + z] = -v;
}

// resid on the fine level (sources.f90:196-216) and restriction onto the
// coarse one (:118-137), fused: each coarse cell q forms its 8 children's
// residuals; its own error starts the cycle's way down at 0 (:146-148).
// (The reference's ret array of the fine level is not kept: it is
// overwritten before anything reads it.)  The FP64 pipe bounds it: 8
// operations a fine cell are left on it, the division by dxl**2 and the
// product 6 E run on the integer pipe beside them.  128^3 fine cells: 72 -> 30 us.
__device__ __forceinline__ void mg_resid_restrict(const double* __restrict__ E, const double* __restrict__ Rf, int n,
                                                  double dxl, double* Ec, double* Rc, double* Tc, int q) {
  const int nc = n / 2, s1 = n + 2, s2 = (n + 2) * (n + 2);
  const int i = 1 + q % nc, j = 1 + (q / nc) % nc, k = 1 + q / (nc * nc);
  const long long o0 = mgi(n, 2 * i - 1, 2 * j - 1, 2 * k - 1);
  const double d2 = dxl * dxl;
  auto cell = [&](int di, int dj, int dk) {
    const long long o = o0 + di + s1 * dj + s2 * dk;
    double g = E[o - 1] + E[o + 1];
    g = g + E[o - s1];
    g = g + E[o + s1];
    g = g + E[o - s2];
    g = g + E[o + s2];
    g = sf::div(g - sf::mul(6.0, E[o]), d2);
    return Rf[o] - g;
  };
  double a = cell(0, 0, 0) + cell(1, 0, 0);
  a = a + cell(0, 1, 0);
  a = a + cell(0, 0, 1);
  a = a + cell(1, 1, 0);
  a = a + cell(1, 0, 1);
  a = a + cell(0, 1, 1);
  a = a + cell(1, 1, 1);
  const double r = (1.0 / 8.0) * a, dc = dxl * 2.0;  // (the coarse level's dxl: (xr - xl) / (n/2), exactly twice)
  Rc[mgi(nc, i, j, k)] = r;
  Tc[mgi(nc, i, j, k)] = r * (dc * dc);
  mg_put(Ec, nc, i, j, k, 0.0);
}

__global__ void k_mg_resid_restrict(const MgCtl* c, MgLevel f, MgLevel co) {
  if (!c->active) return;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < co.n * co.n * co.n) mg_resid_restrict(f.E, f.R, f.n, f.dxl, co.E, co.R, co.T, q);
}

// prolongation (sources.f90:139-194), then Error = Error + ret (:181) and,
// on a coarse level (ghosts), the error's ghosts: each coarse cell q serves
// its 8 children, whose sums begin alike (27 V + 9 Vx for four of them, with
// 9 Vy for two): 54 additions and 19 products where 8 separate sums take 64
// and 64, the products on the integer pipe beside the additions, which
// bound it.  The last two operations are one fused one: (1/64) r is exact
// (unless it is subnormal: then as two).  128^3 fine cells: 72 -> 34 us (and
// 12.6 us less per coarse level, the launch that set the ghosts).
__device__ __forceinline__ void mg_prolong_add(const double* __restrict__ V, double* E, int nc, int q, bool ghosts) {
  const int n = 2 * nc;
  const long long s1 = nc + 2, s2 = (long long)(nc + 2) * (nc + 2);
  const int i = 1 + q % nc, j = 1 + (q / nc) % nc, k = 1 + q / (nc * nc);
  const long long o = mgi(nc, i, j, k);
  const double v27 = sf::mul(27.0, V[o]);
  double vy[2], vz[2], vyz[2][2];
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    vy[b] = sf::mul(9.0, V[o + (b ? s1 : -s1)]);
    vz[b] = sf::mul(9.0, V[o + (b ? s2 : -s2)]);
#pragma unroll
    for (int g = 0; g < 2; ++g) vyz[b][g] = sf::mul(3.0, V[o + (b ? s1 : -s1) + (g ? s2 : -s2)]);
  }
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const long long ox = o + (a ? 1 : -1);
    const double ax = v27 + sf::mul(9.0, V[ox]);
    double vxz[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) vxz[g] = sf::mul(3.0, V[ox + (g ? s2 : -s2)]);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const long long oxy = ox + (b ? s1 : -s1);
      const double axy = ax + vy[b], vxy = sf::mul(3.0, V[oxy]);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        double r = axy + vz[g];
        r = r + vxy;
        r = r + vxz[g];
        r = r + vyz[b][g];
        r = r + V[oxy + (g ? s2 : -s2)];
        const int fi = 2 * i - 1 + a, fj = 2 * j - 1 + b, fk = 2 * k - 1 + g;
        const double old = E[mgi(n, fi, fj, fk)];
        const bool small = ((unsigned)__double2hiint(r) & 0x7fffffffu) < 0x00800000u;  // |r| < 2^-1015
        const double v = small ? old + (1.0 / 64.0) * r : fma(1.0 / 64.0, r, old);
        if (ghosts)
          mg_put(E, n, fi, fj, fk, v);
        else
          E[mgi(n, fi, fj, fk)] = v;
      }
    }
  }
}

__global__ void k_mg_prolong_add(const MgCtl* c, MgLevel co, MgLevel f, bool ghosts) {
  if (!c->active) return;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < co.n * co.n * co.n) mg_prolong_add(co.E, f.E, co.n, q, ghosts);
}

// ---------------------------------------------------------------------------
// Levels of at most MG_COARSE_N cells of one V-cycle in one block, in shared
// memory.  A relax's ten half-sweeps overlap as in k_mg_relax_plane, a skew
// of two diagonals apart (a value is there after the step's barrier): step t
// holds the cells of half-sweep hs on diagonal i + j = 2 + t - 2 hs of every
// plane, 2n + 17 steps instead of ten waves of 2n - 1.  The steps' cells lie
// in a table, packed: at most 128 of them on 8 cells, one per thread, so
// that four warps' FP64 operations (8 x 4 x 19 cycles a step) take no longer
// than one cell's chain of eight (8 x 79), which bounds it.  Levels 8 to 1:
// 130 us a cycle (from level arrays, wave after wave: 195 us for 4 to 1
// alone, and 68 us and four launches more for the 8-cell level's relaxes).
// ---------------------------------------------------------------------------
constexpr int MG_CT = 128;
static_assert(MG_CT == 2 * MG_COARSE_N * MG_COARSE_N, "a step's cells, one per thread");

struct alignas(16) MgCoarseSched {
  unsigned short first[3][40];               // per level size (8, 4, 2): the first entry of each step, and the end
  unsigned short cell[(512 + 64 + 8) * 5];   // offset in the level's array; bit 15: the last pass
};

void mg_coarse_sched(MgCoarseSched* s) {
  int at = 0;
  for (int lv = 0; lv < 3; ++lv) {
    const int n = 8 >> lv;
    for (int t = 0; t < 2 * n + 17; ++t) {
      s->first[lv][t] = (unsigned short)at;
      for (int hs = 0; hs < 10; ++hs)
        for (int k = 1; k <= n; ++k)
          for (int i = 1; i <= n; ++i) {
            const int j = 2 + t - 2 * hs - i;
            const bool s1 = !(i & 1) && (j & 1);
            if (j < 1 || j > n || s1 != (((k ^ hs) & 1) == 1)) continue;
            s->cell[at++] = (unsigned short)(mgi(n, i, j, k) | (hs >= 8 ? 0x8000 : 0));
          }
    }
    s->first[lv][2 * n + 17] = (unsigned short)at;
  }
}

struct MgCoarseMem {
  double E[1307], R[1307], T[1307];  // levels of 8, 4, 2 and 1 cells
  MgCoarseSched sched;
};
template <int N>
constexpr int MG_COARSE_AT = N == 8 ? 0 : N == 4 ? 1000 : N == 2 ? 1216 : 1280;

// 5 passes of 2 half-sweeps; returns the thread's part of the last pass's
// |change| (track).
template <int N>
__device__ __forceinline__ double mg_relax_shared(MgCoarseMem& m, bool track) {
  constexpr int LV = N == 8 ? 0 : N == 4 ? 1 : 2, STEPS = 2 * N + 17, s1 = N + 2, s2 = s1 * s1;
  double* E = m.E + MG_COARSE_AT<N>;
  const double* T = m.T + MG_COARSE_AT<N>;
  const unsigned short* first = m.sched.first[LV];
  double acc = 0.0;
  int at = first[0] + (int)threadIdx.x, end = first[1];
  int e = at < end ? m.sched.cell[at] : -1;
  for (int t = 0; t < STEPS; ++t) {
    const int cur = e;
    if (t + 1 < STEPS) {
      at = end + (int)threadIdx.x;
      end = first[t + 2];
      e = at < end ? m.sched.cell[at] : -1;
    }
    if (cur >= 0) {
      double* p = E + (cur & 0x7fff);
      const double old = p[0];
      const double v = mg_new(p[1], p[-1], p[s1], p[-s1], p[s2], p[-s2], T[cur & 0x7fff], old);
      p[0] = v;
      if (track && (cur & 0x8000)) acc += fabs(v - old);
    }
    __syncthreads();
  }
  return acc;
}

// Gauss-Seidel on the coarsest level, one cell, until the change is
// <= 0.001 (sources.f90:337-396); its ghosts are not set anew.
__device__ void mg_solve_shared(MgCoarseMem& m, MgCtl* c) {
  if (threadIdx.x == 0) {
    double* p = m.E + MG_COARSE_AT<1> + 13;
    const double sdx = m.T[MG_COARSE_AT<1> + 13];
    double Dif = 1000.0;
    int passes = 0;
    while (Dif > 0.001) {
      if (++passes > MG_SOLVE_LIMIT) {
        atomicOr(&c->status, MG_ST_SOLVE);
        break;
      }
      const double old = p[0];
      p[0] = mg_new(p[1], p[-1], p[3], p[-3], p[9], p[-9], sdx, old);
      Dif = fabs(p[0] - old);
    }
  }
  __syncthreads();
}

// Levels N .. 1 of one V-cycle: relax, residual + restriction, the levels
// below, prolongation + add, relax.
template <int N>
__device__ __forceinline__ double mg_cycle_shared(MgCoarseMem& m, MgCtl* c, double dxl, bool whole) {
  if constexpr (N == 1) {
    mg_solve_shared(m, c);
    return 0.0;
  } else {
    constexpr int f = MG_COARSE_AT<N>, g = MG_COARSE_AT<N / 2>, CELLS = N * N * N / 8;
    mg_relax_shared<N>(m, false);
    if (threadIdx.x < CELLS)
      mg_resid_restrict(m.E + f, m.R + f, N, dxl, m.E + g, m.R + g, m.T + g, (int)threadIdx.x);
    __syncthreads();
    mg_cycle_shared<N / 2>(m, c, 2.0 * dxl, false);
    if (threadIdx.x < CELLS) mg_prolong_add(m.E + g, m.E + f, N / 2, (int)threadIdx.x, !whole);
    __syncthreads();
    return mg_relax_shared<N>(m, whole);
  }
}

// WHOLE: the mesh itself has N cells; the kernel is the cycle and also forms
// Dif's sum.
template <int N, bool WHOLE>
__global__ void __launch_bounds__(MG_CT) k_mg_coarse(MgCtl* c, MgLevel top, const MgCoarseSched* sched) {
  __shared__ MgCoarseMem m;
  __shared__ double red[32];
  if (!c->active) return;
  constexpr int f = MG_COARSE_AT<N>, CELLS = (N + 2) * (N + 2) * (N + 2);
  for (int q = threadIdx.x; q < (int)(sizeof(MgCoarseSched) / 16); q += MG_CT)
    reinterpret_cast<uint4*>(&m.sched)[q] = reinterpret_cast<const uint4*>(sched)[q];
  for (int q = threadIdx.x; q < CELLS; q += MG_CT) {
    m.E[f + q] = top.E[q];
    m.R[f + q] = top.R[q];
    m.T[f + q] = top.T[q];
  }
  __syncthreads();
  const double acc = mg_cycle_shared<N>(m, c, top.dxl, WHOLE);
  for (int q = threadIdx.x; q < CELLS; q += MG_CT) top.E[q] = m.E[f + q];
  if (WHOLE) {
    const double d = block_sum(acc, red);
    if (threadIdx.x == 0) c->part[0] = d;
  }
}

void launch_coarse(MgCtl* c, const MgLevel& top, const void* sched, cudaStream_t s) {
  const MgCoarseSched* t = static_cast<const MgCoarseSched*>(sched);
  switch (top.n) {
    case 8: k_mg_coarse<8, true><<<1, MG_CT, 0, s>>>(c, top, t); break;
    case 4: k_mg_coarse<4, true><<<1, MG_CT, 0, s>>>(c, top, t); break;
    default: k_mg_coarse<2, true><<<1, MG_CT, 0, s>>>(c, top, t);
  }
}

// One half-sweep launch: a block per plane, a thread per i (n of them).
void launch_half(const MgCtl* c, const MgLevel& lv, int half, double* part, cudaStream_t s) {
  const int nt = lv.n < 32 ? 32 : lv.n;  // whole warps (threads past n idle)
  if (lv.n <= 256) {
    if (part)
      k_mg_half<256, true><<<lv.n, nt, 0, s>>>(c, lv, half, part);
    else
      k_mg_half<256, false><<<lv.n, nt, 0, s>>>(c, lv, half, part);
  } else {
    if (part)
      k_mg_half<1024, true><<<lv.n, nt, 0, s>>>(c, lv, half, part);
    else
      k_mg_half<1024, false><<<lv.n, nt, 0, s>>>(c, lv, half, part);
  }
}

int log2i(int n) {
  int l = 0;
  while ((1 << l) < n) ++l;
  return l;
}

// Whether a level's relax runs as one cooperative launch: every plane's
// block resident at once (checked with the occupancy calculator, once per
// context, level size and kernel: the answer, and the shared memory a kernel
// may use, belong to the context's device; levels of at most 256 cells),
// unless TLQ_MG_PIPELINE=0 asks for the per-half-sweep kernels.
bool resident(signed char* fit, const void* kernel, int n, int threads, size_t smem) {
  if (!*fit) {
    int dev = 0, sms = 0, per = 0;
    bool ok = cudaGetDevice(&dev) == cudaSuccess &&
              cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess;
    ok = ok && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess;
    ok = ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) == cudaSuccess;
    if (!ok) cudaGetLastError();
    *fit = (ok && (long long)per * sms >= n) ? 1 : -1;
  }
  return *fit > 0;
}

// A relax's cooperative launch; false (and no error left behind) if refused.
template <class Kernel, class... Args>
bool launch_resident(Kernel kernel, int n, int threads, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess) return true;
  cudaGetLastError();
  return false;
}

template <int NT, int MINB, int HG, int G, int CH, bool TRACK>
bool launch_pipe(tlq_ctx* ctx, MgCtl* c, const MgLevel& lv, double* part, cudaStream_t s) {
  const int nt = (lv.n * HG + 31) / 32 * 32;
  const auto kernel = k_mg_relax_pipe<NT, MINB, HG, G, CH, TRACK>;
  if (!resident(&ctx->mg_fit[1][TRACK][log2i(lv.n)], (const void*)kernel, lv.n, nt, pipe_smem(lv.n))) return false;
  k_mg_prog_reset<<<1, 256, 0, s>>>(c, lv.n);
  return launch_resident(kernel, lv.n, nt, pipe_smem(lv.n), s, c, lv, part);
}

// The shared-memory-plane relax: one block per plane, all resident at once.
template <int N, bool TRACK>
bool launch_plane(tlq_ctx* ctx, MgCtl* c, const MgLevel& lv, int leg, double* part, cudaStream_t s) {
  using G = PlaneGeo<N>;
  const auto kernel = k_mg_relax_plane<N, TRACK>;
  if (!lv.X || !resident(&ctx->mg_fit[0][TRACK][log2i(N)], (const void*)kernel, N, G::NT + G::NH, G::smem)) return false;
  return launch_resident(kernel, N, G::NT + G::NH, G::smem, s, c, lv, leg, part);
}

template <bool TRACK>
bool launch_plane_any(tlq_ctx* ctx, MgCtl* c, const MgLevel& lv, int leg, double* part, cudaStream_t s) {
  switch (lv.n) {
    case 16: return launch_plane<16, TRACK>(ctx, c, lv, leg, part, s);
    case 32: return launch_plane<32, TRACK>(ctx, c, lv, leg, part, s);
    case 64: return launch_plane<64, TRACK>(ctx, c, lv, leg, part, s);
    case 128: return launch_plane<128, TRACK>(ctx, c, lv, leg, part, s);
    default: return false;
  }
}

// One relax of a level above MG_COARSE_N cells (sources.f90:398-471); part:
// where the last pass's per-plane |change| sums go (null: not needed).
// Levels up to 128 cells hold their planes in shared memory
// (k_mg_relax_plane) unless TLQ_MG_PLANE=0; the others, and those, then use
// k_mg_relax_pipe.  Its threads per plane (measured on the gravitating
// cloud): 128-cell levels 5 x 128 (two half-sweeps each), 64 down to 16:
// 10 x n; neighbour checks every 8 steps on 128 and 64 cells, 4 on 32, 2
// on 16 (a relax takes 2n + 9 (CH + 1) steps); 256-cell levels need two
// blocks per SM: 2 x 256, checks every 4 steps.
template <bool TRACK>
bool launch_pipe_any(tlq_ctx* ctx, MgCtl* c, const MgLevel& lv, int leg, double* part, cudaStream_t s) {
  const char* env = std::getenv("TLQ_MG_PLANE");
  const bool plane = !(env && env[0] == '0');
  if (plane && launch_plane_any<TRACK>(ctx, c, lv, leg, part, s)) return true;
  switch (lv.n) {
    case 16: return launch_pipe<160, 1, 10, 1, 2, TRACK>(ctx, c, lv, part, s);
    case 32: return launch_pipe<320, 1, 10, 1, 4, TRACK>(ctx, c, lv, part, s);
    case 64: return launch_pipe<640, 1, 10, 1, 8, TRACK>(ctx, c, lv, part, s);
    case 128: return launch_pipe<640, 1, 5, 1, 8, TRACK>(ctx, c, lv, part, s);
    case 256: return launch_pipe<512, 2, 2, 1, 4, TRACK>(ctx, c, lv, part, s);
    default: return false;
  }
}

// leg: 0 on the way down, 1 on the way up.
void launch_relax(tlq_ctx* ctx, MgCtl* c, const MgLevel& lv, int leg, double* part, cudaStream_t s) {
  const char* env = std::getenv("TLQ_MG_PIPELINE");
  const bool pipe = !(env && env[0] == '0');
  if (pipe && (part ? launch_pipe_any<true>(ctx, c, lv, leg, part, s) : launch_pipe_any<false>(ctx, c, lv, leg, part, s))) return;
  for (int h = 0; h < 10; ++h) launch_half(c, lv, h & 1, (part && h >= 8) ? part + (h - 8) * lv.n : nullptr, s);
}

int grid_for(long long work, int threads) {
  return (int)std::max<long long>(1, std::min<long long>((work + threads - 1) / threads, 152LL * 8));
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// The solver's buffers: E of every level (contiguous, so that the coarse
// ones zero in one pass), then R, then T; the control block; the moments'
// block partials.
int mg_levels_of(const tlq_config& c) {
  if (c.nx != c.ny || c.nx != c.nz || c.nx < 2 || (c.nx & (c.nx - 1))) return -1;
  return log2i(c.nx);
}

cudaError_t mg_alloc(tlq_ctx* ctx) {
  const int L = mg_levels_of(ctx->cfg);
  long long cells = 0;
  for (int l = 0; l <= L; ++l) {
    const long long m = (ctx->cfg.nx >> l) + 2;
    cells += m * m * m;
  }
  cudaError_t e = cudaMalloc(&ctx->mg_work, (size_t)cells * 3 * sizeof(double));
  if (e != cudaSuccess) return e;
  e = cudaMalloc(&ctx->mg_ctl, sizeof(MgCtl));
  if (e != cudaSuccess) return e;
  e = cudaMemset(ctx->mg_ctl, 0, sizeof(MgCtl));
  if (e != cudaSuccess) return e;
  long long limit = MG_WAIT_LIMIT;
  if (const char* env = std::getenv("TLQ_MG_WAIT_LIMIT")) {
    char* end = nullptr;
    const long long v = std::strtoll(env, &end, 10);
    if (end != env && *end == '\0' && v >= 0) limit = v;
  }
  e = cudaMemcpy(reinterpret_cast<char*>(ctx->mg_ctl) + offsetof(MgCtl, wait_limit), &limit, sizeof limit,
                 cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return e;
  MgCoarseSched coarse;
  mg_coarse_sched(&coarse);
  e = cudaMalloc(&ctx->mg_coarse, sizeof(MgCoarseSched));
  if (e != cudaSuccess) return e;
  e = cudaMemcpy(ctx->mg_coarse, &coarse, sizeof(MgCoarseSched), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return e;
  long long xc = 0, sc = 0;
  for (int l = 0; l <= L; ++l)
    if (exch_level(ctx->cfg.nx >> l)) {
      xc += exch_cells(ctx->cfg.nx >> l);
      sc += 2 * sched_entries(ctx->cfg.nx >> l);
    }
  if (xc) {
    e = cudaMalloc(&ctx->mg_sched, (size_t)sc * sizeof(MgSched));
    if (e != cudaSuccess) return e;
    MgSched* at = static_cast<MgSched*>(ctx->mg_sched);
    for (int l = 0; l <= L; ++l) {
      const int n = ctx->cfg.nx >> l;
      if (!exch_level(n)) continue;
      const int nt = (5 * n + 31) / 32 * 32, rows = (int)(sched_entries(n) / nt);
      k_mg_sched<<<(unsigned)((2 * sched_entries(n) + 255) / 256), 256>>>(n, at, rows, nt);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      at += 2 * sched_entries(n);
    }
    e = cudaMalloc(&ctx->mg_exch, (size_t)xc * sizeof(Tagged));
    if (e != cudaSuccess) return e;
    e = cudaMemset(ctx->mg_exch, 0, (size_t)xc * sizeof(Tagged));  // (no call's tag)
    if (e != cudaSuccess) return e;
  }
  e = cudaMalloc(&ctx->mg_mom, (size_t)MG_MOM_BLOCKS * 25 * sizeof(double));
  if (e != cudaSuccess) return e;
  e = cudaMallocHost(&ctx->mg_go, 2 * sizeof(int));
  if (e != cudaSuccess) return e;
  for (cudaEvent_t& ev : ctx->mg_seen) {
    e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
  }
  e = cudaStreamCreateWithFlags(&ctx->mg_body, cudaStreamNonBlocking);
  if (e != cudaSuccess) return e;
  const long long m0 = ctx->cfg.nx + 2;
  e = cudaMalloc(&ctx->phig, (size_t)(m0 * m0 * m0) * sizeof(double));
  if (e != cudaSuccess) return e;
  e = cudaMemset(ctx->phig, 0, (size_t)(m0 * m0 * m0) * sizeof(double));
  if (e != cudaSuccess) return e;
  e = cudaMalloc(&ctx->phit, (size_t)ctx->L.plane * sizeof(double));
  if (e != cudaSuccess) return e;
  e = cudaMemset(ctx->phit, 0, (size_t)ctx->L.plane * sizeof(double));
  if (e != cudaSuccess) return e;
  return cudaMemset(ctx->mg_work, 0, (size_t)cells * 3 * sizeof(double));
}

void mg_free(tlq_ctx* ctx) {
  cudaFree(ctx->mg_exch); cudaFree(ctx->mg_sched); cudaFree(ctx->mg_coarse);
  ctx->mg_exch = nullptr; ctx->mg_coarse = nullptr; ctx->mg_sched = nullptr;
  cudaFree(ctx->mg_work); cudaFree(ctx->mg_ctl); cudaFree(ctx->mg_mom); cudaFree(ctx->phig); cudaFree(ctx->phit);
  if (ctx->mg_body) cudaStreamDestroy(ctx->mg_body);
  for (cudaEvent_t& ev : ctx->mg_seen) {
    if (ev) cudaEventDestroy(ev);
    ev = nullptr;
  }
  cudaFreeHost(ctx->mg_go);
  ctx->mg_go = nullptr;
  ctx->mg_work = nullptr; ctx->mg_ctl = nullptr; ctx->mg_mom = nullptr; ctx->phig = nullptr; ctx->phit = nullptr;
  ctx->mg_body = nullptr;
}

namespace {

struct MgLevels {
  MgLevel lv[MG_MAXL];
};

MgLevels mg_plan(const tlq_ctx* ctx, int L) {
  MgLevels v{};
  long long total = 0;
  for (int l = 0; l <= L; ++l) {
    const long long m = (ctx->cfg.nx >> l) + 2;
    total += m * m * m;
  }
  double* base = static_cast<double*>(ctx->mg_work);
  long long off = 0, xoff = 0, soff = 0;
  for (int l = 0; l <= L; ++l) {
    const int n = ctx->cfg.nx >> l;
    const long long m = n + 2;
    v.lv[l].n = n;
    v.lv[l].X = exch_level(n) ? static_cast<Tagged*>(ctx->mg_exch) + xoff : nullptr;
    v.lv[l].sched = exch_level(n) ? static_cast<MgSched*>(ctx->mg_sched) + soff : nullptr;
    if (exch_level(n)) {
      xoff += exch_cells(n);
      soff += 2 * sched_entries(n);
    }
    v.lv[l].E = base + off;
    v.lv[l].R = base + total + off;
    v.lv[l].T = base + 2 * total + off;
    v.lv[l].dxl = (ctx->cfg.xr - ctx->cfg.xl) / (double)n;
    off += m * m * m;
  }
  return v;
}

template <class Dens>
cudaError_t enqueue_mg(tlq_ctx* ctx, Dens rho, const Clock* clk, double* phit, cudaStream_t s) {
  const int L = mg_levels_of(ctx->cfg);
  const MgLevels v = mg_plan(ctx, L);
  MgCtl* c = static_cast<MgCtl*>(ctx->mg_ctl);
  const int n = ctx->cfg.nx;
  const bool multipole = ctx->cfg.grav_bc == TLQ_GBC_MULTIPOLE;
  int lc = 0;
  while (lc < L && v.lv[lc].n > MG_COARSE_N) ++lc;
  const long long m0 = n + 2;
  // Captured into a graph: the cycles are the body of a while node whose
  // condition the loop test sets on the device (before the node and at the
  // end of each cycle), captured on the context's second stream.  Run
  // directly (or with TLQ_MG_GRAPH_LOOP=0): a sequence of up to 31 slots.
  cudaStreamCaptureStatus cst = cudaStreamCaptureStatusNone;
  cudaGraph_t cg = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t nd = 0;
  cudaError_t e = cudaStreamGetCaptureInfo(s, &cst, nullptr, &cg, &deps, nullptr, &nd);
  if (e != cudaSuccess) return e;
  const char* env = std::getenv("TLQ_MG_GRAPH_LOOP");
  const bool loop = cst == cudaStreamCaptureStatusActive && ctx->mg_body && !(env && env[0] == '0');
  cudaGraphConditionalHandle h = {};
  if (loop) {
    e = cudaGraphConditionalHandleCreate(&h, cg, 0, 0);
    if (e != cudaSuccess) return e;
  }
  k_mg_begin<<<1, 1, 0, s>>>(c, clk, loop, h);
  if (multipole) {
    k_mg_moments<<<MG_MOM_BLOCKS, MG_MOM_THREADS, 0, s>>>(c, clk, ctx->P, rho, static_cast<double*>(ctx->mg_mom));
    k_mg_moments_final<<<1, 25 * 32, 0, s>>>(c, clk, static_cast<const double*>(ctx->mg_mom), MG_MOM_BLOCKS);
    k_mg_faces<<<grid_for(6LL * n * n, 256), 256, 0, s>>>(c, clk, ctx->P, ctx->phig);
  }
  k_mg_init<<<grid_for(m0 * m0 * m0, 256), 256, 0, s>>>(c, rho, n, ctx->phig, v.lv[0].E, v.lv[0].R, v.lv[0].T,
                                                        v.lv[0].dxl);
  double* part = reinterpret_cast<double*>(reinterpret_cast<char*>(c) + offsetof(MgCtl, part));
  // a level operator's launch: a thread per coarse cell; blocks of one warp
  // where 128 threads would leave most SMs without one
  auto blocks = [](int nc) { return nc >= 64 ? 128 : 32; };
  // One V-cycle slot (sources.f90:140-187): k_mg_begin or the cycle before
  // evaluated the loop test, and every kernel of a slot that does not run
  // returns.
  auto cycle = [&](cudaStream_t st) {
    if (lc == 0) {
      launch_coarse(c, v.lv[0], ctx->mg_coarse, st);
      k_mg_cycle_end<<<1, 32, 0, st>>>(c, 1, loop, h);
      return;
    }
    // down: level 0 .. lc-1 on the large kernels
    for (int l = 0; l < lc; ++l) {
      launch_relax(ctx, c, v.lv[l], 0, nullptr, st);
      const int nc = v.lv[l + 1].n, nt = blocks(nc);
      k_mg_resid_restrict<<<(nc * nc * nc + nt - 1) / nt, nt, 0, st>>>(c, v.lv[l], v.lv[l + 1]);
    }
    k_mg_coarse<MG_COARSE_N, false><<<1, MG_CT, 0, st>>>(c, v.lv[lc],
                                                         static_cast<const MgCoarseSched*>(ctx->mg_coarse));
    // up: level lc-1 .. 0
    for (int l = lc - 1; l >= 0; --l) {
      const int nc = v.lv[l + 1].n, nt = blocks(nc);
      k_mg_prolong_add<<<(nc * nc * nc + nt - 1) / nt, nt, 0, st>>>(c, v.lv[l + 1], v.lv[l], l > 0);
      // the last pass of the level-0 relax forms Dif (sources.f90:465-471)
      launch_relax(ctx, c, v.lv[l], 1, l == 0 ? part : nullptr, st);
    }
    k_mg_cycle_end<<<1, 32, 0, st>>>(c, 2 * n, loop, h);
  };
  if (loop) {
    e = cudaStreamGetCaptureInfo(s, &cst, nullptr, &cg, &deps, nullptr, &nd);
    if (e != cudaSuccess) return e;
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node = nullptr;
    e = cudaGraphAddNode(&node, cg, deps, nullptr, nd, &np);
    if (e != cudaSuccess) return e;
    e = cudaStreamBeginCaptureToGraph(ctx->mg_body, np.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                      cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    cycle(ctx->mg_body);
    cudaGraph_t body = nullptr;
    e = cudaStreamEndCapture(ctx->mg_body, &body);
    if (e != cudaSuccess) return e;
    e = cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1, cudaStreamSetCaptureDependencies);
    if (e != cudaSuccess) return e;
  } else {
    // Outside a capture the slots are enqueued two ahead of the cycle that the
    // host has seen to go on, so that at most two slots run empty (of about
    // 17 launches each, 1.5 us a launch; its callers wait for the result).
    const bool look = cst == cudaStreamCaptureStatusNone;
    for (int cyc = 0; cyc < MG_CYCLES; ++cyc) {
      if (look && cyc >= 2) {
        e = cudaEventSynchronize(ctx->mg_seen[cyc & 1]);
        if (e != cudaSuccess) return e;
        if (!ctx->mg_go[cyc & 1]) break;
      }
      cycle(s);
      if (!look) continue;
      e = cudaMemcpyAsync(ctx->mg_go + (cyc & 1), &c->active, sizeof(int), cudaMemcpyDeviceToHost, s);
      if (e != cudaSuccess) return e;
      e = cudaEventRecord(ctx->mg_seen[cyc & 1], s);
      if (e != cudaSuccess) return e;
    }
  }
  k_mg_end<<<grid_for(m0 * m0 * m0, 256), 256, 0, s>>>(c, const_cast<Clock*>(clk), n, v.lv[0].E, ctx->phig, ctx->phi,
                                                       phit, phit ? ctx->phif : nullptr, ctx->L);
  return cudaGetLastError();
}

}  // namespace

cudaError_t enqueue_multigrid_soa(tlq_ctx* ctx, const double* U, cudaStream_t s) {
  return enqueue_mg(ctx, DensSoA{U, ctx->L}, ctx->clk, ctx->phit, s);
}

cudaError_t enqueue_multigrid_aos(tlq_ctx* ctx, const double* U, const Clock* clk, cudaStream_t s) {
  return enqueue_mg(ctx, DensAoS{U, ctx->A}, clk, nullptr, s);
}

int mg_cycles_and_status(tlq_ctx* ctx, int* cycles, int* status) {
  MgCtl h;
  if (cudaMemcpy(&h, ctx->mg_ctl, sizeof(MgCtl), cudaMemcpyDeviceToHost) != cudaSuccess) return TLQ_ERR_CUDA;
  if (cycles) *cycles = h.iter;
  if (status) *status = h.status;
  return TLQ_OK;
}

}  // namespace tlq
