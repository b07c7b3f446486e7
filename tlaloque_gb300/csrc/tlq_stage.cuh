// tlq_stage.cuh -- the two fused stage kernels of one hydrodynamic step.
//
// STAGE 1 = HLL[C]Fluxes(U, ..., 1) + Godunov(UPP, U, ..., dt/2) + borders(UPP, 2)
//           (source/mainHD.f90:76-82)
// STAGE 2 = calc_prims(UPP) + HLL[C]Fluxes(UPP, ..., 2) + Godunov(UP, U, ..., dt)
//           + borders(UP, 1) + step + calc_prims(U) + cooling + time_step
//           (source/mainHD.f90:84-97 and the next iteration's :74)
//
// A block owns a TX x TY column tile of interior cells and marches along z
// through a chunk of planes.  One elected thread streams planes of the input
// state (all 5 conserved variables, tile + 2-cell halo) into a 4-slot shared
// ring with 4-D TMA tensor loads completing on mbarriers; the block converts
// each plane to primitives once, computes every x/y/z face flux of the plane
// once (one flat, direction-generic task list), and applies the conservative
// update, sources, ghost fill, viscosity and cooling per cell.
#pragma once

#include "tlq_device.cuh"

namespace tlq {

constexpr int TX = 16, TY = 8, NT = TX * TY;

// Tile of the mixed-form kernels (its own constants, so that it can be tuned
// apart from the plain form's): MTX x MTY columns on MNT threads, a multiple
// of 16 columns wide (the FP32 box of a tile starts on a 64-byte boundary).
#ifndef TLQ_MTX
#define TLQ_MTX 16
#endif
#ifndef TLQ_MTY
#define TLQ_MTY 8
#endif
#ifndef TLQ_MNT
#define TLQ_MNT 128
#endif
constexpr int MTX = TLQ_MTX, MTY = TLQ_MTY, MNT = TLQ_MNT;
static_assert(MTX * MTY <= MNT, "one cell per thread");
static_assert(MTX % 16 == 0 && MNT % 32 == 0, "tile shape");
constexpr int NRING = 3;
constexpr long long WAIT_LIMIT = 1LL << 24;  // mbarrier polls before giving up

struct StageArgs {
  Params p;
  Layout L;
  const double* uold;  // STAGE 2: U at the start of the step (Godunov centre, viscosity)
  double* out;         // STAGE 1: UPP; STAGE 2: U of the next step
  double* pout;        // STAGE 2 with cooling: carried (cooled) interior pressure
  const double* phi;   // point-mass potential plane (null without gravity)
  const float* phif;   // mixed form: the same potential rounded to FP32 (what its kernels read)
  Clock* clk;          // time, and the CFL reduction's ticket and maxima
  int zlen;            // planes per block
  int use_p;           // STAGE 1 with cooling: interior pressure from the P plane
  float* lapf;         // mixed form: eta * Laplacian of U (FP32, written by stage 1, read by stage 2)
  float* uppf;         // mixed form, STAGE 1: UPP as FP32 primitives (rho, u, v, w, p), read by stage 2
  unsigned* cqueue;    // mixed form with the cooling surrogate: stage 2 queues the cells that cool
  unsigned* cqcount;   // (beyond a single step of the exact integrator, which it takes itself)
  unsigned long long* cool_counts;  // [2]: the cells stage 2 cooled in a single step
};

// Geometry of the planes the plain form stages in shared memory (x fastest,
// tile cell (tx, ty) at (OY + ty, 2 + tx)): 2 halo cells in x (a TMA box of
// FP64 values starts on an even cell), in y the faces' own reach (1 in stage
// 1, 2 in stage 2).
template <int S>
struct Geo {
  static constexpr int OY = S, PX = TX + 4, PY = TY + 2 * OY, PB = PX * PY;
};

// Shared memory of the plain form's kernels: three planes of conserved
// values (the TMA's landing slots), the primitives of the plane whose x and y
// faces are evaluated, and the x and y fluxes.  What the z faces need of
// their own column lives in the column's thread, so a block takes 62 KB and
// 3 blocks fit an SM (107 KB and 2 with four planes of both forms and every
// flux in shared memory).
template <int S>
struct StageSmem {
  static constexpr int NP = (S == 1) ? 8 : 5;  // stage 1 adds the cell's sound speed, E/rho and enthalpy
  // (slots padded to 128 bytes, the TMA's destination alignment)
  double raw[NRING][(5 * Geo<S>::PB + 15) / 16 * 16];
  double praw[S == 1 ? NRING : 1][S == 1 ? (Geo<S>::PB + 15) / 16 * 16 : 16];  // the carried pressure (stage 1 with cooling)
  double prm[NP][Geo<S>::PB];
  double sx[S == 2 ? 5 : 1][S == 2 ? TY * (TX + 2) : 1];  // x and y slopes of the plane's cells
  double sy[S == 2 ? 5 : 1][S == 2 ? (TY + 2) * TX : 1];
  double fx[5][TY][TX + 1];
  double fy[5][TY + 1][TX];
  uint64_t bar[NRING];
  double red[96];
  TileSpecial tspec;  // the tile's boundary/wind pre-test
  int flag;
  int abort;
};

// The face-ghost images of interior cell (i, j, k) (boundaries.f90 non-MPI
// branches; layers = 1: boundariesI :183-257, layers = 2: boundariesII
// :433-531): put(axis, flip, gi, gj, gk) for each ghost cell that takes this
// cell's value (flip: with the momentum along the axis negated).  Rolled
// loops: few cells come here, and unrolled this code (with what put inlines)
// was most of a stage kernel's 0.5-0.9 MB of instructions (now 0.12-0.36).
template <class Put>
__device__ __forceinline__ void ghost_images(const Params& p, int layers, int i, int j, int k, Put put) {
#pragma unroll 1
  for (int f = 0; f < 6; ++f) {
    const int ax = f >> 1, hi = f & 1, bc = p.bc[f];
    const int c = ax == 0 ? i : (ax == 1 ? j : k), n = ax == 0 ? p.nx : (ax == 1 ? p.ny : p.nz);
#pragma unroll 1
    for (int l = 0; l < layers; ++l) {
      // the interior cell ghost layer l of this side copies
      const bool from_hi = (bc == BC_PERIODIC) != (hi != 0);
      const int off = bc == BC_OUTFLOW ? 0 : l;
      if (c != (from_hi ? n - off : 1 + off)) continue;
      const int g = hi ? n + 1 + l : -l;
      put(ax, bc == BC_REFLECTIVE, ax == 0 ? g : i, ax == 1 ? g : j, ax == 2 ? g : k);
    }
  }
}

// Write the face-ghost images of cell (i, j, k), whose value (before the
// wind overwrite) is v, into `out`, then apply the winds at each ghost cell
// (borders applies user_boundaries after the face fill).
__device__ __forceinline__ void write_ghosts(const Params& p, const Layout& L, double* out, int layers, int i, int j,
                                             int k, const double* v) {
  ghost_images(p, layers, i, j, k, [&](int ax, bool flip, int gi, int gj, int gk) {
    double g[5];
#pragma unroll
    for (int e = 0; e < 5; ++e) g[e] = (flip && e == ax + 1) ? -v[e] : v[e];
    winds_cell(p, gi, gj, gk, g);
    const long long o = L.at(gi, gj, gk);
#pragma unroll
    for (int e = 0; e < 5; ++e) out[e * L.plane + o] = g[e];
  });
}

// The face-ghost images (ghost_images) of the interior cell (i, j, k) at c
// where no wind reaches a ghost cell: its value v, the momentum along the
// axis negated at a reflective face.  FP32 primitives as well: negating a
// momentum negates its velocity and leaves the others, so they are what
// mixed_cell would form of the image.
//   A tile at an x or y face has such cells in every warp and plane: with
// each image formed anew from FP64 (winds, mixed_cell) it took twice an
// interior tile's time in stage 1 and 1.45 times in stage 2 (16-plane chunks,
// 290 k and 142 k cycles, 340 k and 235 k); now 1.3 and 1.15 times.  Bubble
// 256^3: stage 1 0.97 -> 0.83 ms, stage 2 1.42 -> 1.34; diagonal Sod 150^3:
// 0.235 -> 0.198 and 0.281 -> 0.265.  The axes rolled in stage 1 (less code:
// 3 % on the bubble), unrolled in stage 2 (1 %).
template <int LAYERS, class T>
__device__ __forceinline__ void store_ghosts(const Params& p, const Layout& L, T* out, int i, int j, int k,
                                             long long c, const T* v) {
#pragma unroll(LAYERS == 2 ? 1 : 3)
  for (int ax = 0; ax < 3; ++ax) {
    const int q = ax == 0 ? i : ax == 1 ? j : k, n = ax == 0 ? p.nx : ax == 1 ? p.ny : p.nz;
    if (q > LAYERS && q <= n - LAYERS) continue;
    const long long st = ax == 0 ? 1 : ax == 1 ? (long long)L.px : (long long)L.px * L.nyg;
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      const int bc = p.bc[2 * ax + side];
      const bool flip = bc == BC_REFLECTIVE, from_hi = (bc == BC_PERIODIC) != (side != 0);
#pragma unroll
      for (int l = 0; l < LAYERS; ++l) {
        const int off = bc == BC_OUTFLOW ? 0 : l;  // the cell that layer l copies
        if (q != (from_hi ? n - off : 1 + off)) continue;
        T* o = out + c + (long long)((side ? n + 1 + l : -l) - q) * st;
#pragma unroll
        for (int e = 0; e < 5; ++e) o[e * L.plane] = (flip && e == ax + 1) ? -v[e] : v[e];
      }
    }
  }
}

// Where a wind may reach the cell or its ghost images: the images of v (the
// value before the winds) with the winds applied at the ghost cells, and v
// with the winds.  Calls: few tiles come here.
struct Cons {
  double u[5];
};
static __device__ __noinline__ Cons windy_ghosts(const Params& p, const Layout& L, double* out, int layers, int i, int j,
                                              int k, Cons v) {
  write_ghosts(p, L, out, layers, i, j, k, v.u);
  winds_cell(p, i, j, k, v.u);
  return v;
}
// ---------------------------------------------------------------------------
// One face's flux in direction d from the states beside it: HLL[C] of
// riemann (tlq_physics.cuh) operation for operation, with what the cells
// share formed once per cell instead of once per face.  cl, cr: the sound
// speeds; el, er: E/rho of the two sides (0.0 in stage 2, which forms the
// chosen side's); hl, hr: (1/2) rho v^2 + g1 p, likewise; UL, UR: the
// cell-centred conserved states, `us` doubles between variables.
//   Every 0.5 x is exact, so its sum with the next term takes one FMA, the
// rounding unchanged.  prod: a multiplication on the integer pipe.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double enthalpy(double g1, const double* w) {
  return __fma_rn(0.5, w[0] * ((w[1] * w[1] + w[2] * w[2]) + w[3] * w[3]), g1 * w[4]);
}

// prim2f of tlq_physics.cuh with the mass flux m = rho un and h given.
__device__ __forceinline__ void flux_of(double* ff, const double* w, double un, double m, double h, int d) {
  ff[0] = m;
#pragma unroll
  for (int e = 1; e <= 3; ++e) {
    // (rho u_lo) u_hi, lo < hi the two component indices
    const double t = ((e < d) ? w[0] * w[e] : m) * ((e < d) ? un : w[e]);
    ff[e] = (e == d) ? t + w[4] : t;
  }
  ff[4] = un * h;
}

template <int STAGE, int SOLV>
__device__ __forceinline__ void face_flux(const Params& p, double* ff, const double* wl, const double* wr, double cl,
                                          double cr, double el, double er, double hl, double hr, const double* UL,
                                          const double* UR, int us, int d) {
  const double ul = comp(wl, d), ur = comp(wr, d);
  const double sl = mn(ul - cl, ur - cr);
  const double sr = mx(ul + cl, ur + cr);
  const double ml = prod(wl[0], ul), mr = prod(wr[0], ur);
  if (SOLV == SOLVER_HLL || (SOLV < 0 && p.solver == SOLVER_HLL)) {
    if (ge0(sl) || le0(sr)) {
      const bool left = ge0(sl);
      double w[5];
#pragma unroll
      for (int e = 0; e < 5; ++e) w[e] = left ? wl[e] : wr[e];
      flux_of(ff, w, left ? ul : ur, left ? ml : mr, STAGE == 1 ? (left ? hl : hr) : enthalpy(p.g1, w), d);
    } else {
      double fl[5], fr[5];
      flux_of(fl, wl, ul, ml, STAGE == 1 ? hl : enthalpy(p.g1, wl), d);
      flux_of(fr, wr, ur, mr, STAGE == 1 ? hr : enthalpy(p.g1, wr), d);
      const auto ds = divisor(sr - sl);
      const double ss = prod(sl, sr);
#pragma unroll
      for (int e = 0; e < 5; ++e) 
        ff[e] = quot(prod(sr, fl[e]) - prod(sl, fr[e]) + prod(ss, UR[e * us] - UL[e * us]), ds);
    }
    return;  // NaN speeds take the HLL average branch, as in the reference
  }
  const double dl = sl - ul, dr = sr - ur;
  const double al = prod(wl[0], dl), ar = prod(wr[0], dr);
  const double sst = quot(wr[4] - wl[4] + prod(ml, dl) - prod(mr, dr), al - ar);
  // Branch order of the reference: sl>=0, sr<=0, sst>=0, sst<=0; a face with
  // NaN speeds takes none (NaN here)
  bool star, left;
  if (ge0(sl)) { star = false; left = true; }
  else if (le0(sr)) { star = false; left = false; }
  else if (ge0(sst)) { star = true; left = true; }
  else if (le0(sst)) { star = true; left = false; }
  else {
#pragma unroll
    for (int e = 0; e < 5; ++e) ff[e] = NAN;
    return;
  }
  double w[5];
#pragma unroll
  for (int e = 0; e < 5; ++e) w[e] = left ? wl[e] : wr[e];
  const double un = left ? ul : ur;
  flux_of(ff, w, un, left ? ml : mr, STAGE == 1 ? (left ? hl : hr) : enthalpy(p.g1, w), d);
  if (star) {
    const double* uc = left ? UL : UR;
    const double s = left ? sl : sr;
    const double a = left ? al : ar;  // rho (s - un)
    const double rhostr = quot(a, s - sst);
    const double eor = STAGE == 1 ? (left ? el : er) : quot(uc[4 * us], w[0]);
    double u[5];
    u[0] = rhostr;
#pragma unroll
    for (int e = 1; e <= 3; ++e) u[e] = prod(rhostr, (e == d) ? sst : w[e]);
    u[4] = prod(rhostr, eor + prod(sst - un, sst + quot(w[4], a)));
#pragma unroll
    for (int e = 0; e < 5; ++e) ff[e] = ff[e] + prod(s, u[e] - uc[e * us]);
  }
}

// The plain FP64 step's kernels.  What bounds them: the FP64 pipe (18.6 SM
// cycles per warp instruction), so every operation whose result another face
// or cell also needs is done once --
//   stage 1: the sound speed, E/rho and enthalpy per cell (each was formed
//     for all six faces of a cell);
//   stage 2: the limited slopes per cell (the slope right of a face is the
//     one left of the next face: one per cell and direction instead of two
//     per face);
// divisions and square roots run on the integer pipe (tlq_softfp.cuh).
//   A thread owns a column of the tile.  Per plane: it converts the column's
// next plane (kept in registers for the z direction), the block converts the
// plane's halo, then (stage 2) the slopes, then the faces -- each thread its
// cell's left x, lower y and upper z face, one warp in turn the tile's right
// and upper edges -- through one copy of the code, then the cells' update.
// The z flux stays in its thread.
//   Measured, Sedov 128^3, 8-plane chunks: stage 1 2.90 -> 0.98 ms, stage 2
// 5.09 -> 1.90 ms per launch against one face task list with the limiter and
// sound speeds per face and hardware divisions (1.44 and 2.80 ms with those
// off the FP64 pipe; 1.01 and 2.08 before the sign tests moved to the bits
// and the z differences were carried).  The FP64 pipe's counter: 197
// instructions a cell in stage 1 and 407 in stage 2 before those two, at 70-73
// % of its rate, in a quarter of the issue slots.  Which multiplications go to the
// integer pipe is measured too: all of them, or none, is 3-12 % slower than
// the star state's, the wave speeds', the limiter's and the update's.
template <int STAGE, int LIM, int SOLV>
__global__ void __launch_bounds__(NT, STAGE == 1 ? 4 : 3)
    stage_kernel(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_p,
                 const __grid_constant__ StageArgs a) {
  using G = Geo<STAGE>;
  using Smem = StageSmem<STAGE>;
  constexpr int H = STAGE, OY = G::OY, PX = G::PX, PB = G::PB, NP = Smem::NP;
  extern __shared__ __align__(128) unsigned char smem_bytes[];
  Smem& s = *reinterpret_cast<Smem*>(smem_bytes);
  const Params& p = a.p;
  const Layout& L = a.L;
  const int tid = threadIdx.x;
  const int bx = blockIdx.x, by = blockIdx.y;
  const int i0 = 1 + bx * TX, j0 = 1 + by * TY;
  const int k0 = 1 + (int)blockIdx.z * a.zlen;
  const int k1 = min(p.nz, k0 + a.zlen - 1);
  const int lim = LIM >= 0 ? LIM : p.limiter;
  Clock* clk = a.clk;

  if (!(clk->t < clk->tfin)) return;  // the loop condition of mainHD.f90:61 (uniform)
  const double dtstep = clk->dt;
  const double dt = (STAGE == 1) ? dtstep / 2.0 : dtstep;  // dth = dt/2.0 (mainHD.f90:78)
  const double dtdx = dt / p.dx, dtdy = dt / p.dy, dtdz = dt / p.dz;
  const bool use_p = STAGE == 1 && a.use_p;
  const uint32_t box_bytes = 5u * PB * 8u + (use_p ? PB * 8u : 0u);
  const int last_plane = k1 + H;

  if (tid == 0) {
    for (int q = 0; q < NRING; ++q) mbar_init(&s.bar[q], 1);
    s.abort = 0;
    s.tspec = tile_special(p, i0, min(i0 + TX - 1, p.nx), j0, min(j0 + TY - 1, p.ny));
    fence_mbar_init();
  }
  __syncthreads();

  // Plane q lives in slot (q - (k0 - H)) mod 3.
  auto slot_of = [&](int q) { return (unsigned)(q - (k0 - H)) % (unsigned)NRING; };
  int issued = k0 - H - 1;  // last plane issued (meaningful in thread 0)
  auto issue = [&](int q) {  // thread 0
    const int slot = slot_of(q);
    fence_proxy_async();
    mbar_arrive_expect_tx(&s.bar[slot], box_bytes);
    tma_load_4d(s.raw[slot], &tm_in, &s.bar[slot], bx * TX, by * TY + 2 - OY, q + 1, 0);
    if (use_p) tma_load_4d(s.praw[slot], &tm_p, &s.bar[slot], bx * TX, by * TY + 2 - OY, q + 1, 0);
    issued = q;
  };
  // Every thread waits for every plane in order and tracks the slot phases.
  uint32_t phase = 0;
  int waited = k0 - H - 1;  // last plane this thread saw land
  bool failed = false;
  auto wait_plane = [&](int q) {
    if (failed) return;
    const int slot = slot_of(q);
    if (!mbar_wait_bounded(&s.bar[slot], (phase >> slot) & 1u, WAIT_LIMIT)) {
      failed = true;
      s.abort = 1;
      return;
    }
    phase ^= 1u << slot;
    waited = q;
  };

  const int tx = tid % TX, ty = tid / TX;
  const int i = i0 + tx, j = j0 + ty;
  const bool cell_ok = (i <= p.nx) && (j <= p.ny);
  const int oc = (ty + OY) * PX + tx + 2;

  // Primitives (and stage 1's derived values) of the cell at offset o of
  // landed plane q, mesh indices (ii, jj).
  auto convert = [&](int q, int o, int ii, int jj, double* w) {
    if (ii > p.nx + 2 || jj > p.ny + 2) {  // beyond the mesh: no face reads it
#pragma unroll
      for (int e = 0; e < NP; ++e) w[e] = 1.0;
      return;
    }
    const int slot = slot_of(q);
    double u[5];
#pragma unroll
    for (int e = 0; e < 5; ++e) u[e] = s.raw[slot][e * PB + o];
    cons2prim(p.gamma, u, w);
    if constexpr (STAGE == 1) {
      if (use_p && ii >= 1 && ii <= p.nx && jj >= 1 && jj <= p.ny && q >= 1 && q <= p.nz) w[4] = s.praw[slot][o];
      const auto r = divisor(u[0]);
      w[5] = root(quot(p.gamma * w[4], r));
      w[6] = quot(u[4], r);
      w[7] = enthalpy(p.g1, w);
    }
  };

  // ---- prologue: the column's first planes ---------------------------------
  if (tid == 0)
    for (int q = k0 - H; q < k0 - H + NRING && q <= last_plane; ++q) issue(q);
  // the column's primitives of plane k and k+1, its slope of plane k in z
  // (stage 2) and its lower z flux
  double w0[NP], w1[NP], sz[5], fz[5];
  double dz[5];  // w1 - w0 (stage 2)
#pragma unroll
  for (int e = 0; e < 5; ++e) sz[e] = fz[e] = 0.0;
  bool aborted = false;
  for (int q = k0 - H; q < k0; ++q) {  // (stage 1: k0-1; stage 2: k0-2, k0-1)
#pragma unroll
    for (int e = 0; e < NP; ++e) w0[e] = w1[e];
    wait_plane(q);
    convert(q, oc, i, j, w1);
  }
  if (STAGE == 1) {
#pragma unroll
    for (int e = 0; e < NP; ++e) w0[e] = w1[e];
  }
  if (STAGE == 2) {
#pragma unroll
    for (int e = 0; e < 5; ++e) dz[e] = w1[e] - w0[e];
  }
  unsigned long long m0 = 0ull, m1 = 0ull, m2 = 0ull;  // CFL maxima as max_key keys (STAGE 2)

  // Stage 1 starts at k0-1 (its z face k0-1/2), stage 2 at k0-2 (the z slope
  // of k0-1).  At plane k: w0 = plane k (stage 2: w1 = plane k+1).
  for (int k = k0 - H; k <= k1; ++k) {
    const bool cells = k >= k0, zface = k >= k0 - 1;
    const int slot = slot_of(k), slot1 = slot_of(k + 1);
    double w2[NP];  // plane k + H
    wait_plane(k + H);
    convert(k + H, oc, i, j, w2);  // (garbage if the wait gave up; discarded below)
    if (cells) {
#pragma unroll
      for (int e = 0; e < NP; ++e) s.prm[e][oc] = w0[e];
      constexpr int NROW = 2 * H * TY, NCOL = 2 * H * TX;
      if (tid < NROW + NCOL) {  // the plane's halo
        int lx, ly;
        if (tid < NROW) {
          const int c = tid / TY;
          lx = c < H ? 2 - H + c : TX + 2 + c - H;
          ly = OY + tid % TY;
        } else {
          const int u = tid - NROW, c = u / TX;
          lx = 2 + u % TX;
          ly = c < H ? OY - H + c : TY + OY + c - H;
        }
        double w[NP];
        convert(k, ly * PX + lx, i0 - 2 + lx, j0 - OY + ly, w);
#pragma unroll
        for (int e = 0; e < NP; ++e) s.prm[e][ly * PX + lx] = w[e];
      }
    }
    __syncthreads();  // the plane's primitives
    if (s.abort) { aborted = true; break; }
    if (STAGE == 1 && tid == 0 && k + 2 <= last_plane && k + 2 > issued) issue(k + 2);  // plane k-1's slot

    double sz1[5];  // the z slope of plane k+1
    if constexpr (STAGE == 2) {
#pragma unroll 1
      for (int r = cells ? 0 : 3; r < 4; ++r) {
        double dm[5], dp[5];
        double* out = nullptr;
        int os = 0;
        if (r == 3) {
#pragma unroll
          for (int e = 0; e < 5; ++e) {
            dm[e] = dz[e];
            dp[e] = w2[e] - w1[e];
            dz[e] = dp[e];
          }
        } else {
          // the own cell's x, its y, and the cells beside the tile (48 tasks,
          // on the upper warps when k is odd)
          int o, st, t = (k & 1) ? NT - 1 - tid : tid;
          if (r == 0) { o = oc; st = 1; out = &s.sx[0][ty * (TX + 2) + tx + 1]; }
          else if (r == 1) { o = oc; st = PX; out = &s.sy[0][(ty + 1) * TX + tx]; }
          else if (t < 2 * TY) {
            const int lx = t < TY ? 1 : TX + 2, row = t % TY;
            o = (row + OY) * PX + lx; st = 1; out = &s.sx[0][row * (TX + 2) + lx - 1];
          } else if (t < 2 * TY + 2 * TX) {
            const int u = t - 2 * TY, ly = u < TX ? 1 : TY + 2;
            o = ly * PX + 2 + u % TX; st = PX; out = &s.sy[0][(ly - 1) * TX + u % TX];
          } else continue;
          os = st == 1 ? TY * (TX + 2) : (TY + 2) * TX;
#pragma unroll
          for (int e = 0; e < 5; ++e) {
            const double* c = &s.prm[e][o];
            const double v = c[0];
            dm[e] = v - c[-st];
            dp[e] = c[st] - v;
          }
        }
#pragma unroll
        for (int e = 0; e < 5; ++e) {
          const double v = average(dm[e], dp[e], lim);
          if (r == 3) sz1[e] = v; else out[e * os] = v;
        }
      }
      if (cells) __syncthreads();  // the plane's slopes
    }

    double fz1[5];
    if (zface) {
#pragma unroll 1
      for (int r = cells ? 0 : 2; r < 4; ++r) {
        double wl[NP], wr[NP], ff[5];
        const double *uL, *uR;
        double* out = nullptr;
        int d, fs = 0;
        if (r == 2) {
          d = 3;
          if (!cell_ok) continue;
          if constexpr (STAGE == 1) {
#pragma unroll
            for (int e = 0; e < NP; ++e) { wl[e] = w0[e]; wr[e] = w2[e]; }
          } else {
#pragma unroll
            for (int e = 0; e < 5; ++e) {
              wl[e] = __fma_rn(0.5, sz[e], w0[e]);
              wr[e] = __fma_rn(-0.5, sz1[e], w1[e]);
            }
          }
          uL = &s.raw[slot][oc];
          uR = &s.raw[slot1][oc];
        } else {
          // the left x face, the lower y face; the edges: x = TX (8 faces), y
          // = TY (16), on warp k mod 4
          int fxl = tx, fyl = ty;
          d = r + 1;
          if (r == 3) {
            const int t = tid - 32 * (k & 3);
            if (t < 0 || t >= TY + TX || !cells) continue;
            d = t < TY ? 1 : 2;
            fxl = t < TY ? TX : t - TY;
            fyl = t < TY ? t : TY;
          }
          const int ii = i0 + fxl, jj = j0 + fyl;  // the cell right of (above) the face
          if (!(d == 1 ? (ii - 1 <= p.nx && jj <= p.ny) : (ii <= p.nx && jj - 1 <= p.ny))) continue;
          const int st = d == 1 ? 1 : PX, oR = (fyl + OY) * PX + fxl + 2, oL = oR - st;
#pragma unroll
          for (int e = 0; e < NP; ++e) {
            wl[e] = s.prm[e][oL];
            wr[e] = s.prm[e][oR];
          }
          if constexpr (STAGE == 2) {
            const double* sp = d == 1 ? &s.sx[0][fyl * (TX + 2) + fxl] : &s.sy[0][fyl * TX + fxl];
            const int one = d == 1 ? 1 : TX, ss = d == 1 ? TY * (TX + 2) : (TY + 2) * TX;
#pragma unroll
            for (int e = 0; e < 5; ++e) {
              wl[e] = __fma_rn(0.5, sp[e * ss], wl[e]);
              wr[e] = __fma_rn(-0.5, sp[e * ss + one], wr[e]);
            }
          }
          uL = &s.raw[slot][oL];
          uR = &s.raw[slot][oR];
          out = d == 1 ? &s.fx[0][fyl][fxl] : &s.fy[0][fyl][fxl];
          fs = d == 1 ? TY * (TX + 1) : (TY + 1) * TX;
        }
        if constexpr (STAGE == 1)
          face_flux<1, SOLV>(p, ff, wl, wr, wl[5], wr[5], wl[6], wr[6], wl[7], wr[7], uL, uR, PB, d);
        else
          face_flux<2, SOLV>(p, ff, wl, wr, csound(p.gamma, wl[4], wl[0]), csound(p.gamma, wr[4], wr[0]), 0.0, 0.0,
                             0.0, 0.0, uL, uR, PB, d);
#pragma unroll
        for (int e = 0; e < 5; ++e) {
          if (r == 2) fz1[e] = ff[e]; else out[e * fs] = ff[e];
        }
      }
    }
    __syncthreads();  // the plane's fluxes; (stage 2) plane k's slot is free
    if (STAGE == 2 && tid == 0 && k + 3 <= last_plane && k + 3 > issued) issue(k + 3);

    if (cells && cell_ok) {
      const long long c = L.at(i, j, k);
      double uc[5], up[5];
      if (STAGE == 1) {
#pragma unroll
        for (int e = 0; e < 5; ++e) uc[e] = s.raw[slot][e * PB + oc];
      } else {
#pragma unroll
        for (int e = 0; e < 5; ++e) uc[e] = a.uold[e * L.plane + c];
      }
#pragma unroll
      for (int e = 0; e < 5; ++e)
        up[e] = uc[e] - prod(dtdx, s.fx[e][ty][tx + 1] - s.fx[e][ty][tx]) -
                prod(dtdy, s.fy[e][ty + 1][tx] - s.fy[e][ty][tx]) - prod(dtdz, fz1[e] - fz[e]);
      if (p.gravity) {  // Godunov's + dt*S (source/HLLC.f90:39-41)
        const double* ph = a.phi;
        const long long pxy = (long long)L.px * L.nyg;
        double sv[5];
        gravity_cell(p, w0, ph[c + 1] - ph[c - 1], ph[c + L.px] - ph[c - L.px], ph[c + pxy] - ph[c - pxy], sv);
#pragma unroll
        for (int e = 0; e < 5; ++e) up[e] = up[e] + dt * sv[e];
      }
      // borders: face ghosts from the pre-wind value, then the winds (only
      // cells near a face or in a wind's box can be concerned)
      if (s.tspec.may_be_special(p, k) && near_boundary_or_wind(p, i, j, k)) {
        if (s.tspec.windy(k)) {
          write_ghosts(p, L, a.out, STAGE == 1 ? 2 : 1, i, j, k, up);
          winds_cell(p, i, j, k, up);
        } else {
          store_ghosts<STAGE == 1 ? 2 : 1>(p, L, a.out, i, j, k, c, up);
        }
      }
      if (STAGE == 1) {
#pragma unroll
        for (int e = 0; e < 5; ++e) a.out[e * L.plane + c] = up[e];
      } else {
        // step: U = UP + eta*(sum of the 6 neighbours of the old U - 6 U_old)
        const long long pxy = (long long)L.px * L.nyg;
        double un[5], w[5];
#pragma unroll
        for (int e = 0; e < 5; ++e) {
          const double* uo = a.uold + e * L.plane + c;
          un[e] = up[e] + prod(p.eta, uo[1] + uo[-1] + uo[L.px] + uo[-L.px] + uo[pxy] + uo[-pxy] - prod(6.0, uc[e]));
        }
        cons2prim(p.gamma, un, w);  // calc_prims(UPrim, U)
        if (p.cooling != COOL_NONE) {
          cool_cell(p, w, un[4], dtstep);
          a.pout[c] = w[4];
        }
        if (!gt0(un[0])) atomicOr(&clk->status, ST_NEG_DENSITY);
#pragma unroll
        for (int e = 0; e < 5; ++e) a.out[e * L.plane + c] = un[e];
        double v3[3];
        signal_speeds(p.gamma, w, v3);
        m0 = max(m0, max_key(v3[0]));
        m1 = max(m1, max_key(v3[1]));
        m2 = max(m2, max_key(v3[2]));
      }
    }
    if constexpr (STAGE == 2) {
#pragma unroll
      for (int e = 0; e < 5; ++e) {
        w0[e] = w1[e];
        w1[e] = w2[e];
        sz[e] = sz1[e];
      }
    } else {
#pragma unroll
      for (int e = 0; e < NP; ++e) w0[e] = w2[e];
    }
    if (zface) {
#pragma unroll
      for (int e = 0; e < 5; ++e) fz[e] = fz1[e];
    }
  }

  if (aborted) {
    // Let the copies still in flight land (bounded) before the block exits,
    // and poison this block's CFL maxima so that the step reports it.
    if (tid == 0) {
      atomicOr(&clk->status, ST_TIMEOUT);
      for (int q = waited + 1; q <= issued; ++q) {
        const int slot = slot_of(q);
        mbar_wait_bounded(&s.bar[slot], (phase >> slot) & 1u, WAIT_LIMIT);
        phase ^= 1u << slot;
      }
    }
    m0 = m1 = m2 = ~0ull;
  }
  if (STAGE == 2) cfl_reduce_finalize<NT>(key_value(m0), key_value(m1), key_value(m2), clk, p, true, s.red, &s.flag);
}

}  // namespace tlq
