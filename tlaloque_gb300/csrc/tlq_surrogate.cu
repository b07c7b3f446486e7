// tlq_surrogate.cu -- the learned cooling surrogate in the step (mixed form,
// TLQ_COOL_MLP) and its training driver.
//
// In the step, stage 2 cools the cells the exact integrator takes in one
// step and leaves the other cells that cool (temp >= the table's first
// temperature, cooling.f90:71) and the CFL reduction to three passes
// (k_cool_sort, k_cool_net, k_cool_dt; one launch, k_cool_all, for a single
// mesh): for a cell inside the training box
// the network predicts r with ln(T/T_new) = tau (1 + tau r) from
// (log10 n, log10 T, log10 tau); the prediction is accepted when
// |T_pred - T_ex| <= tol T, T_ex the exact integrator's temperature (the
// closed-form solution of dT/dt = -(gamma-1) n Lambda(T)/k_B for the
// piecewise power-law table, cool_exact_dropf); otherwise, and for a cell
// outside the box, the cell takes T_ex.
// Built with --use_fast_math (FP32 part of the mixed form).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <numeric>
#include <random>

#include "tlq_ctx.h"
#include "tlq_mlp.cuh"
#include "tlq_stage_mixed.cuh"
#include "tlq_umma.cuh"

namespace tlq {
namespace {

struct SurrogateArgs {
  const mlp::SmemWeights* img;  // the network's image (launch_pack_weights)
  float norm[6];        // centre, half-width per feature
  float box[6];         // training box (lo, hi per feature)
  unsigned long long* counts;
};

constexpr int CT = 128;      // threads per block of the network pass
constexpr int ST = 512;      // threads per block of the sort pass
constexpr int FT = 128;      // threads per block of the dt pass
constexpr int PB = 152 * 3;  // blocks of each pass (at most): one resident wave of the network pass

// Blocks of each cooling pass for a mesh: enough for its cells to cool at
// once (2048 cells a block), at most one wave.
int pass_blocks(const Params& p) {
  const long long n = (long long)p.nx * p.ny * p.nz;
  return (int)std::max<long long>(4, std::min<long long>((n + 2047) / 2048, PB));
}

__device__ __forceinline__ void speeds_max(const float* w, float gf, float& m0, float& m1, float& m2) {
  const float cs = sqrtf(gf * w[4] / w[0]);
  const float v0 = fabsf(w[1]) + cs, v1 = fabsf(w[2]) + cs, v2 = fabsf(w[3]) + cs;
  m0 = (v0 != v0 || v0 > m0) ? v0 : m0;
  m1 = (v1 != v1 || v1 > m1) ? v1 : m1;
  m2 = (v2 != v2 || v2 > m2) ? v2 : m2;
}

// (32-bit divisions: a queue entry is one word; 64-bit ones were a third of a
// pass's instructions)
__device__ __forceinline__ long long interior_offset(const Params& p, const Layout& L, unsigned cidx) {
  const unsigned nx = (unsigned)p.nx, ny = (unsigned)p.ny;
  const unsigned r = cidx / nx, k = r / ny;
  return L.at(1 + (int)(cidx - r * nx), 1 + (int)(r - k * ny), 1 + (int)k);
}

// Pass 1 (sort): stage 2 queued the interior cells that cool (temp >= the
// table's first temperature, cooling.f90:71) beyond a single step of the
// exact integrator (it cooled the cells whose tau is at most the
// integrator's single-step limit itself, with this pass's arithmetic).  A
// cell inside the training box goes to the network queue; a cell outside it
// takes the exact integrator here; a queued cell whose tau is at most the
// single-step limit after all takes the single exponential step here.
// Pass 2 (network): the network queue densely, 32 cells to a warp (a warp
// of the sort pass holds a few network cells at most, and its matrix tiles
// would run for all 32 rows): the prediction, accepted when the residual
// check against the exact integrator passes, else the exact integrator's
// temperature (which the check has just computed).
// Both passes fold the block maxima of the signal speeds of the cells they
// cooled into the clock's (stage 2 left out the cells it queued); pass 3
// finishes the dt reduction and empties the queues.
// The state the step just wrote: U1 or U0 by the clock's buffer parity (the
// clock has not advanced yet), so that one captured launch serves both
// parities.
__device__ __forceinline__ double* step_output(double* U0, double* U1, const Clock* clk, long long it_base) {
  return ((clk->it - it_base) & 1LL) ? U0 : U1;
}

// Everything one mesh's cooling passes need (a kernel argument for one
// mesh, a device array entry for a batch of them).
struct CoolJob {
  Params p;  // the run's parameters, cooling = the exact integrator (the fallback)
  Layout L;
  double* U0;
  double* U1;
  long long it_base;
  Clock* clk;
  SurrogateArgs sa;
  const unsigned* cqueue;  // cells stage 2 queued (they cool)
  unsigned* cqcount;
  unsigned* nqueue;  // cells for the network
  unsigned* nqcount;
  unsigned blk0, nblk;  // this mesh's blocks of the dt pass: [blk0, blk0 + nblk)
};

// The mesh block b of a pass works on: the job whose block range holds b
// (ranges ascending, back to back).
__device__ __forceinline__ const CoolJob* job_of_block(const CoolJob* jobs, int njobs, unsigned b) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].blk0 <= b) lo = mid; else hi = mid - 1;
  }
  return &jobs[lo];
}

// A block's copy of its job in shared memory (8-byte words): the passes read
// their arguments from there whichever path launched them.
static_assert(sizeof(CoolJob) % 8 == 0 && alignof(CoolJob) <= 16, "CoolJob copies as 8-byte words");
struct SmemJob {
  alignas(16) unsigned long long w[sizeof(CoolJob) / 8];
};
__device__ __forceinline__ const CoolJob& stage_job(SmemJob& s, const CoolJob* src) {
  const unsigned long long* from = reinterpret_cast<const unsigned long long*>(src);
  for (int q = threadIdx.x; q < (int)(sizeof(CoolJob) / 8); q += blockDim.x) s.w[q] = from[q];
  __syncthreads();
  return *reinterpret_cast<const CoolJob*>(s.w);
}

// The cooling quantities of a queued cell from its state u: primitives w,
// temperature T, whether it cools (need), and for one that does its
// tau = Lambda n^2 dt / E_th, the network's normalised features and whether
// they lie in the training box.  One definition for both passes.
struct CellCool {
  float w[5], T, tau, lam, feat[3];
  bool need, inbox;
};
__device__ __forceinline__ void cell_cool(const Params& p, const SurrogateArgs& sa, const double* u, float dtf,
                                          CellCool& c) {
  const float gm1 = p.f_gamma - 1.0f;
  float cf[5];
  mixed_cell(gm1, u, 1, cf, c.w);
  // (divisions and products as intrinsics: every kernel that inlines this
  // gets the same bits)
  c.T = __fmul_rn(__fdividef(c.w[4], c.w[0]), p.f_cT);
  c.need = cools_at(p, c.T, u);
  c.tau = 0.f;
  c.lam = 0.f;
  c.feat[0] = c.feat[1] = c.feat[2] = 0.f;
  c.inbox = false;
  if (c.need) {
    const float nd = __fmul_rn(c.w[0], p.f_inv_muamu);
    const float eth = __fdividef(c.w[4], gm1);
    c.lam = cool_coef_f(p.cool, c.T);
    c.tau = __fmul_rn(__fmul_rn(__fmul_rn(c.lam, nd), __fdividef(nd, eth)), dtf);
    const float f0 = log10f(nd), f1 = log10f(c.T), f2 = log10f(c.tau);
    // inclusive, with 1e-4 dex of slack for the FP32 logarithms of cells on
    // a face of the box (e.g. a medium at the table's first temperature)
    constexpr float SL = 1e-4f;
    c.inbox = f0 >= sa.box[0] - SL && f0 <= sa.box[1] + SL && f1 >= sa.box[2] - SL && f1 <= sa.box[3] + SL &&
              f2 >= sa.box[4] - SL && f2 <= sa.box[5] + SL;
    c.feat[0] = __fdividef(__fsub_rn(f0, sa.norm[0]), sa.norm[1]);
    c.feat[1] = __fdividef(__fsub_rn(f1, sa.norm[2]), sa.norm[3]);
    c.feat[2] = __fdividef(__fmaf_rn(__log2f(c.tau), 0.301029996f, -sa.norm[4]), sa.norm[5]);  // (f2 - centre, fused)
  }
}

// Append of cell index v to a queue, one atomic for the block's ST threads
// (all of them call it).  A warp's own atomic for its 32 cells bounded the
// sort pass: a mesh's go to one address, 65 k of them for 128^3 cells (batch of
// eight bubbles: 0.287 ms a step, 0.101 so and with interior_offset in 32 bits).
struct SmemAppend {
  unsigned count[ST / 32], base[ST / 32];
};
__device__ __forceinline__ void block_append(SmemAppend& s, bool take, unsigned v, unsigned* queue, unsigned* count) {
  const unsigned qm = __ballot_sync(0xffffffffu, take);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s.count[warp] = (unsigned)__popc(qm);
  __syncthreads();
  if (warp == 0) {
    const unsigned c = lane < ST / 32 ? s.count[lane] : 0u;
    unsigned sum = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned below = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += below;
    }
    unsigned at = 0u;
    if (lane == 31 && sum) at = atomicAdd(count, sum);
    at = __shfl_sync(0xffffffffu, at, 31);
    if (lane < ST / 32) s.base[lane] = at + sum - c;
  }
  __syncthreads();
  if (take) queue[s.base[warp] + __popc(qm & ((1u << lane) - 1u))] = v;
}

// The counters of the three outcomes (network, fallback, single step).
__device__ __forceinline__ void add_counts(const SurrogateArgs& sa, unsigned used, unsigned fell, unsigned one) {
  used = __reduce_add_sync(0xffffffffu, used);
  fell = __reduce_add_sync(0xffffffffu, fell);
  one = __reduce_add_sync(0xffffffffu, one);
  if ((threadIdx.x & 31) == 0) {
    if (used) atomicAdd(&sa.counts[0], (unsigned long long)used);
    if (fell) atomicAdd(&sa.counts[1], (unsigned long long)fell);
    if (one) atomicAdd(&sa.counts[2], (unsigned long long)one);
  }
}

// Tiles [first, end) of ST queued cells of one mesh (block-uniform).
__device__ void cool_sort_mesh(const CoolJob& j, double* red, SmemAppend& app, long long first, long long end) {
  const Params& p = j.p;
  const Layout& L = j.L;
  const Clock* clk = j.clk;
  const long long n = (long long)*j.cqcount;
  double* __restrict__ U = step_output(j.U0, j.U1, clk, j.it_base);
  const float gm1 = p.f_gamma - 1.0f, gf = p.f_gamma;
  const float dtf = d2f(clk->dt);
  float m0 = 0.f, m1 = 0.f, m2 = 0.f;
  unsigned fell = 0, one = 0;
  for (long long tile = first; tile < end; ++tile) {
    const long long q = tile * ST + threadIdx.x;
    const bool valid = q < n;
    long long o = 0;
    unsigned cidx = 0;
    double u[5] = {1.0, 0.0, 0.0, 0.0, 1.0};
    if (valid) {
      cidx = j.cqueue[q];
      o = interior_offset(p, L, cidx);
#pragma unroll
      for (int e = 0; e < 5; ++e) u[e] = U[e * L.plane + o];
    }
    CellCool c;
    cell_cool(p, j.sa, u, dtf, c);
    const bool need = valid && c.need;
    // tau at most the single-step limit: the exact integrator is a single
    // exponential step, and the network has nothing to gain; outside the
    // training box the exact integrator's closed form (p.cooling: COOL_EXACT)
    const bool single = need && !(c.tau > p.f_cool_sub_frac);
    const bool net = need && !single && c.inbox;
    const bool ext = need && !single && !c.inbox;
    if (single || ext) {
      cool_cell_f(p, p.f_cT, p.f_inv_muamu, gm1, c.w, u[4], dtf, u);
      U[4 * L.plane + o] = u[4];
      speeds_max(c.w, gf, m0, m1, m2);
    }
    block_append(app, net, cidx, j.nqueue, j.nqcount);
    fell += ext ? 1 : 0;
    one += single ? 1 : 0;
  }
  add_counts(j.sa, 0, fell, one);
  cfl_contribute<ST>(m0, m1, m2, j.clk, red);
}

// A network cell: the prediction y's change where the residual check accepts
// it, else the exact integrator's; u[4] and the primitives updated.  tc: the
// tensor-core path is healthy.
__device__ __forceinline__ bool cool_net_cell(const Params& p, CellCool& c, double* u, float y, bool tc, float dtf) {
  const CoolTable& tab = p.cool;
  const float T = c.T, tau = c.tau, gm1 = p.f_gamma - 1.0f;
  // the exact integrator's change and the network's, T_new/T - 1 (the
  // network's r: ln(T_new/T) = -(tau + tau^2 r); clamped at the table's
  // first temperature, where cooling stops).  A cell whose cooling
  // reaches that temperature within the step (the exact change is the
  // floor's, T_0/T - 1) takes the exact integrator: training leaves those
  // pairs out, and the network's prediction, clamped at the floor, could
  // only err on one side.
  const float qfloor = __fsub_rn(__fdividef(tab.Tf[0], T), 1.0f);
  const float qx = cool_exact_dropf(tab, T, c.lam, tau);
  const float qf = fmaxf(expm1f(__fmul_rn(-__fmaf_rn(tau, y, 1.0f), tau)), qfloor);
  const bool ok = tc && qx > qfloor && fabsf(qf - qx) <= p.f_mlp_tol;
  if (ok) {
    const float dp = __fmul_rn(c.w[4], qf);
    c.w[4] = __fadd_rn(c.w[4], dp);
    u[4] = u[4] + f2d(__fdividef(dp, gm1));
  } else {
    cool_cell_f(p, p.f_cT, p.f_inv_muamu, gm1, c.w, u[4], dtf, u);
  }
  return ok;
}

// Tiles [first, end) of 128 queued cells of one mesh (block-uniform).
__device__ void cool_net_mesh(const CoolJob& j, umma::Smem& S, double* red, long long first, long long end, bool& tc,
                              uint32_t& phase) {
  const Params& p = j.p;
  const Layout& L = j.L;
  const Clock* clk = j.clk;
  const SurrogateArgs& sa = j.sa;
  const long long n = (long long)*j.nqcount;
  double* __restrict__ U = step_output(j.U0, j.U1, clk, j.it_base);
  umma::load_weights(sa.img, S);
  __syncthreads();
  const float gf = p.f_gamma;
  const float dtf = d2f(clk->dt);
  float m0 = 0.f, m1 = 0.f, m2 = 0.f;
  unsigned used = 0, fell = 0;
  for (long long tile = first; tile < end; ++tile) {
    const long long q = tile * CT + threadIdx.x;
    const bool valid = q < n;
    long long o = 0;
    unsigned cidx = 0;
    double u[5] = {1.0, 0.0, 0.0, 0.0, 1.0};
    if (valid) {
      cidx = j.nqueue[q];
      o = interior_offset(p, L, cidx);
#pragma unroll
      for (int e = 0; e < 5; ++e) u[e] = U[e * L.plane + o];
    }
    CellCool c;
    cell_cool(p, sa, u, dtf, c);
    float y = 0.f;
    if (tc) tc = umma::forward(S, c.feat, y, phase);
    bool ok = false;
    if (valid) {
      ok = cool_net_cell(p, c, u, y, tc, dtf);
      U[4 * L.plane + o] = u[4];
      speeds_max(c.w, gf, m0, m1, m2);
    }
    used += ok ? 1 : 0;
    fell += (valid && !ok) ? 1 : 0;
  }
  // an MMA wait ran out: the cells above took the exact integrator; the step
  // reports the timeout
  if (!tc && threadIdx.x == 0) atomicOr(&const_cast<Clock*>(clk)->status, ST_TIMEOUT);
  add_counts(sa, used, fell, 0);
  cfl_contribute<CT>(m0, m1, m2, j.clk, red);
}

// The meshes' tiles (TILE cells of a queue, its length at *count(job)) end
// to end, an equal run of them to each block of NT threads: run(job, first,
// end) for each mesh in this block's run, after begin().  (A mesh whose step
// does not run, mainHD.f90:61, has empty queues.)  Returns whether the block
// had any.  On ranges of blocks by the meshes' sizes half of the blocks were
// idle on average, the queues differing widely: batch of eight bubbles, the
// network pass 0.79 ms a step, 0.47 so (the sort pass 0.10 both ways).
template <int NT, int TILE, class Count, class Begin, class Run>
__device__ __forceinline__ bool for_runs(const CoolJob* __restrict__ jobs, int njobs, SmemJob& sj, Count count,
                                         Begin begin, Run run) {
  __shared__ unsigned tiles[NT];
  __shared__ unsigned long long total;
  const int tid = threadIdx.x;
  auto tiles_of = [&](int q) { return q < njobs ? (*count(jobs[q]) + TILE - 1u) / TILE : 0u; };
  if (tid == 0) total = 0ull;
  __syncthreads();
  unsigned mine = 0u;
  for (int q = tid; q < njobs; q += NT) mine += tiles_of(q);
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((tid & 31) == 0 && mine) atomicAdd(&total, (unsigned long long)mine);
  __syncthreads();
  const long long T = (long long)total, B = gridDim.x, b = blockIdx.x;
  const long long lo = T * b / B, hi = T * (b + 1) / B;  // this block's tiles
  if (lo == hi) return false;
  begin();
  long long at = 0;  // tiles of the meshes before
  for (int q0 = 0; q0 < njobs && at < hi; q0 += NT) {
    __syncthreads();
    tiles[tid] = tiles_of(q0 + tid);
    __syncthreads();
    for (int q = q0; q < min(q0 + NT, njobs) && at < hi; ++q) {
      const long long nt = tiles[q - q0];
      if (nt && at + nt > lo) {
        __syncthreads();  // the mesh before is done
        run(stage_job(sj, &jobs[q]), max(lo - at, 0LL), min(hi - at, nt));
      }
      at += nt;
    }
  }
  return true;
}

// The sort pass of njobs meshes.
__global__ void __launch_bounds__(ST) k_cool_sort(const CoolJob* __restrict__ jobs, int njobs) {
  __shared__ double red[96];
  __shared__ SmemAppend app;
  __shared__ SmemJob sj;
  for_runs<ST, ST>(
      jobs, njobs, sj, [](const CoolJob& j) { return j.cqcount; }, [] {},
      [&](const CoolJob& j, long long first, long long end) { cool_sort_mesh(j, red, app, first, end); });
}

// The network pass.
__global__ void __launch_bounds__(CT, 3) k_cool_net(const CoolJob* __restrict__ jobs, int njobs) {
  __shared__ umma::Smem S;
  __shared__ double red[96];
  __shared__ SmemJob sj;
  bool tc = true;  // the tensor-core path is healthy (block-wide)
  uint32_t phase = 0;
  const bool any = for_runs<CT, CT>(
      jobs, njobs, sj, [](const CoolJob& j) { return j.nqcount; }, [&] { umma::setup(S); },
      [&](const CoolJob& j, long long first, long long end) { cool_net_mesh(j, S, red, first, end, tc, phase); });
  if (!any) return;
  if (!tc) umma::drain(S, phase);
  umma::teardown(S);
}

__device__ void cool_dt_mesh(const CoolJob& j, double* red, int* flag, unsigned nblocks) {
  Clock* clk = j.clk;
  if (!(clk->t < clk->tfin)) return;
  cfl_reduce_finalize_n<FT>(0.0f, 0.0f, 0.0f, clk, j.p, true, red, flag, nblocks);
  if (*flag && threadIdx.x == 0) {
    *j.cqcount = 0u;
    *j.nqcount = 0u;
  }
}

// Pass 3: the dt reduction over the block maxima of stage 2 and the two
// cooling passes (this pass's blocks only take their tickets); the last
// block of a mesh empties its queues.
__global__ void __launch_bounds__(FT) k_cool_dt(const CoolJob* __restrict__ jobs, int njobs) {
  __shared__ double red[96];
  __shared__ int flag;
  __shared__ SmemJob sj;
  const CoolJob& j = stage_job(sj, job_of_block(jobs, njobs, blockIdx.x));
  cool_dt_mesh(j, red, &flag, j.nblk);
}

// The single-mesh step's cooling in one launch: the three passes' work on
// stage 2's queue directly, the last block to finish closing the dt reduction
// and emptying the queue.  Nearly every queued cell is the network's (stage 2
// cools the others), so sorting them first gains no density here, and the
// passes were latency: three launches of a few tiles each, 49 us of a 48^3
// clumpy step (the stages take 56) and 72 us at 128^3.  (The batched step
// keeps the three passes; one launch over its members' queues is not tried.)
__global__ void __launch_bounds__(2 * CT, 2) k_cool_all(const __grid_constant__ CoolJob j) {
  __shared__ umma::Smem S;
  __shared__ float x3[3][CT], acc[CT];
  __shared__ double red[96];
  __shared__ int flag;
  const Params& p = j.p;
  const Layout& L = j.L;
  Clock* clk = j.clk;
  const SurrogateArgs& sa = j.sa;
  // launched before stage 2 has ended (programmatic dependent launch): the
  // weights and the TMEM columns come in beside its last wave
  umma::load_weights(sa.img, S);
  umma::setup(S);
  // and the cooling table's FP32 columns into L1 (a cell walks them in a dozen
  // dependent loads)
  {
    const CoolTable& t = p.cool;
    const float* cols[5] = {t.Tf, t.logTf, t.Cf, t.slopef, t.gcumf};
#pragma unroll
    for (int e = 0; e < 5; ++e)
      for (int q = 32 * (int)threadIdx.x; q < t.n; q += 32 * 2 * CT)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(cols[e] + q));
  }
  cudaGridDependencySynchronize();
  if (!(clk->t < clk->tfin)) {  // the step did not run (mainHD.f90:61)
    umma::teardown(S);
    return;
  }
  const long long n = (long long)*j.cqcount;
  double* __restrict__ U = step_output(j.U0, j.U1, clk, j.it_base);
  const float gm1 = p.f_gamma - 1.0f, gf = p.f_gamma;
  const float dtf = d2f(clk->dt);
  float m0 = 0.f, m1 = 0.f, m2 = 0.f;
  unsigned used = 0, fell = 0, one = 0;
  uint32_t phase = 0;
  bool tc = true;
  for (long long base = (long long)blockIdx.x * CT; base < n; base += (long long)gridDim.x * CT) {
    // the lower 128 threads hold a cell each, the upper ones help with the network
    const long long q = base + threadIdx.x;
    const bool valid = threadIdx.x < CT && q < n;
    long long o = 0;
    double u[5] = {1.0, 0.0, 0.0, 0.0, 1.0};
    if (valid) {
      o = interior_offset(p, L, j.cqueue[q]);
#pragma unroll
      for (int e = 0; e < 5; ++e) u[e] = U[e * L.plane + o];
    }
    CellCool c;
    c.need = false;
    if (threadIdx.x < CT) {
      cell_cool(p, sa, u, dtf, c);
#pragma unroll
      for (int e = 0; e < 3; ++e) x3[e][threadIdx.x] = c.feat[e];
    }
    const bool need = valid && c.need;
    const bool single = need && !(c.tau > p.f_cool_sub_frac);
    const bool net = need && !single && c.inbox;
    if (__syncthreads_or(net) && tc) {
      tc = umma::forward2(S, x3, acc, phase);
      __syncthreads();
    }
    if (need) {
      const float y = acc[threadIdx.x];
      bool ok = false;
      if (net)
        ok = cool_net_cell(p, c, u, y, tc, dtf);
      else
        cool_cell_f(p, p.f_cT, p.f_inv_muamu, gm1, c.w, u[4], dtf, u);
      U[4 * L.plane + o] = u[4];
      speeds_max(c.w, gf, m0, m1, m2);
      used += ok ? 1 : 0;
      one += single ? 1 : 0;
      fell += (!ok && !single) ? 1 : 0;
    }
  }
  if (!tc) {
    // an MMA wait ran out: the cells took the exact integrator; the step
    // reports the timeout
    if (threadIdx.x == 0) atomicOr(&clk->status, ST_TIMEOUT);
    umma::drain(S, phase);
  }
  umma::teardown(S);
  add_counts(sa, used, fell, one);
  cfl_reduce_finalize_n<2 * CT>(m0, m1, m2, clk, p, true, red, &flag, gridDim.x);
  if (flag && threadIdx.x == 0) *j.cqcount = 0u;
}

}  // namespace

size_t cool_job_bytes() { return sizeof(CoolJob); }

void fill_cool_job(void* dst, const Params& p, const Layout& L, double* U0, double* U1, long long it_base, Clock* clk,
                   const void* img, const float norm[6], const double box[6], unsigned long long* counts,
                   const unsigned* cqueue, unsigned* cqcount, unsigned* nqueue, unsigned* nqcount, int blk0,
                   int nblk) {
  CoolJob j{};
  j.p = p;
  j.p.cooling = COOL_EXACT;  // the fallback: the exact integrator (single step up to the run's cool_sub_frac)
  j.L = L;
  j.U0 = U0;
  j.U1 = U1;
  j.it_base = it_base;
  j.clk = clk;
  j.sa.img = static_cast<const mlp::SmemWeights*>(img);
  for (int q = 0; q < 6; ++q) {
    j.sa.norm[q] = norm[q];
    j.sa.box[q] = (float)box[q];
  }
  j.sa.counts = counts;
  j.cqueue = cqueue;
  j.cqcount = cqcount;
  j.nqueue = nqueue;
  j.nqcount = nqcount;
  j.blk0 = (unsigned)blk0;
  j.nblk = (unsigned)nblk;
  std::memcpy(dst, &j, sizeof j);
}

cudaError_t launch_cool_mlp_dt(const Params& p, const Layout& L, double* U0, double* U1, long long it_base,
                               Clock* clk, const void* img, const float norm[6], const double box[6],
                               unsigned long long* counts, const unsigned* cqueue, unsigned* cqcount,
                               cudaStream_t s) {
  // a 128-cell tile for every 512 cells (a tenth to a quarter of a clumpy
  // medium is queued), at most one resident wave (2 blocks per SM)
  const long long n = (long long)p.nx * p.ny * p.nz;
  const int nb = (int)std::min<long long>((n + 511) / 512, 152 * 2);
  CoolJob j;
  fill_cool_job(&j, p, L, U0, U1, it_base, clk, img, norm, box, counts, cqueue, cqcount, nullptr, nullptr, 0, nb);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nb);
  cfg.blockDim = dim3(2 * CT);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_cool_all, j);
}

int cool_pass_blocks(const Params& p) { return pass_blocks(p); }

cudaError_t launch_cool_mlp_dt_batch(const void* jobs, int njobs, int nblocks, cudaStream_t s) {
  const CoolJob* d = static_cast<const CoolJob*>(jobs);
  k_cool_sort<<<nblocks, ST, 0, s>>>(d, njobs);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_cool_net<<<nblocks, CT, 0, s>>>(d, njobs);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_cool_dt<<<nblocks, FT, 0, s>>>(d, njobs);
  return cudaGetLastError();
}


}  // namespace tlq

// ===========================================================================
// Host side
// ===========================================================================
namespace {

int sfail(tlq_ctx* c, int code, const std::string& m) {
  if (c) c->err = m;
  return code;
}

#define SCK(call)                                                                                  \
  do {                                                                                             \
    cudaError_t e_ = (call);                                                                       \
    if (e_ != cudaSuccess) return sfail(ctx, TLQ_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Parameters of the training pairs' integrator (the context's physics and
// table): the exact integrator's closed form when sub_frac is 0, else the
// sub-cycled integrator with the given sub-steps (extrapolated).
Params exact_params(const tlq_ctx* ctx, double sub_frac, int max_sub) {
  Params p = ctx->P;
  p.cooling = sub_frac > 0.0 ? COOL_SUBCYCLE : COOL_EXACT;
  p.cool_sub_frac = sub_frac;
  p.cool_max_sub = max_sub;
  return p;
}

// Initial parameters: uniform(-a, a) with a = sqrt(6/(fan_in + fan_out)).
void init_params(std::vector<float>& P, unsigned long long seed) {
  using namespace tlq::mlp;
  std::mt19937_64 rng(seed ^ 0x5eedULL);
  auto fill = [&](int off, int fo, int fi) {
    const float a = std::sqrt(6.0f / (float)(fi + fo));
    std::uniform_real_distribution<float> d(-a, a);
    for (int q = 0; q < fo * fi; ++q) P[off + q] = d(rng);
  };
  std::fill(P.begin(), P.end(), 0.0f);
  fill(OFF_W1, HID, IN);
  fill(OFF_W2, HID, HID);
  fill(OFF_W3, HID, HID);
  fill(OFF_W4, 1, HID);
  P[OFF_B4] = 0.0f;
}

}  // namespace

extern "C" {

void tlq_surrogate_opts_default(tlq_surrogate_opts* o) {
  if (!o) return;
  std::memset(o, 0, sizeof(*o));
  o->nsamples = 20000000LL;
  o->epochs = 30;
  o->batch = 4096;
  o->lr = 3e-3f;
  o->seed = 12345ULL;
  const double box[6] = {-4.0, 4.0, 4.0, 8.5, -8.0, 1.0};
  for (int q = 0; q < 6; ++q) o->box[q] = box[q];
  o->sub_frac = 0.0;  // the exact integrator's closed form
  o->max_sub = 20000;
}

int tlq_cooling_pairs(tlq_ctx* ctx, long long n, unsigned long long seed, const double* box6, double sub_frac,
                      int max_sub, float* X, float* Y, double* raw) {
  if (!ctx || n <= 0 || !box6 || !X || !Y || !(sub_frac >= 0.0) || max_sub < 1) return TLQ_ERR_ARG;
  if (!ctx->dT) return sfail(ctx, TLQ_ERR_STATE, "cooling table not set");
  float *dX = nullptr, *dY = nullptr;
  double* dR = nullptr;
  SCK(cudaMalloc(&dX, 3 * n * sizeof(float)));
  SCK(cudaMalloc(&dY, n * sizeof(float)));
  if (raw) SCK(cudaMalloc(&dR, 4 * n * sizeof(double)));
  const Params p = exact_params(ctx, sub_frac, max_sub);
  cudaError_t e = launch_cool_pairs(p, n, seed, box6, dX, dY, nullptr, dR, ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(X, dX, 3 * n * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(Y, dY, n * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess && raw) e = cudaMemcpyAsync(raw, dR, 4 * n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  cudaFree(dX);
  cudaFree(dY);
  cudaFree(dR);
  if (e != cudaSuccess) return sfail(ctx, TLQ_ERR_CUDA, std::string("cooling pairs: ") + cudaGetErrorString(e));
  return TLQ_OK;
}

int tlq_train_cooling_surrogate(tlq_ctx* ctx, const tlq_surrogate_opts* opts, tlq_surrogate_report* rep) {
  using namespace tlq::mlp;
  if (!ctx) return TLQ_ERR_ARG;
  tlq_surrogate_opts o;
  if (opts) o = *opts; else tlq_surrogate_opts_default(&o);
  if (o.nsamples < 2 * o.batch || o.batch < 16 || o.epochs < 1) return sfail(ctx, TLQ_ERR_ARG, "bad training options");
  if (!ctx->dT) return sfail(ctx, TLQ_ERR_STATE, "cooling table not set");
  const long long N = o.nsamples;
  const long long Nval = std::max<long long>(o.batch, N / 100);
  const long long Ntr = N - Nval;
  float norm[6];
  for (int q = 0; q < 3; ++q) {
    norm[2 * q] = (float)(0.5 * (o.box[2 * q] + o.box[2 * q + 1]));
    norm[2 * q + 1] = (float)(0.5 * (o.box[2 * q + 1] - o.box[2 * q]));
  }
  cudaStream_t s = ctx->stream;
  float *X = nullptr, *Y = nullptr, *X2 = nullptr, *Y2 = nullptr, *P = nullptr, *m = nullptr, *v = nullptr,
        *grad = nullptr, *loss = nullptr, *Yp = nullptr, *Wt = nullptr, *Wt2 = nullptr;
  long long* perm = nullptr;
  int rc = TLQ_OK;
  auto t0 = std::chrono::steady_clock::now();
  auto cleanup = [&]() {
    cudaFree(X); cudaFree(Y); cudaFree(X2); cudaFree(Y2); cudaFree(m); cudaFree(v); cudaFree(grad);
    cudaFree(Wt); cudaFree(Wt2);
    cudaFree(loss); cudaFree(Yp); cudaFree(perm);
  };
#define TCK(call)                                                                              \
  do {                                                                                         \
    cudaError_t e_ = (call);                                                                   \
    if (e_ != cudaSuccess) {                                                                   \
      cleanup();                                                                               \
      cudaFree(P);                                                                             \
      return sfail(ctx, TLQ_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));     \
    }                                                                                          \
  } while (0)
  TCK(cudaMalloc(&X, 3 * N * sizeof(float)));
  TCK(cudaMalloc(&Y, N * sizeof(float)));
  TCK(cudaMalloc(&X2, 3 * N * sizeof(float)));
  TCK(cudaMalloc(&Y2, N * sizeof(float)));
  TCK(cudaMalloc(&Wt, N * sizeof(float)));
  TCK(cudaMalloc(&Wt2, N * sizeof(float)));
  TCK(cudaMalloc(&perm, N * sizeof(long long)));
  TCK(cudaMalloc(&P, NPARAM * sizeof(float)));
  TCK(cudaMalloc(&m, NPARAM * sizeof(float)));
  TCK(cudaMalloc(&v, NPARAM * sizeof(float)));
  TCK(cudaMalloc(&grad, NPARAM * sizeof(float)));
  TCK(cudaMalloc(&loss, sizeof(float)));
  TCK(cudaMalloc(&Yp, Nval * sizeof(float)));
  // pairs (stratified in tau), shuffled, normalised
  const Params pe = exact_params(ctx, o.sub_frac, o.max_sub);
  TCK(launch_cool_pairs(pe, N, o.seed, o.box, X, Y, Wt, nullptr, s));
  {
    std::vector<long long> hp(N);
    std::iota(hp.begin(), hp.end(), 0LL);
    std::mt19937_64 rng(o.seed * 2654435761ULL + 7);
    std::shuffle(hp.begin(), hp.end(), rng);
    TCK(cudaMemcpyAsync(perm, hp.data(), N * sizeof(long long), cudaMemcpyHostToDevice, s));
    TCK(launch_gather_pairs(X, Y, Wt, perm, N, X2, Y2, Wt2, s));
    TCK(cudaStreamSynchronize(s));
  }
  auto t1 = std::chrono::steady_clock::now();
  TCK(launch_normalise(X2, N, norm, s));
  std::vector<float> hP(NPARAM);
  init_params(hP, o.seed);
  TCK(cudaMemcpyAsync(P, hP.data(), NPARAM * sizeof(float), cudaMemcpyHostToDevice, s));
  TCK(cudaMemsetAsync(m, 0, NPARAM * sizeof(float), s));
  TCK(cudaMemsetAsync(v, 0, NPARAM * sizeof(float), s));
  const long long steps_per_epoch = Ntr / o.batch;
  const long long total = steps_per_epoch * o.epochs;
  float lfirst = 0.f, llast = 0.f;
  long long t = 0;
  for (int ep = 0; ep < o.epochs; ++ep) {
    for (long long b = 0; b < steps_per_epoch; ++b) {
      ++t;
      const float lr = o.lr * (0.05f + 0.95f * 0.5f * (1.0f + std::cos(3.14159265f * (float)(t - 1) / (float)total)));
      TCK(cudaMemsetAsync(grad, 0, NPARAM * sizeof(float), s));
      TCK(cudaMemsetAsync(loss, 0, sizeof(float), s));
      TCK(launch_mlp_grad(P, X2 + 3 * b * o.batch, Y2 + b * o.batch, Wt2 + b * o.batch, o.batch, grad, loss, s));
      TCK(launch_adam(P, m, v, grad, NPARAM, lr, 0.9f, 0.999f, 1e-8f, (int)t, s));
      if (t == 1) {
        TCK(cudaMemcpyAsync(&lfirst, loss, sizeof(float), cudaMemcpyDeviceToHost, s));
        TCK(cudaStreamSynchronize(s));
      }
    }
  }
  TCK(cudaMemcpyAsync(&llast, loss, sizeof(float), cudaMemcpyDeviceToHost, s));
  // held-out pairs
  TCK(launch_mlp_infer(P, X2 + 3 * Ntr, (int)Nval, Yp, s));
  std::vector<float> hx(3 * Nval), hy(Nval), hyp(Nval), hw(Nval);
  TCK(cudaMemcpyAsync(hw.data(), Wt2 + Ntr, Nval * sizeof(float), cudaMemcpyDeviceToHost, s));
  TCK(cudaMemcpyAsync(hx.data(), X2 + 3 * Ntr, 3 * Nval * sizeof(float), cudaMemcpyDeviceToHost, s));
  TCK(cudaMemcpyAsync(hy.data(), Y2 + Ntr, Nval * sizeof(float), cudaMemcpyDeviceToHost, s));
  TCK(cudaMemcpyAsync(hyp.data(), Yp, Nval * sizeof(float), cudaMemcpyDeviceToHost, s));
  TCK(cudaStreamSynchronize(s));
  auto t2 = std::chrono::steady_clock::now();
  // held-out pairs that do not complete (the step's network cells): T_new/T
  // as the step forms it (clamped at the table's first temperature)
  double se = 0.0, mx = 0.0;
  std::vector<double> rel;
  rel.reserve(Nval);
  for (long long q = 0; q < Nval; ++q) {
    if (!(hw[q] > 0.0f)) continue;
    const double T = std::pow(10.0, (double)hx[3 * q + 1] * norm[3] + norm[2]);
    const double tau = std::pow(10.0, (double)hx[3 * q + 2] * norm[5] + norm[4]);
    const double d = tau * ((double)hyp[q] - (double)hy[q]);  // error of y = 1 + tau r
    se += d * d;
    // network output r: T_new/T = exp(-(tau + tau^2 r))
    const double pred = std::max(std::exp(-(tau + tau * tau * (double)hyp[q])), ctx->cool_tmin / T);
    rel.push_back(std::fabs(pred - std::exp(-(tau + tau * tau * (double)hy[q]))));  // |dT|/T
    mx = std::max(mx, rel.back());
  }
  if (rel.empty()) rel.push_back(0.0);
  std::sort(rel.begin(), rel.end());
  if (!ctx->mlp_image && cudaMalloc(&ctx->mlp_image, tlq::mlp_image_bytes()) != cudaSuccess) {
    cleanup();
    cudaFree(P);
    return sfail(ctx, TLQ_ERR_NOMEM, "network image");  // (the previous network, if any, stays)
  }
  cudaFree(ctx->mlp_params);
  ctx->mlp_params = P;
  if (tlq::launch_pack_weights(P, ctx->mlp_image, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) {
    cleanup();
    ctx->mlp_ready = false;
    return sfail(ctx, TLQ_ERR_CUDA, "network image");
  }
  for (int q = 0; q < 6; ++q) {
    ctx->mlp_norm[q] = norm[q];
    ctx->mlp_box[q] = o.box[q];
  }
  ctx->mlp_ready = true;
  invalidate_graphs(ctx);
  if (rep) {
    rep->loss_first = lfirst;
    rep->loss_last = llast;
    rep->val_rmse_y = std::sqrt(se / (double)rel.size());
    rep->val_max_rel_T = mx;
    rep->val_p99_rel_T = rel[(size_t)(0.99 * (double)(rel.size() - 1))];
    rep->val_accept = (double)(std::upper_bound(rel.begin(), rel.end(), 1e-3) - rel.begin()) / (double)rel.size();
    rep->ms_generate = std::chrono::duration<double, std::milli>(t1 - t0).count();
    rep->ms_train = std::chrono::duration<double, std::milli>(t2 - t1).count();
    rep->steps = t;
  }
  cleanup();
#undef TCK
  return rc;
}

int tlq_get_cooling_surrogate(tlq_ctx* ctx, float* params, float* norm6, double* box6) {
  if (!ctx) return TLQ_ERR_ARG;
  if (!ctx->mlp_ready) return sfail(ctx, TLQ_ERR_STATE, "no cooling surrogate");
  if (params) SCK(cudaMemcpy(params, ctx->mlp_params, tlq::mlp::NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
  if (norm6) std::memcpy(norm6, ctx->mlp_norm, 6 * sizeof(float));
  if (box6) std::memcpy(box6, ctx->mlp_box, 6 * sizeof(double));
  return TLQ_OK;
}

int tlq_set_cooling_surrogate(tlq_ctx* ctx, const float* params, const float* norm6, const double* box6) {
  if (!ctx || !params || !norm6 || !box6) return TLQ_ERR_ARG;
  ctx->mlp_ready = false;  // until the parameters and their image are the new network's
  if (!ctx->mlp_params) SCK(cudaMalloc(&ctx->mlp_params, tlq::mlp::NPARAM * sizeof(float)));
  // (on the stream of the kernel that packs them: see tlq_set_cooling_table)
  SCK(cudaMemcpyAsync(ctx->mlp_params, params, tlq::mlp::NPARAM * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
  if (!ctx->mlp_image) SCK(cudaMalloc(&ctx->mlp_image, tlq::mlp_image_bytes()));
  SCK(tlq::launch_pack_weights(ctx->mlp_params, ctx->mlp_image, ctx->stream));
  SCK(cudaStreamSynchronize(ctx->stream));
  std::memcpy(ctx->mlp_norm, norm6, 6 * sizeof(float));
  std::memcpy(ctx->mlp_box, box6, 6 * sizeof(double));
  ctx->mlp_ready = true;
  invalidate_graphs(ctx);
  return TLQ_OK;
}

int tlq_mlp_loss_grad(const float* params, const float* X, const float* Y, const float* Wt, int n, float* grad,
                      float* loss) {
  if (!params || !X || !Y || n < 1 || !grad || !loss) return TLQ_ERR_ARG;
  // One allocation a call (the gradient and the loss first, so that they
  // clear and return in one copy each): six took 83 us and as many frees 69,
  // one takes 40 and 34.
  using tlq::mlp::NPARAM;
  constexpr size_t OUT = (NPARAM + 1 + 63) / 64 * 64;  // floats, whole 256-byte lines
  const size_t m = ((size_t)n + 63) / 64 * 64;
  float* d = nullptr;
  cudaError_t e = cudaMalloc(&d, (2 * OUT + (Wt ? 5 : 4) * m) * sizeof(float));
  if (e != cudaSuccess) return TLQ_ERR_CUDA;
  float *dP = d + OUT, *dX = dP + OUT, *dY = dX + 3 * m, *dW = Wt ? dY + m : nullptr;
  float out[NPARAM + 1];
  if (Wt) e = cudaMemcpy(dW, Wt, (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dP, params, NPARAM * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dX, X, 3 * (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dY, Y, (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(d, 0, (NPARAM + 1) * sizeof(float));
  if (e == cudaSuccess) e = launch_mlp_grad(dP, dX, dY, dW, n, d, d + NPARAM, 0);
  if (e == cudaSuccess) e = cudaMemcpy(out, d, (NPARAM + 1) * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return TLQ_ERR_CUDA;
  std::memcpy(grad, out, NPARAM * sizeof(float));
  *loss = out[NPARAM];
  return TLQ_OK;
}

int tlq_mlp_infer(const float* params, const float* X, int n, float* Yout) {
  if (!params || !X || n < 1 || !Yout) return TLQ_ERR_ARG;
  float *dP = nullptr, *dX = nullptr, *dY = nullptr;
  cudaError_t e = cudaMalloc(&dP, tlq::mlp::NPARAM * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&dX, 3 * (size_t)n * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&dY, (size_t)n * sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(dP, params, tlq::mlp::NPARAM * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dX, X, 3 * (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = launch_mlp_infer(dP, dX, n, dY, 0);
  if (e == cudaSuccess) e = cudaMemcpy(Yout, dY, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(dP); cudaFree(dX); cudaFree(dY);
  return e == cudaSuccess ? TLQ_OK : TLQ_ERR_CUDA;
}

}  // extern "C"
