// tlq_mlp.cu -- training and inference kernels of the cooling surrogate, and
// the generator of its training pairs (the exact, finely sub-cycled form of
// the reference's cooling step, source/cooling.f90:64-112, in FP64).
//
// Numerics (mirrored by the CPU oracle oracle/mlp_oracle.py): the weights of
// the hidden layers 2 and 3 and every activation fed to a tensor-core
// product are rounded to BF16; products accumulate in FP32; the input and
// output layers, biases, pre-activations, SiLU derivatives, the loss
// gradient, the layer-1 and layer-4 weight gradients are FP32.
#include <algorithm>

#include "tlq_internal.h"
#include "tlq_mlp.cuh"
#include "tlq_umma.cuh"

namespace tlq {
namespace mlp {

constexpr int TW = 8;        // warps per training block: one per (layer, 16 rows) of the two 64 x 64 gradients
constexpr int TT = TW * 32;  // threads per training block
constexpr int TS = 16;       // samples per warp tile
constexpr int NVEC = 7;      // 64-wide gradients: W4, b3, b2, b1 and W1's three columns

struct TrainSmem {
  SmemWeights W;
  // Each warp's tile for the weight gradients, sample by feature: dZ3, H2, dZ2, H1
  alignas(16) __nv_bfloat16 st[4][TW][TS][LD];
  float vec[TW][NVEC][HID];
  float b4[TW], loss[TW];
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t r[4], uint32_t addr) {
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

// acc = bias + A W^T (the layer), or A W (BACK: the layer's transpose), 64 x
// 64, for one m16 tile; the operand fragments two k-tiles at a time, the
// eight column tiles' products of a k-tile one after another (independent).
template <bool BACK>
__device__ __forceinline__ void train_dense(float acc[8][4], const uint32_t a[4][4], const __nv_bfloat16 (*w)[LD],
                                            const float* bias, int lane) {
  const int tig = lane & 3;
  // lane l gives the address of row l % 8 of 8 x 8 matrix l / 8
  const uint32_t base = smem_addr(BACK ? &w[lane][0] : &w[lane & 7][8 * (lane >> 3)]);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float b0 = bias ? bias[8 * j + 2 * tig] : 0.0f, b1 = bias ? bias[8 * j + 2 * tig + 1] : 0.0f;
    acc[j][0] = b0; acc[j][1] = b1; acc[j][2] = b0; acc[j][3] = b1;
  }
#pragma unroll
  for (int kp = 0; kp < 2; ++kp) {
    uint32_t b[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      ldmatrix4<BACK>(b[j], base + (uint32_t)sizeof(__nv_bfloat16) *
                                       (BACK ? 32 * kp * LD + 8 * j : 8 * j * LD + 32 * kp));
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) mma_bf16(acc[j], a[2 * kp + k], b[j][2 * k], b[j][2 * k + 1]);
  }
}

// A fragment set (rows g, g+8; 64 columns) into a staging tile.
__device__ __forceinline__ void stage(__nv_bfloat16 (*dst)[LD], const uint32_t a[4][4], int g, int tig) {
#pragma unroll
  for (int kt = 0; kt < 4; ++kt) {
    *reinterpret_cast<uint32_t*>(&dst[g][16 * kt + 2 * tig]) = a[kt][0];
    *reinterpret_cast<uint32_t*>(&dst[g + 8][16 * kt + 2 * tig]) = a[kt][1];
    *reinterpret_cast<uint32_t*>(&dst[g][16 * kt + 8 + 2 * tig]) = a[kt][2];
    *reinterpret_cast<uint32_t*>(&dst[g + 8][16 * kt + 8 + 2 * tig]) = a[kt][3];
  }
}

__device__ __forceinline__ void frag_plain(uint32_t a[4][4], const float d[8][4]) {
#pragma unroll
  for (int kt = 0; kt < 4; ++kt) {
    a[kt][0] = pack_bf16(d[2 * kt][0], d[2 * kt][1]);
    a[kt][1] = pack_bf16(d[2 * kt][2], d[2 * kt][3]);
    a[kt][2] = pack_bf16(d[2 * kt + 1][0], d[2 * kt + 1][1]);
    a[kt][3] = pack_bf16(d[2 * kt + 1][2], d[2 * kt + 1][3]);
  }
}

// z -> silu(z) and silu'(z), with one sigmoid.
__device__ __forceinline__ void silu_both(float h[8][4], float ds[8][4], const float z[8][4]) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float sg = recip_ge1(1.0f + __expf(-z[j][q]));
      h[j][q] = z[j][q] * sg;
      ds[j][q] = sg * (1.0f + z[j][q] * (1.0f - sg));
    }
}

// v[2 j + h] over the 8 lanes that share tig, each adding its column sums 8 j
// + 2 tig + h: lane g keeps j = g (14 exchanges for 16 sums, where a sum
// per column takes 48), added to acc[0..1].
__device__ __forceinline__ void add_column_sums(float acc[2], const float v[16], int lane) {
  float a[8], b[4];
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
  for (int q = 0; q < 8; ++q)
    a[q] = (h4 ? v[8 + q] : v[q]) + __shfl_xor_sync(0xffffffffu, h4 ? v[q] : v[8 + q], 16);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    b[q] = (h3 ? a[4 + q] : a[q]) + __shfl_xor_sync(0xffffffffu, h3 ? a[q] : a[4 + q], 8);
#pragma unroll
  for (int q = 0; q < 2; ++q)
    acc[q] += (h2 ? b[2 + q] : b[q]) + __shfl_xor_sync(0xffffffffu, h2 ? b[q] : b[2 + q], 4);
}

// One pass over a minibatch: loss sum_i |w_i| e_i^2 / nb and its gradient
// w.r.t. the FP32 parameters P, on features X (3 per sample, normalised),
// targets Y and weights Wt (all 1 when null), e_i = y_i - t_i, or
// min(y_i - t_i, 0) where w_i < 0 (a one-sided target: y_i >= t_i).  grad and
// loss are accumulated with global atomics, once per block.
//
// A warp takes 16 samples through the forward and the backward pass in
// registers and stages dZ and H of the two 64 x 64 layers; the block's eight
// warps then share those layers' weight gradients, 16 rows of one layer
// each over the block's 128 samples, and hold them in registers until the
// end (added with FP32 additions every 16 samples, as the products' own
// accumulator starts at zero).  Each pre-activation's sigmoid is evaluated
// once, for the activation and its derivative.  262,144 samples: 637 us with
// shared-memory atomics for every 16 samples' gradient, a sum over lanes per
// column and three sigmoids, 105 us now.  Latency bounds it: one block of 8
// warps an SM (255 registers a thread) uses 46 % of the issue slots, the tensor
// pipe is 22 % busy, and a warp waits on fixed latencies (0.83 of its cycles per
// issue) and on loads (0.78).
__global__ void __launch_bounds__(TT) k_mlp_grad(const float* __restrict__ P, const float* __restrict__ X,
                                                 const float* __restrict__ Y, const float* __restrict__ Wt, int nb,
                                                 float* grad, float* loss) {
  extern __shared__ __align__(16) unsigned char sm_[];
  TrainSmem& s = *reinterpret_cast<TrainSmem*>(sm_);
  load_weights(P, s.W);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  const float inv_nb = 1.0f / (float)nb;
  const int ntiles = (nb + TS - 1) / TS;
  float gw[8][4], vec[NVEC][2], gb4 = 0.0f, part = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) gw[j][q] = 0.0f;
#pragma unroll
  for (int q = 0; q < NVEC; ++q) vec[q][0] = vec[q][1] = 0.0f;
  for (int tile0 = blockIdx.x * TW; tile0 < ntiles; tile0 += gridDim.x * TW) {
    const int tile = tile0 + warp;
    if (tile < ntiles) {
      const int r0 = tile * TS + g, r1 = r0 + 8;
      const bool v0 = r0 < nb, v1 = r1 < nb;
      float xg[3] = {0.f, 0.f, 0.f}, xg8[3] = {0.f, 0.f, 0.f};
      if (v0) for (int f = 0; f < 3; ++f) xg[f] = X[3 * (size_t)r0 + f];
      if (v1) for (int f = 0; f < 3; ++f) xg8[f] = X[3 * (size_t)r1 + f];
      float d[8][4], h[8][4], ds1[8][4], ds2[8][4], ds3[8][4], v[16];
      uint32_t a[4][4];
      input_layer(d, s.W, xg, xg8, tig);
      silu_both(h, ds1, d);
      frag_plain(a, h);
      stage(s.st[3][warp], a, g, tig);
      train_dense<false>(d, a, s.W.w2, s.W.b2, lane);
      silu_both(h, ds2, d);
      frag_plain(a, h);
      stage(s.st[1][warp], a, g, tig);
      train_dense<false>(d, a, s.W.w3, s.W.b3, lane);
      silu_both(h, ds3, d);
      // output layer in FP32: this lane's 16 columns, then the sum over tig
      float y0 = 0.0f, y1 = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = 8 * j + 2 * tig;
        y0 += s.W.w4[c] * h[j][0] + s.W.w4[c + 1] * h[j][1];
        y1 += s.W.w4[c] * h[j][2] + s.W.w4[c + 1] * h[j][3];
      }
      y0 += __shfl_xor_sync(0xffffffffu, y0, 1);
      y1 += __shfl_xor_sync(0xffffffffu, y1, 1);
      y0 += __shfl_xor_sync(0xffffffffu, y0, 2);
      y1 += __shfl_xor_sync(0xffffffffu, y1, 2);
      y0 = s.W.b4 + y0;  // row g
      y1 = s.W.b4 + y1;  // row g + 8
      // d loss / d y = 2 w (y - t) / nb (rows outside the batch contribute 0)
      float dy0 = 0.f, dy1 = 0.f;
      if (tig == 0) {
        float w0 = v0 ? (Wt ? Wt[r0] : 1.0f) : 0.0f, w1 = v1 ? (Wt ? Wt[r1] : 1.0f) : 0.0f;
        float e0 = v0 ? y0 - Y[r0] : 0.0f, e1 = v1 ? y1 - Y[r1] : 0.0f;
        if (w0 < 0.0f) { w0 = -w0; e0 = fminf(e0, 0.0f); }
        if (w1 < 0.0f) { w1 = -w1; e1 = fminf(e1, 0.0f); }
        dy0 = 2.0f * w0 * e0 * inv_nb;
        dy1 = 2.0f * w1 * e1 * inv_nb;
        part += (w0 * e0 * e0 + w1 * e1 * e1) * inv_nb;
        gb4 += dy0 + dy1;
      }
      dy0 = __shfl_sync(0xffffffffu, dy0, lane & ~3);
      dy1 = __shfl_sync(0xffffffffu, dy1, lane & ~3);
      // layer 4: dW4 = dy H3, dZ3 = dy W4 * silu'(z3)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = 8 * j + 2 * tig;
        const float w0 = s.W.w4[c], w1 = s.W.w4[c + 1];
        v[2 * j] = dy0 * h[j][0] + dy1 * h[j][2];
        v[2 * j + 1] = dy0 * h[j][1] + dy1 * h[j][3];
        d[j][0] = dy0 * w0 * ds3[j][0];
        d[j][1] = dy0 * w1 * ds3[j][1];
        d[j][2] = dy1 * w0 * ds3[j][2];
        d[j][3] = dy1 * w1 * ds3[j][3];
      }
      add_column_sums(vec[0], v, lane);
      // layers 3 and 2: db = sum dZ; dH = dZ W (tensor cores)
#pragma unroll
      for (int L = 0; L < 2; ++L) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[2 * j] = d[j][0] + d[j][2];
          v[2 * j + 1] = d[j][1] + d[j][3];
        }
        add_column_sums(vec[1 + L], v, lane);
        frag_plain(a, d);
        stage(s.st[2 * L][warp], a, g, tig);
        train_dense<true>(h, a, L == 0 ? s.W.w3 : s.W.w2, nullptr, lane);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) d[j][q] = h[j][q] * (L == 0 ? ds2[j][q] : ds1[j][q]);
      }
      // layer 1: db1 = sum dZ1, dW1 = dZ1^T X (K = 3, FP32)
#pragma unroll
      for (int f = -1; f < 3; ++f) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[2 * j] = f < 0 ? d[j][0] + d[j][2] : d[j][0] * xg[f] + d[j][2] * xg8[f];
          v[2 * j + 1] = f < 0 ? d[j][1] + d[j][3] : d[j][1] * xg[f] + d[j][3] * xg8[f];
        }
        add_column_sums(vec[4 + f], v, lane);
      }
    }
    __syncthreads();
    // dW = dZ^T H (tensor cores) of layer 3 (warps 0-3) or 2, rows 16 (warp & 3) ..
    const int nt = min(TW, ntiles - tile0), L = warp >> 2, mt = warp & 3;
    for (int t = 0; t < nt; ++t) {
      uint32_t a[4];
      // (matrices: samples 0-7 of features 0-7, 0-7 of 8-15, 8-15 of 0-7, 8-15 of 8-15)
      ldmatrix4<true>(a, smem_addr(&s.st[2 * L][t][(lane & 7) + 8 * (lane >> 4)][16 * mt + 8 * ((lane >> 3) & 1)]));
#pragma unroll
      for (int jp = 0; jp < 4; ++jp) {
        uint32_t b[4];
        ldmatrix4<true>(b, smem_addr(&s.st[2 * L + 1][t][(lane & 7) + 8 * ((lane >> 3) & 1)][16 * jp + 8 * (lane >> 4)]));
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          float acc[4] = {0.f, 0.f, 0.f, 0.f};
          mma_bf16(acc, a, b[2 * q], b[2 * q + 1]);
#pragma unroll
          for (int e = 0; e < 4; ++e) gw[2 * jp + q][e] += acc[e];
        }
      }
    }
    __syncthreads();
  }
  float* gW = grad + ((warp >> 2) ? OFF_W2 : OFF_W3) + (16 * (warp & 3) + g) * HID + 2 * tig;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    atomicAdd(reinterpret_cast<float2*>(gW + 8 * j), make_float2(gw[j][0], gw[j][1]));
    atomicAdd(reinterpret_cast<float2*>(gW + 8 * HID + 8 * j), make_float2(gw[j][2], gw[j][3]));
  }
#pragma unroll
  for (int q = 0; q < NVEC; ++q) {
    s.vec[warp][q][8 * g + 2 * tig] = vec[q][0];
    s.vec[warp][q][8 * g + 2 * tig + 1] = vec[q][1];
  }
  for (int o = 16; o > 0; o >>= 1) {
    gb4 += __shfl_xor_sync(0xffffffffu, gb4, o);
    part += __shfl_xor_sync(0xffffffffu, part, o);
  }
  if (lane == 0) {
    s.b4[warp] = gb4;
    s.loss[warp] = part;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < NVEC * HID + 2; q += TT) {
    float sum = 0.0f;
    for (int w = 0; w < TW; ++w)
      sum += q < NVEC * HID ? s.vec[w][q / HID][q % HID] : q == NVEC * HID ? s.b4[w] : s.loss[w];
    const int c = q % HID, k = q / HID;
    if (q == NVEC * HID + 1)
      atomicAdd(loss, sum);
    else
      atomicAdd(&grad[q == NVEC * HID ? OFF_B4
                      : k == 0       ? OFF_W4 + c
                      : k == 1       ? OFF_B3 + c
                      : k == 2       ? OFF_B2 + c
                      : k == 3       ? OFF_B1 + c
                                     : OFF_W1 + c * IN + (k - 4)],
                sum);
  }
}

// Adam on the FP32 master parameters.
__global__ void k_adam(float* P, float* m, float* v, const float* grad, int n, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const float gq = grad[q];
  const float mq = b1 * m[q] + (1.0f - b1) * gq;
  const float vq = b2 * v[q] + (1.0f - b2) * gq * gq;
  m[q] = mq;
  v[q] = vq;
  P[q] -= lr * (mq / c1) / (sqrtf(vq / c2) + eps);
}

// Batch inference on the tcgen05 path of the step's network pass
// (tlq_umma.cuh): 128 samples per tile, one per thread.  A tile whose MMA
// wait ran out writes NaN (the caller sees it), and the block stops.
__global__ void __launch_bounds__(umma::ROWS) k_mlp_infer_umma(const float* __restrict__ P,
                                                               const float* __restrict__ X, int n,
                                                               float* __restrict__ Yout) {
  __shared__ umma::Smem S;
  const int ntiles = (n + umma::ROWS - 1) / umma::ROWS;
  if ((int)blockIdx.x >= ntiles) return;
  umma::load_weights_fp32(P, S);
  umma::setup(S);
  uint32_t phase = 0;
  bool tc = true;
  for (int tile = blockIdx.x; tile < ntiles && tc; tile += gridDim.x) {
    const int r = tile * umma::ROWS + (int)threadIdx.x;
    float x[3] = {0.f, 0.f, 0.f};
    if (r < n)
      for (int f = 0; f < 3; ++f) x[f] = X[3 * r + f];
    float y = 0.f;
    tc = umma::forward(S, x, y, phase);
    if (r < n) Yout[r] = tc ? y : NAN;
  }
  if (!tc) umma::drain(S, phase);
  umma::teardown(S);
}

// ---------------------------------------------------------------------------
// Training pairs from the exact integrator.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t x) {  // splitmix64 finaliser
  x += 0x9e3779b97f4a7c15ULL;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
  return x ^ (x >> 31);
}
__device__ __forceinline__ double uniform01(uint64_t seed, uint64_t i, int stream) {
  return (double)(mix64(seed ^ mix64(i * 4 + stream)) >> 11) * (1.0 / 9007199254740992.0);
}

// Sample i of N: log10 n and log10 T uniform in the box, log10 tau (the
// step's cooling number Lambda(T) n^2 dt / E_th) stratified in i so that the
// 32 samples of a warp need similar numbers of sub-steps; dt follows from
// tau.  The pair is (features, r) with r = (y - 1)/tau, y = ln(T/T_new)/tau,
// T_new from the exact integrator's closed form (params' cooling
// COOL_EXACT, FP64) or from the finely sub-cycled FP64 integrator (cool_cell
// with the params' sub-step settings).  ln(T/T_new) = tau + tau^2 r is exact to first
// order whatever r is (y -> 1 as tau -> 0; r -> -(s-1)/2, s the local slope
// of the table), and r is O(1) everywhere; below tau ~ 1e-5 r is lost to
// FP64 round-off (ln(T/T_new) - tau ~ 1e-16 against tau^2), so those pairs
// are weighted (tau/1e-5)^2 -- their tau^2 r is negligible in the step.
// The sub-cycled exponential step is first order in its sub-step, so it is
// run with sub-steps of frac and frac/2 and extrapolated (Richardson):
// ln T_new = 2 ln T_(frac/2) - ln T_(frac), second order -- which still
// leaves it ~1e-5 of T above the exact solution on average (up to 3e-4)
// where cooling runs away (tau ~ 0.1-1: the cooling coefficient grows by
// decades within the step), a one-sided error a network trained on it
// inherits; hence the closed form by default.  A pair whose
// cooling reaches the table's first temperature within the step (cooling
// stops there, cooling.f90:71) is "completed": its target is the y that
// lands exactly on that temperature, with weight 0 (the step hands such
// cells to the integrator, whose last sub-step decides where below that
// temperature they end), so the network need not follow the kink at
// completion.  Other pairs have weight 1.
__global__ void k_cool_pairs(Params p, long long N, uint64_t seed, double lnlo, double lnhi, double ltlo,
                             double lthi, double lclo, double lchi, float* __restrict__ X, float* __restrict__ Y,
                             float* __restrict__ Wt, double* __restrict__ raw) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double ln = lnlo + (lnhi - lnlo) * uniform01(seed, i, 0);
  const double lt = ltlo + (lthi - ltlo) * uniform01(seed, i, 1);
  const double lc = lclo + (lchi - lclo) * (((double)i + uniform01(seed, i, 2)) / (double)N);
  const double n = pow(10.0, ln), T = pow(10.0, lt), tau = pow(10.0, lc);
  // state with density n mu0 AMU and temperature T at rest
  double w[5];
  w[0] = n * p.mu0 * AMU;
  w[1] = w[2] = w[3] = 0.0;
  w[4] = w[0] * KB * T / (p.mu0 * AMU);
  const double eth = w[4] / (p.gamma - 1.0);
  const double lam = cool_coef(p.cool, T);
  const double ce = lam * (n * n) / eth;
  const double dt = tau / ce;
  const double Tmin = p.cool.T[0];
  double Tn;
  bool completed;
  if (p.cooling == COOL_EXACT) {
    Tn = cool_exact_T(p.cool, T, lam, tau);
    completed = !(Tn > Tmin);
  } else {
    const double p0 = w[4];
    double u4 = eth;
    cool_cell(p, w, u4, dt);
    const double T1 = w[4] * p.mu0 * AMU / (w[0] * KB);
    Params ph = p;
    ph.cool_sub_frac = 0.5 * p.cool_sub_frac;
    w[4] = p0;
    u4 = eth;
    cool_cell(ph, w, u4, dt);
    const double T2 = w[4] * p.mu0 * AMU / (w[0] * KB);
    Tn = exp(2.0 * log(T2) - log(T1));
    completed = T2 < Tmin || Tn < Tmin;
  }
  if (completed) Tn = Tmin;
  X[3 * i + 0] = (float)ln;
  X[3 * i + 1] = (float)lt;
  X[3 * i + 2] = (float)lc;
  // target r = (y - 1) / tau with y = ln(T / T_new) / tau
  const double r = (-log(Tn / T) - tau) / (tau * tau);
  Y[i] = completed ? 0.0f : (float)r;
  if (Wt) Wt[i] = completed ? 0.0f : (float)fmin(1.0, (tau / 1e-5) * (tau / 1e-5));
  if (raw) {
    raw[4 * i + 0] = n;
    raw[4 * i + 1] = T;
    raw[4 * i + 2] = Tn;
    raw[4 * i + 3] = dt;
  }
}

// Gather a permutation of the pairs (shuffles the stratified order).
__global__ void k_gather_pairs(const float* __restrict__ X, const float* __restrict__ Y, const float* __restrict__ Wt,
                               const long long* perm, long long N, float* __restrict__ X2, float* __restrict__ Y2,
                               float* __restrict__ Wt2) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  const long long j = perm[i];
  X2[3 * i + 0] = X[3 * j + 0];
  X2[3 * i + 1] = X[3 * j + 1];
  X2[3 * i + 2] = X[3 * j + 2];
  Y2[i] = Y[j];
  Wt2[i] = Wt[j];
}

// Normalise raw features (log10 n, log10 T, log10 tau) to [-1, 1] over the box.
__global__ void k_normalise(float* X, long long N, float c0, float h0, float c1, float h1, float c2, float h2) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= N) return;
  X[3 * i + 0] = (X[3 * i + 0] - c0) / h0;
  X[3 * i + 1] = (X[3 * i + 1] - c1) / h1;
  X[3 * i + 2] = (X[3 * i + 2] - c2) / h2;
}

}  // namespace mlp

cudaError_t launch_cool_pairs(const Params& p, long long N, unsigned long long seed, const double box[6], float* X,
                              float* Y, float* Wt, double* raw, cudaStream_t s) {
  const int bt = 128;
  mlp::k_cool_pairs<<<(unsigned)((N + bt - 1) / bt), bt, 0, s>>>(p, N, seed, box[0], box[1], box[2], box[3], box[4],
                                                                  box[5], X, Y, Wt, raw);
  return cudaGetLastError();
}

cudaError_t launch_gather_pairs(const float* X, const float* Y, const float* Wt, const long long* perm, long long N,
                                float* X2, float* Y2, float* Wt2, cudaStream_t s) {
  mlp::k_gather_pairs<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(X, Y, Wt, perm, N, X2, Y2, Wt2);
  return cudaGetLastError();
}

cudaError_t launch_normalise(float* X, long long N, const float norm[6], cudaStream_t s) {
  mlp::k_normalise<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(X, N, norm[0], norm[1], norm[2], norm[3], norm[4],
                                                                norm[5]);
  return cudaGetLastError();
}

cudaError_t launch_mlp_grad(const float* P, const float* X, const float* Y, const float* Wt, int nb, float* grad,
                            float* loss, cudaStream_t s) {
  // (set on every call: the attribute belongs to the current device)
  const cudaError_t e = cudaFuncSetAttribute(mlp::k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(mlp::TrainSmem));
  if (e != cudaSuccess) return e;
  // a warp per 16 samples, at most a block per SM (98 KB and 256 threads of up to 255 registers)
  const int nblocks = std::max(1, std::min(152, (nb + mlp::TS * mlp::TW - 1) / (mlp::TS * mlp::TW)));
  mlp::k_mlp_grad<<<nblocks, mlp::TT, sizeof(mlp::TrainSmem), s>>>(P, X, Y, Wt, nb, grad, loss);
  return cudaGetLastError();
}

cudaError_t launch_adam(float* P, float* m, float* v, const float* grad, int n, float lr, float b1, float b2,
                        float eps, int t, cudaStream_t s) {
  const float c1 = 1.0f - powf(b1, (float)t), c2 = 1.0f - powf(b2, (float)t);
  mlp::k_adam<<<(n + 255) / 256, 256, 0, s>>>(P, m, v, grad, n, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError();
}

namespace {
__global__ void k_pack_weights(const float* __restrict__ P, mlp::SmemWeights* img) { mlp::load_weights(P, *img); }
}  // namespace

size_t mlp_image_bytes() { return sizeof(mlp::SmemWeights); }

cudaError_t launch_pack_weights(const float* P, void* img, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(img, 0, sizeof(mlp::SmemWeights), s);  // (struct padding too)
  if (e != cudaSuccess) return e;
  k_pack_weights<<<1, 256, 0, s>>>(P, static_cast<mlp::SmemWeights*>(img));
  return cudaGetLastError();
}

cudaError_t launch_mlp_infer(const float* P, const float* X, int n, float* Y, cudaStream_t s) {
  // the step's forward pass (tcgen05, TMEM accumulators)
  const int tiles = (n + umma::ROWS - 1) / umma::ROWS;
  const int blocks = std::max(1, std::min(tiles, 152 * 3));
  mlp::k_mlp_infer_umma<<<blocks, umma::ROWS, 0, s>>>(P, X, n, Y);
  return cudaGetLastError();
}

}  // namespace tlq
