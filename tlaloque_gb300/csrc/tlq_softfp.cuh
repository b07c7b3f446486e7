// tlq_softfp.cuh -- IEEE FP64 division, square root and multiplication on the
// integer pipe, correctly rounded (round to nearest even): the bits of the
// hardware operations.
//
// Why: GB300 runs FP64 at 1/64 of the FP32 rate.  Measured with 16 warps per
// SM of independent chains, an addition, multiplication or FMA takes 18.6 SM
// cycles per warp, a division 133 and a square root 139 (their Newton steps
// are FMAs on the same pipe); below, a division takes 23, a square root 33
// and a multiplication 15, on pipes that run beside the FP64 one (4
// multiplications here beside 4 FP64 additions: 75 cycles, the additions
// alone 72).  Dependent: a division 103 ns (280 on the FP64 pipe), a square
// root 148 (299), a multiplication 75 (39).
//
// How: schoolbook long division and digit-by-digit square root on the
// 53-bit significands with ~30-bit digits.  An FP32 reciprocal (square
// root) approximation seeds a 32-bit fixed-point one, improved by one Newton
// step; the digits it gives are taken low, so that every remainder stays
// non-negative and an exact integer remainder decides the last bit.  The
// quotient and the root are formed with one extra bit, which rounds: neither
// can be a tie (a 54-bit odd quotient times the divisor's significand, or a
// 54-bit odd root squared, has more significant bits than the operand).
// Zeros over normals are exact; subnormals, infinities, NaNs and results
// near the ends of the exponent range take the hardware operation.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define TLQ_SF __device__ __forceinline__
#else
#include <cmath>
#define TLQ_SF static inline
#endif
#ifndef TLQ_SF_HOST_SEED  // compiled for the host: lets a caller move the seeds within the GPU's error
#define TLQ_SF_HOST_SEED(y) (y)
#endif

namespace tlq {
namespace sf {

TLQ_SF uint32_t hi32(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2hiint(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return (uint32_t)(b >> 32);
#endif
}
TLQ_SF uint32_t lo32(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2loint(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return (uint32_t)b;
#endif
}
TLQ_SF double make(uint32_t hi, uint32_t lo) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
TLQ_SF uint32_t mulhi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
TLQ_SF int32_t mulhis(int32_t a, int32_t b) {
#if defined(__CUDA_ARCH__)
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
TLQ_SF uint64_t mulw(uint32_t a, uint32_t b) { return (uint64_t)a * b; }
TLQ_SF float fbits(uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}
TLQ_SF uint32_t ubits(float f) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(f);
#else
  uint32_t b;
  memcpy(&b, &f, 4);
  return b;
#endif
}
TLQ_SF float rcp_seed(float x) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return TLQ_SF_HOST_SEED(1.0f / x);
#endif
}
TLQ_SF float rsqrt_seed(float x) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return TLQ_SF_HOST_SEED((float)(1.0 / std::sqrt((double)x)));
#endif
}

// The upper word of (hi:lo) << n, 0 < n < 32.
TLQ_SF uint32_t shl2(uint32_t hi, uint32_t lo, uint32_t n) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, n);
#else
  return (hi << n) | (lo >> (32u - n));
#endif
}
// (h:l) rounded to nearest even by the 32 bits f that follow (their lowest
// sticky): plus the carry of f + (2^31 - 1) + odd.
TLQ_SF double round_up(uint32_t h, uint32_t l, uint32_t f) {
  const uint32_t c = 0x7fffffffu + (l & 1u);
#if defined(__CUDA_ARCH__)
  asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %0, %0, 0;\n\t}"
      : "+r"(h), "+r"(l)
      : "r"(f), "r"(c));
#else
  const uint64_t up = ((uint64_t)f + c) >> 32;
  const uint64_t v = (((uint64_t)h << 32) | l) + up;
  h = (uint32_t)(v >> 32);
  l = (uint32_t)v;
#endif
  return make(h, l);
}

// Reciprocal of a normal double's significand: V ~ 2^63 / Bt, Bt = the
// significand's top 32 bits (leading one at bit 31), V <= the true value and
// within 2^-29 of it.
struct Recip {
  uint32_t v;         // V
  uint32_t mh, ml;    // the significand (53 bits)
};
TLQ_SF Recip recip(uint32_t bh, uint32_t bl) {
  Recip r;
  r.mh = (bh & 0xfffffu) | 0x100000u;
  r.ml = bl;
  const uint32_t bt = (r.mh << 11) | (bl >> 21);
  // y ~ 2^31/bt in (1/2, 1), a little below it
  const float y = fmaxf(rcp_seed(fbits((bt >> 8) + 0x3f000000u)) * (1.0f - 8.0f / 16777216.0f), 0.5f);
  const uint32_t v0 = (ubits(y) << 8) | 0x80000000u;
  // one Newton step in fixed point: v0 + v0 (2^63 - v0 bt) / 2^63
  const uint64_t e = 0x8000000000000000ull - mulw(v0, bt);
  r.v = v0 + (mulhi(v0, (uint32_t)(e >> 12)) >> 19);
  return r;
}

// a / b for the significand's reciprocal; ah, al: a's words, eb, bs: b's
// exponent field and sign word.  Both normal, the quotient's exponent field
// within [2, 2045].
TLQ_SF double div_core(uint32_t ah, uint32_t al, const Recip& r, int e, uint32_t sign) {
  const uint32_t amh = (ah & 0xfffffu) | 0x100000u;
  const uint64_t B = ((uint64_t)r.mh << 32) | r.ml;
  uint64_t A = ((uint64_t)amh << 32) | al;
  if (A < B) {
    A <<= 1;
    e -= 1;
  }
  // first digit: q1 ~ (A/B) 2^30, 1 to 7 below it (so that R1 >= B)
  const uint32_t q1 = mulhi((uint32_t)(A >> 22), r.v) - 2u;
  const uint64_t R1 = (A << 30) - (mulw(q1, r.ml) + ((uint64_t)(q1 * r.mh) << 32));
  // second digit: q2 = floor((R1/B) 2^23) or one below it
  const uint32_t q2 = (mulhi((uint32_t)(R1 >> 24), r.v) - 2u) >> 5;
  const uint64_t R2 = (R1 << 23) - (mulw(q2, r.ml) + ((uint64_t)(q2 * r.mh) << 32));
  uint64_t Q = ((uint64_t)q1 << 23) + q2 + (R2 >= B ? 1u : 0u);  // floor(A 2^53 / B): 54 bits
  Q = (Q + 1) >> 1;                                              // the last bit rounds (no ties)
  return make((uint32_t)(Q >> 32) + ((uint32_t)(e - 1) << 20) + sign, (uint32_t)Q);
}

#if defined(__CUDACC__)
static __device__ __noinline__ double div_slow(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_slow(double a) { return sqrt(a); }
static __device__ __noinline__ double mul_slow(double a, double b) { return a * b; }
#else
TLQ_SF double div_slow(double a, double b) { return a / b; }
TLQ_SF double sqrt_slow(double a) { return std::sqrt(a); }
TLQ_SF double mul_slow(double a, double b) { return a * b; }
#endif

// A divisor with its reciprocal, for several quotients by it.
struct Divisor {
  double b;
  Recip r;
};
TLQ_SF Divisor divisor(double b) { return Divisor{b, recip(hi32(b), lo32(b))}; }

TLQ_SF double div(double a, const Divisor& d) {
  const uint32_t ah = hi32(a), al = lo32(a), bh = hi32(d.b);
  const int ea = (int)((ah >> 20) & 0x7ffu), eb = (int)((bh >> 20) & 0x7ffu);
  const int e = ea - eb + 1023;
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  const bool bok = (uint32_t)(eb - 1) < 2046u;
  if (!(bok && (uint32_t)(ea - 1) < 2046u && (uint32_t)(e - 2) < 2044u)) {
    if (bok && ((ah & 0x7fffffffu) | al) == 0u) return make(sign, 0u);  // 0 / b
    return div_slow(a, d.b);
  }
  return div_core(ah, al, d.r, e, sign);
}
TLQ_SF double div(double a, double b) { return div(a, divisor(b)); }

// sqrt(a) for a normal and positive.
TLQ_SF double sqrt_rn(double a) {
  const uint32_t ah = hi32(a), al = lo32(a);
  if ((uint32_t)(ah - 0x00100000u) >= 0x7fe00000u) return sqrt_slow(a);  // zero, subnormal, negative, inf, NaN
  const uint32_t ex = ah >> 20;
  const uint32_t odd = (ex & 1u) ^ 1u;  // unbiased exponent odd
  uint64_t M = (((uint64_t)((ah & 0xfffffu) | 0x100000u) << 32) | al) << odd;  // [2^52, 2^54)
  const uint32_t ft = (uint32_t)(M >> 22);                                     // f = ft / 2^30 in [1, 4)
  float ff = fbits(0x3f800000u | ((ah & 0xfffffu) << 3) | (al >> 29));
  ff = odd ? ff + ff : ff;
  const float y = fmaxf(rsqrt_seed(ff) * (1.0f - 8.0f / 16777216.0f), 0.5f);  // in [1/2, 1)
  const uint32_t w0 = (ubits(y) << 8) | 0x80000000u;
  // one Newton step of w = 1/sqrt(f) in fixed point: w0 + w0 (1 - f w0^2) / 2
  const uint64_t E = 0x4000000000000000ull - mulw(ft, mulhi(w0, w0));
  const int32_t es = (int32_t)((int64_t)E >> 12);
  const uint32_t w = w0 + (uint32_t)(mulhis((int32_t)(w0 >> 1), es) >> 18);
  // the root's first 31 bits, at most 7 below, then 23 more, at most 2 below
  const uint32_t s1 = mulhi(ft, w) - 2u;
  const uint64_t R1 = (M << 8) - mulw(s1, s1);
  const uint32_t s2 = (mulhi((uint32_t)(R1 >> 4), w) >> 4) - 1u;
  uint64_t R2 = (R1 << 46) - (mulw(s1, s2) << 24) - mulw(s2, s2);
  uint64_t S = ((uint64_t)s1 << 23) + s2;
  uint64_t D = 2 * S + 1;
  if ((int64_t)(R2 - D) >= 0) {
    R2 -= D;
    S += 1;
    D += 2;
  }
  if ((int64_t)(R2 - D) >= 0) {
    R2 -= D;
    S += 1;
  }
  S = (S + 1) >> 1;
  const uint32_t er = (ex + 1023u - odd) >> 1;
  return make((uint32_t)(S >> 32) + ((er - 1u) << 20), (uint32_t)S);
}

// a * b.
TLQ_SF double mul(double a, double b) {
  const uint32_t ah = hi32(a), al = lo32(a), bh = hi32(b), bl = lo32(b);
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  // exponent fields less 512: in range while below 2^10, the product's too
  // while their sum stays below 2045
  const uint32_t ea = (ah & 0x7ff00000u) - 0x20000000u, eb = (bh & 0x7ff00000u) - 0x20000000u;
  if (((ea | eb) & 0xc0000000u) || ea + eb >= 0x7fd00000u) {
    const uint32_t za = (ah & 0x7fffffffu) | al, zb = (bh & 0x7fffffffu) | bl;
    if ((za == 0u && (bh & 0x7ff00000u) != 0x7ff00000u) || (zb == 0u && (ah & 0x7ff00000u) != 0x7ff00000u))
      return make(sign, 0u);  // 0 * finite
    return mul_slow(a, b);
  }
  const uint32_t mh = (ah & 0xfffffu) | 0x100000u, nh = (bh & 0xfffffu) | 0x100000u;
  // the product's words w0..w3 (106 bits, the leading one at bit 104 or 105)
  const uint64_t p0 = mulw(al, bl);
  const uint64_t p1 = mulw(al, nh) + (p0 >> 32);
  const uint64_t p2 = mulw(mh, bl) + (uint32_t)p1;
  const uint64_t p3 = mulw(mh, nh) + (p1 >> 32) + (p2 >> 32);
  const uint32_t w0 = (uint32_t)p0, w1 = (uint32_t)p2, w2 = (uint32_t)p3, w3 = (uint32_t)(p3 >> 32);
  const uint32_t one = w3 >> 9;  // 1: the product of the significands is 2 or more
  const uint32_t sh = 12u - one;
  const uint32_t h = shl2(w3, w2, sh), l = shl2(w2, w1, sh);
  // the next 32 bits, the rest as a sticky bit (w0's bits that moved into f
  // are zero wherever f is the tie 2^31, so w0 != 0 says the same)
  const uint32_t f = shl2(w1, w0, sh) | (w0 != 0u ? 1u : 0u);
  const uint32_t e = ea + eb + (one << 20) + sign;  // (h holds the leading one)
  return round_up(h + e, l, f);
}

}  // namespace sf
}  // namespace tlq
