// Correctly rounded double division and square root, and exact comparisons and
// uniform draws, on the integer pipes.
//
// The trajectory's doubles must be the reference's bit for bit.  On GB300 an
// FP64 warp instruction holds a sub-partition's pipe for 76 cycles, and a
// division or square root is eight to ten of them; the same correctly rounded
// result takes some 60 integer instructions (1-2 cycles each): an approximate
// reciprocal (root) refined by Newton's iteration in 64-bit fractions, the
// quotient's bits, and one exact remainder that settles the last bit and the
// rounding.  Operands or results that are zero, subnormal, infinite, NaN or
// (root) negative take the hardware's operation.  Calls, not inlined: one copy of
// each keeps the trajectory's code small, which instruction supply rewards.
// Compiled for the host too, for tests.
#pragma once

#include "st_fixed.cuh"

namespace st {
namespace sfp {
using fx::bits_f64;
using fx::clz64;
using fx::f64_bits;
using fx::i64;
using fx::recip;
using fx::u64;
using fx::umul;

#ifdef __CUDA_ARCH__
static __device__ __noinline__ double hw_div(double a, double b) { return __ddiv_rn(a, b); }
static __device__ __noinline__ double hw_sqrt(double a) { return __dsqrt_rn(a); }
// Leading bits of 1/sqrt(x), relative error below 2^-20.
__device__ __forceinline__ uint32_t rsqrt_hi(double x) {
  double r;
  asm("rsqrt.approx.f64 %0, %1;" : "=d"(r) : "d"(x));
  return (uint32_t)(f64_bits(r) >> 32);
}
#else
inline double hw_div(double a, double b) { return a / b; }
inline double hw_sqrt(double a) { return sqrt(a); }
inline uint32_t rsqrt_hi(double x) { return (uint32_t)(f64_bits(1.0 / sqrt(x) * fx::seed_error(x)) >> 32); }
#endif

using fx::kFrac;
using fx::kOne;
constexpr u64 kSign = 0x8000000000000000ull;

// The quotient's last step: q = floor(2^54 (a < b ? 2 : 1) a / b) from its approximation
// (one or two units off) and the exact remainder, rounded to 53 bits to even.
__device__ __forceinline__ double div_finish(u64 ma, u64 mb, u64 y, int e, u64 sign) {
  const bool less = ma < mb;
  e -= less ? 1 : 0;
  // a y in units of 2^-62 of the quotient in [1, 2) (in [1/2, 1), doubled, when ma < mb): 55 bits
  u64 q = umul(ma << 11, y) >> (less ? 7 : 8);
  i64 r = (i64)((ma << (less ? 55 : 54)) - q * mb);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (r < 0) {
      --q;
      r += (i64)mb;
    } else if (r >= (i64)mb) {
      ++q;
      r -= (i64)mb;
    }
  }
  // q in [2^54, 2^55): one bit below the result's 54th counts as the rounding bit, r as sticky
  const u64 h = q >> 2, low = ((q & 3) << 1) | (r != 0 ? 1 : 0);
  const u64 m = h + ((low > 4 || (low == 4 && (h & 1))) ? 1 : 0);
  return bits_f64((((u64)(i64)e << 52) + (m - kOne)) | sign);
}

// a / b, correctly rounded.
static __device__ __noinline__ double div_rn(double a, double b) {
  const u64 ba = f64_bits(a), bb = f64_bits(b);
  const int ea = (int)((ba >> 52) & 0x7ff), eb = (int)((bb >> 52) & 0x7ff);
  const int e = ea - eb + 1023;
  if ((unsigned)(ea - 1) >= 0x7feu || (unsigned)(eb - 1) >= 0x7feu || (unsigned)(e - 2) >= 0x7fbu) return hw_div(a, b);
  const u64 ma = (ba & kFrac) | kOne, mb = (bb & kFrac) | kOne;
  return div_finish(ma, mb, recip(mb << 11), e, (ba ^ bb) & kSign);
}

// a / g, correctly rounded, for the constant g = -9.81 (its reciprocal is a constant too).
static __device__ __noinline__ double div_g(double a) {
  const double g = -9.81;
  const u64 ba = f64_bits(a);
  const int ea = (int)((ba >> 52) & 0x7ff), e = ea - 3;  // 9.81 = 1.22625 2^3
  if ((unsigned)(ea - 1) >= 0x7feu || e < 2) return hw_div(a, g);
  return div_finish((ba & kFrac) | kOne, (f64_bits(9.81) & kFrac) | kOne, 0x68621ecb0686206full, e, (ba ^ kSign) & kSign);
}

// sqrt(a), correctly rounded.
static __device__ __noinline__ double sqrt_rn(double a) {
  const u64 ba = f64_bits(a);
  const int ea = (int)(ba >> 52);
  if ((unsigned)(ea - 1) >= 0x7feu) return hw_sqrt(a);  // zero, subnormal, infinite, NaN, negative
  const int odd = (ea & 1) ^ 1;                          // a = m 2^(2 k) with m in [1, 4)
  const u64 m = ((ba & kFrac) | kOne) << odd;            // m 2^52
  const u64 x = m << 9;                                  // m / 8 as a 64-bit fraction, in [1/8, 1/2)
  // y = 1 / sqrt(m) in (1/2, 1]: 32 bits, 2^31 = 1
  const uint32_t s = rsqrt_hi(bits_f64((ba & kFrac) | ((u64)(0x3ff + odd) << 52)));
  const uint32_t y0 = s >= 0x3ff00000u ? 0x80000000u : (s < 0x3fe00000u ? 0x40000000u : ((s & 0xfffffu) | 0x100000u) << 10);
  // e = 1 - m y0^2 in units of 2^-59; y1 = y0 + y0 e / 2, twice
  const u64 t0 = umul(x, (u64)y0 * y0);                  // m y0^2 / 8 2^62 = (m y0^2) 2^59
  const i64 e0 = (i64)(0x0800000000000000ull - t0);      // |e0| < 2^40
  const u64 y1 = ((u64)y0 << 31) + (u64)((e0 >> 10) * (i64)(y0 >> 1) >> 18);  // 2^62 = 1
  const u64 t1 = umul(x, umul(y1, y1) << 2);             // (m y1^2) 2^59
  const i64 e1 = (i64)(0x0800000000000000ull - t1);
  const u64 y2 = y1 + (u64)((e1 * (i64)(y1 >> 40)) >> 20);  // y1 e1 / 2 in units of 2^-62
  // root = m y in [1, 2): r in units of 2^-53 (54 bits), remainder exact
  u64 r = umul(x, y2 << 1) >> 7;                         // m / 8 y 2^63 = root 2^60
  i64 d = (i64)((m << 54) - r * r);                      // (m - root^2) 2^106, modulo 2^64
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (d < 0) {
      --r;
      d += (i64)(2 * r + 1);
    } else if (d > (i64)(2 * r)) {
      d -= (i64)(2 * r + 1);
      ++r;
    }
  }
  const u64 h = r >> 1;
  const u64 v = h + ((r & 1) && (d != 0 || (h & 1)) ? 1 : 0);
  return bits_f64(((u64)((ea - odd + 1023) >> 1) << 52) + (v - kOne));
}

// The top 53 bits of u scaled by 2^-53, exactly (src/particle.cpp:72-83).
__device__ __forceinline__ double unit_53(u64 u) {
  const u64 m = u >> 11;
  const int z = clz64(m);  // 11..64
  return m == 0 ? 0.0 : bits_f64(((u64)(1022 + 11 - z) << 52) + ((m << (z - 11)) - kOne));
}

// 2 u - 1 of that draw, exactly (the product and the difference round to nothing).
__device__ __forceinline__ double signed_unit_53(u64 u) {
  const i64 j = (i64)((u >> 11) << 1) - (1ll << 53);
  const u64 m = (u64)(j < 0 ? -j : j);
  const int z = clz64(m);  // 10..64
  return m == 0 ? 0.0 : bits_f64((((u64)(1023 + 10 - z) << 52) + ((m << (z - 10)) >> 1) - kOne) | (j < 0 ? kSign : 0));
}

// x + 0: -0 becomes 0.
__device__ __forceinline__ double plus0(double x) { return f64_bits(x) == kSign ? 0.0 : x; }

// ---------------------------------------------------------------- comparisons
// Integer order of a double: key(a) < key(b) exactly when a < b for numbers (-0 equals 0).
__device__ __forceinline__ i64 key(double x) {
  const i64 b = (i64)f64_bits(x);
  return b < 0 ? (i64)(kSign - (u64)b) : b;
}
__device__ __forceinline__ bool is_nan(double x) { return (f64_bits(x) & ~kSign) > 0x7ff0000000000000ull; }
__device__ __forceinline__ bool is_finite(double x) { return (f64_bits(x) & ~kSign) < 0x7ff0000000000000ull; }
__device__ __forceinline__ bool is_inf(double x) { return (f64_bits(x) & ~kSign) == 0x7ff0000000000000ull; }
__device__ __forceinline__ bool lt(double a, double b) { return key(a) < key(b) && !is_nan(a) && !is_nan(b); }
__device__ __forceinline__ bool le(double a, double b) { return key(a) <= key(b) && !is_nan(a) && !is_nan(b); }
__device__ __forceinline__ bool eq(double a, double b) { return key(a) == key(b) && !is_nan(a) && !is_nan(b); }
__device__ __forceinline__ bool negative(double x) { return f64_bits(x) > kSign && !is_nan(x); }  // x < 0
// |a| > b (any b: a limit below zero is exceeded by every number)
__device__ __forceinline__ bool abs_gt(double a, double b) { return lt(b, bits_f64(f64_bits(a) & ~kSign)); }

}  // namespace sfp
}  // namespace st
