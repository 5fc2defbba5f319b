// DOP853 and quaternion step arithmetic in 64-bit fixed point on the integer pipes.
//
// GB300 issues one FP64 warp instruction per 64 or more cycles on each SM
// sub-partition (measured: 76 cycles per DFMA, DADD, DMUL or DSETP), while a
// 32 x 32 + 64 bit multiply-add (IMAD.WIDE) takes 2.1 cycles and a 32-bit add
// about 1.  A spin step is a few hundred multiply-adds on values whose size is
// known (the spin's norm is constant, the stage derivatives are h Omega times
// it), so it runs in block fixed point: three IMAD.WIDE replace one DFMA, and
// every value keeps 58 or more bits of its block's scale, five more than a
// double's significand.
//
// Numbers are Q63: an int64 m stands for m 2^-63, |m 2^-63| < 1, times a power
// of two kept beside it (one per block: spin, field, step).  A factor of a
// product is split into limbs, m 2^-63 = (h 2^27 + l) 2^-58 with 0 <= l < 2^27
// (|l| <= 2^26 for tableau entries), rounded to 58 fractional bits.  A sum of
// products accumulates the h h terms (weight 2^-62) and the h l + l h terms
// (weight 2^-89) in one int64 each; the l l terms (below 2^-62 each, 2^-64 on
// average) are left out.  Up to 15 terms fit the second accumulator whatever their
// size, and the first one while the sum of the products' magnitudes stays
// below 2.
//
// A block's power of two is that of its norm, so a component that is small beside the
// norm would have fewer bits than a double.  In the usual geometry components
// are small: fields lie along one axis but for 1e-4 or less of them, spins (and
// adjoints) along that axis or across it.  The words are therefore turned so that
// component 0 is the axis, and graded: the field's components 1 and 2 are kept times
// 2^ok, a spin's times 2^sk where it lies along the axis (sk > 0), its component 0 times
// 2^-sk where it lies across (sk < 0), with |sk| <= ok.  Of the terms of a cross product,
// those that stay small have the grade of the component they go to, and the others
// need one shift (Grade).  Ungraded, a spin within 1e-5 of its axis lost its
// transverse part at 5e-17 of the norm per step of 0.13 rad, where FP64 loses 6e-21.
//
// The stages run as one rolled loop over tables in constant memory, with the
// stage derivatives in shared (or local) memory: the hot code has to stay
// within the ~16 KB of instructions that a sub-partition holds close by.
// Beyond that, instructions arrive at 8 bytes per cycle and SM, one per 8
// cycles and sub-partition; the same step fully unrolled (40 KB) waited for
// them most of the time and was slower than FP64 (867 ms against 643 on 1,048,576 particles x 0.1 s).
//
// Steps whose rotation angle h |Omega| reaches 1, whose stage values leave the
// checked range, or whose tolerances do not fit return false: the caller
// takes them in FP64 (dop_attempt_f64 in st_device.cuh).  Also compiled for the
// host, for tests.
#pragma once

#include <math.h>
#include <stdint.h>

#include "st_tableau.h"

namespace st {

// DOP853 stage structure as constexpr functions of compile-time stage and
// term indices (they fold to constants inside unrolled loops).
namespace dopst {
// earlier stages summed into stage s (2..12): stage 1, then 2 (s = 3),
// 3.. (s = 4, 5) or 4.. (s >= 6)
__device__ __forceinline__ constexpr int src(int s, int j) { return j == 0 ? 1 : (s == 3 ? 2 : (s <= 5 ? j + 2 : j + 3)); }
__device__ __forceinline__ constexpr int cnt(int s) { return s <= 2 ? s - 1 : (s <= 4 ? 2 : (s == 5 ? 3 : s - 3)); }
// coefficient of term j of stage s (the a_{s,src(s,j)} of the tableau)
__device__ __forceinline__ constexpr double a(int s, int j) {
  switch (s * 16 + j) {
    case 32: return dop::A21;
    case 48: return dop::A31;
    case 49: return dop::A32;
    case 64: return dop::A41;
    case 65: return dop::A43;
    case 80: return dop::A51;
    case 81: return dop::A53;
    case 82: return dop::A54;
    case 96: return dop::A61;
    case 97: return dop::A64;
    case 98: return dop::A65;
    case 112: return dop::A71;
    case 113: return dop::A74;
    case 114: return dop::A75;
    case 115: return dop::A76;
    case 128: return dop::A81;
    case 129: return dop::A84;
    case 130: return dop::A85;
    case 131: return dop::A86;
    case 132: return dop::A87;
    case 144: return dop::A91;
    case 145: return dop::A94;
    case 146: return dop::A95;
    case 147: return dop::A96;
    case 148: return dop::A97;
    case 149: return dop::A98;
    case 160: return dop::A101;
    case 161: return dop::A104;
    case 162: return dop::A105;
    case 163: return dop::A106;
    case 164: return dop::A107;
    case 165: return dop::A108;
    case 166: return dop::A109;
    case 176: return dop::A111;
    case 177: return dop::A114;
    case 178: return dop::A115;
    case 179: return dop::A116;
    case 180: return dop::A117;
    case 181: return dop::A118;
    case 182: return dop::A119;
    case 183: return dop::A1110;
    case 192: return dop::A121;
    case 193: return dop::A124;
    case 194: return dop::A125;
    case 195: return dop::A126;
    case 196: return dop::A127;
    case 197: return dop::A128;
    case 198: return dop::A129;
    case 199: return dop::A1210;
    case 200: return dop::A1211;
    default: return 0.0;
  }
}
// node of stage s (stage 12 at x + h)
__device__ __forceinline__ constexpr double c(int s) {
  switch (s) {
    case 2: return dop::C2;
    case 3: return dop::C3;
    case 4: return dop::C4;
    case 5: return dop::C5;
    case 6: return dop::C6;
    case 7: return dop::C7;
    case 8: return dop::C8;
    case 9: return dop::C9;
    case 10: return dop::C10;
    case 11: return dop::C11;
    case 12: return 1.0;
    default: return 0.0;
  }
}
// 8th-order weight of stage s
__device__ __forceinline__ constexpr double b(int s) {
  switch (s) {
    case 1: return dop::B1;
    case 6: return dop::B6;
    case 7: return dop::B7;
    case 8: return dop::B8;
    case 9: return dop::B9;
    case 10: return dop::B10;
    case 11: return dop::B11;
    case 12: return dop::B12;
    default: return 0.0;
  }
}
}  // namespace dopst

namespace fx {

typedef long long i64;
typedef unsigned long long u64;

#ifdef __CUDA_ARCH__
__device__ __forceinline__ int clz64(u64 x) { return __clzll((long long)x); }
__device__ __forceinline__ int clz32(unsigned x) { return __clz((int)x); }
__device__ __forceinline__ float lg2f_approx(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float ex2f_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// Leading bits of 1/x, relative error below 2^-20.
__device__ __forceinline__ uint32_t rcp_hi(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return (uint32_t)((unsigned long long)__double_as_longlong(r) >> 32);
}
__device__ __forceinline__ float rcpf_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ uint32_t f32_bits(float x) { return __float_as_uint(x); }
__device__ __forceinline__ float bits_f32(uint32_t b) { return __uint_as_float(b); }
// a * b + c in one IMAD.WIDE (left to the compiler, factors that it proves
// non-negative turn into 64 x 64 bit products).
__device__ __forceinline__ i64 madw(int a, int b, i64 c) {
  i64 r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
__device__ __forceinline__ i64 mulw(int a, int b) {
  i64 r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ u64 f64_bits(double x) { return (u64)__double_as_longlong(x); }
__device__ __forceinline__ double bits_f64(u64 b) { return __longlong_as_double((long long)b); }
#else
inline int clz64(u64 x) { return x ? __builtin_clzll(x) : 64; }
inline int clz32(unsigned x) { return x ? __builtin_clz(x) : 32; }
inline float lg2f_approx(float x) { return log2f(x); }
inline float ex2f_approx(float x) { return exp2f(x); }
inline float rcpf_approx(float x) { return 1.0f / x; }
inline i64 madw(int a, int b, i64 c) { return (i64)a * b + c; }
inline i64 mulw(int a, int b) { return (i64)a * b; }
inline uint32_t f32_bits(float x) {
  uint32_t b;
  __builtin_memcpy(&b, &x, 4);
  return b;
}
inline float bits_f32(uint32_t b) {
  float x;
  __builtin_memcpy(&x, &b, 4);
  return x;
}
inline u64 f64_bits(double x) {
  u64 b;
  __builtin_memcpy(&b, &x, 8);
  return b;
}
inline double bits_f64(u64 b) {
  double x;
  __builtin_memcpy(&x, &b, 8);
  return x;
}
// (for tests: seeds off by up to 1.5 x 2^-21)
inline double seed_error(double x) { return 1.0 + ((int)(f64_bits(x) >> 20 & 3) - 1.5) * 0x1p-21; }
inline uint32_t rcp_hi(double x) { return (uint32_t)(f64_bits(1.0 / x * seed_error(x)) >> 32); }
#endif

__device__ __forceinline__ i64 shl(i64 a, int k) { return (i64)((u64)a << k); }
__device__ __forceinline__ i64 add(i64 a, i64 b) { return (i64)((u64)a + (u64)b); }  // modulo 2^64

// ---------------------------------------------------------------- conversions
// Biased exponent of x (0: zero or subnormal, 0x7ff: infinite or NaN).
__device__ __forceinline__ int bexp(double x) { return (int)((f64_bits(x) >> 52) & 0x7ff); }

// x 2^-E as Q63, for |x| < 2^E (and E within the exponents of normal doubles);
// rounded to nearest, ties away from zero.  Subnormal x give 0.
__device__ __forceinline__ i64 to_q63(double x, int E) {
  const u64 b = f64_bits(x);
  const int e = (int)((b >> 52) & 0x7ff);
  const u64 m = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 11;  // x = m 2^(e - 1023 - 63)
  int s = E + 1023 - e;  // x 2^-E 2^63 = m >> s
  s = s > 63 ? 63 : s;
  u64 q = (m >> s) + ((m >> (s > 0 ? s - 1 : 0)) & (s > 0 ? 1u : 0u));
  if (e == 0) q = 0;
  return (i64)b < 0 ? -(i64)q : (i64)q;
}

// m 2^(E - 63), rounded to nearest.
__device__ __forceinline__ double from_q63(i64 m, int E) {
  const double d = (double)m;  // correctly rounded
  const u64 b = f64_bits(d);
  return m == 0 ? 0.0 : bits_f64(b + ((u64)(i64)(E - 63) << 52));
}

// m 2^-n, rounded.
__device__ __forceinline__ i64 rsh(i64 m, int n) { return (m + ((i64)((1ull << n) >> 1))) >> n; }
// |m| or one less, for its leading zeros
__device__ __forceinline__ unsigned mag(int m) { return (unsigned)(m ^ (m >> 31)); }

// ---------------------------------------------------------------- products
struct Limb {
  int h, l;
};
// m to 58 fractional bits, rounded down (callers add 16 units first to round to nearest), and back.
__device__ __forceinline__ Limb limb(i64 m) { return {(int)(m >> 32), (int)((unsigned)m >> 5)}; }
__device__ __forceinline__ i64 unlimb(Limb a) { return (i64)((u64)(unsigned)a.h << 32 | (unsigned)a.l << 5); }
__device__ __forceinline__ Limb neg(Limb a) { return {-a.h, -a.l}; }

struct Acc {
  i64 hh, mid;
};
__device__ __forceinline__ void mac(Acc& a, Limb x, Limb y) {
  a.hh = madw(x.h, y.h, a.hh);
  a.mid = madw(x.h, y.l, a.mid);
  a.mid = madw(x.l, y.h, a.mid);
}
__device__ __forceinline__ Acc mac0(Limb x, Limb y, i64 mid = 0) {  // the first of a sum
  Acc a;
  a.hh = mulw(x.h, y.h);
  a.mid = mid == 0 ? mulw(x.h, y.l) : madw(x.h, y.l, mid);
  a.mid = madw(x.l, y.h, a.mid);
  return a;
}
// Start value of `mid` that makes a following limb split round to nearest.
constexpr i64 kHalfLimb = 1ll << 30;
// The sum as Q63 times 2^k.
__device__ __forceinline__ i64 q63(const Acc& a, int k = 0) { return shl(a.hh, 1 + k) + (a.mid >> (26 - k)); }
__device__ __forceinline__ i64 mulq(Limb x, Limb y, int k = 0) {
  return q63(mac0(x, y, kHalfLimb), k);
}
// x m as Q63 times 2^k, m in 32 and 31 bits of its 63.
__device__ __forceinline__ i64 mulw63(Limb x, i64 m, int k) {
  const int h = (int)(m >> 32), l = (int)((unsigned)m >> 1);
  const i64 mid = madw(x.l, h, madw(x.h, l, 1 << (29 - k)) >> 4);  // (weights 2^-89 and 2^-93; half of the last bit)
  return shl(mulw(x.h, h), 1 + k) + (mid >> (26 - k));
}
// A tableau entry times 2^-p as limbs (folds to immediates).
__device__ __forceinline__ constexpr Limb coef(double a, int p) {
  const double s = a * (double)(1ull << (58 - p));
  const i64 q = (i64)(s + (s < 0.0 ? -0.5 : 0.5));
  const i64 h = (q + (1ll << 26)) >> 27;
  return {(int)h, (int)(q - (i64)((u64)h << 27))};
}
// Half of c^2 as limbs, 2^-5 <= c <= 1 (or 0): squared as an integer, since c^2 rounded to a double
// would cost the second moments of the adjoint up to 5e-16.
__device__ __forceinline__ constexpr Limb coef_sq(double c) {
  const u64 m = (u64)(c * (double)(1ull << 58)), a = m >> 29, b = m & 0x1fffffffull;
  const i64 q = (i64)((a * a + ((2 * a * b + (b * b >> 29)) >> 29) + 1) >> 1), h = (q + (1ll << 26)) >> 27;
  return {(int)h, (int)(q - (i64)((u64)h << 27))};
}
// High 64 bits of the product of two 64-bit fractions, at most 3 units low.
__device__ __forceinline__ u64 umul(u64 a, u64 b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (u64)ah * bh + (((u64)ah * bl) >> 32) + (((u64)al * bh) >> 32);
}

constexpr u64 kFrac = 0x000fffffffffffffull, kOne = 0x0010000000000000ull;

// 2^62 / b to a relative 2^-57 for b in [1/2, 1) as a 64-bit fraction (top bit set).
__device__ __forceinline__ u64 recip(u64 b) {
  // 1/x of the double with b's leading bits lies in (1, 2]: 31 bits, 2^30 = 1
  const double x = bits_f64(((b >> 11) & kFrac) | 0x3fe0000000000000ull);
  const uint32_t s = rcp_hi(x);
  const uint32_t y0 = s >= 0x40000000u ? 0x7fffffffu : (s < 0x3ff00000u ? 0x40000000u : ((s & 0xfffffu) | 0x100000u) << 10);
  // e = 1 - b y0 in units of 2^-62, |e| < 2^43; y1 = y0 + y0 e
  const u64 t = (u64)(uint32_t)(b >> 32) * y0 + (((u64)(uint32_t)b * y0) >> 32);
  const i64 e = (i64)(0x4000000000000000ull - t);
  const u64 y1 = ((u64)y0 << 32) + (u64)(madw((int)y0, (int)(e >> 14), 0) >> 16);
  // once more: |e| < 2^24 now
  const i64 f = (i64)(0x4000000000000000ull - umul(b, y1));
  return y1 + (u64)(madw((int)(y1 >> 32), (int)f, 0) >> 30);
}

// ---------------------------------------------------------------- lanes
// All three spin components on one lane.
struct Lane3 {
  static constexpr int N = 3;
  // kappa = y x w for the lane's components (w's limbs and their negatives)
  __device__ __forceinline__ void cross(const Limb y[3], const Limb w[3], Acc k[3]) const {
    const Limb n[3] = {neg(w[0]), neg(w[1]), neg(w[2])};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int a = c == 2 ? 0 : c + 1, b = c == 0 ? 2 : c - 1;
      k[c] = mac0(y[a], w[b], kHalfLimb);
      mac(k[c], y[b], n[a]);
    }
  }
  __device__ __forceinline__ void gather(const i64 v[3], i64 all[3]) const {
#pragma unroll
    for (int c = 0; c < 3; ++c) all[c] = v[c];
  }
  __device__ __forceinline__ bool any(bool b) const { return b; }
  __device__ __forceinline__ int comp(int c) const { return c; }
  __device__ __forceinline__ void pick(i64 x, i64 y, i64 z, i64 v[3]) const {
    v[0] = x;
    v[1] = y;
    v[2] = z;
  }
};

// Where an attempt keeps its stage derivatives kappa_1..kappa_12: this
// thread's column of two shared-memory arrays, [12][BLOCK] x (16 + 8) bytes
// (conflict-free), or a local array.
struct alignas(16) Limb2 {
  Limb a, b;
};
struct StageSmem {
  Limb2* xy;  // &array[0][thread]
  Limb* z;
  int stride;  // BLOCK
  __device__ __forceinline__ void load(int s, Limb k[3]) const {
    const Limb2 v = xy[s * stride];
    k[0] = v.a;
    k[1] = v.b;
    k[2] = z[s * stride];
  }
  __device__ __forceinline__ void store(int s, const Limb k[3]) {
    xy[s * stride] = {k[0], k[1]};
    z[s * stride] = k[2];
  }
  // a scratch array of 12 words over the same memory
  __device__ __forceinline__ i64 word(int k) const { return *reinterpret_cast<const i64*>(&xy[k * stride]); }
  __device__ __forceinline__ void set_word(int k, i64 v) { *reinterpret_cast<i64*>(&xy[k * stride]) = v; }
};
template <int N>
struct StageLocal {
  Limb v[12][N];
  __device__ __forceinline__ void load(int s, Limb k[N]) const {
#pragma unroll
    for (int c = 0; c < N; ++c) k[c] = v[s][c];
  }
  __device__ __forceinline__ void store(int s, const Limb k[N]) {
#pragma unroll
    for (int c = 0; c < N; ++c) v[s][c] = k[c];
  }
  __device__ __forceinline__ i64 word(int k) const { return ((i64)v[k][0].h << 32) | (uint32_t)v[k][0].l; }
  __device__ __forceinline__ void set_word(int k, i64 x) { v[k][0] = {(int)(x >> 32), (int)x}; }
};

// ---------------------------------------------------------------- pulse
// (pi/2)^2k / (2k)! / 4 with alternating sign as Q63, k = 0..7, and 2^32 times
// it for k = 8..11.
__device__ __forceinline__ constexpr i64 cos_coef(int k) {
  switch (k) {
    case 0: return 2305843009213693952ll;
    case 1: return -2844719788994575541ll;
    case 2: return 584922061444309466ll;
    case 3: return -48107911266041808ll;
    case 4: return 2119669878386351ll;
    case 5: return -58111953223829ll;
    case 6: return 1086253767602ll;
    case 7: return -14726504073ll;
    case 8: return 650261490920323669ll;
    case 9: return -5243319993991956ll;
    case 10: return 34045719795410ll;
    default: return -181827806240ll;
  }
}

// cos(2 pi phi) / 2 as Q63, phi in turns as a 64-bit fraction.  phi is brought
// to a quarter turn either side of 0 (a half turn flips the sign); with
// y = (4 phi)^2 <= 1 the series sum (-1)^k (pi/2)^2k / (2k)! y^k runs to k = 11
// (the next term is below 2^-63).  The terms from k = 8 on sum to less than
// 2^-33 and take one limb product each.  A double's cos costs some 25 FP64
// instructions (1,900 cycles of the pipe); this takes 33 multiply-adds.
__device__ __forceinline__ i64 half_cos_turns(u64 phi) {
  const u64 flip = (phi + 0x4000000000000000ull) >> 63;  // phi in [1/4, 3/4)
  const Limb z = limb((i64)(phi + (flip << 63)));        // 2 phi, in [-1/2, 1/2)
  const Limb y = limb(mulq(z, z, 1));                    // y / 2
  i64 t = cos_coef(11);
#pragma unroll
  for (int k = 2; k >= 0; --k) t = cos_coef(8 + k) + shl(madw((int)(t >> 32), y.h, 0), 2);
  t >>= 32;
#pragma unroll
  for (int k = 7; k >= 0; --k) t = cos_coef(k) + mulq(y, limb(t), 1);
  t = shl(t, 1);
  return flip ? -t : t;
}

// frac(t turns_per_s) as a 64-bit fraction for t >= 0; turns_per_s = wm 2^(we - 64), wm normalised.
__device__ __forceinline__ u64 turns_of(double t, u64 wm, int we) {
  const u64 b = f64_bits(t);
  const int e = (int)(b >> 52);
  if (e == 0) return 0;
  const u64 m = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 11;  // t = m 2^(e - 1022 - 64)
#ifdef __CUDA_ARCH__
  const u64 hi = __umul64hi(m, wm);
#else
  const u64 hi = (u64)(((unsigned __int128)m * wm) >> 64);
#endif
  const u64 lo = m * wm;
  const int s = e - 1022 + we;  // the product's integer bits
  if (s <= 0) return s > -64 ? hi >> -s : 0;
  return s < 64 ? (hi << s) | (lo >> (64 - s)) : lo << (s < 128 ? s - 64 : 63);
}

// ---------------------------------------------------------------- segment
// The field polynomial of a segment in block fixed point: with tau = u 2^te,
// 0 <= u < 1/2 on the segment, Omega(tau) = 2^oe (o0 + u (o1 + u o2)) plus the
// pulse's 2^oe ga cos on z, where the norm of the summed magnitudes lies in
// [1/4, 1/2) (on: that norm).  The spin is 2^se times a vector of norm in
// (1/8, 1/4], so that a spin of norm 1 sits at the top of its range.
struct SegScale {
  int oe, te, se;
  float on;
  int ok = 0, sk = 0;  // grades of the field and the spin
  int pz = 2;          // component of the words along z (the pulse)
};

// What a spin's (or adjoint's) grade g does in a step: components 0, and 1 and 2, are kept
// times 2^e0, 2^e1.
struct Grade {
  int g;
  __device__ __forceinline__ int e0() const { return g < 0 ? -g : 0; }
  __device__ __forceinline__ int e1() const { return g > 0 ? g : 0; }
  // A derivative's component 0 is kept times 2^(e0 + up()): the spin adds it that much further down.
  __device__ __forceinline__ int up() const { return 2 * e1(); }
  // In the derivative's components 1 and 2, component 0 stands this much further down.
  __device__ __forceinline__ int down() const { return 2 * e0(); }
};
// The grade, up to ok, that brings the smaller side's words (leading zeros a along
// the axis, b across) up to [1/8, 1/4), where the larger side's are.
__device__ __forceinline__ int grade_of(int a, int b, int ok) {
  int n = (a > b ? a : b) - 3;
  n = n < 0 ? 0 : (n > ok ? ok : n);
  return b > a ? n : -n;
}

// 31-bit magnitude of x 2^-E (|x| < 2^E), for norms.
__device__ __forceinline__ uint32_t mag31(double x, int E) {
  const u64 b = f64_bits(x);
  const int e = (int)((b >> 52) & 0x7ff);
  const uint32_t m = ((uint32_t)(b >> 32) & 0xfffffu | 0x100000u) << 11;
  const int s = E + 1023 - e;
  return e == 0 || s > 31 ? 0u : m >> s;
}
__device__ __forceinline__ int imax(int a, int b) { return a > b ? a : b; }
__device__ __forceinline__ u64 sq32(uint32_t a) { return (u64)a * a; }

// Scale of the spin: false when a component is infinite or NaN, or all are zero.
__device__ __forceinline__ bool spin_scale(const double S[3], int& se) {
  const int e = imax(imax(bexp(S[0]), bexp(S[1])), bexp(S[2]));
  if (e == 0x7ff || e < 64) return false;
  se = e - 1021;  // the largest component is in [1/4, 1/2), the norm in [1/4, 0.87)
  const u64 n2 = sq32(mag31(S[0], se)) + sq32(mag31(S[1], se)) + sq32(mag31(S[2], se));  // norm^2 2^62
  if (n2 > 0x0405400000000000ull) ++se;  // 0.2506^2: a norm within 0.2% of a power of two rounds down to it
  if (n2 > 0x1015000000000000ull) ++se;  // 0.5012^2
  return true;
}

// Grade of a spin of scale se (its components in the order of the words), up to ok.
__device__ __forceinline__ int spin_grade(const double S[3], int se, int ok) {
  const int top = se + 1023;  // less the biased exponent: the word's leading zeros
  return grade_of(top - bexp(S[0]), top - imax(bexp(S[1]), bexp(S[2])), ok);
}
__device__ __forceinline__ void spin_words(const double S[3], int se, int sk, i64 w[3]) {
  const Grade g{sk};
  w[0] = to_q63(S[0], se - g.e0());
  w[1] = to_q63(S[1], se - g.e1());
  w[2] = to_q63(S[2], se - g.e1());
}
// The words of a spin of grade sk at the grade that fits them best, up to ok (or nearer to it
// where their high halves are zero).
__device__ __forceinline__ void regrade(i64 w[3], int& sk, int ok) {
  const Grade g{sk};
  const int h0 = (int)(w[0] >> 32), h1 = (int)(w[1] >> 32), h2 = (int)(w[2] >> 32);
  const int n = grade_of(clz32(mag(h0)) + g.e0(), clz32(mag(h1) | mag(h2)) + g.e1(), ok);
  if (n == sk) return;
  sk = n;
  const int d0 = g.e0() - Grade{n}.e0(), d1 = g.e1() - Grade{n}.e1();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int d = c == 0 ? d0 : d1;
    w[c] = d >= 0 ? rsh(w[c], d) : shl(w[c], -d);
  }
}

// Scale of the field over a segment of length T, and with `grade` its grade (else 0):
// false when a coefficient is infinite or NaN, T is not positive, or an exponent
// leaves the usual range.  ga is on component q.pz.
__device__ __forceinline__ bool field_scale(const double o0[3], const double o1[3], const double o2[3], double ga,
                                            double T, SegScale& q, bool grade = false) {
  if (!(T > 0.0)) return false;
  const int t = bexp(T) - 1021;  // T < 2^(te - 1)
  int e0 = bexp(ga), e1 = 0, e2 = 0;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    e0 = imax(e0, bexp(o0[c]));
    e1 = imax(e1, bexp(o1[c]));
    e2 = imax(e2, bexp(o2[c]));
  }
  if (e0 == 0x7ff || e1 == 0x7ff || e2 == 0x7ff || t < -900 || t > 900) return false;
  int e = e0;
  if (e1) e = imax(e, e1 + t);
  if (e2) e = imax(e, e2 + 1 + 2 * t);
  if (e < 64) e = 64;  // no field to speak of: every coefficient rounds to zero
  if (e > 1900) return false;
  const int E = e - 1023 + 3;  // each term below 1/4, the sum of a component's below 1
  u64 n2 = 0, axis2 = 0;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const u64 m = (u64)mag31(o0[c], E) + mag31(o1[c], E - t) + 2ull * mag31(o2[c], E - 2 * t) +
                  (c == q.pz ? mag31(ga, E) : 0u) + 4u;  // units of 2^-31, rounded up
    n2 += (m * m) >> 2;
    if (c == 0) axis2 = n2;
  }
  const float n = sqrtf((float)n2) * 0x1p-30f;  // norm of 2^-E Omega, below 1.8
  const uint32_t nb = f32_bits(n);
  const int ne = (int)(nb >> 23) - 125;  // n 2^-ne in [1/4, 1/2)
  q.oe = E + ne;
  q.te = t;
  q.on = bits_f32(nb - ((uint32_t)ne << 23)) * 1.00001f;
  q.ok = 0;
  if (grade)  // the words across grow no larger than the norm: all to sqrt 2 times it at most
    q.ok = imax((int)(f32_bits((float)n2) - f32_bits((float)(n2 - axis2))) >> 24, 0);  // (at most 28: the sums are 4 units or more)
  return true;
}

// ---------------------------------------------------------------- step
// Tolerances of a set: sk = atol + rtol |S| = rtol (atol / rtol + |S|).
struct StepTol {
  double rtol, ratio;  // ratio = atol / rtol
};
// Whether a spin of scale se can be stepped with this ratio.  A component near
// zero is weighted by atol alone, while its error estimate carries the rounding
// of the whole spin (2^-58 of its norm): up to norm / ratio = 16 the estimate was
// better than the FP64 step's in the median (spins of any direction, and along and across the
// field's axis), at 64 it spoiled the growth of tiny steps (14 of 20,000).
__device__ __forceinline__ bool ratio_fits(double ratio, int se) {
  const int e = bexp(ratio) - 1023;  // ratio >= 2^e
  return ratio > 0.0 && e >= se - 6 && e < se + 40;
}

// Result of an attempt.
struct StepOut {
  bool accept;   // err <= 1
  double root8;  // err^(-1/8); infinite when err = 0
};

// Powers of two p >= the sums of the magnitudes of a stage's coefficients.
__device__ __forceinline__ constexpr int stage_p(int s) { return s <= 4 || s == 6 || s == 7 || s == 8 ? -1 : (s == 5 ? 2 : 7); }

// Row s of the stage loop: its terms' first coefficient in kStageCoef, their
// number, the first source after kappa_1, p, and the halves of its node and of
// the node's square.
struct StageRow {
  int off, n, src, p;
  Limb c, c2;
};
#define ST_ROW(s, off) {off, dopst::cnt(s), (s) == 3 ? 1 : ((s) <= 5 ? 2 : 3), stage_p(s), \
                        coef(dopst::c(s), 1), coef_sq(dopst::c(s))}
static __constant__ StageRow kStageRows[12] = {ST_ROW(1, 0),  ST_ROW(2, 0),  ST_ROW(3, 1),  ST_ROW(4, 3),
                                               ST_ROW(5, 5),  ST_ROW(6, 8),  ST_ROW(7, 11), ST_ROW(8, 15),
                                               ST_ROW(9, 20), ST_ROW(10, 26), ST_ROW(11, 33), ST_ROW(12, 41)};
#undef ST_ROW
#define ST_A(s, j) coef(dopst::a(s, j), stage_p(s))
static __constant__ Limb kStageCoef[50] = {
    ST_A(2, 0),  ST_A(3, 0),  ST_A(3, 1),  ST_A(4, 0),  ST_A(4, 1),  ST_A(5, 0),  ST_A(5, 1),  ST_A(5, 2),
    ST_A(6, 0),  ST_A(6, 1),  ST_A(6, 2),  ST_A(7, 0),  ST_A(7, 1),  ST_A(7, 2),  ST_A(7, 3),  ST_A(8, 0),
    ST_A(8, 1),  ST_A(8, 2),  ST_A(8, 3),  ST_A(8, 4),  ST_A(9, 0),  ST_A(9, 1),  ST_A(9, 2),  ST_A(9, 3),
    ST_A(9, 4),  ST_A(9, 5),  ST_A(10, 0), ST_A(10, 1), ST_A(10, 2), ST_A(10, 3), ST_A(10, 4), ST_A(10, 5),
    ST_A(10, 6), ST_A(11, 0), ST_A(11, 1), ST_A(11, 2), ST_A(11, 3), ST_A(11, 4), ST_A(11, 5), ST_A(11, 6),
    ST_A(11, 7), ST_A(12, 0), ST_A(12, 1), ST_A(12, 2), ST_A(12, 3), ST_A(12, 4), ST_A(12, 5), ST_A(12, 6),
    ST_A(12, 7), ST_A(12, 8)};
#undef ST_A
// The 8th-order weights b / 16, the third-order error row (b - bhh) / 16 and the
// fifth-order one er / 8 of kappa_1, kappa_6..kappa_12.
static __constant__ Limb kSumCoef[8][3] = {
    {coef(dop::B1, 4), coef(dop::B1 - dop::BHH1, 4), coef(dop::ER1, 3)},
    {coef(dop::B6, 4), coef(dop::B6, 4), coef(dop::ER6, 3)},
    {coef(dop::B7, 4), coef(dop::B7, 4), coef(dop::ER7, 3)},
    {coef(dop::B8, 4), coef(dop::B8, 4), coef(dop::ER8, 3)},
    {coef(dop::B9, 4), coef(dop::B9 - dop::BHH2, 4), coef(dop::ER9, 3)},
    {coef(dop::B10, 4), coef(dop::B10, 4), coef(dop::ER10, 3)},
    {coef(dop::B11, 4), coef(dop::B11, 4), coef(dop::ER11, 3)},
    {coef(dop::B12, 4), coef(dop::B12 - dop::BHH3, 4), coef(dop::ER12, 3)}};

// (b / (a 2^i))^(1/16) / 2 as a 64-bit fraction, for fractions a >= b and 0 <= i < 16:
// Newton's iteration for r^16 a 2^i = b, the powers of two of i fed in between the
// squarings so that every intermediate stays in [1/4, 1].  From a seed good to
// 2^-20 two steps reach 2^-60.
__device__ __forceinline__ u64 root16(u64 a, u64 b, int i) {
  const float af = (float)(uint32_t)(a >> 32), bf = (float)(uint32_t)(b >> 32);
  const float lg = lg2f_approx(bf) - lg2f_approx(af) - (float)i;
  u64 r = (u64)(ex2f_approx(0.0625f * lg) * 0x1.fffff8p62f);
  const float ib = rcpf_approx(bf) * 0x1p-35f;  // 2 / (16 b), b in units of 2^-64
#pragma unroll 1
  for (int it = 0; it < 2; ++it) {
    u64 v = r;
#pragma unroll 1
    for (int q = 3; q >= 0; --q) v = umul(v, v) << 1 << ((i >> q) & 1);  // half of the square times a bit of 2^i
    const i64 d = (i64)((b >> 1) - umul(v, a));  // (b - r^16 2^i a) / 2
    const float f = (float)d * ib * (float)(uint32_t)(r >> 32);  // the correction of r / 2 in units of 2^-32
    r += (u64)(i64)(f * 0x1p32f);
  }
  return r;
}

// h Omega over a step, as 2^ez (w(c)) with the norm of w in [1/4, 1/2): at the node
// c (0 <= c <= 1) w = 4 w0 + c w1 + c^2 w2, and on z the pulse's 2 hg cos(2 pi (phi0 + c dphi)).
template <int N>
struct StepField {
  i64 w0[N];
  Limb w1[N], w2[N], hg, dphi;
  u64 phi0;
  int ez, pz, dk;
  bool pulse;
  // without the pulse; the halves of the node and of its square
  __device__ __forceinline__ i64 at(int k, Limb c, Limb c2) const {
    Acc o;
    o.hh = madw(c.h, w1[k].h, w0[k]);
    o.mid = madw(c.h, w1[k].l, kHalfLimb >> 1);
    o.mid = madw(c.l, w1[k].h, o.mid);
    mac(o, c2, w2[k]);
    return q63(o, 1);
  }
  template <class V>
  __device__ __forceinline__ void add_pulse(const V& view, i64 p, i64* w) const {
#pragma unroll
    for (int c = 0; c < N; ++c)
      if (view.comp(c) == pz) w[c] += p;
  }
  // the pulse's phase at a node, in turns
  __device__ __forceinline__ u64 phase_at(Limb c) const { return phi0 + ((u64)mulq(c, dphi, 1) << dk); }
  __device__ __forceinline__ i64 pulse_at(Limb c) const {
    return mulq(hg, limb(half_cos_turns(phase_at(c)) + 16), 1);
  }
};
// Components 1 and 2 come out at the grade ok - kw.  False: the step leaves the
// segment, reaches 2^max_ez / 2 rad or passes 16 of the pulse's turns.
template <class V>
__device__ __forceinline__ bool step_field(const V& view, const SegScale& q, int kw, const i64* o0, const i64* o1,
                                           const i64* o2, i64 ga, u64 wm, int we, double x, double tx, double h, int max_ez,
                                           StepField<V::N>& f) {
  constexpr int N = V::N;
  // ---- the step in segment units
  if ((i64)f64_bits(h) <= 0 || (i64)f64_bits(tx) < 0) return false;  // (a NaN is out of range below)
  const int eh = bexp(h) - 1021;  // h = hm 2^eh, hm in [1/4, 1/2)
  if (bexp(tx) - 1022 >= q.te || eh - 1 > q.te || bexp(h) < 64) return false;
  const i64 u = to_q63(tx, q.te);
  const i64 hm = to_q63(h, eh);
  const int sh = q.te - eh + 1;  // eta = h 2^-te = 2 hm 2^-sh
  if ((u64)u + ((u64)hm << 1 >> (sh > 63 ? 63 : sh)) > 0x4010000000000000ull) return false;  // past the segment's end
  // ---- h Omega = 2^ez omega, |omega| in [1/4, 1/2)
  const bool small = (float)(uint32_t)(hm >> 32) * q.on < 0x1.ff8p-4f * 0x1p31f;
  const i64 hs = small ? hm << 1 : hm;
  f.ez = eh + q.oe - 1 - (small ? 1 : 0);
  if (f.ez > max_ez) return false;
  const Limb hsl = limb(hs), hml = limb(hm), ul = limb(u);
  const int s63 = sh > 63 ? 63 : sh;
  const i64 g1 = mulq(hsl, hml, 1) >> s63;  // hs eta
  const Limb g1l = limb(g1);
  const i64 g2 = mulq(g1l, hml, 1) >> s63;  // hs eta^2
  const Limb g2l = limb(g2);
#pragma unroll
  for (int c = 0; c < N; ++c) {
    const Limb o2l = limb(o2[c]);
    const i64 t1 = mulq(ul, o2l);
    const int d = view.comp(c) == 0 ? 0 : kw;
    f.w0[c] = mulq(hsl, limb(o0[c] + mulq(ul, limb(o1[c] + t1))), -1) >> d;  // a quarter of it
    f.w1[c] = limb(mulq(g1l, limb(o1[c] + shl(t1, 1)), 1) >> d);
    f.w2[c] = limb(mulq(g2l, o2l, 1) >> d);
  }
  f.pulse = ga != 0;
  f.pz = q.pz;
  f.hg = f.dphi = {0, 0};
  f.phi0 = 0;
  f.dk = 0;
  if (f.pulse) {
    f.hg = limb(mulq(hsl, limb(ga), 1) >> (q.pz == 0 ? 0 : kw));
    // the step's turns times 2^-dk, below a half
    const int top = bexp(h) - 1022 + we;  // (below 2^top turns)
    f.dk = top < -1 ? 0 : top + 2;
    if (f.dk > 6) return false;  // 16 turns and more
    f.dphi = limb((i64)turns_of(h, wm, we - f.dk));
    const u64 p = turns_of(fabs(x), wm, we);
    f.phi0 = x < 0.0 ? 0ull - p : p;
  }
  return true;
}

// ys of dop_stages where the stage states are not kept.
struct StageNone {
  __device__ __forceinline__ void store(int, const Limb*) {}
};
// The stages of a step from a spin of grade g, the field at the grade |g| + wd: kappa_1..
// kappa_12 in ks, the states Y in ys; not zero: a sum left its range.
template <class V, class KS, class YS>
__device__ __forceinline__ unsigned dop_stages(const V& view, KS& ks, YS& ys, const StepField<V::N>& f, const i64* S, int r,
                                               Grade g, int wd = 0) {
  constexpr int N = V::N;
  const int r0 = r + g.up() > 63 ? 63 : r + g.up();
  // ---- stages: kappa_s = Y_s x omega_s, Y_s = S + 2^ez sum a_sj kappa_j
  i64 Sr[N];
#pragma unroll
  for (int c = 0; c < N; ++c) Sr[c] = S[c] + 16;  // rounds the limb split
  unsigned bad = 0;  // set where a sum leaves the range in which nothing overflows
#pragma unroll 1
  for (int s = 0; s < 12; ++s) {
    const StageRow& row = kStageRows[s];
    Acc a[N];
#pragma unroll
    for (int c = 0; c < N; ++c) a[c] = {0, 0};
    // two terms a pass, each loaded one ahead (the last load unused, within the array)
    Limb k[N], k2[N];
    ks.load(0, k);
    int src = row.src, j = 0;
#pragma unroll 1
    for (; j + 1 < row.n; j += 2) {
      const Limb f = kStageCoef[row.off + j], f2 = kStageCoef[row.off + j + 1];
      ks.load(src, k2);
#pragma unroll
      for (int c = 0; c < N; ++c) mac(a[c], f, k[c]);
      ks.load(src + 1, k);
      src += 2;
#pragma unroll
      for (int c = 0; c < N; ++c) mac(a[c], f2, k2[c]);
    }
    if (j < row.n) {
      const Limb f = kStageCoef[row.off + j];
#pragma unroll
      for (int c = 0; c < N; ++c) mac(a[c], f, k[c]);
    }
    Limb Yg[N], Y[N], W[N];
    const i64 pulse = f.pulse ? f.pulse_at(row.c) : 0;  // (one copy of its code)
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const int p = row.p;
      const bool axis = view.comp(c) == 0;
      // |2 sum a kappa| < 1/2: neither the shift below nor Y can overflow
      bad |= ((unsigned)(int)(a[c].hh >> 32) + (1u << (28 - p))) & ~((1u << (29 - p)) - 1u);
      const i64 y = Sr[c] + (q63(a[c], 1 + p) >> (axis ? r0 : r));
      Yg[c] = limb(y);
      Y[c] = limb(axis ? y >> g.down() : y);
      i64 w = f.at(c, row.c, row.c2);
      if (view.comp(c) == f.pz) w += pulse;
      W[c] = limb(axis ? w : w >> wd);
    }
    view.cross(Y, W, a);
#pragma unroll
    for (int c = 0; c < N; ++c) k[c] = limb(q63(a[c]));
    ks.store(s, k);
    ys.store(s, Yg);
  }
  return bad;
}

// One attempted DOP853 step of size h at tau = tx (t = x) over a scaled
// segment: new spin in S (on any outcome the caller decides whether to keep
// it: Sn), the error's verdict in out.  False: outside the fixed-point range.
template <class V, class KS>
__device__ __forceinline__ bool dop_step(const V& view, KS& ks, const SegScale& q, const i64* o0, const i64* o1, const i64* o2,
                                         i64 ga, u64 wm, int we, double x, double tx, double h, const StepTol& tol,
                                         const i64* S, i64* Sn, StepOut& out) {
  using namespace dop;
  constexpr int N = V::N;
  const Grade g{q.sk};
  const int k = g.e0() + g.e1();
  StepField<N> f;
  if (!step_field(view, q, q.ok - k, o0, o1, o2, ga, wm, we, x, tx, h, 1, f)) return false;  // (1: up to 1 rad)
  const int ez = f.ez, r = 1 - ez > 63 ? 63 : 1 - ez, r0 = r + g.up() > 63 ? 63 : r + g.up();
  StageNone none;
  const unsigned stages_bad = dop_stages(view, ks, none, f, S, r, g);
  unsigned bad = stages_bad;
  // ---- 8th-order sum, new spin, the two error rows
  Acc sb[N], s3[N], s5[N];
#pragma unroll
  for (int c = 0; c < N; ++c) sb[c] = s3[c] = s5[c] = {0, 0};
  {
    Limb k[N];
    ks.load(0, k);
#pragma unroll 1
    for (int j = 0; j < 8; j += 2) {
      Limb k2[N];
      ks.load(5 + j, k2);
#pragma unroll
      for (int c = 0; c < N; ++c) {
        mac(sb[c], kSumCoef[j][0], k[c]);
        mac(s3[c], kSumCoef[j][1], k[c]);
        mac(s5[c], kSumCoef[j][2], k[c]);
      }
      ks.load(j < 6 ? 6 + j : 11, k);
#pragma unroll
      for (int c = 0; c < N; ++c) {
        mac(sb[c], kSumCoef[j + 1][0], k2[c]);
        mac(s3[c], kSumCoef[j + 1][1], k2[c]);
        mac(s5[c], kSumCoef[j + 1][2], k2[c]);
      }
    }
  }
  i64 e3[N], e5[N], big[N];
#pragma unroll
  for (int c = 0; c < N; ++c) {
    bad |= ((unsigned)(int)(sb[c].hh >> 32) + (1u << 24)) & ~((1u << 25) - 1u);
    Sn[c] = S[c] + rsh(q63(sb[c], 5), view.comp(c) == 0 ? r0 : r);
    e3[c] = q63(s3[c]);  // 2^-4 of the row
    e5[c] = q63(s5[c]);  // 2^-3 of the row
    const i64 m0 = S[c] < 0 ? -S[c] : S[c], m1 = Sn[c] < 0 ? -Sn[c] : Sn[c];
    big[c] = m0 > m1 ? m0 : m1;
  }
  if (view.any(bad != 0)) return false;
  // ---- err^2 = 2^2(ee - sa) N5^2 / (3 rtol^2 (N5 + N3 / 100)), N = sum (e_c / G_c)^2 with
  // G_c = |S_c| + atol / rtol in units of 2^(se + sa); one component after another in a
  // rolled loop, their words in the stage array
  i64 E5[3], E3[3], Mx[3];
  view.gather(e5, E5);
  view.gather(e3, E3);
  view.gather(big, Mx);
  if (((u64)(Mx[0] | Mx[1] | Mx[2]) >> 62) != 0) return false;  // a spin twice its norm: a step far too long
  // the spin at grade 0, the errors times 2^e1: component 0's were kept times 2^k more
  Mx[0] >>= g.e0();
  Mx[1] >>= g.e1();
  Mx[2] >>= g.e1();
  E5[0] >>= k;
  E3[0] >>= k;
  const int ee = ez - g.e1();
  u64 all5 = 0, all3 = 0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const u64 m5 = (u64)(E5[c] < 0 ? -E5[c] : E5[c]), m3 = (u64)(E3[c] < 0 ? -E3[c] : E3[c]);
    all5 |= m5;
    all3 |= m3;
    ks.set_word(c, (i64)m5);
    ks.set_word(3 + c, (i64)m3);
    ks.set_word(6 + c, Mx[c]);
  }
  const int be = bexp(tol.ratio);
  int sa = be - 1021 - q.se;  // atol / rtol < 2^(se + sa - 1)
  sa = sa < 0 ? 0 : sa;
  const i64 ar = to_q63(tol.ratio, q.se + sa);
  out.accept = true;
  out.root8 = bits_f64(0x7ff0000000000000ull);
  if (all5 == 0) return true;
  const int l5 = clz64(all5), l3 = all3 ? clz64(all3) : 63;
  u64 n5 = 0, n3 = 0;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    // 2^-8 / G, G in [2^-7, 1): 2^62 / (G 2^z) shifted by z
    const u64 G = (u64)((ks.word(6 + c) >> sa) + ar) << 1;
    const int z = clz64(G);
    const u64 y = recip(G << z) >> (6 - z);
    const u64 t5 = umul((u64)ks.word(c) << l5, y), t3 = umul((u64)ks.word(3 + c) << l3, y);
    n5 += umul(t5, t5);
    n3 += umul(t3, t3);
  }
  n3 = umul(n3, 184467440737095516ull);  // N3 / 100
  // e5 = n 2^(1 - l5) 2^3, e3 = n 2^(1 - l3) 2^4, and 2^8 from 1 / G: the two blocks' scales
  const int d2 = 2 * (l5 - l3 + 1);  // N3's block is 2^d2 of N5's
  u64 t;
  int et;  // N5 + N3 / 100 = t 2^(et - 64) in units of N5's block
  if (d2 >= 0) {
    t = n3 + (d2 > 63 ? 0 : n5 >> d2);
    et = d2;
  } else {
    t = n5 + (d2 < -63 ? 0 : n3 >> -d2);
    et = 0;
  }
  if (n5 == 0 || t == 0) return false;
  const int z5 = clz64(n5), zt = clz64(t);
  n5 <<= z5;
  t <<= zt;
  const u64 rb = f64_bits(tol.rtol);
  const u64 rt = ((rb & kFrac) | kOne) << 11;  // rtol = rt 2^(bexp - 1022 - 64)
  const u64 A = umul(n5, n5);                  // in [1/4, 1)
  const u64 B = umul(umul(rt, rt), t);         // times 3 / 16: in [2^-7, 1/4)
  const u64 b = (B >> 3) + (B >> 4);
  // X = err^2 = 2^kx A / b, A >= b
  const int kx = 2 * (ee - sa) + 24 - 2 * l5 - 2 * z5 - et + zt - 2 * (bexp(tol.rtol) - 1022) - 4;
  out.accept = kx <= 0 && (kx < -10 || (A >> -kx) <= b);
  const int i = kx & 15, j = kx >> 4;  // kx = 16 j + i
  const u64 rr = root16(A, b, i);
  const int zr = clz64(rr);  // rr / 2^64 = r / 2, to the nearest double
  out.root8 = bits_f64(((u64)(1022 + 1 - zr - j) << 52) + ((rr << zr) >> 11) + (((rr << zr) >> 10) & 1) - kOne);
  return true;
}

// ---------------------------------------------------------------- adjoint step
// Column s of the tableau, from stage s's side: the stages r = s + 1 .. s + n that read
// kappa_s (their a_rs from kAdjCoef[off], over 2^7 for r >= 9 and 2^2 below) and b_s / 2^3.
namespace adjcol {
__device__ __forceinline__ constexpr int last_reader(int s) { return s == 2 ? 3 : (s == 3 ? 5 : 12); }
__device__ __forceinline__ constexpr double col(int s, int r) {
  return dopst::a(r, s == 1 ? 0 : (r == 3 ? 1 : (r <= 5 ? s - 2 : s - 3)));
}
}  // namespace adjcol
struct AdjRow {
  int off, n;
  Limb b;
};
#define ST_ROW(s, off) {off, adjcol::last_reader(s) - (s), coef(dopst::b(s), 3)}
static __constant__ AdjRow kAdjRows[12] = {ST_ROW(1, 0),  ST_ROW(2, 11),  ST_ROW(3, 12),  ST_ROW(4, 14),
                                           ST_ROW(5, 22), ST_ROW(6, 29),  ST_ROW(7, 35),  ST_ROW(8, 40),
                                           ST_ROW(9, 44), ST_ROW(10, 47), ST_ROW(11, 49), ST_ROW(12, 50)};
#undef ST_ROW
#define ST_A(s, r) coef(adjcol::col(s, r), (r) >= 9 ? 7 : 2)
static __constant__ Limb kAdjCoef[51] = {
    ST_A(1, 2), ST_A(1, 3), ST_A(1, 4), ST_A(1, 5), ST_A(1, 6), ST_A(1, 7), ST_A(1, 8), ST_A(1, 9),
    ST_A(1, 10), ST_A(1, 11), ST_A(1, 12), ST_A(2, 3), ST_A(3, 4), ST_A(3, 5), ST_A(4, 5), ST_A(4, 6),
    ST_A(4, 7), ST_A(4, 8), ST_A(4, 9), ST_A(4, 10), ST_A(4, 11), ST_A(4, 12), ST_A(5, 6), ST_A(5, 7),
    ST_A(5, 8), ST_A(5, 9), ST_A(5, 10), ST_A(5, 11), ST_A(5, 12), ST_A(6, 7), ST_A(6, 8), ST_A(6, 9),
    ST_A(6, 10), ST_A(6, 11), ST_A(6, 12), ST_A(7, 8), ST_A(7, 9), ST_A(7, 10), ST_A(7, 11), ST_A(7, 12),
    ST_A(8, 9), ST_A(8, 10), ST_A(8, 11), ST_A(8, 12), ST_A(9, 10), ST_A(9, 11), ST_A(9, 12), ST_A(10, 11),
    ST_A(10, 12), ST_A(11, 12), {0, 0}};
#undef ST_A

// What a step adds to the gradient moments, times 2^(exp + scales of spin and adjoint) / h:
// the sums over the stages of z, c z, c^2 z with z = (dL/dk_s / h) x Y_s at the node c, and with
// the pulse's phase of cos z_z, sin z_z, c sin z_z (halved).
struct AdjMoments {
  i64 z0[3], z1[3], z2[3], cz, sz, scz;
  int exp;
  int e[3] = {0, 0, 0};  // less these, by component (the pulse's: component pz's)
};

// Scale and grade of an adjoint: as a spin's, but graded, its words' norm may be sqrt 3 times
// that of the vector and the field's sqrt 2 times, so its scale is one bit up (dop_adjoint's bounds).
__device__ __forceinline__ bool adjoint_scale(const double l[3], int ok, int& le, int& gl) {
  if (!spin_scale(l, le)) return false;
  gl = spin_grade(l, le, ok);
  if (gl >= -1 && gl <= 1) gl = 0;  // (a grade of 1 would gain nothing)
  le += gl != 0 ? 1 : 0;
  return true;
}

// Backward through one DOP853 step of size h at tau = tx from the spin S: the adjoint lam (a
// scaled vector like S) of the step's result becomes that of S.  With kh_s = (dL/dk_s) / h
//   kh_s = b_s lam + sum_{r > s} a_rs yb_r,  yb_s = h Omega_s x kh_s,  dL/dS = lam + sum_s yb_s;
// kh is kept as kh 2^-K: sum |a_rs| |yb_r| + |b_s| stays under 17, 10, 7.5 |lam| (|lam| <= 1/4)
// for steps below 1/4, 1/8, 1/16 rad; above that the growing K costs more bits than FP64
// loses.  For s >= 9 it stays under 0.6, and
// the large coefficients of the tableau multiply these: they have a K of their own, -1.
// The adjoint has a grade gl of its own (adjoint_scale).
// The stages' 12 states Y go to ys, kappa and then yb to ks.  In FP64 a step takes some 850
// instructions of 76 cycles.  False: out of range, the caller takes FP64.
template <class KS>
__device__ __forceinline__ bool dop_adjoint(KS& ks, KS& ys, const SegScale& q, const i64* o0, const i64* o1, const i64* o2,
                                            i64 ga, u64 wm, int we, double x, double tx, double h, bool pulse_grads,
                                            const i64* S, i64* lam, AdjMoments& m, int gl = 0) {
  const Lane3 view;
  const Grade gs{q.sk}, g{gl};
  StepField<3> f;
  // the field at the larger of the two grades, shifted down where the other needs it
  const int ks0 = gs.e0() + gs.e1(), kl0 = g.e0() + g.e1(), wk = imax(ks0, kl0), wl = wk - kl0;
  if (!step_field(view, q, q.ok - wk, o0, o1, o2, ga, wm, we, x, tx, h, -1, f)) return false;  // (-1: up to 1/4 rad)
  if (pulse_grads && !f.pulse) return false;
  const int ez = f.ez, r = 1 - ez > 63 ? 63 : 1 - ez;
  if (dop_stages(view, ks, ys, f, S, r, gs, wk - ks0) != 0) return false;
  const int K = ez < -3 ? 1 : 4 + ez;
  const int up = g.up() > 63 ? 63 : g.up();
  // z = kh x Y: in components 1 and 2, Y_0 and kh_0 meet the other's components 1 and 2
  const int zd = (g.e1() + gs.e0()) - (g.e0() + gs.e1()), zy = zd > 0 ? zd : 0, zk = zd < 0 ? -zd : 0;
  m.e[0] = g.e1() + gs.e1();
  m.e[1] = m.e[2] = g.e1() + gs.e0() - zy;
  Limb ll[3];
  i64 ln[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    ll[c] = limb(lam[c] + 16);
    ln[c] = lam[c];
    m.z0[c] = m.z1[c] = m.z2[c] = 0;
  }
  m.cz = m.sz = m.scz = 0;
  // A stage's z may pass the words' range (sum |kh| |Y| up to 6), the sums do not: they are
  // mean values of lam x Y over the step, below 0.1.  So the sums run modulo 2^64, without shifts down.
  m.exp = -2;
#pragma unroll 1
  for (int s = 11; s >= 0; --s) {
    const AdjRow& row = kAdjRows[s];
    const Limb nc = kStageRows[s].c, nc2 = kStageRows[s].c2;
    const bool late = s >= 8;
    Acc a[3];
    i64 kq[3];
    // the stages r >= 9, then those below
#pragma unroll
    for (int c = 0; c < 3; ++c) a[c] = {0, 0};
    int j = row.n;
#pragma unroll 1
    for (const int j0 = late ? 0 : 7 - s; j > j0;) {
      Limb yb[3];
      --j;
      const Limb g = kAdjCoef[row.off + j];
      ks.load(s + 1 + j, yb);
#pragma unroll
      for (int c = 0; c < 3; ++c) mac(a[c], g, yb[c]);
    }
    const int ls = late ? 6 + ez : 5 + ez - K;  // (at most 7)
    const int bs = late ? 0 : K - 1;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const i64 t = late ? q63(mac0(row.b, ll[c]), 4) : q63(mac0(row.b, ll[c]), 2) >> bs;
      const i64 sum = ls >= 0 ? q63(a[c], ls) : q63(a[c]) >> (ls < -63 ? 63 : -ls);
      kq[c] = t + (c == 0 ? sum >> up : sum);
      a[c] = {0, 0};
    }
#pragma unroll 1
    while (j > 0) {
      Limb yb[3];
      --j;
      const Limb g = kAdjCoef[row.off + j];
      ks.load(s + 1 + j, yb);
#pragma unroll
      for (int c = 0; c < 3; ++c) mac(a[c], g, yb[c]);
    }
    Limb kl[3], kc[3], W[3], Y[3];
    i64 hc = 0, hs = 0, pulse = 0;
    if (f.pulse) {
      const u64 phi = f.phase_at(nc);
      hc = half_cos_turns(phi);
      pulse = mulq(f.hg, limb(hc + 16), 1);
      if (pulse_grads) hs = half_cos_turns(phi - 0x4000000000000000ull);
    }
    ys.load(s, Y);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const i64 sum = ez >= -1 ? q63(a[c], 1 + ez) : q63(a[c]) >> (ez < -64 ? 63 : -1 - ez);
      const i64 kh = kq[c] + (c == 0 ? sum >> up : sum);
      kc[c] = limb((c == 0 ? kh >> g.down() : kh) + 16);
      kl[c] = c == 0 ? limb((kh >> zk) + 16) : kc[c];
      if (c == 0) Y[c] = limb(unlimb(Y[c]) >> zy);
      i64 w = f.at(c, nc, nc2);
      if (c == f.pz) w += pulse;
      W[c] = limb(c == 0 ? w : w >> wl);
    }
    view.cross(W, kc, a);  // half of yb 2^-(K + ez)
    const int us = ez - 1 + (late ? -1 : K), zs = late ? 0 : K + 1;
    Limb yb[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const i64 y2 = q63(a[c], 1) - 32;
      const i64 add = us >= 0 ? shl(y2, us) : y2 >> (us < -63 ? 63 : -us);
      yb[c] = limb(y2 + 16);
      ln[c] += c == 0 ? add >> up : add;
    }
    ks.store(s, yb);
    view.cross(kl, Y, a);
    i64 zz = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      a[c].mid -= kHalfLimb - (1 << 24);  // (half of the last bit in the place of half a limb)
      const i64 z = q63(a[c], 1);         // |kq| < 0.95, |Y| < 0.44
      m.z0[c] = add(m.z0[c], shl(z, zs));
      m.z1[c] = add(m.z1[c], shl(mulw63(nc, z, 1), zs));
      m.z2[c] = add(m.z2[c], shl(mulw63(nc2, z, 1), zs));
      if (c == f.pz) zz = z;
    }
    if (pulse_grads) {
      m.cz = add(m.cz, shl(mulw63(limb(hc + 16), zz, 0), zs));
      const i64 t = mulw63(limb(hs + 16), zz, 0);
      m.sz = add(m.sz, shl(t, zs));
      m.scz = add(m.scz, shl(mulw63(nc, t, 1), zs));
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) lam[c] = ln[c];
  return true;
}

// ---------------------------------------------------------------- rotations
// 1 / (2k + 3)! and 1 / (2k + 2)! as Q63: sin b / b = 1 - z (1/3! - z/5! ...), cos b = 1 - z (1/2! - z/4! ...), z = b^2
static __constant__ i64 kHalfAngle[8][2] = {
    {1537228672809129301ll, 4611686018427387904ll}, {76861433640456465ll, 384307168202282325ll},
    {1830034134296583ll, 12810238940076078ll}, {25417140754119ll, 228754266787073ll},
    {231064915947ll, 2541714075412ll}, {1481185359ll, 19255409662ll},
    {7053264ll, 105798954ll}, {25931ll, 440829ll}};

// One rotation: y (of grade g, kappa at the grade |g|) by 2^ez |kappa| about -kappa, |kappa| < 0.73, |y| < 0.251 (ungraded).  With k = 2^ez kappa
// and b = |k|/2, v' = v + S (w (v x k) + S/2 (v x k) x k), S = sin b / b and w = cos b: both are
// even series in b, so neither a square root nor a division is needed; above 1 rad the series
// run at b 2^-m and are doubled m times.  In FP64 a rotation is some 100 instructions of 76 cycles,
// its sincos more than half of them; here it is about 400 of 2 to 4.  False: kappa is zero.
__device__ __forceinline__ bool rotate(int ez, const Limb* k, i64* y, Grade g) {
  const Lane3 view;
  constexpr i64 kHalf = 1ll << 62;
  const int ps = ez < -60 ? 62 : (ez < 1 ? 1 - ez : 0);
  Acc t[3];
  Limb v[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) v[c] = limb((c == 0 ? y[c] >> g.down() : y[c]) + 16);
  Acc a = mac0(k[1], k[1]);
  mac(a, k[2], k[2]);
  const int kg = g.e0() + g.e1(), x2 = 2 * kg;
  const i64 k2 = q63(mac0(k[0], k[0])) + (q63(a) >> x2);
  // z = |kappa|^2 4^(ez - 1) 4^-doublings <= 1/4
  const int lead = clz64((u64)k2), dbl = 2 * ez + 2 - lead, doublings = dbl > 0 ? dbl >> 1 : 0;
  const int zs = 2 - 2 * ez + 2 * doublings;
  const i64 zw = zs >= 0 ? k2 >> (zs > 62 ? 62 : zs) : shl(k2, -zs);
  const Limb z = limb(zw + 16);
  // z < 2^-n: the first term left out is below 2^-65
  const int nz = clz64((u64)zw) - 1;
  const int terms = nz >= 20 ? 2 : (nz >= 13 ? 3 : (nz >= 9 ? 4 : (nz >= 7 ? 5 : (nz >= 5 ? 6 : 8))));
  i64 sb = kHalfAngle[terms - 1][0], cb = kHalfAngle[terms - 1][1];
#pragma unroll 1
  for (int i = terms - 2; i >= 0; --i) {
    sb = kHalfAngle[i][0] - mulq(z, limb(sb));
    cb = kHalfAngle[i][1] - mulq(z, limb(cb));
  }
  i64 s2 = kHalf - q63(mac0(z, limb(sb)), -1), w2 = kHalf - q63(mac0(z, limb(cb)), -1);  // S / 2, w / 2
#pragma unroll 1
  for (int i = 0; i < doublings; ++i) {
    const Limb sl = limb(s2 + 16), wl = limb(w2 + 16);
    s2 = q63(mac0(sl, wl), 1);
    w2 = (i64)((u64)q63(mac0(wl, wl), 2) - (u64)kHalf);
  }
  const Limb sl = limb(s2 + 16);
  const Limb fs = limb(mulq(sl, limb(w2 + 16), 1)), fp = limb(mulq(sl, sl, 1));  // S w / 2, S^2 / 2
  // tau = 2^ts v x kappa, as large as |v| < 0.251 and |kappa| < 2^((1 - lead) / 2) let it be
  // (and b times that)
  const int tb = ez - (lead >> 1);
  // (graded, |v| < 0.44 and kappa's words up to 1.42 times as large)
  const int ts = (lead < 30 ? 2 + ((lead > 2 ? lead - 2 : 0) >> 1) : 16) - (tb > 0 ? tb : 0) - (kg ? 1 : 0);
  const int us = ts - ez > 62 ? 62 : ts - ez;
  const i64 half = us > 0 ? (1ll << us) >> 1 : 0;
  const int up = g.up() > 63 ? 63 : g.up();
  view.cross(v, k, t);
  // tau's component 0 is kept times 2^(e0 + up()), and so is that of tau x kappa; in the others it
  // stands 2^2k further down
  Limb tau[3], tc[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const i64 x = ts >= 0 ? q63(t[c], ts) - (16 << ts) : (q63(t[c]) - 16) >> -ts;  // (the limb's half was shifted with the product)
    tau[c] = limb(x + 16);
    tc[c] = c == 0 ? limb((x >> x2) + 16) : tau[c];
  }
  view.cross(tc, k, t);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const i64 p = q63(t[c]) - 16;  // 2^(ez - 1) tau x kappa
    Acc d = mac0(fs, tau[c]);
    mac(d, fp, limb((ez >= 1 ? shl(p, ez - 1) : p >> ps) + 16));
    const i64 u = q63(d, 1);
    const i64 add = us < 0 ? shl(u, -us) : (u + half) >> us;
    y[c] += c == 0 ? add >> up : add;
  }
  return k2 != 0;
}


// The quaternion steppers' rotations in the order they are applied, each at a node (the halves of
// it and of its square) by a weight: RK45's proposal (5), its comparison (4); RKF45's 5, whose
// first four are the comparison.
struct QuatRow {
  Limb c, c2, w;
};
#define ST_Q(node, w) {coef(node, 1), coef_sq(node), coef(w, 0)}
static __constant__ QuatRow kQuatRows[14] = {
    ST_Q(0.0, rk45::CH1),      ST_Q(rk45::A3, rk45::CH3),   ST_Q(rk45::A4, rk45::CH4),   ST_Q(rk45::A5, rk45::CH5),
    ST_Q(rk45::A6, rk45::CH6), ST_Q(0.0, rk45::C1),         ST_Q(rk45::A3, rk45::C3),    ST_Q(rk45::A4, rk45::C4),
    ST_Q(rk45::A5, rk45::C5),  ST_Q(0.0, rkf45::C1),        ST_Q(rkf45::A3, rkf45::C3),  ST_Q(rkf45::A4, rkf45::C4),
    ST_Q(rkf45::A5, rkf45::C5), ST_Q(rkf45::A6, rkf45::C6)};
#undef ST_Q

// One step of RK45 (F: RKF45) with quaternions: the rotations turn the spin one after another,
// which is what the product of their quaternions does.  Proposal in w, its difference from the
// comparison in e.  False: out of range (above 4 rad, off the segment, no field): the caller takes FP64.
template <bool F>
__device__ __forceinline__ bool quat_step(const SegScale& q, const i64* o0, const i64* o1, const i64* o2, i64 ga, u64 wm, int we,
                                          double x, double tx, double h, const i64* S, i64* w, i64* e) {
  const Grade g{q.sk};
  StepField<3> f;
  if (!step_field(Lane3(), q, q.ok - g.e0() - g.e1(), o0, o1, o2, ga, wm, we, x, tx, h, 3, f)) return false;
  i64 y[3] = {S[0], S[1], S[2]}, y0[3] = {S[0], S[1], S[2]};
  bool ok = true;
  constexpr int kFirst = F ? 9 : 0, kLast = F ? 14 : 9, kSwap = F ? 13 : 5;
#pragma unroll 1
  for (int n = kFirst; n < kLast; ++n) {
    if (n == kSwap) {  // RK45: proposal done, comparison from S; RKF45: comparison done
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        y0[c] = y[c];
        if (!F) y[c] = S[c];
      }
    }
    const QuatRow& row = kQuatRows[n];
    Limb k[3];
    i64 o[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) o[c] = f.at(c, row.c, row.c2);
    if (f.pulse) f.add_pulse(Lane3(), f.pulse_at(row.c), o);
#pragma unroll
    for (int c = 0; c < 3; ++c) k[c] = limb(mulq(row.w, limb(o[c])));
    ok &= rotate(f.ez, k, y, g);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    w[c] = F ? y[c] : y0[c];
    e[c] = F ? y[c] - y0[c] : y0[c] - y[c];
  }
  return ok;
}

}  // namespace fx
}  // namespace st
