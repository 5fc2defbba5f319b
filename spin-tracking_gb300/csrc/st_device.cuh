// Device building blocks of the hot path: the RNG, the ballistic trajectory
// events, the field polynomial and single step attempts of DOP853, RK45 and
// the integrator types 2-5 (Magnus CFET8, RK45 / RKF45 with quaternions, RKF45).
//
// Two arithmetic regimes:
//  * Trajectory and RNG code reproduces the reference's doubles bit for bit
//    (same operation order, no FMA contraction: every add and mul is an
//    explicit round-to-nearest intrinsic, every division and square root the
//    correctly rounded one of st_softfp.cuh), so event times, bounce/collision
//    counts and RNG draws match the CPU build exactly.  Its log, acos, cos and
//    sin are the correctly rounded ones of st_crmath.cuh (equal to the host C
//    library's wherever those are correctly rounded), or CUDA's with
//    ST_TRAJ_CORRECTLY_ROUNDED 0 (st_fields.cuh).
//  * The spin steppers are restated: the field as a polynomial in segment time,
//    reciprocal-form error weights and step controller.  DOP853 steps run in
//    64-bit fixed point (st_fixed.cuh), the rest (and DOP853 steps outside the
//    fixed-point range) in FMA-contracted FP64.  Results agree with the
//    reference to the integration tolerance, not bit for bit.
#pragma once

#include <float.h>
#include <stdint.h>
#include "st_internal.h"
#include "st_fields.cuh"
#include "st_tableau.h"
#include "st_crmath.cuh"
#include "st_fixed.cuh"
#include "st_softfp.cuh"

namespace st {
// The trajectory's transcendental functions (ST_TRAJ_CORRECTLY_ROUNDED, st_fields.cuh).
__device__ __forceinline__ double traj_log(double x) {
#if ST_TRAJ_CORRECTLY_ROUNDED
  double y;
  return crm::cr_log_fast(x, y) ? y : crm::log_accurate(x);
#else
  return log(x);
#endif
}
// acos(x) and the sin and cos of the result
__device__ __forceinline__ void traj_acos_sincos(double x, double& y, double& sy, double& cy) {
#if ST_TRAJ_CORRECTLY_ROUNDED
  if (!crm::cr_acos_sincos_fast(x, y, sy, cy)) crm::cr_acos_sincos(x, y, sy, cy);
#else
  y = acos(x);
  sy = sin(y);
  cy = cos(y);
#endif
}
__device__ __forceinline__ void traj_sincos(double x, double& s, double& c) {
#if ST_TRAJ_CORRECTLY_ROUNDED
  if (!crm::cr_sincos_fast(x, s, c)) crm::sincos_accurate(x, s, c);
#else
  s = sin(x);
  c = cos(x);
#endif
}
}  // namespace st

namespace st {

// ------------------------------------------------------------------ exact ops
__device__ __forceinline__ double xadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double xsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double xmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double xdiv(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double xsqrt(double a) { return __dsqrt_rn(a); }
// sgn with sgn(0) = +1 (src/particle.cpp:24-31)
__device__ __forceinline__ double sgn1(double v) { return v < 0.0 ? -1.0 : 1.0; }
// std::min / std::max argument conventions
__device__ __forceinline__ double std_min(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double std_max(double a, double b) { return (a < b) ? b : a; }
// min_d / max_d (src/integrator.cpp:25-33)
__device__ __forceinline__ double min_d(double a, double b) { return (a < b) ? a : b; }
__device__ __forceinline__ double max_d(double a, double b) { return (a > b) ? a : b; }

// ------------------------------------------------------------ fast FP64 roots
// Approximate hardware seeds (PTX rcp.approx / rsqrt.approx, ~2^-22 relative)
// refined by FMA Newton steps on the FP64 pipe.
__device__ __forceinline__ double rcp_seed(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
}
__device__ __forceinline__ double rsqrt_seed(double x) {
  double r;
  asm("rsqrt.approx.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
}
// 1/x to full double precision for finite nonzero x; 0 and inf pass through.
__device__ __forceinline__ double rcp_full(double x) {
  const double r = rcp_seed(x);
  const double e = fma(-x, r, 1.0);
  const double r2 = fma(r, fma(e, e, e), r);  // third-order correction
  return (e == e) ? r2 : r;
}
// 1/sqrt(x) to full double precision for finite positive x.
__device__ __forceinline__ double rsqrt_full(double x) {
  const double y = rsqrt_seed(x);
  const double e = fma(-x * y, y, 1.0);
  const double y2 = fma(y * e, fma(0.375, e, 0.5), y);  // third-order correction
  return (e == e) ? y2 : y;
}
// x^(-1/8) for 1e-300 < x < 1e300: chained rsqrt seeds, two Newton steps on
// r^8 x = 1.
__device__ __forceinline__ double rroot8(double x) {
  double r = rsqrt_seed(rsqrt_seed(rsqrt_seed(x)));
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double r2 = r * r, r4 = r2 * r2;
    const double u = (r4 * r4) * x;
    r = fma(r, fma(u, -0.125, 0.125), r);
  }
  return r;
}

// ------------------------------------------------------------------------ RNG
// Reference rngState (include/particle.h:52-59) and its generator.
struct Rng {
  uint64_t x, y, z, w;
  double spare;
  bool has;
};

// xoshiro256+ as the reference implements it (src/particle.cpp:59-70): the
// last word is re-derived from the third, not rotated in place.
__device__ __forceinline__ uint64_t rng_next(Rng& r) {
  const uint64_t out = r.x + r.z;
  const uint64_t t = r.y << 17;
  r.z ^= r.x;
  r.w ^= r.y;
  r.y ^= r.z;
  r.x ^= r.w;
  r.z ^= t;
  r.w = (r.z << 45) | (r.z >> 19);
  return out;
}
// top 53 bits scaled by 2^-53 (exact), src/particle.cpp:72-83
__device__ __forceinline__ double rng_uniform(Rng& r) { return sfp::unit_53(rng_next(r)); }

// The uniform pairs of the Marsaglia polar method until 0 < s = u^2 + v^2 < 1,
// and the factor sqrt(-2 log s / s) from log s.
__device__ __forceinline__ void marsaglia_draw(Rng& r, double& u, double& v, double& s) {
  do {
    u = sfp::signed_unit_53(rng_next(r));
    v = sfp::signed_unit_53(rng_next(r));
    s = xadd(xmul(u, u), xmul(v, v));
  } while (sfp::f64_bits(s) >= 0x3ff0000000000000ull || s == 0.0);  // s >= 1 or s = 0
}
__device__ __forceinline__ double marsaglia_factor(double s, double log_s) { return sfp::sqrt_rn(sfp::div_rn(xmul(-2.0, log_s), s)); }

// Marsaglia polar normal with cached spare (src/particle.cpp:89-107).
__device__ __forceinline__ double rng_normal(Rng& r, double mean, double sd) {
  if (r.has) {
    r.has = false;
    return xadd(xmul(r.spare, sd), mean);
  }
  double u, v, s;
  marsaglia_draw(r, u, v, s);
  const double f = marsaglia_factor(s, traj_log(s));
  r.spare = xmul(v, f);
  r.has = true;
  return xadd(mean, xmul(xmul(sd, u), f));
}
// Three standard normals, in a rolled loop (one copy of the draw's code).
__device__ __forceinline__ void rng_normals(Rng& r, double& n0, double& n1, double& n2) {
#pragma unroll 1
  for (int k = 0; k < 3; ++k) {
    n0 = n1;
    n1 = n2;
    n2 = rng_normal(r, 0.0, 1.0);
  }
}
__device__ __forceinline__ double rng_exponential(Rng& r, double tc) {
  return xmul(-tc, traj_log(xsub(1.0, rng_uniform(r))));
}

// Seeding of initParticlesCPU (src/particle.cpp:648-663): splitmix64 of the
// 32-bit sum seed + ipart, two outputs split into 32-bit halves, three
// discarded draws.
__device__ __forceinline__ uint64_t splitmix_next(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ Rng rng_seed(unsigned int seed, unsigned int ipart) {
  uint64_t s = (uint64_t)(uint32_t)(seed + ipart);
  Rng r;
  const uint64_t a = splitmix_next(s);
  r.x = (uint32_t)a;
  r.y = (uint32_t)(a >> 32);
  const uint64_t b = splitmix_next(s);
  r.z = (uint32_t)b;
  r.w = (uint32_t)(b >> 32);
  r.spare = 0.0;
  r.has = false;
  rng_next(r);
  rng_next(r);
  rng_next(r);
  return r;
}

// ------------------------------------------------------------ particle state
struct PState {
  double t, px, py, pz, vx, vy, vz, Sx, Sy, Sz, h, next_gas;
  Rng rng;
  uint64_t n_coll, n_bounce, n_steps;
  int fail;
  int turns;  // precession turns about x (see count_turn)
  bool stop;
  char coll, wall;
};

__device__ __forceinline__ PState load_state(const DeviceState& s, int64_t i) {
  PState p;
  p.t = s.t[i];
  p.px = s.px[i]; p.py = s.py[i]; p.pz = s.pz[i];
  p.vx = s.vx[i]; p.vy = s.vy[i]; p.vz = s.vz[i];
  p.Sx = s.Sx[i]; p.Sy = s.Sy[i]; p.Sz = s.Sz[i];
  p.h = s.h[i];
  p.next_gas = s.next_gas[i];
  p.rng.x = s.rx[i]; p.rng.y = s.ry[i]; p.rng.z = s.rz[i]; p.rng.w = s.rw[i];
  p.rng.spare = s.rspare[i];
  p.rng.has = s.rhas[i] != 0;
  p.n_coll = s.n_coll[i]; p.n_bounce = s.n_bounce[i]; p.n_steps = s.n_steps[i];
  p.fail = s.fail[i];
  p.turns = s.turns[i];
  p.stop = s.stop[i] != 0;
  p.coll = (char)s.coll[i];
  p.wall = (char)s.wall[i];
  return p;
}

__device__ __forceinline__ void store_state(const DeviceState& s, int64_t i, const PState& p) {
  s.t[i] = p.t;
  s.px[i] = p.px; s.py[i] = p.py; s.pz[i] = p.pz;
  s.vx[i] = p.vx; s.vy[i] = p.vy; s.vz[i] = p.vz;
  s.Sx[i] = p.Sx; s.Sy[i] = p.Sy; s.Sz[i] = p.Sz;
  s.h[i] = p.h;
  s.next_gas[i] = p.next_gas;
  s.rx[i] = p.rng.x; s.ry[i] = p.rng.y; s.rz[i] = p.rng.z; s.rw[i] = p.rng.w;
  s.rspare[i] = p.rng.spare;
  s.rhas[i] = p.rng.has ? 1 : 0;
  s.n_coll[i] = p.n_coll; s.n_bounce[i] = p.n_bounce; s.n_steps[i] = p.n_steps;
  s.fail[i] = p.fail;
  s.turns[i] = p.turns;
  s.stop[i] = p.stop ? 1 : 0;
  s.coll[i] = (uint8_t)p.coll;
  s.wall[i] = (uint8_t)p.wall;
}

// initParticlesCPU for one particle (src/particle.cpp:646-708).
__device__ inline PState init_particle(const SetParams& P, unsigned int ipart) {
  PState p;
  Rng r = rng_seed(P.seed, ipart);
  p.px = xsub(xmul(rng_uniform(r), P.Lx), P.Lx / 2.0);
  p.py = xsub(xmul(rng_uniform(r), P.Ly), P.Ly / 2.0);
  p.pz = xsub(xmul(rng_uniform(r), P.Lz), P.Lz / 2.0);
  p.next_gas = P.gas ? rng_exponential(r, P.tc) : DBL_MAX;
  p.vx = p.vy = p.vz = 0.0;
  if (P.dist == 'C') {
    // the CPU build draws three normals even for V == 0 (src/particle.cpp:677-684)
    const double dx = rng_normal(r, 0.0, 1.0);
    const double dy = rng_normal(r, 0.0, 1.0);
    const double dz = rng_normal(r, 0.0, 1.0);
    const double nrm = xsqrt(xadd(xadd(xmul(dx, dx), xmul(dy, dy)), xmul(dz, dz)));
    p.vx = xdiv(xmul(dx, P.V), nrm);
    p.vy = xdiv(xmul(dy, P.V), nrm);
    p.vz = xdiv(xmul(dz, P.V), nrm);
  } else if (P.dist == 'M') {
    p.vx = xmul(rng_normal(r, 0.0, 1.0), P.sqrtKT_m);
    p.vy = xmul(rng_normal(r, 0.0, 1.0), P.sqrtKT_m);
    p.vz = xmul(rng_normal(r, 0.0, 1.0), P.sqrtKT_m);
  }
  p.rng = r;
  p.Sx = P.yi_x; p.Sy = P.yi_y; p.Sz = P.yi_z;
  p.t = P.t0;
  p.h = P.h0;
  p.stop = false;
  p.coll = 'W';
  p.wall = 0;
  p.fail = 0;
  p.turns = 0;
  p.n_coll = p.n_bounce = p.n_steps = 0;
  return p;
}

// Start of the current ballistic segment (t_old, pos_old, v_old).
struct SegStart {
  double t, px, py, pz, vx, vy, vz;
};

// A trajectory event whose draws were taken but whose logarithms, sines and
// cosines are not yet computed (traj_event<true>): a cosine-law diffuse
// reflection, or a gas collision.
//   reflection: x[0] = u1, x[1] = u2 (their sqrt and 2 pi, and |v|, are taken later too)
//   gas:        x[0] = 1 - u of the gas clock's exponential draw, then the
//               Marsaglia pairs drawn for the three velocity normals, (u, v, s)
//               in x[1..3] and x[4..6]: one pair when the first normal is the
//               cached spare (spare_first), two otherwise
struct EventDefer {
  double x[7];
  char wall;
  bool pending, gas, spare_first;
};

// New velocity of a cosine-law diffuse reflection off wall w from the sin and
// cos of phi = acos(sqrt u1) and of theta = 2 pi u2 (src/particle.cpp:309-328).
__device__ __forceinline__ void diffuse_apply(PState& p, double sp, double cp, double stt, double ct, double speed,
                                              char w) {
  if (w == 'x') {
    p.vx = xmul(xmul(xmul(-1.0, sgn1(p.vx)), speed), cp);
    p.vy = xmul(xmul(-speed, sp), ct);
    p.vz = xmul(xmul(speed, sp), stt);
  } else if (w == 'y') {
    p.vx = xmul(xmul(speed, sp), ct);
    p.vy = xmul(xmul(xmul(-1.0, sgn1(p.vy)), speed), cp);
    p.vz = xmul(xmul(speed, sp), stt);
  } else {
    p.vx = xmul(xmul(speed, sp), ct);
    p.vy = xmul(xmul(speed, sp), stt);
    p.vz = xmul(xmul(xmul(-1.0, sgn1(p.vz)), speed), cp);
  }
}

// A reflection's arguments from its draws: sqrt(u1), theta = 2 pi u2 and |v|.
__device__ __forceinline__ double norm3(double x, double y, double z) {
  return sfp::sqrt_rn(xadd(xadd(xmul(x, x), xmul(y, y)), xmul(z, z)));
}
__device__ __forceinline__ double theta_of(double u2) { return xmul(xmul(u2, 2.0), 3.141592653589793); }

// New velocity of a cosine-law diffuse reflection off wall w (src/particle.cpp:309-328).
__device__ __forceinline__ void diffuse_velocity(PState& p, double u1, double u2, char w) {
  const double su = sfp::sqrt_rn(u1), theta = theta_of(u2), speed = norm3(p.vx, p.vy, p.vz);
  double phi, cp, sp, ct, stt;
  traj_acos_sincos(su, phi, sp, cp);
  traj_sincos(theta, stt, ct);
  diffuse_apply(p, sp, cp, stt, ct, speed, w);
}

// Position of the k-th set bit of m, counting from 0 (k < popc(m)).
__device__ __forceinline__ int nth_set_bit(unsigned m, int k) {
  int p = 0;
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const int c = __popc(m & ((1u << s) - 1u));
    if (k >= c) {
      k -= c;
      m >>= s;
      p += s;
    }
  }
  return p;
}

// The velocity after a gas collision from its three normals: Maxwell-Boltzmann
// ('M'), or the old speed in their direction ('C') (src/particle.cpp:373-391).
__device__ __forceinline__ void gas_velocity(PState& p, const SetParams& P, double n1, double n2, double n3) {
  if (P.dist == 'M') {
    p.vx = xmul(n1, P.sqrtKT_m);
    p.vy = xmul(n2, P.sqrtKT_m);
    p.vz = xmul(n3, P.sqrtKT_m);
  } else {
    const double speed = norm3(p.vx, p.vy, p.vz), nrm = norm3(n1, n2, n3);
    p.vx = sfp::div_rn(xmul(n1, speed), nrm);
    p.vy = sfp::div_rn(xmul(n2, speed), nrm);
    p.vz = sfp::div_rn(xmul(n3, speed), nrm);
  }
}

// The rest of a deferred gas collision from the logarithms of its draws
// (log_a of the gas clock's 1 - u, log_s0 and log_s1 of the Marsaglia pairs):
// the gas clock as rng_exponential advances it, the three normals and the
// cached spare as three rng_normal calls leave them, and the new velocity
// (src/particle.cpp:117-119, 89-111, 373-391).
__device__ __forceinline__ void gas_finish(PState& p, const SetParams& P, const EventDefer& dd, double log_a,
                                           double log_s0, double log_s1) {
  p.next_gas = xadd(p.next_gas, xmul(-P.tc, log_a));
  const double f0 = marsaglia_factor(dd.x[3], log_s0);
  const double pair0 = xadd(0.0, xmul(xmul(1.0, dd.x[1]), f0));
  const double spare0 = xmul(dd.x[2], f0);
  double n1, n2, n3;
  if (dd.spare_first) {
    n1 = xadd(xmul(p.rng.spare, 1.0), 0.0);
    n2 = pair0;
    n3 = xadd(xmul(spare0, 1.0), 0.0);
    p.rng.spare = spare0;
  } else {
    const double f1 = marsaglia_factor(dd.x[6], log_s1);
    n1 = pair0;
    n2 = xadd(xmul(spare0, 1.0), 0.0);
    n3 = xadd(0.0, xmul(xmul(1.0, dd.x[4]), f1));
    p.rng.spare = xmul(dd.x[5], f1);
  }
  gas_velocity(p, P, n1, n2, n3);
}

// The deferred events of a warp, lanes `pend`, computed by all 32 lanes
// together (the warp must be converged).  A diffuse reflection needs the sin
// and cos of two angles (the argument of its acos Newton step and theta), a
// gas collision the logarithms of up to three of its draws.  Those
// evaluations are dealt out one per lane per pass (one pass for up to 16
// reflections, another for up to 10 gas collisions) instead of running one
// after the other on each pending lane; each pending lane then finishes its
// own event from the shuffled results.  Every value is computed by the code of
// the per-lane path (diffuse_velocity, rng_exponential, rng_normal), so the
// results are the same bit for bit.
template <bool GAS>
__device__ __forceinline__ void deferred_events_warp(PState& p, const SetParams& P, EventDefer& dd, unsigned pend,
                                                     int lane) {
#if ST_TRAJ_CORRECTLY_ROUNDED
  const unsigned FULL = 0xffffffffu;
  const unsigned below = (1u << lane) - 1u;
  const unsigned refl = GAS ? __ballot_sync(FULL, dd.pending && !dd.gas) : pend;
  if (refl) {
    const int np = __popc(refl);
    const bool mine = dd.pending && !dd.gas;
    double x = 0.0, theta = 0.0, y0 = 0.0, arg_a = 0.0;
    if (mine) {
      x = sfp::sqrt_rn(dd.x[0]);
      theta = theta_of(dd.x[1]);
      y0 = acos(x);
      arg_a = x < 1.0 ? crm::acos_newton_arg(x, y0) : 0.0;  // NaN and 1 use none
    }
    const int rank = __popc(refl & below);
    crm::DD sa{0.0, 0.0}, ca{1.0, 0.0}, st{0.0, 0.0}, ct{1.0, 0.0};
    for (int base = 0; base < 2 * np; base += 32) {
      // job j = base + lane: the Newton argument of reflection j (j < np) or
      // the theta of reflection j - np
      const int j = base + lane;
      const int src = nth_set_bit(refl, min(j < np ? j : j - np, np - 1));
      const double a1 = __shfl_sync(FULL, arg_a, src), a2 = __shfl_sync(FULL, theta, src);
      crm::DD sn, cs;
      crm::sincos_dd(j < np ? a1 : a2, sn, cs);
      // the reflection of rank r takes jobs r and np + r
      const int ja = rank - base, jb = np + rank - base;
      const double v0 = __shfl_sync(FULL, sn.hi, ja & 31), v1 = __shfl_sync(FULL, sn.lo, ja & 31);
      const double v2 = __shfl_sync(FULL, cs.hi, ja & 31), v3 = __shfl_sync(FULL, cs.lo, ja & 31);
      const double w0 = __shfl_sync(FULL, sn.hi, jb & 31), w1 = __shfl_sync(FULL, sn.lo, jb & 31);
      const double w2 = __shfl_sync(FULL, cs.hi, jb & 31), w3 = __shfl_sync(FULL, cs.lo, jb & 31);
      if (ja >= 0 && ja < 32) {
        sa = {v0, v1};
        ca = {v2, v3};
      }
      if (jb >= 0 && jb < 32) {
        st = {w0, w1};
        ct = {w2, w3};
      }
    }
    if (mine) {
      double phi, sp, cp;
      if (!crm::acos_sincos_given(x, y0, sa, ca, phi, sp, cp)) crm::cr_acos_sincos(x, phi, sp, cp);
      double stt = st.hi, ctt = ct.hi;
      if (!(crm::trig_sure(st) && crm::trig_sure(ct))) crm::sincos_accurate(theta, stt, ctt);
      diffuse_apply(p, sp, cp, stt, ctt, norm3(p.vx, p.vy, p.vz), dd.wall);
      dd.pending = false;
    }
  }
  if (GAS) {
    const unsigned gm = pend & ~refl;
    if (gm) {
      const int ng = __popc(gm);
      const bool mine = dd.pending && dd.gas;
      const double third = dd.spare_first ? 1.0 : dd.x[6];  // log 1 = 0 fills the unused job
      const int rank = __popc(gm & below);
      double l0 = 0.0, l1 = 0.0, l2 = 0.0;
      for (int base = 0; base < 3 * ng; base += 32) {
        // job j = base + lane: draw j % 3 (1 - u, s of pair 0, s of pair 1)
        // of gas collision j / 3
        const int j = base + lane;
        const int q = min(j / 3, ng - 1), k = j - 3 * (j / 3);
        const int src = nth_set_bit(gm, q);
        const double a0 = __shfl_sync(FULL, dd.x[0], src), a1 = __shfl_sync(FULL, dd.x[3], src);
        const double a2 = __shfl_sync(FULL, third, src);
        const double arg = k == 0 ? a0 : (k == 1 ? a1 : a2);
        double y;
        if (!crm::cr_log_fast(arg, y)) y = crm::log_accurate(arg);
        // the collision of rank r takes jobs 3r, 3r + 1, 3r + 2
        const int jr = 3 * rank - base;
        const double r0 = __shfl_sync(FULL, y, jr & 31), r1 = __shfl_sync(FULL, y, (jr + 1) & 31);
        const double r2 = __shfl_sync(FULL, y, (jr + 2) & 31);
        if (jr >= 0 && jr < 32) l0 = r0;
        if (jr + 1 >= 0 && jr + 1 < 32) l1 = r1;
        if (jr + 2 >= 0 && jr + 2 < 32) l2 = r2;
      }
      if (mine) {
        gas_finish(p, P, dd, l0, l1, l2);
        dd.pending = false;
        dd.gas = false;
      }
    }
  }
#else
  if (dd.pending) {
    if (GAS && dd.gas)
      gas_finish(p, P, dd, traj_log(dd.x[0]), traj_log(dd.x[3]), dd.spare_first ? 0.0 : traj_log(dd.x[6]));
    else
      diffuse_velocity(p, dd.x[0], dd.x[1], dd.wall);
    dd.pending = false;
    dd.gas = false;
  }
#endif
}

// The ballistic move in the reference's own operations, for a dt that is not finite.
static __device__ __noinline__ void move_any(double* x, double dt, double ay) {
  const double hax = xmul(xmul(0.5 * 0.0, dt), dt), hay = xmul(xmul(0.5 * ay, dt), dt);
  x[0] = xadd(xadd(x[0], xmul(x[3], dt)), hax);
  x[1] = xadd(xadd(x[1], xmul(x[4], dt)), hay);
  x[2] = xadd(xadd(x[2], xmul(x[5], dt)), hax);
  x[3] = xadd(x[3], xmul(0.0, dt));
  x[4] = xadd(x[4], xmul(ay, dt));
  x[5] = xadd(x[5], xmul(0.0, dt));
}

// The nearest wall and its time; NaN when every comparison fails.
__device__ __forceinline__ double first_wall(double dtx, double dty, double dtz, char& wall) {
  double tb = __longlong_as_double(0x7ff8000000000000ll);
  if (sfp::is_nan(dtx) || sfp::is_nan(dty) || sfp::is_nan(dtz)) {  // a NaN loses every comparison
    if (dtx == dty) {
      tb = dtx; wall = 'b';  // x-y edge
    } else if (dtx == dtz) {
      tb = dtx; wall = 'c';  // x-z edge
    } else if (dty == dtz) {
      tb = dty; wall = 'd';  // y-z edge
    }
    return tb;
  }
  const fx::i64 x = sfp::key(dtx), y = sfp::key(dty), z = sfp::key(dtz);
  if (x < y && x < z) {
    tb = dtx; wall = 'x';
  } else if (y < x && y < z) {
    tb = dty; wall = 'y';
  } else if (z < x && z < y) {
    tb = dtz; wall = 'z';
  } else if (x == y && x == z) {
    tb = dtx; wall = 'a';  // corner
  } else if (x == y) {
    tb = dtx; wall = 'b';  // x-y edge
  } else if (x == z) {
    tb = dtx; wall = 'c';  // x-z edge
  } else if (y == z) {
    tb = dty; wall = 'd';  // y-z edge
  }
  return tb;
}

// One trajectory event: calc_next_collision_time, update_position_and_velocity
// and sanity_check (src/particle.cpp:121-444).  Returns `finished` (the window
// end tf was reached).  Fills the segment start.
//
// DEFER: a diffuse reflection's draws are taken here (the RNG sequence is
// unchanged) but its velocity is left to deferred_events_warp, called later by
// the trajectory-ahead kernel for many lanes at once.  The sanity check then
// sees the velocity before the reflection; that gives the same outcome: the
// reflected velocity is |v| times sines and cosines that are finite and, for
// the draws possible here, non-zero except cos(phi) at u1 = 0, so it is NaN
// or infinite only when the velocity before it already was, which fails the
// same check (NaN) or the position check before it (infinite).  A gas
// collision is deferred the same way: its uniform draws are taken here in the
// reference's order, the logarithms (of the gas clock and of the Marsaglia
// pairs) later.  Its new velocity is the product of finite normals and a finite
// sqrt(kT/m), or the old speed in the direction of the normals, so the NaN check
// gives the outcome it gives on the velocity before the collision (which it
// also tests).
//
// GAS = false: compiled for launches in which no parameter set has gas
// collisions.  Their gas clock is DBL_MAX and never moves, so the gas
// collision is never the next event: either the wall time is finite and
// smaller, or it is infinite and the step ends at the maxPosStep / window
// limit either way.
//
// What bounds it: latency and issue of the integer code.  Divisions, square roots,
// comparisons and draws run on the integer pipes (st_softfp.cuh), and the
// reference's additions of a zero acceleration's terms are left out where they
// change nothing (finite dt; -0 becomes 0 as they make it): some 35 FP64
// instructions remain of about 180.
template <bool DEFER = false, bool GAS = true>
__device__ __forceinline__ bool traj_event(PState& p, const SetParams& P, double tf, SegStart& s0,
                                           EventDefer* dd = nullptr) {
  const double G = kGravity;
  double dtx, dty, dtz;
  // ---- time to the next wall (calc_next_collision_time)
  dtx = sfp::div_rn(xsub(sfp::negative(p.vx) ? -P.hLx : P.hLx, p.px), p.vx);
  dtz = sfp::div_rn(xsub(sfp::negative(p.vz) ? -P.hLz : P.hLz, p.pz), p.vz);
  if (P.gravity) {
    const double y2 = xmul(p.vy, p.vy);
    // Moving down meets the floor; moving up meets the ceiling unless the apex
    // is below it (then rise and fall to the floor).  Floor and ceiling share
    // one root pair: the reference's ceiling roots (-vy + sq)/G, (-vy - sq)/G
    // are bit for bit its floor roots (sq - vy)/G, -(sq + vy)/G in swapped
    // order (IEEE addition commutes, negation is exact), and min(|r1|, |r2|)
    // does not depend on the order (both roots are NaN together), so both
    // branches run the same sqrt and divisions, once.  The apex branch shares
    // them too: its sqrt argument and its one division are chosen first.
    bool apex = false;
    double arg, t1 = 0.0;
    if (sfp::negative(p.vy)) {
      const double dy = xadd(p.py, P.hLy);
      arg = xadd(xmul(-2.0 * G, dy), y2);
    } else {
      const double top = xadd(sfp::div_g(xmul(-0.5, y2)), p.py);
      apex = sfp::lt(top, P.hLy);
      if (apex) {
        t1 = sfp::div_g(-p.vy);
        const double ap = xadd(xadd(p.py, xmul(p.vy, t1)), xmul(xmul(0.5 * G, t1), t1));
        arg = sfp::div_g(xmul(xsub(-P.hLy, ap), 2.0));
      } else {
        arg = xsub(y2, xmul(2.0 * G, xsub(p.py, P.hLy)));
      }
    }
    const double sq = sfp::sqrt_rn(arg);
    if (apex) {
      dty = xadd(t1, sq);
    } else {
      const double a1 = fabs(sfp::div_g(xadd(sq, p.vy))), a2 = fabs(sfp::div_g(xsub(sq, p.vy)));
      dty = sfp::f64_bits(a2) < sfp::f64_bits(a1) ? a2 : a1;
    }
    if (!sfp::le(1e-16, dtx))  // only the first offending axis is replaced (below 1e-16, or NaN)
      dtx = 1e6;
    else if (!sfp::le(1e-16, dty))
      dty = 1e6;
    else if (!sfp::le(1e-16, dtz))
      dtz = 1e6;
  } else {
    dty = sfp::div_rn(xsub(sfp::negative(p.vy) ? -P.hLy : P.hLy, p.py), p.vy);
    if (sfp::lt(dtx, 1e-16))
      dtx = 1e6;
    else if (sfp::lt(dty, 1e-16))
      dty = 1e6;
    else if (sfp::lt(dtz, 1e-16))
      dtz = 1e6;
  }
  const double tb = first_wall(dtx, dty, dtz, p.wall);
  // ---- gas collision, wall, window end or maxPosStep
  bool gas_next = false;
  double to_col = tb;
  const double to_gas = GAS ? xsub(p.next_gas, p.t) : 0.0;
  if (!GAS) {
    // no gas collisions in this launch
  } else if (sfp::lt(to_gas, tb)) {
    gas_next = true;
    to_col = to_gas;
  } else if (sfp::eq(to_gas, tb)) {  // tie: the wall wins and the gas clock is redrawn
    p.next_gas = xadd(p.next_gas, rng_exponential(p.rng, P.tc));
    to_col = to_gas;
  }
  const double left = xsub(tf, p.t);
  const bool window_end = sfp::le(left, P.maxPosStep);
  const double to_free = window_end ? left : P.maxPosStep;
  bool finished = false;
  double dt;
  if (sfp::le(to_col, to_free)) {
    dt = to_col;
    if (gas_next) {
      p.coll = 'G';
      p.n_coll += 1;
      if (DEFER && (P.dist != 'M' || sfp::is_finite(P.sqrtKT_m))) {
        dd->x[0] = xsub(1.0, rng_uniform(p.rng));  // rng_exponential's draw; its log later
        dd->gas = true;
      } else {
        p.next_gas = xadd(p.next_gas, rng_exponential(p.rng, P.tc));
      }
    } else {
      p.n_bounce += 1;
      p.coll = 'W';
    }
    if (window_end && sfp::eq(to_col, to_free)) finished = true;
  } else {
    p.coll = 'N';
    dt = to_free;
    if (window_end) finished = true;
  }
  // ---- ballistic move (update_position_and_velocity)
  s0.t = p.t;
  s0.px = p.px; s0.py = p.py; s0.pz = p.pz;
  s0.vx = p.vx; s0.vy = p.vy; s0.vz = p.vz;
  p.t = xadd(p.t, dt);
  if (sfp::is_finite(dt)) {
    p.px = sfp::plus0(xadd(s0.px, xmul(s0.vx, dt)));
    p.py = xadd(s0.py, xmul(s0.vy, dt));
    p.pz = sfp::plus0(xadd(s0.pz, xmul(s0.vz, dt)));
    p.vx = sfp::plus0(p.vx);
    p.vz = sfp::plus0(p.vz);
    if (P.gravity) {
      p.py = xadd(p.py, xmul(xmul(0.5 * G, dt), dt));
      p.vy = xadd(p.vy, xmul(G, dt));
    } else {
      p.py = sfp::plus0(p.py);
      p.vy = sfp::plus0(p.vy);
    }
  } else {
    double x[6] = {p.px, p.py, p.pz, p.vx, p.vy, p.vz};
    move_any(x, dt, P.gravity ? G : 0.0);
    p.px = x[0]; p.py = x[1]; p.pz = x[2];
    p.vx = x[3]; p.vy = x[4]; p.vz = x[5];
  }
  if (p.coll == 'W') {
    const char w = p.wall;
    const bool sx = (w == 'x' || w == 'a' || w == 'b' || w == 'c');
    const bool sy = (w == 'y' || w == 'a' || w == 'b' || w == 'd');
    const bool sz = (w == 'z' || w == 'a' || w == 'c' || w == 'd');
    if (sx) p.px = sfp::negative(p.px) ? -P.hLx : P.hLx;
    if (sy) p.py = sfp::negative(p.py) ? -P.hLy : P.hLy;
    if (sz) p.pz = sfp::negative(p.pz) ? -P.hLz : P.hLz;
    bool diffuse = false;
    if (sfp::lt((double)FLT_MIN, P.diffuse)) diffuse = sfp::lt(rng_uniform(p.rng), P.diffuse);
    if (diffuse) {
      // cosine-law diffuse reflection (src/particle.cpp:309-328): both draws
      // now, the roots and the trigonometry now or (DEFER) batched later
      const double u1 = rng_uniform(p.rng), u2 = rng_uniform(p.rng);
      if (w == 'x' || w == 'y' || w == 'z') {
        if (DEFER) {
          dd->x[0] = u1;
          dd->x[1] = u2;
          dd->wall = w;
          dd->gas = false;
          dd->pending = true;
        } else {
          diffuse_velocity(p, u1, u2, w);
        }
      } else {
        p.stop = true;  // a diffuse hit on an edge or corner stops the particle
      }
    } else {
      if (sx) p.vx = -p.vx;
      if (sy) p.vy = -p.vy;
      if (sz) p.vz = -p.vz;
    }
  } else if (GAS && p.coll == 'G') {
    if (DEFER && dd->gas) {
      // the three normals' uniform draws now, in rng_normal's order: the first
      // normal is the cached spare or opens pair 0, whose spare is the second;
      // the third opens pair 1 (its spare stays cached) or is pair 0's spare
      dd->spare_first = p.rng.has;
#pragma unroll 1
      for (int k = dd->spare_first ? 1 : 0; k < 2; ++k) {
        double u, v, s;
        marsaglia_draw(p.rng, u, v, s);
        const bool first = k == 0 || dd->spare_first;
        dd->x[first ? 1 : 4] = u;
        dd->x[first ? 2 : 5] = v;
        dd->x[first ? 3 : 6] = s;
      }
      p.rng.has = !dd->spare_first;
      dd->pending = true;
    } else {
      double n0 = 0.0, n1 = 0.0, n2 = 0.0;
      rng_normals(p.rng, n0, n1, n2);
      gas_velocity(p, P, n0, n1, n2);
    }
  }
  // ---- sanity_check (limits: the half edges plus 1e-15)
  if (sfp::abs_gt(p.px, P.limx) || sfp::abs_gt(p.py, P.limy) || sfp::abs_gt(p.pz, P.limz)) {
    p.stop = true; p.fail = 1;  // out of bounds
  } else if (sfp::is_inf(s0.t) || sfp::is_inf(p.t)) {
    p.stop = true; p.fail = 2;  // infinite time
  } else if (sfp::is_nan(s0.px) || sfp::is_nan(s0.py) || sfp::is_nan(s0.pz) || sfp::is_nan(p.px) ||
             sfp::is_nan(p.py) || sfp::is_nan(p.pz)) {
    p.stop = true; p.fail = 3;  // NaN position
  } else if (sfp::is_nan(p.vx) || sfp::is_nan(p.vy) || sfp::is_nan(p.vz) || sfp::is_nan(s0.vx) ||
             sfp::is_nan(s0.vy) || sfp::is_nan(s0.vz)) {
    p.stop = true; p.fail = 4;  // NaN velocity
  }
  return finished;
}

// ------------------------------------------------------------ field model
// Integrator state of the current segment.  Omega(tau) = gamma*B at time
// t0 + tau is the quadratic o0 + tau*(o1 + tau*o2) (plus the pulse).  For
// DOP853 in fixed point (fx) the same fields hold the Q63 words of st_fixed.cuh
// (as bits): the scaled polynomial and pulse amplitude, and the spin in k.
struct Seg {
  double o0x, o0y, o0z, o1x, o1y, o1z, o2x, o2y, o2z;
#if !ST_GRAD_IS_LINEAR
  double p0x, p0y, p0z, v0x, v0y, v0z;
#endif
  double gpa;          // gamma * pulse amplitude (0: no pulse)
  double t0, xf, x, h, posneg, facold;
  double kx, ky, kz;   // DOP853: the spin (fx) or the derivative at (x, y) (FSAL); RK45: last stage-6 state
  double lastH, lnprev;
  double hu;           // step size of the last accepted attempt (read by the adjoint replay)
  unsigned int nstep;
  int turns;           // precession turns of the segment's accepted steps (count_turn)
  bool reject, last;
  bool acc;            // the last attempt was accepted
  bool fx;             // DOP853 in fixed point, scaled by sc
  bool carry;          // k holds the spin in fixed point (kept from segment to segment; false at a window's start)
  fx::SegScale sc;
};

// Precession phase accumulation: the phase phi = atan2(Sz, Sy) about x jumps
// by 2 pi where the spin's (y, z) projection crosses the cut at phi = +-pi
// (Sy < 0, Sz changing sign).  While accepted steps turn the spin by less than a
// quarter turn about x (DOP853 at rtol 1e-12: some 0.13 rad), a crossing is a sign
// change of Sz with Sy < 0 at both ends; longer steps (Magnus passes a radian on long
// smooth segments) and spins that cross near Sy = 0 can miss one.  Counted +1 from
// phi near +pi to near -pi (phi increasing) and -1 back; atan2(Sz, Sy) + 2 pi * turns
// is then continuous along the run.
__device__ __forceinline__ int count_turn(double y0, double z0, double y1, double z1) {
  if (!(y0 < 0.0 && y1 < 0.0)) return 0;
  const bool s0 = signbit(z0), s1 = signbit(z1);
  return (s0 == s1) ? 0 : (s1 ? 1 : -1);
}

// The per-set field constants (launch_prepare_sets): gamma * B0, the gradient
// tensor's columns through the st_grad hook, gamma * E / c^2 and the gravity
// terms of the segment polynomial.
__device__ inline void prepare_set(SetParams& P) {
  const double gm = P.gamma;
  const double g_ = P.gravity ? kGravity : 0.0;
  // the pulse's turns per second |w| / 2 pi = wturn_m 2^(wturn_e - 64) to 64 bits
  P.wturn_m = 0;
  P.wturn_e = 0;
  if (P.w != 0.0 && isfinite(P.w)) {
    const double w = fabs(P.w), p = w * 0.15915494309189535;  // 1 / (2 pi) = 0.15915494309189535 -9.839338337591243e-18
    const double e = fma(w, -9.839338337591243e-18, fma(w, 0.15915494309189535, -p));
    const int x = fx::bexp(p) - 1022;  // p in [1/2, 1) 2^x
    if (x > -900 && x < 900) {
      const uint64_t m = (uint64_t)(fx::to_q63(p, x)) << 1;
      const uint64_t de = (uint64_t)(long long)rint(ldexp(e, 64 - x));
      P.wturn_m = (de >> 63) == 0 && m + de < m ? ~0ull : m + de;
      P.wturn_e = x;
    }
  }
  P.gB0[0] = gm * P.B0x; P.gB0[1] = gm * P.B0y; P.gB0[2] = gm * P.B0z;
  P.axis = fabs(P.gB0[1]) > fabs(P.gB0[0]) ? 1 : 0;
  if (fabs(P.gB0[2]) > fabs(P.gB0[P.axis])) P.axis = 2;
  P.pz = (5 - P.axis) % 3;
  const Vec3 ex = {1.0, 0.0, 0.0}, ey = {0.0, 1.0, 0.0}, ez = {0.0, 0.0, 1.0};
  const Vec3 c0 = st_grad(ex, P), c1 = st_grad(ey, P), c2 = st_grad(ez, P);
  P.gGc[0][0] = gm * c0.x; P.gGc[0][1] = gm * c0.y; P.gGc[0][2] = gm * c0.z;
  P.gGc[1][0] = gm * c1.x; P.gGc[1][1] = gm * c1.y; P.gGc[1][2] = gm * c1.z;
  P.gGc[2][0] = gm * c2.x; P.gGc[2][1] = gm * c2.y; P.gGc[2][2] = gm * c2.z;
  P.gEc[0] = gm * P.inv_c2 * P.Ex; P.gEc[1] = gm * P.inv_c2 * P.Ey; P.gEc[2] = gm * P.inv_c2 * P.Ez;
  // d/dtau of v x E along the parabola: (g yhat) x E = g (Ez, 0, -Ex)
  P.o1g[0] = gm * P.inv_c2 * g_ * P.Ez; P.o1g[1] = 0.0; P.o1g[2] = -gm * P.inv_c2 * g_ * P.Ex;
#if ST_GRAD_IS_LINEAR
  P.o2c[0] = 0.5 * g_ * P.gGc[1][0]; P.o2c[1] = 0.5 * g_ * P.gGc[1][1]; P.o2c[2] = 0.5 * g_ * P.gGc[1][2];
#else
  P.o2c[0] = P.o2c[1] = P.o2c[2] = 0.0;  // the hook is evaluated at every stage instead
#endif
  for (int c = 0; c < 3; ++c) P.o2w[c] = P.o2c[(c + P.axis) % 3];
}

// Coefficients o0, o1 of the field polynomial of a segment starting at (p0, v0).
__device__ __forceinline__ void seg_field(const SetParams& P, double px, double py, double pz, double vx, double vy,
                                          double vz, double o0[3], double o1[3]) {
  const double* e = P.gEc;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    // v0 x gEc, component c
    const double cr = (c == 0) ? fma(vy, e[2], -vz * e[1]) : (c == 1) ? fma(vz, e[0], -vx * e[2]) : fma(vx, e[1], -vy * e[0]);
#if ST_GRAD_IS_LINEAR
    o0[c] = P.gB0[c] + fma(px, P.gGc[0][c], fma(py, P.gGc[1][c], fma(pz, P.gGc[2][c], cr)));
    o1[c] = fma(vx, P.gGc[0][c], fma(vy, P.gGc[1][c], fma(vz, P.gGc[2][c], P.o1g[c])));
#else
    o0[c] = P.gB0[c] + cr;
    o1[c] = P.o1g[c];
#endif
  }
}

// Fill the integrator's segment from its field coefficients and time span.
__device__ __forceinline__ void seg_begin(Seg& g, const SetParams& P, double t0, double t_end, const double o0[3],
                                          const double o1[3]) {
  g.o0x = o0[0]; g.o0y = o0[1]; g.o0z = o0[2];
  g.o1x = o1[0]; g.o1y = o1[1]; g.o1z = o1[2];
  g.o2x = P.o2c[0]; g.o2y = P.o2c[1]; g.o2z = P.o2c[2];
  g.gpa = P.gamma * P.a;
  g.t0 = t0;
  g.xf = t_end;
  g.x = t0;
  g.posneg = (t_end - t0 < 0.0) ? -1.0 : 1.0;
}

// The fixed-point words of a segment's state, kept in its double fields.
__device__ __forceinline__ double as_f64(fx::i64 m) { return __longlong_as_double(m); }
__device__ __forceinline__ fx::i64 as_i64(double x) { return __double_as_longlong(x); }

// Components turned n places (0 to 2): x becomes component n.  Words have the set's axis first
// (n = P.axis); back with unturn.
template <class T>
__device__ __forceinline__ void turn_by(T& x, T& y, T& z, int n) {
#pragma unroll 1
  for (; n > 0; --n) {
    const T t = x;
    x = y;
    y = z;
    z = t;
  }
}
__device__ __forceinline__ void unturn(double& x, double& y, double& z, int axis) { turn_by(x, y, z, axis == 0 ? 0 : 3 - axis); }

// The field of a segment as the trajectory side hands it to the spin side:
// the polynomial's o0 and o1, for DOP853 and quaternion sets scaled to fixed point where they
// have a scale there (fx; then o0, o1 and o2 hold Q63 words, the set's axis first).
struct SegPoly {
  double o0[3], o1[3], o2[3];
  fx::SegScale sc;
  bool fx;
};
// Scale a polynomial given in doubles over a segment of length T.
// FX (here and below): an instantiation for runs with sets that step in fixed point; without it
// every step is inlined in FP64 (the FP64 form as a call beside the fixed-point one takes 1.25 times
// as long: 65,536 particles x 0.1 s with beta 0.04, 105 ms against 83).
template <bool FX>
__device__ __forceinline__ void seg_scale(SegPoly& q, const SetParams& P, double T, bool backward = false) {
  q.fx = false;
  if (!FX) return;
  const double gpa = P.gamma * P.a;
  if (((P.integrator == 0 && (P.tol_ratio >= 0.0 || (backward && P.tol_ratio == -2.0))) || P.integrator == 3 || P.integrator == 5) && (gpa == 0.0 || isfinite(P.w)))
  {
    turn_by(q.o0[0], q.o0[1], q.o0[2], P.axis);
    turn_by(q.o1[0], q.o1[1], q.o1[2], P.axis);
    q.sc.pz = P.pz;
    q.fx = fx::field_scale(q.o0, q.o1, P.o2w, gpa, T, q.sc, true);
    if (!q.fx) {
      unturn(q.o0[0], q.o0[1], q.o0[2], P.axis);
      unturn(q.o1[0], q.o1[1], q.o1[2], P.axis);
    }
  }
  if (q.fx) {
#pragma unroll 1  // rolled: less code
    for (int c = 0; c < 3; ++c) {
      const int e0 = q.sc.oe - (c == 0 ? 0 : q.sc.ok), e1 = e0 - q.sc.te, e2 = e1 - q.sc.te;
      q.o0[c] = as_f64(fx::to_q63(q.o0[c], e0));
      q.o1[c] = as_f64(fx::to_q63(q.o1[c], e1));
      q.o2[c] = as_f64(fx::to_q63(P.o2w[c], e2));
    }
  }
}
template <bool FX>
__device__ __forceinline__ void seg_poly(SegPoly& q, const SetParams& P, const SegStart& s0, double t_end) {
  seg_field(P, s0.px, s0.py, s0.pz, s0.vx, s0.vy, s0.vz, q.o0, q.o1);
  seg_scale<FX>(q, P, t_end - s0.t);
}

// Fill the integrator's segment from the handed-over field.
template <bool FX>
__device__ __forceinline__ void seg_open(Seg& g, const SetParams& P, const SegPoly& q, double t0, double t_end) {
  seg_begin(g, P, t0, t_end, q.o0, q.o1);
  g.fx = FX && q.fx;
  if (!FX) return;
  const int se = g.sc.se, sk = g.sc.sk;  // the spin's own scale and grade go on
  g.sc = q.sc;
  g.sc.se = se;
  g.sc.sk = sk;
  if (q.fx) {
    g.o2x = q.o2[0]; g.o2y = q.o2[1]; g.o2z = q.o2[2];
    g.gpa = as_f64(fx::to_q63(g.gpa, q.sc.oe - (P.pz == 0 ? 0 : q.sc.ok)));
  }
}

template <bool FX>
__device__ __forceinline__ void seg_setup(Seg& g, const SetParams& P, const SegStart& s0, double t_end) {
  SegPoly q;
  seg_poly<FX>(q, P, s0, t_end);
  seg_open<FX>(g, P, q, s0.t, t_end);
#if !ST_GRAD_IS_LINEAR
  g.p0x = s0.px; g.p0y = s0.py; g.p0z = s0.pz;
  g.v0x = s0.vx; g.v0y = s0.vy; g.v0z = s0.vz;
#endif
}

// Omega = gamma * B at tau = t - t0.
__device__ __forceinline__ void omega_at(const Seg& g, const SetParams& P, double tau, double& Ox, double& Oy,
                                         double& Oz) {
  Ox = fma(fma(g.o2x, tau, g.o1x), tau, g.o0x);
  Oy = fma(fma(g.o2y, tau, g.o1y), tau, g.o0y);
  Oz = fma(fma(g.o2z, tau, g.o1z), tau, g.o0z);
#if !ST_GRAD_IS_LINEAR
  {
    const double gy = P.gravity ? 0.5 * kGravity : 0.0;
    const Vec3 pos = {fma(g.v0x, tau, g.p0x), fma(fma(gy, tau, g.v0y), tau, g.p0y), fma(g.v0z, tau, g.p0z)};
    const Vec3 Gp = st_grad(pos, P);
    Ox = fma(P.gamma, Gp.x, Ox);
    Oy = fma(P.gamma, Gp.y, Oy);
    Oz = fma(P.gamma, Gp.z, Oz);
  }
#endif
#if ST_PULSE_IS_Z_COS
  if (g.gpa != 0.0) Oz = fma(g.gpa, cos(P.w * (g.t0 + tau)), Oz);
#else
  {
    const Vec3 pu = st_pulse(g.t0 + tau, P);
    Ox = fma(P.gamma, pu.x, Ox);
    Oy = fma(P.gamma, pu.y, Oy);
    Oz = fma(P.gamma, pu.z, Oz);
  }
#endif
}

// Bloch right-hand side f = y x Omega (src/integrator.cpp:83-88).
__device__ __forceinline__ void bloch(double yx, double yy, double yz, double Ox, double Oy, double Oz, double& fx,
                                      double& fy, double& fz) {
  fx = fma(yy, Oz, -yz * Oy);
  fy = fma(yz, Ox, -yx * Oz);
  fz = fma(yx, Oy, -yy * Ox);
}

__device__ __forceinline__ void feval(const Seg& g, const SetParams& P, double tau, double yx, double yy, double yz,
                                      double& fx, double& fy, double& fz) {
  double Ox, Oy, Oz;
  omega_at(g, P, tau, Ox, Oy, Oz);
  bloch(yx, yy, yz, Ox, Oy, Oz, fx, fy, fz);
}

// The field polynomial scaled by a step size h, so that a stage's Bloch
// evaluation gives h k directly and its state y + sum a_j (h k_j) is an FMA
// chain from y (ten multiplications per attempt instead of one per stage and
// component).
struct HPoly {
  double o0x, o0y, o0z, o1x, o1y, o1z, o2x, o2y, o2z, gpa, h;
};
__device__ __forceinline__ HPoly hpoly_of(const Seg& g, double h) {
  return {h * g.o0x, h * g.o0y, h * g.o0z, h * g.o1x, h * g.o1y, h * g.o1z,
          h * g.o2x, h * g.o2y, h * g.o2z, h * g.gpa, h};
}
// h Omega at tau = t - t0 (omega_at, scaled).
__device__ __forceinline__ void homega_at(const HPoly& q, const Seg& g, const SetParams& P, double tau, double& Ox,
                                          double& Oy, double& Oz) {
  Ox = fma(fma(q.o2x, tau, q.o1x), tau, q.o0x);
  Oy = fma(fma(q.o2y, tau, q.o1y), tau, q.o0y);
  Oz = fma(fma(q.o2z, tau, q.o1z), tau, q.o0z);
#if !ST_GRAD_IS_LINEAR
  {
    const double gy = P.gravity ? 0.5 * kGravity : 0.0;
    const Vec3 pos = {fma(g.v0x, tau, g.p0x), fma(fma(gy, tau, g.v0y), tau, g.p0y), fma(g.v0z, tau, g.p0z)};
    const Vec3 Gp = st_grad(pos, P);
    const double hg = q.h * P.gamma;
    Ox = fma(hg, Gp.x, Ox);
    Oy = fma(hg, Gp.y, Oy);
    Oz = fma(hg, Gp.z, Oz);
  }
#endif
#if ST_PULSE_IS_Z_COS
  if (g.gpa != 0.0) Oz = fma(q.gpa, cos(P.w * (g.t0 + tau)), Oz);
#else
  {
    const Vec3 pu = st_pulse(g.t0 + tau, P);
    const double hg = q.h * P.gamma;
    Ox = fma(hg, pu.x, Ox);
    Oy = fma(hg, pu.y, Oy);
    Oz = fma(hg, pu.z, Oz);
  }
#endif
}

// ------------------------------------------------------------ DOP853
// A fixed-point segment's field back in doubles.
__device__ __forceinline__ void seg_unscale(Seg& g, const SetParams& P) {
  const int e0 = g.sc.oe, e1 = e0 - g.sc.te, e2 = e1 - g.sc.te, ok = g.sc.ok;
  g.o0x = fx::from_q63(as_i64(g.o0x), e0);
  g.o0y = fx::from_q63(as_i64(g.o0y), e0 - ok);
  g.o0z = fx::from_q63(as_i64(g.o0z), e0 - ok);
  g.o1x = fx::from_q63(as_i64(g.o1x), e1);
  g.o1y = fx::from_q63(as_i64(g.o1y), e1 - ok);
  g.o1z = fx::from_q63(as_i64(g.o1z), e1 - ok);
  g.o2x = fx::from_q63(as_i64(g.o2x), e2);
  g.o2y = fx::from_q63(as_i64(g.o2y), e2 - ok);
  g.o2z = fx::from_q63(as_i64(g.o2z), e2 - ok);
  unturn(g.o0x, g.o0y, g.o0z, P.axis);
  unturn(g.o1x, g.o1y, g.o1z, P.axis);
  unturn(g.o2x, g.o2y, g.o2z, P.axis);
  g.gpa = fx::from_q63(as_i64(g.gpa), e0 - (P.pz == 0 ? 0 : ok));
  g.fx = false;
}

// The spin of a fixed-point segment in progress as doubles.
__device__ __forceinline__ void dop_spin(const Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz) {
  const fx::Grade k{g.sc.sk};
  Sx = fx::from_q63(as_i64(g.kx), g.sc.se - k.e0());
  Sy = fx::from_q63(as_i64(g.ky), g.sc.se - k.e1());
  Sz = fx::from_q63(as_i64(g.kz), g.sc.se - k.e1());
  unturn(Sx, Sy, Sz, P.axis);
}

// A spin in fixed point stays there from segment to segment (g.carry): it becomes
// doubles again at a window end, or where a segment runs in FP64.
template <bool FX>
__device__ __forceinline__ void spin_settle(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz) {
  if (!FX) return;
  if (g.carry) dop_spin(g, P, Sx, Sy, Sz);
  g.carry = false;
}

// A spin as words: ok false where it has no scale, the tolerances do not fit, or a word
// would lose its sign (-0, or less than half a unit: turns count signs).
struct SpinWords {
  fx::i64 w[3];
  int se, sk;
  bool ok;
};
static __device__ __noinline__ SpinWords spin_words_of(const SetParams& P, int field_grade, double Sx, double Sy, double Sz) {
  SpinWords r;
  turn_by(Sx, Sy, Sz, P.axis);
  const double S[3] = {Sx, Sy, Sz};
  r.ok = fx::spin_scale(S, r.se) && fx::ratio_fits(P.tol_ratio, r.se);
  if (r.ok) {
    r.sk = fx::spin_grade(S, r.se, field_grade);
    fx::spin_words(S, r.se, r.sk, r.w);
#pragma unroll
    for (int c = 0; c < 3; ++c) r.ok &= r.w[c] != 0 || !signbit(S[c]);
  }
  return r;
}

// The derivative at the start of an FP64 segment, taking the segment out of fixed point first.
static __device__ __noinline__ void dop_begin_f64(Seg& g, const SetParams& P, double Sx, double Sy, double Sz) {
  if (g.fx) seg_unscale(g, P);
  feval(g, P, 0.0, Sx, Sy, Sz, g.kx, g.ky, g.kz);
}

// Start a DOP853 call over the segment (src/integrator.cpp:102-119).
template <bool FX>
__device__ __forceinline__ void dop_begin(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz, double h) {
  g.h = h;
  g.facold = 1.0e-4;
  g.nstep = 0;
  g.turns = 0;
  g.reject = false;
  g.last = false;
  if (!FX) {
    feval(g, P, 0.0, Sx, Sy, Sz, g.kx, g.ky, g.kz);
    return;
  }
  if (g.fx && !g.carry) {
    const SpinWords r = spin_words_of(P, g.sc.ok, Sx, Sy, Sz);
    if (r.ok) {
      g.kx = as_f64(r.w[0]);
      g.ky = as_f64(r.w[1]);
      g.kz = as_f64(r.w[2]);
      g.sc.se = r.se;
      g.sc.sk = r.sk;
      g.carry = true;
    }
  }
  if (!(g.fx && g.carry)) {
    spin_settle<FX>(g, P, Sx, Sy, Sz);
    Seg t = g;  // the call takes its address: g itself stays in registers
    dop_begin_f64(t, P, Sx, Sy, Sz);
    g = t;
  }
}

// FP64 stage derivatives k2..k11.
struct StageF64 {
  double v[12][3];
  __device__ __forceinline__ double& k(int s, int c) { return v[s][c]; }
};

// One attempted DOP853 step (one pass of the loop at src/integrator.cpp:128-247)
// in FP64.  Returns 0 to continue, 1 when the segment's last
// step was accepted (g.h then holds that step, as the reference returns it),
// -1 after more than nmax attempts.
__device__ __forceinline__ int dop_attempt_f64(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz) {
  using namespace dop;
  StageF64 ks;
  if (g.nstep > P.nmax) return -1;
  double h = g.h;
  bool last = g.last;
  if ((g.x + 1.01 * h - g.xf) * g.posneg > 0.0) {
    h = g.xf - g.x;
    last = true;
  }
  if (h < P.hmin && !last) h = P.hmin;
  g.nstep++;
  g.acc = false;
  const double tx = g.x - g.t0;
  const double S0[3] = {Sx, Sy, Sz};
  // stage derivatives are carried scaled by h (ks holds h k_s)
  const HPoly hp = hpoly_of(g, h);
  const double k1[3] = {h * g.kx, h * g.ky, h * g.kz};
  // stages 2..11: y + sum_j a_sj (h k_j), then h k_s = Y x (h Omega(x + c_s h))
#pragma unroll
  for (int s = 2; s <= 11; ++s) {
    double Y[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double acc = fma(dopst::a(s, 0), k1[c], S0[c]);
#pragma unroll
      for (int j = 1; j < dopst::cnt(s); ++j) acc = fma(dopst::a(s, j), ks.k(dopst::src(s, j), c), acc);
      Y[c] = acc;
    }
    double Ox, Oy, Oz, kx, ky, kz;
    homega_at(hp, g, P, fma(dopst::c(s), h, tx), Ox, Oy, Oz);
    bloch(Y[0], Y[1], Y[2], Ox, Oy, Oz, kx, ky, kz);
    ks.k(s, 0) = kx;
    ks.k(s, 1) = ky;
    ks.k(s, 2) = kz;
  }
  // stage 12 at x + h; its unscaled Omega is reused for the FSAL derivative
  double Y12[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double acc = fma(dopst::a(12, 0), k1[c], S0[c]);
#pragma unroll
    for (int j = 1; j < dopst::cnt(12); ++j) acc = fma(dopst::a(12, j), ks.k(dopst::src(12, j), c), acc);
    Y12[c] = acc;
  }
  const double tph = tx + h;
  double Ox12, Oy12, Oz12, k12[3];
  omega_at(g, P, tph, Ox12, Oy12, Oz12);
  bloch(Y12[0], Y12[1], Y12[2], h * Ox12, h * Oy12, h * Oz12, k12[0], k12[1], k12[2]);
  // 8th-order combination and the new state
  double bsum[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double acc = B1 * k1[c];
    acc = fma(B6, ks.k(6, c), acc);
    acc = fma(B7, ks.k(7, c), acc);
    acc = fma(B8, ks.k(8, c), acc);
    acc = fma(B9, ks.k(9, c), acc);
    acc = fma(B10, ks.k(10, c), acc);
    acc = fma(B11, ks.k(11, c), acc);
    bsum[c] = fma(B12, k12[c], acc);
  }
  const double bx = bsum[0], by = bsum[1], bz = bsum[2];
  const double nx = Sx + bx, ny = Sy + by, nz = Sz + bz;
  // error estimates: 3rd-order (bhh) and 5th-order (er) rows, h times the
  // reference's; the scale cancels in err = |h| err_5 / sqrt(3 (err_5 + 0.01 err_3))
  const double e1x = fma(-BHH3, k12[0], fma(-BHH2, ks.k(9, 0), fma(-BHH1, k1[0], bx)));
  const double e1y = fma(-BHH3, k12[1], fma(-BHH2, ks.k(9, 1), fma(-BHH1, k1[1], by)));
  const double e1z = fma(-BHH3, k12[2], fma(-BHH2, ks.k(9, 2), fma(-BHH1, k1[2], bz)));
  double er[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double acc = ER1 * k1[c];
    acc = fma(ER6, ks.k(6, c), acc);
    acc = fma(ER7, ks.k(7, c), acc);
    acc = fma(ER8, ks.k(8, c), acc);
    acc = fma(ER9, ks.k(9, c), acc);
    acc = fma(ER10, ks.k(10, c), acc);
    acc = fma(ER11, ks.k(11, c), acc);
    er[c] = fma(ER12, k12[c], acc);
  }
  const double ax = er[0], ay = er[1], az = er[2];
  const double wx = rcp_full(fma(P.rtol, max_d(fabs(Sx), fabs(nx)), P.atol));
  const double wy = rcp_full(fma(P.rtol, max_d(fabs(Sy), fabs(ny)), P.atol));
  const double wz = rcp_full(fma(P.rtol, max_d(fabs(Sz), fabs(nz)), P.atol));
  const double q1x = e1x * wx, q1y = e1y * wy, q1z = e1z * wz;
  const double q2x = ax * wx, q2y = ay * wy, q2z = az * wz;
  const double err2 = fma(q1z, q1z, fma(q1y, q1y, q1x * q1x));
  double err = fma(q2z, q2z, fma(q2y, q2y, q2x * q2x));
  double deno = fma(0.01, err2, err);
  if (deno <= 0.0) deno = 1.0;
  err = err * rsqrt_full(deno * 3.0);
  // step-size controller (Lund-stabilised, clamped to [1/fac2, 1/fac1])
  double hnew;
  const bool fast = (P.beta == 0.0) && (err > 1e-300) && (err < 1e300);
  double rr = 0.0, fac11 = 0.0;
  if (fast) {
    rr = rroot8(err);  // 1 / fac11
    hnew = h * min_d(P.fac2, max_d(P.fac1, P.safe * rr));
  } else {
    fac11 = pow(err, P.expo1);
    double fac = fac11 / pow(g.facold, P.beta);
    fac = max_d(P.facc2, min_d(P.facc1, fac / P.safe));
    hnew = h / fac;
  }
  int ret = 0;
  if (err <= 1.0 || P.fixed) {
    g.acc = true;
    g.hu = h;
    g.facold = max_d(err, 1.0e-4);
    bloch(nx, ny, nz, Ox12, Oy12, Oz12, g.kx, g.ky, g.kz);  // FSAL: f(x + h, y_new)
    g.turns += count_turn(Sy, Sz, ny, nz);
    Sx = nx; Sy = ny; Sz = nz;
    g.x = g.x + h;
    if (last) {
      g.h = h;
      g.last = true;
      return 1;
    }
    if (fabs(hnew) > P.hmax) hnew = g.posneg * P.hmax;
    if (g.reject) hnew = g.posneg * min_d(fabs(hnew), fabs(h));
    g.reject = false;
  } else {
    hnew = fast ? h * max_d(P.fac1, P.safe * rr) : h / min_d(P.facc1, fac11 / P.safe);
    g.reject = true;
    last = false;
  }
  g.last = last;
  g.h = P.fixed ? h : hnew;
  return ret;
}


// The FP64 attempt for any segment, beside the fixed-point step, which takes all but a few (a
// call, not inlined).  A segment in fixed point goes on in FP64 after an
// accepted step; a rejected one changes its step size only.
static __device__ __noinline__ int dop_attempt_slow(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz) {
  if (!g.fx) return dop_attempt_f64(g, P, Sx, Sy, Sz);
  Seg t = g;
  double x, y, z;
  dop_spin(g, P, x, y, z);
  seg_unscale(t, P);
  feval(t, P, t.x - t.t0, x, y, z, t.kx, t.ky, t.kz);
  const int r = dop_attempt_f64(t, P, x, y, z);
  if (t.acc) {
    t.carry = false;
    g = t;
    Sx = x;
    Sy = y;
    Sz = z;
  } else {
    g.h = t.h;
    g.reject = t.reject;
    g.last = t.last;
    g.nstep = t.nstep;
    g.acc = false;
  }
  return r;
}

// One attempted DOP853 step (one pass of the loop at src/integrator.cpp:128-247),
// spin components over the lanes of `view`, stage derivatives in `ks`.  While
// the segment is in fixed point Sx..Sz stay behind (spin_settle).
// Returns as dop_attempt_f64.
//
// What bounds it: latency and supply of instructions at two warps per sub-partition (one
// issued per 3.3 cycles; 298 warp instructions per attempt of a lane in the trajectory-ahead
// kernel, the trajectory's and idle lanes' included), against ~510 FP64 instructions of 76 cycles
// before: 1,048,576 particles x 0.1 s, 642 ms in FP64, 345 in fixed point.
template <bool FX, class V, class KS>
__device__ __forceinline__ int dop_attempt_v(const V& view, KS& ks, Seg& g, const SetParams& P, double& Sx, double& Sy,
                                             double& Sz) {
  if (!FX) return dop_attempt_f64(g, P, Sx, Sy, Sz);
  if (g.nstep > P.nmax) return -1;
  double h = g.h;
  bool last = g.last;
  const double over = g.x + 1.01 * h - g.xf;
  if (g.posneg < 0.0 ? sfp::negative(over) : sfp::lt(0.0, over)) {
    h = g.xf - g.x;
    last = true;
  }
  if (!last && sfp::lt(h, P.hmin)) h = P.hmin;
  fx::i64 Sn[V::N];
  fx::StepOut out;
  bool fixed = g.fx;
  if (fixed) {
    fx::i64 o0[V::N], o1[V::N], o2[V::N], S[V::N], K[3] = {as_i64(g.kx), as_i64(g.ky), as_i64(g.kz)};
    fx::regrade(K, g.sc.sk, g.sc.ok);
    g.kx = as_f64(K[0]);
    g.ky = as_f64(K[1]);
    g.kz = as_f64(K[2]);
    view.pick(as_i64(g.o0x), as_i64(g.o0y), as_i64(g.o0z), o0);
    view.pick(as_i64(g.o1x), as_i64(g.o1y), as_i64(g.o1z), o1);
    view.pick(as_i64(g.o2x), as_i64(g.o2y), as_i64(g.o2z), o2);
    view.pick(K[0], K[1], K[2], S);
    const fx::StepTol tol = {P.rtol, P.tol_ratio};
    fx::SegScale sc = g.sc;
    sc.pz = P.pz;
    fixed = fx::dop_step(view, ks, sc, o0, o1, o2, as_i64(g.gpa), (fx::u64)P.wturn_m, P.wturn_e, g.x, g.x - g.t0, h,
                         tol, S, Sn, out);
  }
  if (!fixed) {  // rare: on copies, so that g itself stays in registers
    Seg t = g;
    double x = Sx, y = Sy, z = Sz;
    const int r = dop_attempt_slow(t, P, x, y, z);
    g = t;
    Sx = x;
    Sy = y;
    Sz = z;
    return r;
  }
  g.nstep++;
  g.acc = false;
  // step-size controller (clamped to [fac1, fac2]; beta = 0)
  // (comparisons on the integer pipes; fac1 and fac2 are numbers)
  const double raw = P.safe * out.root8;
  double grow = sfp::lt(raw, P.fac1) ? P.fac1 : raw;
  if ((out.accept || P.fixed) && sfp::lt(P.fac2, grow)) grow = P.fac2;
  double hnew = h * grow;
  if (out.accept || P.fixed) {
    g.acc = true;
    g.hu = h;
    fx::i64 N3[3];
    view.gather(Sn, N3);
    // count_turn; y is word 1 - axis, z word 2 - axis, modulo 3
    int y0 = (int)(as_i64(g.ky) >> 32), z0 = (int)(as_i64(g.kz) >> 32), y1 = (int)(N3[1] >> 32), z1 = (int)(N3[2] >> 32);
    if (P.axis != 0) {
      const int x0 = (int)(as_i64(g.kx) >> 32), x1 = (int)(N3[0] >> 32);
      const bool one = P.axis == 1;
      const int u0 = one ? y0 : x0, u1 = one ? y1 : x1;
      y0 = one ? x0 : z0;
      y1 = one ? x1 : z1;
      z0 = u0;
      z1 = u1;
    }
    if ((y0 & y1 & (z0 ^ z1)) < 0) g.turns += z0 < 0 ? -1 : 1;
    g.kx = as_f64(N3[0]);
    g.ky = as_f64(N3[1]);
    g.kz = as_f64(N3[2]);
    g.x = g.x + h;
    if (last) {
      g.h = h;
      g.last = true;
      return 1;
    }
    if (sfp::lt(P.hmax, fabs(hnew))) hnew = g.posneg * P.hmax;
    if (g.reject) hnew = g.posneg * (sfp::lt(fabs(hnew), fabs(h)) ? fabs(hnew) : fabs(h));
    g.reject = false;
  } else {
    g.reject = true;
    last = false;
  }
  g.last = last;
  g.h = P.fixed ? h : hnew;
  return 0;
}

// One attempted DOP853 step on one lane, stage derivatives in local memory.
template <bool FX>
__device__ __forceinline__ int dop_attempt(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz) {
  fx::StageLocal<3> ks;
  return dop_attempt_v<FX>(fx::Lane3(), ks, g, P, Sx, Sy, Sz);
}

// ------------------------------------------------------------ RK45
__device__ __forceinline__ void rk45_begin(Seg& g, double h) {
  g.h = h;
  g.lastH = h;
  g.lnprev = 0.0;  // log(prev_ratio = 1)
  g.kx = g.ky = g.kz = 0.0;  // the stage state a fresh call starts from
  g.nstep = 0;
  g.turns = 0;
  g.last = false;
}

// One attempt of integrateRK45 (src/integrator.cpp:267-335), including its
// first-stage quirk: k1 is evaluated at the previous attempt's last stage
// state (zero on the first attempt of a call).  Returns 0 to continue, 1 when
// the segment end was reached (g.h then holds the carried step), -1 when
// h < hmin, -2 after more than nmax attempts.
__device__ __forceinline__ int rk45_attempt_inl(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz) {
  using namespace rk45;
  g.nstep++;
  if (g.nstep > P.nmax) return -2;
  const double endDt = g.xf - g.x;
  double h = g.h;
  g.lastH = h;
  if (P.fixed) {
    h = P.h0;
  } else {
    if (h > P.hmax)
      h = std_min(h, P.hmax);
    else if (h < P.hmin)
      return -1;
  }
  bool stop;
  if (h >= endDt) {
    h = endDt;
    stop = true;
  } else {
    g.lastH = h;
    stop = false;
  }
  const double tx = g.x - g.t0;
  // stage derivatives scaled by h (k below is h f), as in the DOP853 attempt
  const HPoly hp = hpoly_of(g, h);
  double k1x, k1y, k1z, k2x, k2y, k2z, k3x, k3y, k3z, k4x, k4y, k4z, k5x, k5y, k5z, k6x, k6y, k6z;
  double yx, yy, yz, Ox, Oy, Oz;
  homega_at(hp, g, P, tx, Ox, Oy, Oz);
  bloch(g.kx, g.ky, g.kz, Ox, Oy, Oz, k1x, k1y, k1z);
  yx = fma(B21, k1x, Sx); yy = fma(B21, k1y, Sy); yz = fma(B21, k1z, Sz);
  homega_at(hp, g, P, fma(A2, h, tx), Ox, Oy, Oz);
  bloch(yx, yy, yz, Ox, Oy, Oz, k2x, k2y, k2z);
  yx = fma(B32, k2x, fma(B31, k1x, Sx));
  yy = fma(B32, k2y, fma(B31, k1y, Sy));
  yz = fma(B32, k2z, fma(B31, k1z, Sz));
  homega_at(hp, g, P, fma(A3, h, tx), Ox, Oy, Oz);
  bloch(yx, yy, yz, Ox, Oy, Oz, k3x, k3y, k3z);
  yx = fma(B43, k3x, fma(B42, k2x, fma(B41, k1x, Sx)));
  yy = fma(B43, k3y, fma(B42, k2y, fma(B41, k1y, Sy)));
  yz = fma(B43, k3z, fma(B42, k2z, fma(B41, k1z, Sz)));
  homega_at(hp, g, P, fma(A4, h, tx), Ox, Oy, Oz);
  bloch(yx, yy, yz, Ox, Oy, Oz, k4x, k4y, k4z);
  yx = fma(B54, k4x, fma(B53, k3x, fma(B52, k2x, fma(B51, k1x, Sx))));
  yy = fma(B54, k4y, fma(B53, k3y, fma(B52, k2y, fma(B51, k1y, Sy))));
  yz = fma(B54, k4z, fma(B53, k3z, fma(B52, k2z, fma(B51, k1z, Sz))));
  homega_at(hp, g, P, fma(A5, h, tx), Ox, Oy, Oz);
  bloch(yx, yy, yz, Ox, Oy, Oz, k5x, k5y, k5z);
  yx = fma(B65, k5x, fma(B64, k4x, fma(B63, k3x, fma(B62, k2x, fma(B61, k1x, Sx)))));
  yy = fma(B65, k5y, fma(B64, k4y, fma(B63, k3y, fma(B62, k2y, fma(B61, k1y, Sy)))));
  yz = fma(B65, k5z, fma(B64, k4z, fma(B63, k3z, fma(B62, k2z, fma(B61, k1z, Sz)))));
  homega_at(hp, g, P, fma(A6, h, tx), Ox, Oy, Oz);
  bloch(yx, yy, yz, Ox, Oy, Oz, k6x, k6y, k6z);
  g.kx = yx; g.ky = yy; g.kz = yz;  // the next attempt's first stage sees this state
  // CH2 and CT2 are zero: k2 does not enter the weights; the new state adds
  // the small weighted sum to S in one rounding
  const double wx = fma(CH6, k6x, fma(CH5, k5x, fma(CH4, k4x, fma(CH3, k3x, CH1 * k1x))));
  const double wy = fma(CH6, k6y, fma(CH5, k5y, fma(CH4, k4y, fma(CH3, k3y, CH1 * k1y))));
  const double wz = fma(CH6, k6z, fma(CH5, k5z, fma(CH4, k4z, fma(CH3, k3z, CH1 * k1z))));
  const double tex = fma(CT6, k6x, fma(CT5, k5x, fma(CT4, k4x, fma(CT3, k3x, CT1 * k1x))));
  const double tey = fma(CT6, k6y, fma(CT5, k5y, fma(CT4, k4y, fma(CT3, k3y, CT1 * k1y))));
  const double tez = fma(CT6, k6z, fma(CT5, k5z, fma(CT4, k4z, fma(CT3, k3z, CT1 * k1z))));
  double error = sqrt(fma(tez, tez, fma(tey, tey, tex * tex)));
  error = std_max(error, 1.0e-16);
  const double ratio = P.rtol / error;
  const double lnr = log(ratio);
  double q = exp(E1 * lnr + E2 * g.lnprev);  // ratio^E1 * prev_ratio^E2
  q = std_min(q, 4.0);
  if ((q > 0.81 && error < 2.0 * P.rtol) || P.fixed) {
    const double ny = Sy + wy, nz = Sz + wz;
    g.turns += count_turn(Sy, Sz, ny, nz);
    Sx = Sx + wx; Sy = ny; Sz = nz;
    g.x += h;
    if (stop) {
      g.h = g.lastH;
      return 1;
    }
  }
  g.h = P.fixed ? h : h * q;
  g.lnprev = lnr;
  return 0;
}

// Beside the fixed-point step a call on copies: the caller's segment and spin stay in registers.
static __device__ __noinline__ int rk45_attempt_call(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz) {
  return rk45_attempt_inl(g, P, Sx, Sy, Sz);
}
template <bool FX>
__device__ __forceinline__ int rk45_attempt(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz) {
  if (!FX) return rk45_attempt_inl(g, P, Sx, Sy, Sz);
  Seg t = g;
  double x = Sx, y = Sy, z = Sz;
  const int r = rk45_attempt_call(t, P, x, y, z);
  g = t;
  Sx = x;
  Sy = y;
  Sz = z;
  return r;
}

// ------------------------------------------------------------ integrator types 2-5
// Magnus CFET8 (src/integrator.cpp:625-722), RK45 with quaternions (:441-528),
// RKF45 (:339-439) and RKF45 with quaternions (:530-623).
namespace cfetc {
__device__ __forceinline__ constexpr double x(int i) {
  return i == 0 ? cfet::X1 : i == 1 ? cfet::X2 : i == 2 ? cfet::X3 : i == 3 ? cfet::X4 : cfet::X5;
}
// CFET8 row r (0-5), node j (0-4)
__device__ __forceinline__ constexpr double g(int r, int j) {
  switch (r * 8 + j) {
    case 0: return cfet::G11;  case 1: return cfet::G12;  case 2: return cfet::G13;
    case 3: return cfet::G14;  case 4: return cfet::G15;
    case 8: return cfet::G21;  case 9: return cfet::G22;  case 10: return cfet::G23;
    case 11: return cfet::G24; case 12: return cfet::G25;
    case 16: return cfet::G31; case 17: return cfet::G32; case 18: return cfet::G33;
    case 19: return cfet::G34; case 20: return cfet::G35;
    case 24: return cfet::G41; case 25: return cfet::G42; case 26: return cfet::G43;
    case 27: return cfet::G44; case 28: return cfet::G45;
    case 32: return cfet::G51; case 33: return cfet::G52; case 34: return cfet::G53;
    case 35: return cfet::G54; case 36: return cfet::G55;
    case 40: return cfet::G61; case 41: return cfet::G62; case 42: return cfet::G63;
    case 43: return cfet::G64; default: return cfet::G65;
  }
}
// CFET6 row r (0-2), node j (0-4)
__device__ __forceinline__ constexpr double hh(int r, int j) {
  switch (r * 8 + j) {
    case 0: return cfet::H11;  case 1: return cfet::H12;  case 2: return cfet::H13;
    case 3: return cfet::H14;  case 4: return cfet::H15;
    case 8: return cfet::H21;  case 9: return cfet::H22;  case 10: return cfet::H23;
    case 11: return cfet::H24; case 12: return cfet::H25;
    case 16: return cfet::H31; case 17: return cfet::H32; case 18: return cfet::H33;
    case 19: return cfet::H34; default: return cfet::H35;
  }
}
}  // namespace cfetc

// v rotated by the angle |k| about -k/|k|: Rodrigues' formula
// v cos + (v x k) sin/|k| + k (k.v)(1 - cos)/|k|^2 (rodriguez, src/quaternion.cpp).
// One reciprocal square root gives |k|, 1/|k| and 1/|k|^2 (the reference
// takes a square root and two divisions).
__device__ __forceinline__ void rodrigues(double kx, double ky, double kz, double& vx, double& vy, double& vz) {
  const double a2 = fma(kz, kz, fma(ky, ky, kx * kx));
  const double r = rsqrt(a2);
  const double angle = a2 * r;
  double s, c;
  sincos(angle, &s, &c);
  const double sa = s * r;
  const double d = fma(kz, vz, fma(ky, vy, kx * vx)) * (1.0 - c) * (r * r);
  const double cx = fma(vy, kz, -vz * ky), cy = fma(vz, kx, -vx * kz), cz = fma(vx, ky, -vy * kx);
  vx = fma(kx, d, fma(cx, sa, vx * c));
  vy = fma(ky, d, fma(cy, sa, vy * c));
  vz = fma(kz, d, fma(cz, sa, vz * c));
}

struct Quat {
  double w, x, y, z;
};

// Rotation by the angle |k| dt about -k/|k| as a unit quaternion
// (rodriguezQuat, src/quaternion.cpp).
__device__ __forceinline__ Quat rot_quat(double kx, double ky, double kz, double dt) {
  const double a2 = fma(kz, kz, fma(ky, ky, kx * kx));
  const double r = rsqrt(a2);
  double s, c;
  sincos(a2 * r * dt * 0.5, &s, &c);
  const double f = -s * r;
  return {c, kx * f, ky * f, kz * f};
}

// a b (qMult, src/quaternion.cpp)
__device__ __forceinline__ Quat qmul(const Quat& a, const Quat& b) {
  return {a.w * b.w - a.x * b.x - a.y * b.y - a.z * b.z, a.w * b.x + a.x * b.w + a.y * b.z - a.z * b.y,
          a.w * b.y + a.y * b.w + a.z * b.x - a.x * b.z, a.w * b.z + a.z * b.w + a.x * b.y - a.y * b.x};
}

// q (0, v) q* (qv_mult, src/quaternion.cpp), the terms of the pure
// quaternion's zero real part left out.
__device__ __forceinline__ void qrotate(const Quat& q, double vx, double vy, double vz, double& ox, double& oy,
                                        double& oz) {
  const double tw = -(q.x * vx + q.y * vy + q.z * vz);
  const double tx = q.w * vx + q.y * vz - q.z * vy;
  const double ty = q.w * vy + q.z * vx - q.x * vz;
  const double tz = q.w * vz + q.x * vy - q.y * vx;
  // (tw, tx, ty, tz) (q.w, -q.x, -q.y, -q.z)
  ox = -tw * q.x + tx * q.w - ty * q.z + tz * q.y;
  oy = -tw * q.y + ty * q.w - tz * q.x + tx * q.z;
  oz = -tw * q.z + tz * q.w - tx * q.y + ty * q.x;
}

// The Magnus stepper's 16 exponents in the order they are applied: the
// CFET8 exponents 11 down to 1 (rows 1..5 with the node order reversed, then
// rows 6..1), then the CFET6 exponents 5 down to 1 (rows 1, 2 reversed, then
// rows 3..1); entry [n][j] weights the field at node j.  The stepper reads
// them in a rolled loop, so the rotation code (with its sincos) appears once
// in the kernel instead of 16 times: the unrolled form stalled on
// instruction fetch.
constexpr int magnus_row(int n) { return n < 5 ? n : (n < 11 ? 10 - n : (n < 13 ? n - 11 : 15 - n)); }
constexpr bool magnus_rev(int n) { return n < 5 || n == 11 || n == 12; }
#define ST_MAGNUS_ROW(n)                                                                                      \
  {n < 11 ? cfetc::g(magnus_row(n), magnus_rev(n) ? 4 : 0) : cfetc::hh(magnus_row(n), magnus_rev(n) ? 4 : 0), \
   n < 11 ? cfetc::g(magnus_row(n), magnus_rev(n) ? 3 : 1) : cfetc::hh(magnus_row(n), magnus_rev(n) ? 3 : 1), \
   n < 11 ? cfetc::g(magnus_row(n), 2) : cfetc::hh(magnus_row(n), 2),                                        \
   n < 11 ? cfetc::g(magnus_row(n), magnus_rev(n) ? 1 : 3) : cfetc::hh(magnus_row(n), magnus_rev(n) ? 1 : 3), \
   n < 11 ? cfetc::g(magnus_row(n), magnus_rev(n) ? 0 : 4) : cfetc::hh(magnus_row(n), magnus_rev(n) ? 0 : 4)}
static __constant__ double kMagnusExp[16][5] = {
    ST_MAGNUS_ROW(0),  ST_MAGNUS_ROW(1),  ST_MAGNUS_ROW(2),  ST_MAGNUS_ROW(3),  ST_MAGNUS_ROW(4),  ST_MAGNUS_ROW(5),
    ST_MAGNUS_ROW(6),  ST_MAGNUS_ROW(7),  ST_MAGNUS_ROW(8),  ST_MAGNUS_ROW(9),  ST_MAGNUS_ROW(10), ST_MAGNUS_ROW(11),
    ST_MAGNUS_ROW(12), ST_MAGNUS_ROW(13), ST_MAGNUS_ROW(14), ST_MAGNUS_ROW(15)};
#undef ST_MAGNUS_ROW

// Magnus: the CFET8 product (exponents 11 down to 1, each a combination of h
// times the field at the five Gauss-Legendre nodes) gives the proposal, the
// CFET6 product beside it the error vector.
__device__ __forceinline__ void magnus_stages(const Seg& g, const SetParams& P, double tx, double h, double Sx,
                                              double Sy, double Sz, double w[3], double e[3]) {
  double B[5][3];  // h Omega at the nodes: the exponents are combinations of these
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    omega_at(g, P, fma(cfetc::x(i), h, tx), B[i][0], B[i][1], B[i][2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) B[i][c] *= h;
  }
  double y[3] = {Sx, Sy, Sz}, y8[3];
#pragma unroll 1
  for (int n = 0; n < 16; ++n) {
    if (n == 11) {  // CFET8 done: start CFET6 from S
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        y8[c] = y[c];
        y[c] = c == 0 ? Sx : (c == 1 ? Sy : Sz);
      }
    }
    const double* cf = kMagnusExp[n];
    double k[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double s = cf[0] * B[0][c];
#pragma unroll
      for (int j = 1; j < 5; ++j) s = fma(cf[j], B[j][c], s);
      k[c] = s;
    }
    rodrigues(k[0], k[1], k[2], y[0], y[1], y[2]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    w[c] = y8[c];
    e[c] = y8[c] - y[c];
  }
}

// Per stage m (stages 1, 3, 4, 5, 6; stage 2's weights are zero): node,
// weight of the proposal's rotation, weight of the comparison's (RK45 only).
static __constant__ double kQuatStages[2][5][3] = {
    {{0.0, rk45::CH1, rk45::C1}, {rk45::A3, rk45::CH3, rk45::C3}, {rk45::A4, rk45::CH4, rk45::C4},
     {rk45::A5, rk45::CH5, rk45::C5}, {rk45::A6, rk45::CH6, 0.0}},
    {{0.0, rkf45::C1, 0.0}, {rkf45::A3, rkf45::C3, 0.0}, {rkf45::A4, rkf45::C4, 0.0}, {rkf45::A5, rkf45::C5, 0.0},
     {rkf45::A6, rkf45::C6, 0.0}}};

// RK45 / RKF45 with quaternions: the field at the stages' nodes, each turned
// into a rotation by h times a weight and composed (the first factor onto the
// identity, which is exact); the proposal uses the higher-order weights
// (RK45: CH1..CH6, RKF45: C1..C6), the comparison rotation the first five
// lower-order ones (RK45: C1..C5; RKF45: its own C1..C5, so the two products
// share all but the last factor).  A rolled loop keeps one copy of the
// rotation code in the kernel.
template <bool F>
__device__ __forceinline__ void quat_stages(const Seg& g, const SetParams& P, double tx, double h, double Sx,
                                            double Sy, double Sz, double w[3], double e[3]) {
  Quat qw = {1.0, 0.0, 0.0, 0.0}, qe = {1.0, 0.0, 0.0, 0.0};
#pragma unroll 1
  for (int m = 0; m < 5; ++m) {
    const double* cf = kQuatStages[F ? 1 : 0][m];
    double Ox, Oy, Oz;
    omega_at(g, P, fma(cf[0], h, tx), Ox, Oy, Oz);
    if (F) {
      const Quat r = rot_quat(Ox, Oy, Oz, h * cf[1]);
      if (m < 4)
        qe = qmul(r, qe);
      else
        qw = qmul(r, qe);
    } else {
      qw = qmul(rot_quat(Ox, Oy, Oz, h * cf[1]), qw);
      if (m < 4) qe = qmul(rot_quat(Ox, Oy, Oz, h * cf[2]), qe);
    }
  }
  double cx, cy, cz;
  qrotate(qw, Sx, Sy, Sz, w[0], w[1], w[2]);
  qrotate(qe, Sx, Sy, Sz, cx, cy, cz);
  e[0] = w[0] - cx;
  e[1] = w[1] - cy;
  e[2] = w[2] - cz;
}

// RKF45 with RK45's first-stage quirk (k1 at the previous attempt's last
// stage state, kept in g.k); its error vector is h times the whole
// fourth-order combination, as the reference computes it.
__device__ __forceinline__ void rkf45_stages(Seg& g, const SetParams& P, double tx, double h, double Sx, double Sy,
                                             double Sz, double w[3], double e[3]) {
  using namespace rkf45;
  double k1x, k1y, k1z, k2x, k2y, k2z, k3x, k3y, k3z, k4x, k4y, k4z, k5x, k5y, k5z, k6x, k6y, k6z;
  double yx, yy, yz;
  feval(g, P, tx, g.kx, g.ky, g.kz, k1x, k1y, k1z);
  yx = fma(h * B21, k1x, Sx); yy = fma(h * B21, k1y, Sy); yz = fma(h * B21, k1z, Sz);
  feval(g, P, fma(A2, h, tx), yx, yy, yz, k2x, k2y, k2z);
  yx = fma(h, fma(B32, k2x, B31 * k1x), Sx);
  yy = fma(h, fma(B32, k2y, B31 * k1y), Sy);
  yz = fma(h, fma(B32, k2z, B31 * k1z), Sz);
  feval(g, P, fma(A3, h, tx), yx, yy, yz, k3x, k3y, k3z);
  yx = fma(h, fma(B43, k3x, fma(B42, k2x, B41 * k1x)), Sx);
  yy = fma(h, fma(B43, k3y, fma(B42, k2y, B41 * k1y)), Sy);
  yz = fma(h, fma(B43, k3z, fma(B42, k2z, B41 * k1z)), Sz);
  feval(g, P, fma(A4, h, tx), yx, yy, yz, k4x, k4y, k4z);
  yx = fma(h, fma(B54, k4x, fma(B53, k3x, fma(B52, k2x, B51 * k1x))), Sx);
  yy = fma(h, fma(B54, k4y, fma(B53, k3y, fma(B52, k2y, B51 * k1y))), Sy);
  yz = fma(h, fma(B54, k4z, fma(B53, k3z, fma(B52, k2z, B51 * k1z))), Sz);
  feval(g, P, fma(A5, h, tx), yx, yy, yz, k5x, k5y, k5z);
  yx = fma(h, fma(B65, k5x, fma(B64, k4x, fma(B63, k3x, fma(B62, k2x, B61 * k1x)))), Sx);
  yy = fma(h, fma(B65, k5y, fma(B64, k4y, fma(B63, k3y, fma(B62, k2y, B61 * k1y)))), Sy);
  yz = fma(h, fma(B65, k5z, fma(B64, k4z, fma(B63, k3z, fma(B62, k2z, B61 * k1z)))), Sz);
  feval(g, P, fma(A6, h, tx), yx, yy, yz, k6x, k6y, k6z);
  g.kx = yx; g.ky = yy; g.kz = yz;
  w[0] = fma(h, fma(C6, k6x, fma(C5, k5x, fma(C4, k4x, fma(C3, k3x, C1 * k1x)))), Sx);
  w[1] = fma(h, fma(C6, k6y, fma(C5, k5y, fma(C4, k4y, fma(C3, k3y, C1 * k1y)))), Sy);
  w[2] = fma(h, fma(C6, k6z, fma(C5, k5z, fma(C4, k4z, fma(C3, k3z, C1 * k1z)))), Sz);
  e[0] = h * fma(CR5, k5x, fma(CR4, k4x, fma(CR3, k3x, CR1 * k1x)));
  e[1] = h * fma(CR5, k5y, fma(CR4, k4y, fma(CR3, k3y, CR1 * k1y)));
  e[2] = h * fma(CR5, k5z, fma(CR4, k4z, fma(CR3, k3z, CR1 * k1z)));
}

// The same in FP64 for a segment that may be in fixed point; a call, not inlined: the
// fixed-point step takes all but a few.
static __device__ __noinline__ void quat_slow(const Seg& g, const SetParams& P, double tx, double h, double Sx, double Sy,
                                                  double Sz, double w[3], double e[3]) {
  Seg t = g;
  if (t.fx) seg_unscale(t, P);
  if (P.integrator == 3)
    quat_stages<false>(t, P, tx, h, Sx, Sy, Sz, w, e);
  else
    quat_stages<true>(t, P, tx, h, Sx, Sy, Sz, w, e);
}

// The proposal and error vector of a quaternion step: in fixed point where it fits.  In FP64 an
// attempt of the quaternion RKF45 takes 700 FP64 instructions of 76 cycles: RK45, RKF45 and both
// quaternion forms, 4,096 particles each, 92 ms, 44 with the quaternion forms in fixed point.
// (The Magnus stepper stays in FP64: its error estimate is rounding noise on smooth fields, so
// its steps of a radian and more, and the turns counted at their ends, hang on the noise's bits.)
template <bool FX>
__device__ __forceinline__ void quat_step(const Seg& g, const SetParams& P, double tx, double h, double Sx, double Sy,
                                              double Sz, double w[3], double e[3]) {
  if (!FX) {
    if (P.integrator == 3)
      quat_stages<false>(g, P, tx, h, Sx, Sy, Sz, w, e);
    else
      quat_stages<true>(g, P, tx, h, Sx, Sy, Sz, w, e);
    return;
  }
  if (g.fx) {
    double S[3] = {Sx, Sy, Sz};
    turn_by(S[0], S[1], S[2], P.axis);
    const fx::i64 o0[3] = {as_i64(g.o0x), as_i64(g.o0y), as_i64(g.o0z)};
    const fx::i64 o1[3] = {as_i64(g.o1x), as_i64(g.o1y), as_i64(g.o1z)};
    const fx::i64 o2[3] = {as_i64(g.o2x), as_i64(g.o2y), as_i64(g.o2z)};
    fx::SegScale sc = g.sc;
    sc.pz = P.pz;
    if (fx::spin_scale(S, sc.se)) {
      fx::i64 q[3], y[3], d[3];
      sc.sk = fx::spin_grade(S, sc.se, sc.ok);
      fx::spin_words(S, sc.se, sc.sk, q);
      const fx::i64 ga = as_i64(g.gpa);
      const bool ok = P.integrator == 3 ? fx::quat_step<false>(sc, o0, o1, o2, ga, P.wturn_m, P.wturn_e, g.x, tx, h, q, y, d)
                                        : fx::quat_step<true>(sc, o0, o1, o2, ga, P.wturn_m, P.wturn_e, g.x, tx, h, q, y, d);
      if (ok) {
        const fx::Grade k{sc.sk};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int E = sc.se - (c == 0 ? k.e0() : k.e1());
          w[c] = fx::from_q63(y[c], E);
          e[c] = fx::from_q63(d[c], E);
        }
        unturn(w[0], w[1], w[2], P.axis);
        unturn(e[0], e[1], e[2], P.axis);
        return;
      }
    }
  }
  const Seg t = g;  // (their addresses go to the call: g, w and e stay in registers)
  double ws[3], es[3];
  quat_slow(t, P, tx, h, Sx, Sy, Sz, ws, es);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    w[c] = ws[c];
    e[c] = es[c];
  }
}

// Start a type 2-5 call over the segment: the same state as RK45's.
__device__ __forceinline__ void ext_begin(Seg& g, double h) { rk45_begin(g, h); }

// One attempt of integrator type 2-5 (P.integrator).  Their shared step
// controller differs from RK45's: the segment end is tested before the hmax
// and hmin limits, and a fixed step never looks at the segment end (such a
// segment ends after nmax attempts, -2).  Returns 0 to continue, 1 at the
// segment end (g.h then holds the carried step), -1 when h < hmin, -2 after
// more than nmax attempts.
template <bool FX>
__device__ __forceinline__ int ext_attempt(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz) {
  g.nstep++;
  if (g.nstep > P.nmax) return -2;
  g.acc = false;
  const double endDt = g.xf - g.x;
  double h = g.h;
  g.lastH = h;
  bool stop = false;
  if (P.fixed) {
    h = P.h0;
  } else if (h >= endDt) {
    h = endDt;
    stop = true;
  } else if (h > P.hmax) {
    h = std_min(h, P.hmax);
  } else if (h < P.hmin) {
    return -1;
  }
  const double tx = g.x - g.t0;
  double w[3], e[3];
  if (P.integrator == 2)
    magnus_stages(g, P, tx, h, Sx, Sy, Sz, w, e);
  else if (P.integrator != 4)
    quat_step<FX>(g, P, tx, h, Sx, Sy, Sz, w, e);
  else
    rkf45_stages(g, P, tx, h, Sx, Sy, Sz, w, e);
  double error = sfp::sqrt_rn(fma(e[2], e[2], fma(e[1], e[1], e[0] * e[0])));
  error = std_max(error, 1.0e-16);
  const double ratio = sfp::div_rn(P.rtol, error);
  const double lnr = log(ratio);
  double q = exp(rk45::E1 * lnr + rk45::E2 * g.lnprev);  // ratio^E1 * prev_ratio^E2
  q = std_min(q, 4.0);
  if ((q > 0.81 && error < 2.0 * P.rtol) || P.fixed) {
    g.acc = true;  // read by the adjoint's tape writer
    g.hu = h;
    g.turns += count_turn(Sy, Sz, w[1], w[2]);
    Sx = w[0]; Sy = w[1]; Sz = w[2];
    g.x += h;
    if (stop) {
      g.h = g.lastH;
      return 1;
    }
  }
  g.h = P.fixed ? h : h * q;
  g.lnprev = lnr;
  return 0;
}

}  // namespace st
