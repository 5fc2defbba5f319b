// Host build of the fixed-point quaternion steps (spin-tracking_gb300/csrc/
// st_fixed.cuh) for tests: one RK45 or RKF45 step with quaternions from seeded random
// segments against the same step in binary128, beside the FP64 form of the step (a product
// of unit quaternions).  Arguments: count, seed, kind (0 static field, 1 strongly varying field, 2
// pulse), rotation angle of the step, spin norm, stepper (0 RK45, 1 RKF45).  Prints the number of steps taken
// in fixed point and refused, and the largest errors of either form's spin and
// error vector, relative to the norm.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#if defined(__LDBL_MANT_DIG__) && __LDBL_MANT_DIG__ == 113
typedef long double quad;
static quad q_cos(quad x) { return cosl(x); }
static quad q_sqrt(quad x) { return sqrtl(x); }
static quad q_sin(quad x) { return sinl(x); }
static quad q_frexp(quad x, int* e) { return frexpl(x, e); }
static const quad kPi = acosl(-1.0L);
#else
#include <quadmath.h>
typedef __float128 quad;
static quad q_cos(quad x) { return cosq(x); }
static quad q_sqrt(quad x) { return sqrtq(x); }
static quad q_sin(quad x) { return sinq(x); }
static quad q_frexp(quad x, int* e) { return frexpq(x, e); }
static const quad kPi = acosq(-1);
#endif

#define __device__
#define __constant__ const
#define __forceinline__ inline
#include "st_fixed.cuh"

using namespace st;
using namespace st::fx;

static uint64_t g_state = 0x9E3779B97F4A7C15ull;
static double uniform() {
  g_state ^= g_state >> 12;
  g_state ^= g_state << 25;
  g_state ^= g_state >> 27;
  return (double)((g_state * 0x2545F4914F6CDD1Dull) >> 11) * 0x1p-53;
}


static double mad(double a, double b, double c) { return std::fma(a, b, c); }
static quad mad(quad a, quad b, quad c) { return a * b + c; }
static double cosine(double x) { return std::cos(x); }
static quad cosine(quad x) { return q_cos(x); }
static double sine(double x) { return std::sin(x); }
static quad sine(quad x) { return q_sin(x); }
static double root(double x) { return std::sqrt(x); }
static quad root(quad x) { return q_sqrt(x); }

struct Case {
  double o0[3], o1[3], o2[3], ga, w, t0, tx, h, S[3];
};

template <class R>
struct Quat {
  R w, x, y, z;
};
template <class R>
static Quat<R> mul(const Quat<R>& a, const Quat<R>& b) {
  return {a.w * b.w - a.x * b.x - a.y * b.y - a.z * b.z, a.w * b.x + a.x * b.w + a.y * b.z - a.z * b.y,
          a.w * b.y + a.y * b.w + a.z * b.x - a.x * b.z, a.w * b.z + a.z * b.w + a.x * b.y - a.y * b.x};
}
template <class R>
static void turn(const Quat<R>& q, const double S[3], R o[3]) {
  const Quat<R> v{0, (R)S[0], (R)S[1], (R)S[2]}, p = mul(mul(q, v), Quat<R>{q.w, -q.x, -q.y, -q.z});
  o[0] = p.x;
  o[1] = p.y;
  o[2] = p.z;
}

static const double kStages[2][5][3] = {
    {{0.0, rk45::CH1, rk45::C1}, {rk45::A3, rk45::CH3, rk45::C3}, {rk45::A4, rk45::CH4, rk45::C4},
     {rk45::A5, rk45::CH5, rk45::C5}, {rk45::A6, rk45::CH6, 0.0}},
    {{0.0, rkf45::C1, rkf45::C1}, {rkf45::A3, rkf45::C3, rkf45::C3}, {rkf45::A4, rkf45::C4, rkf45::C4},
     {rkf45::A5, rkf45::C5, rkf45::C5}, {rkf45::A6, rkf45::C6, 0.0}}};
static int g_stepper = 0;

// One step in arithmetic R: the proposal and its difference from the comparison.
template <class R>
static void step(const Case& q, R w[3], R e[3]) {
  Quat<R> p[2] = {{1, 0, 0, 0}, {1, 0, 0, 0}};
  for (int m = 0; m < 5; ++m) {
    const double* cf = kStages[g_stepper][m];
    R B[3];
    const R tau = mad((R)cf[0], (R)q.h, (R)q.tx);
    for (int c = 0; c < 3; ++c) {
      B[c] = mad(mad((R)q.o2[c], tau, (R)q.o1[c]), tau, (R)q.o0[c]);
      if (c == 2 && q.ga != 0.0) B[c] = B[c] + (R)q.ga * cosine((R)q.w * ((R)q.t0 + tau));
    }
    const R a = root(mad(B[2], B[2], mad(B[1], B[1], B[0] * B[0])));
    for (int j = 0; j < (m < 4 ? 2 : 1); ++j) {
      const R half = a * (R)q.h * (R)cf[1 + j] * (R)0.5, s = -sine(half) / a;
      p[j] = mul(Quat<R>{cosine(half), B[0] * s, B[1] * s, B[2] * s}, p[j]);
    }
  }
  R y[3];
  turn(p[0], q.S, w);
  turn(p[1], q.S, y);
  for (int c = 0; c < 3; ++c) e[c] = w[c] - y[c];
}

static quad word(i64 m, int E) {  // m 2^(E - 63), exactly
  return ((quad)(double)(m >> 32) * 4294967296.0 + (quad)(double)(uint32_t)m) * (quad)std::ldexp(1.0, E - 63);
}

int main(int argc, char** argv) {
  if (argc < 7) return 1;
  const long n = std::atol(argv[1]);
  g_state = std::strtoull(argv[2], nullptr, 10) * 2 + 1;
  const int kind = std::atoi(argv[3]);
  const double angle = std::atof(argv[4]), norm = std::atof(argv[5]);
  g_stepper = std::atoi(argv[6]);
  for (int k = 0; k < 8; ++k) uniform();
  long taken = 0, refused = 0;
  double sf = 0, sd = 0, ef = 0, ed = 0;
  for (long it = 0; it < n; ++it) {
    Case q{};
    for (int c = 0; c < 3; ++c) {
      const double a = kind == 1 ? 1000.0 : 1e-2, b = kind == 1 ? 1e5 : 0.1, d = kind == 1 ? 1e7 : 0.1;
      q.o0[c] = (uniform() - 0.5) * a;
      q.o1[c] = (uniform() - 0.5) * b;
      q.o2[c] = (uniform() - 0.5) * d;
    }
    if (kind != 1) q.o0[0] = -611.4;
    if (kind == 2) {
      q.ga = -2.038e8 * 5e-6;
      q.w = 6283.185307179586;
    }
    const double T = (angle > 0.4 ? 1e-2 : 7e-4) * (0.1 + uniform());
    const double O = std::sqrt(q.o0[0] * q.o0[0] + q.o0[1] * q.o0[1] + q.o0[2] * q.o0[2]) + std::fabs(q.ga);
    q.t0 = uniform();
    q.h = angle / O * (0.5 + uniform());
    if (q.h > T) q.h = T * uniform();
    const double x = q.t0 + (T - q.h) * uniform();
    q.tx = x - q.t0;
    const double z = 2.0 * uniform() - 1.0, f = 2.0 * M_PI * uniform();
    q.S[0] = norm * z;
    q.S[1] = norm * std::sqrt(1.0 - z * z) * std::cos(f);
    q.S[2] = norm * std::sqrt(1.0 - z * z) * std::sin(f);
    SegScale sc;
    if (!spin_scale(q.S, sc.se) || !field_scale(q.o0, q.o1, q.o2, q.ga, T, sc)) {
      ++refused;
      continue;
    }
    i64 o0[3], o1[3], o2[3], S[3], y8[3], e[3];
    for (int c = 0; c < 3; ++c) {
      o0[c] = to_q63(q.o0[c], sc.oe);
      o1[c] = to_q63(q.o1[c], sc.oe - sc.te);
      o2[c] = to_q63(q.o2[c], sc.oe - 2 * sc.te);
      S[c] = to_q63(q.S[c], sc.se);
    }
    u64 wm = 0;
    int we = 0;
    if (q.w != 0.0) wm = (u64)(q_frexp((quad)q.w / (2 * kPi), &we) * (quad)18446744073709551616.0);
    const i64 ga = to_q63(q.ga, sc.oe);
    if (!(g_stepper ? quat_step<true>(sc, o0, o1, o2, ga, wm, we, x, q.tx, q.h, S, y8, e)
                    : quat_step<false>(sc, o0, o1, o2, ga, wm, we, x, q.tx, q.h, S, y8, e))) {
      ++refused;
      continue;
    }
    ++taken;
    quad wq[3], eq[3];
    double wd[3], eD[3];
    step<quad>(q, wq, eq);
    step<double>(q, wd, eD);
    for (int c = 0; c < 3; ++c) {
      sf = std::fmax(sf, std::fabs((double)(word(y8[c], sc.se) - wq[c])) / norm);
      sd = std::fmax(sd, std::fabs((double)((quad)wd[c] - wq[c])) / norm);
      ef = std::fmax(ef, std::fabs((double)(word(e[c], sc.se) - eq[c])) / norm);
      ed = std::fmax(ed, std::fabs((double)((quad)eD[c] - eq[c])) / norm);
    }
  }
  std::printf("taken %ld refused %ld spin_fixed %.4g spin_fp64 %.4g err_fixed %.4g err_fp64 %.4g\n", taken, refused, sf, sd, ef, ed);
  return 0;
}
