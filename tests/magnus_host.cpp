// Host build of the fixed-point Magnus step (spin-tracking_gb300/csrc/
// st_fixed.cuh) for tests: one CFET8 / CFET6 step from seeded random segments
// against the same step in binary128, beside the FP64 form of the step.
// Arguments: count, seed, kind (0 static field, 1 strongly varying field, 2
// pulse), rotation angle of the step, spin norm.  Prints the number of steps taken
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

// One step in arithmetic R: the proposal and its difference from the companion's.
template <class R>
static void step(const Case& q, R w[3], R e[3]) {
  R B[5][3], y[3] = {(R)q.S[0], (R)q.S[1], (R)q.S[2]};
  for (int i = 0; i < 5; ++i)
    for (int c = 0; c < 3; ++c) {
      const R tau = mad((R)cfx::x[i], (R)q.h, (R)q.tx);
      R o = mad(mad((R)q.o2[c], tau, (R)q.o1[c]), tau, (R)q.o0[c]);
      if (c == 2 && q.ga != 0.0) o = o + (R)q.ga * cosine((R)q.w * ((R)q.t0 + tau));
      B[i][c] = o * (R)q.h;
    }
  for (int n = 0; n < 16; ++n) {
    if (n == 11)
      for (int c = 0; c < 3; ++c) {
        w[c] = y[c];
        y[c] = (R)q.S[c];
      }
    R k[3], x[3];
    for (int c = 0; c < 3; ++c) {
      k[c] = 0;
      for (int j = 0; j < 5; ++j) k[c] = mad((R)cfx::weight(n, j), B[j][c], k[c]);
    }
    const R a2 = mad(k[2], k[2], mad(k[1], k[1], k[0] * k[0])), a = root(a2), s = sine(a) / a, c1 = cosine(a);
    const R d = mad(k[2], y[2], mad(k[1], y[1], k[0] * y[0])) * ((R)1 - c1) / a2;
    for (int c = 0; c < 3; ++c) x[c] = mad(y[(c + 1) % 3], k[(c + 2) % 3], -(y[(c + 2) % 3] * k[(c + 1) % 3]));
    for (int c = 0; c < 3; ++c) y[c] = mad(k[c], d, mad(x[c], s, y[c] * c1));
  }
  for (int c = 0; c < 3; ++c) e[c] = w[c] - y[c];
}

static quad word(i64 m, int E) {  // m 2^(E - 63), exactly
  return ((quad)(double)(m >> 32) * 4294967296.0 + (quad)(double)(uint32_t)m) * (quad)std::ldexp(1.0, E - 63);
}

int main(int argc, char** argv) {
  if (argc < 6) return 1;
  const long n = std::atol(argv[1]);
  g_state = std::strtoull(argv[2], nullptr, 10) * 2 + 1;
  const int kind = std::atoi(argv[3]);
  const double angle = std::atof(argv[4]), norm = std::atof(argv[5]);
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
    if (!magnus_step(sc, o0, o1, o2, to_q63(q.ga, sc.oe), wm, we, x, q.tx, q.h, S, y8, e)) {
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
