// Host build of the fixed-point DOP853 step (spin-tracking_gb300/csrc/
// st_fixed.cuh) for tests: one step from seeded random segments against the
// same step in binary128, beside the FP64 form of the step (fused
// multiply-adds, as the device's FP64 path).  Arguments: count, seed, kind
// (0 static field, 1 strongly varying field, 2 pulse), rotation angle of the
// step, rtol, spin norm.  Prints the number of steps taken in fixed point and
// refused, the largest spin error of either form (relative to the norm), the
// largest relative error of err^(-1/8) of either form over steps whose err is not
// far below the clamp of the controller, and the accept decisions that differ
// from binary128's by more than its rounding.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <vector>

#if defined(__LDBL_MANT_DIG__) && __LDBL_MANT_DIG__ == 113
typedef long double quad;
static quad q_cos(quad x) { return cosl(x); }
static quad q_sqrt(quad x) { return sqrtl(x); }
static quad q_pow(quad x, quad y) { return powl(x, y); }
static quad q_frexp(quad x, int* e) { return frexpl(x, e); }
static const quad kPi = acosl(-1.0L);
#else
#include <quadmath.h>
typedef __float128 quad;
static quad q_cos(quad x) { return cosq(x); }
static quad q_sqrt(quad x) { return sqrtq(x); }
static quad q_pow(quad x, quad y) { return powq(x, y); }
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
static double root(double x) { return std::sqrt(x); }
static quad root(quad x) { return q_sqrt(x); }

struct Case {
  double o0[3], o1[3], o2[3], ga, w, t0, tx, h, S[3], rtol;
};

// One DOP853 step in arithmetic R: the new spin and err.
template <class R>
static R step(const Case& q, R Sn[3]) {
  static const double B[13] = {0, dop::B1, 0, 0, 0, 0, dop::B6, dop::B7, dop::B8, dop::B9, dop::B10, dop::B11, dop::B12};
  static const double E[13] = {0, dop::ER1, 0, 0, 0, 0, dop::ER6, dop::ER7, dop::ER8, dop::ER9, dop::ER10, dop::ER11,
                               dop::ER12};
  R k[13][3];
  for (int s = 1; s <= 12; ++s) {
    R Y[3], O[3];
    for (int c = 0; c < 3; ++c) {
      R a = q.S[c];
      for (int j = 0; j < dopst::cnt(s); ++j) a = mad((R)dopst::a(s, j), k[dopst::src(s, j)][c], a);
      Y[c] = a;
      const R tau = mad((R)(s == 1 ? 0.0 : dopst::c(s)), (R)q.h, (R)q.tx);
      R o = mad(mad((R)q.o2[c], tau, (R)q.o1[c]), tau, (R)q.o0[c]);
      if (c == 2 && q.ga != 0.0) o = o + (R)q.ga * cosine((R)q.w * ((R)q.t0 + tau));
      O[c] = o * (R)q.h;
    }
    for (int c = 0; c < 3; ++c) {
      const int a = (c + 1) % 3, b = (c + 2) % 3;
      k[s][c] = mad(Y[a], O[b], -(Y[b] * O[a]));
    }
  }
  R n5 = 0, n3 = 0;
  for (int c = 0; c < 3; ++c) {
    R b = 0, e = 0;
    for (int s = 1; s <= 12; ++s) {
      b = mad((R)B[s], k[s][c], b);
      e = mad((R)E[s], k[s][c], e);
    }
    Sn[c] = (R)q.S[c] + b;
    const R e3 = b - (R)dop::BHH1 * k[1][c] - (R)dop::BHH2 * k[9][c] - (R)dop::BHH3 * k[12][c];
    const R m = (R)std::fabs(q.S[c]), n = Sn[c] < 0 ? -Sn[c] : Sn[c];
    const R sk = (R)q.rtol + (R)q.rtol * (m > n ? m : n);
    n5 += e / sk * (e / sk);
    n3 += e3 / sk * (e3 / sk);
  }
  return n5 / root((n5 + (R)0.01 * n3) * (R)3);
}

static double median(std::vector<double> v) {
  if (v.empty()) return 0.0;
  std::nth_element(v.begin(), v.begin() + v.size() / 2, v.end());
  return v[v.size() / 2];
}

int main(int argc, char** argv) {
  const long n = std::atol(argv[1]);
  g_state = std::strtoull(argv[2], nullptr, 10) * 2 + 1;
  const int kind = std::atoi(argv[3]);
  const double angle = std::atof(argv[4]), rtol = std::atof(argv[5]), norm = std::atof(argv[6]);
  for (int k = 0; k < 8; ++k) uniform();
  long taken = 0, refused = 0, wrong = 0;
  double sf = 0, sd = 0;
  std::vector<double> rf, rd;
  for (long it = 0; it < n; ++it) {
    Case q{};
    q.rtol = rtol;
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
    const double T = 7e-4 * (0.1 + uniform());
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
    i64 o0[3], o1[3], o2[3], S[3], Sn[3];
    for (int c = 0; c < 3; ++c) {
      o0[c] = to_q63(q.o0[c], sc.oe);
      o1[c] = to_q63(q.o1[c], sc.oe - sc.te);
      o2[c] = to_q63(q.o2[c], sc.oe - 2 * sc.te);
      S[c] = to_q63(q.S[c], sc.se);
    }
    u64 wm = 0;
    int we = 0;
    if (q.w != 0.0) wm = (u64)(q_frexp((quad)q.w / (2 * kPi), &we) * (quad)18446744073709551616.0);
    StageLocal<3> ks;
    StepOut out;
    if (!dop_step(Lane3(), ks, sc, o0, o1, o2, to_q63(q.ga, sc.oe), wm, we, x, q.tx, q.h, StepTol{rtol, 1.0}, S, Sn,
                  out)) {
      ++refused;
      continue;
    }
    ++taken;
    quad Sq[3];
    double Sd[3];
    const quad eq = step<quad>(q, Sq);
    const double ed = step<double>(q, Sd);
    for (int c = 0; c < 3; ++c) {
      const double ef = std::fabs((double)((quad)from_q63(Sn[c], 0) * (quad)std::ldexp(1.0, sc.se) - Sq[c])) / norm;
      // from_q63 rounds to a double: measure the word itself
      const quad word = (quad)(double)(Sn[c] >> 32) * 4294967296.0 + (quad)(double)(uint32_t)Sn[c];
      const double e = std::fabs((double)(word * (quad)std::ldexp(1.0, sc.se - 63) - Sq[c])) / norm;
      if (e > sf) sf = e;
      if (ef > e + 0x1p-53) ++wrong;
      const double d = std::fabs((double)((quad)Sd[c] - Sq[c])) / norm;
      if (d > sd) sd = d;
    }
    if ((double)eq < 2e-7) {  // 0.9 err^(-1/8) is above the largest growth factor 6
      wrong += 0.9 * out.root8 < 6.0 || !out.accept;
      continue;
    }
    const quad rq = q_pow(eq, (quad)-0.125);
    const double ef = std::fabs((double)((quad)out.root8 / rq - 1)), edd = std::fabs((double)(q_pow((quad)ed, (quad)-0.125) / rq - 1));
    rf.push_back(ef);
    rd.push_back(edd);
    if (std::fabs((double)eq - 1.0) > 1e-3) wrong += out.accept != (eq <= 1);
  }
  std::printf("taken %ld refused %ld wrong %ld judged %ld spin_fixed %.4g spin_fp64 %.4g root8_fixed %.4g root8_fp64 %.4g\n", taken, refused,
              wrong, (long)rf.size(), sf, sd, median(rf), median(rd));
  return 0;
}
