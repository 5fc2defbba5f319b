// Host build of the fixed-point DOP853 step adjoint (spin-tracking_gb300/csrc/
// st_fixed.cuh) for tests: the backward pass through one step from seeded random
// segments against the same in binary128, beside its FP64 form.  Arguments:
// count, seed, kind (0 static field, 1 strongly varying field, 2 pulse), rotation
// angle of the step, norm of the spin and of the adjoint.  Prints the steps taken in
// fixed point and refused, and the largest errors of either form's adjoint (relative
// to its norm) and gradient moments (relative to the norms' product).
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

// One step back in arithmetic R: the adjoint lam and the moments sum z, sum c z, sum c^2 z over the
// stages, and with a pulse the sums of cos z_z, sin z_z, c sin z_z.
template <class R>
static void back(const Case& q, const double l[3], R lam[3], R M[12]) {
  R k[13][3], Y[13][3], O[13][3], kh[13][3];
  for (int s = 1; s <= 12; ++s) {
    for (int c = 0; c < 3; ++c) {
      R a = q.S[c];
      for (int j = 0; j < dopst::cnt(s); ++j) a = mad((R)dopst::a(s, j), k[dopst::src(s, j)][c], a);
      Y[s][c] = a;
      const R tau = mad((R)(s == 1 ? 0.0 : dopst::c(s)), (R)q.h, (R)q.tx);
      R o = mad(mad((R)q.o2[c], tau, (R)q.o1[c]), tau, (R)q.o0[c]);
      if (c == 2 && q.ga != 0.0) o = o + (R)q.ga * cosine((R)q.w * ((R)q.t0 + tau));
      O[s][c] = o * (R)q.h;
    }
    for (int c = 0; c < 3; ++c) {
      const int a = (c + 1) % 3, b = (c + 2) % 3;
      k[s][c] = mad(Y[s][a], O[s][b], -(Y[s][b] * O[s][a]));
    }
  }
  for (int s = 1; s <= 12; ++s)
    for (int c = 0; c < 3; ++c) kh[s][c] = (R)dopst::b(s) * (R)l[c];
  for (int c = 0; c < 3; ++c) lam[c] = l[c];
  for (int j = 0; j < 12; ++j) M[j] = 0;
  for (int s = 12; s >= 1; --s) {
    const R cs = s == 1 ? 0.0 : dopst::c(s), ph = (R)q.w * ((R)q.t0 + mad(cs, (R)q.h, (R)q.tx));
    R yb[3], z[3];
    for (int c = 0; c < 3; ++c) {
      const int a = (c + 1) % 3, b = (c + 2) % 3;
      yb[c] = mad(O[s][a], kh[s][b], -(O[s][b] * kh[s][a]));
      z[c] = mad(kh[s][a], Y[s][b], -(kh[s][b] * Y[s][a]));
      lam[c] += yb[c];
      M[c] += z[c];
      M[3 + c] = mad(cs, z[c], M[3 + c]);
      M[6 + c] = mad(cs * cs, z[c], M[6 + c]);
    }
    if (q.ga != 0.0) {
      const R sn = sine(ph);
      M[9] = mad(cosine(ph), z[2], M[9]);
      M[10] = mad(sn, z[2], M[10]);
      M[11] = mad(cs * sn, z[2], M[11]);
    }
    for (int j = 0; j < dopst::cnt(s); ++j)
      for (int c = 0; c < 3; ++c) kh[dopst::src(s, j)][c] = mad((R)dopst::a(s, j), yb[c], kh[dopst::src(s, j)][c]);
  }
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
  double lf = 0, ld = 0, mf = 0, md = 0;
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
    i64 o0[3], o1[3], o2[3], S[3];
    for (int c = 0; c < 3; ++c) {
      o0[c] = to_q63(q.o0[c], sc.oe);
      o1[c] = to_q63(q.o1[c], sc.oe - sc.te);
      o2[c] = to_q63(q.o2[c], sc.oe - 2 * sc.te);
      S[c] = to_q63(q.S[c], sc.se);
    }
    u64 wm = 0;
    int we = 0;
    if (q.w != 0.0) wm = (u64)(q_frexp((quad)q.w / (2 * kPi), &we) * (quad)18446744073709551616.0);
    double l[3];
    const double lz = 2.0 * uniform() - 1.0, lg = 2.0 * M_PI * uniform();
    l[0] = norm * std::sqrt(1.0 - lz * lz) * std::cos(lg);
    l[1] = norm * lz;
    l[2] = norm * std::sqrt(1.0 - lz * lz) * std::sin(lg);
    int le;
    if (!spin_scale(l, le)) return 1;
    i64 lam[3];
    for (int c = 0; c < 3; ++c) lam[c] = to_q63(l[c], le);
    StageLocal<3> ks, ys;
    AdjMoments m;
    if (!dop_adjoint(ks, ys, sc, o0, o1, o2, to_q63(q.ga, sc.oe), wm, we, x, q.tx, q.h, kind == 2, S, lam, m)) {
      ++refused;
      continue;
    }
    ++taken;
    quad lq[3], Mq[12];
    double lD[3], MD[12];
    back<quad>(q, l, lq, Mq);
    back<double>(q, l, lD, MD);
    const i64 Mf[12] = {m.z0[0], m.z0[1], m.z0[2], m.z1[0], m.z1[1], m.z1[2], m.z2[0], m.z2[1], m.z2[2], m.cz, m.sz, m.scz};
    for (int c = 0; c < 3; ++c) {
      lf = std::fmax(lf, std::fabs((double)(word(lam[c], le) - lq[c])) / norm);
      ld = std::fmax(ld, std::fabs((double)((quad)lD[c] - lq[c])) / norm);
    }
    for (int j = 0; j < 12; ++j) {
      mf = std::fmax(mf, std::fabs((double)(word(Mf[j], sc.se + le + m.exp + (j >= 9)) - Mq[j])) / (norm * norm));
      md = std::fmax(md, std::fabs((double)((quad)MD[j] - Mq[j])) / (norm * norm));
    }
  }
  std::printf("taken %ld refused %ld lam_fixed %.4g lam_fp64 %.4g mom_fixed %.4g mom_fp64 %.4g\n", taken, refused, lf, ld, mf, md);
  return 0;
}
