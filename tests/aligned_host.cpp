// Host build of the fixed-point steps (spin-tracking_gb300/csrc/st_fixed.cuh) for tests where
// the field lies along one axis and spin and adjoint along it or across it, but for a small part:
// each component's largest error against binary128, beside that of the step's FP64 form on the
// same inputs.  The steps' other forms are those of the three programs included.  Arguments:
// form (0 DOP853, 1 its adjoint, 2 RK45 and 3 RKF45 with quaternions), count, seed, geometry of
// the spin (0 any direction, 1 along, 2 across), of the adjoint, the small part, rotation angle,
// axis, pulse (0, 1), field (rad/s, 611.4 unless given).  Prints the steps taken and refused, then component by component the
// error in fixed point and in FP64.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>
#if !(defined(__LDBL_MANT_DIG__) && __LDBL_MANT_DIG__ == 113)
#include <quadmath.h>
#endif
#define __device__
#define __constant__ const
#define __forceinline__ inline
#include "st_fixed.cuh"

namespace host_dop {
#define main unused_main
#include "fixed_host.cpp"
}
namespace host_adj {
#include "adjoint_host.cpp"
}
namespace host_quat {
#include "quat_host.cpp"
#undef main
}

using namespace st::fx;
using host_adj::quad;
using host_adj::word;

static double uniform() { return host_adj::uniform(); }

// A vector of the norm: any direction, along the axis or across it but for `small`.
static void draw(int geometry, double small, int axis, double norm, double v[3]) {
  const double z = 2.0 * uniform() - 1.0, f = 2.0 * M_PI * uniform(), s = geometry == 0 ? std::sqrt(1.0 - z * z) : 1.0;
  const double along = geometry == 0 ? z : (geometry == 1 ? (z < 0 ? -1.0 : 1.0) : small * z), across = geometry == 1 ? small : s;
  v[axis] = norm * along;
  v[(axis + 1) % 3] = norm * across * std::cos(f);
  v[(axis + 2) % 3] = norm * across * std::sin(f);
}

int main(int argc, char** argv) {
  if (argc < 10) return 1;
  const int form = std::atoi(argv[1]), gS = std::atoi(argv[4]), gL = std::atoi(argv[5]), axis = std::atoi(argv[8]);
  const long n = std::atol(argv[2]);
  host_adj::g_state = std::strtoull(argv[3], nullptr, 10) * 2 + 1;
  const double small = std::atof(argv[6]), angle = std::atof(argv[7]);
  const bool pulse = std::atoi(argv[9]) != 0;
  const double field = argc > 10 ? std::atof(argv[10]) : 611.4;
  for (int k = 0; k < 8; ++k) uniform();
  host_quat::g_stepper = form == 3;
  long taken = 0, refused = 0, wrong = 0;
  double ef[15] = {}, ed[15] = {};
  std::vector<double> rf, rd;
  auto put = [&](int j, quad exact, quad fixed, double fp64) {
    ef[j] = std::fmax(ef[j], std::fabs((double)(fixed - exact)));
    ed[j] = std::fmax(ed[j], std::fabs((double)((quad)fp64 - exact)));
  };
  for (long it = 0; it < n; ++it) {
    host_dop::Case q{};
    q.rtol = 1e-12;
    double l[3];
    for (int c = 0; c < 3; ++c) {
      const double size = c == axis ? 1e-3 : small;
      q.o0[c] = field * (uniform() - 0.5) * size;
      q.o1[c] = 5.0 * field * (uniform() - 0.5) * size;
      q.o2[c] = 16.0 * field * (uniform() - 0.5) * size;
    }
    q.o0[axis] -= field;
    if (pulse) {
      q.ga = -field * small;
      q.w = argc > 11 ? std::atof(argv[11]) : 6283.185307179586;
    }
    const double T = 7e-4 * (0.1 + uniform());
    q.t0 = uniform();
    q.h = std::fmin(angle / field * (0.5 + uniform()), T * uniform());
    const double x = q.t0 + (T - q.h) * uniform();
    q.tx = x - q.t0;
    draw(gS, small, axis, 1.0, q.S);
    draw(gL, small, axis, 1.0, l);
    // ---- fixed point: the words turned so that the axis is component 0
    double o[3][3], S[3], L[3];
    for (int c = 0; c < 3; ++c) {
      const int p = (c + axis) % 3;
      o[0][c] = q.o0[p];
      o[1][c] = q.o1[p];
      o[2][c] = q.o2[p];
      S[c] = q.S[p];
      L[c] = l[p];
    }
    SegScale sc;
    sc.pz = (5 - axis) % 3;
    if (!spin_scale(S, sc.se) || !field_scale(o[0], o[1], o[2], q.ga, T, sc, true)) {
      ++refused;
      continue;
    }
    i64 w[3][3], Sw[3], Lw[3];
    for (int k = 0; k < 3; ++k)
      for (int c = 0; c < 3; ++c) w[k][c] = to_q63(o[k][c], sc.oe - k * sc.te - (c ? sc.ok : 0));
    const i64 ga = to_q63(q.ga, sc.oe - (sc.pz ? sc.ok : 0));
    sc.sk = spin_grade(S, sc.se, sc.ok);
    spin_words(S, sc.se, sc.sk, Sw);
    u64 wm = 0;
    int we = 0;
    if (q.w != 0.0) wm = (u64)(host_adj::q_frexp((quad)q.w / (2 * host_adj::kPi), &we) * (quad)18446744073709551616.0);
    auto exps = [](int g, int c) { return g < 0 ? (c ? 0 : -g) : (c ? g : 0); };
    if (form == 0) {
      i64 Sn[3];
      StageLocal<3> ks;
      StepOut out;
      if (!dop_step(Lane3(), ks, sc, w[0], w[1], w[2], ga, wm, we, x, q.tx, q.h, StepTol{q.rtol, 1.0}, Sw, Sn, out)) {
        ++refused;
        continue;
      }
      quad Sq[3];
      double Sd[3];
      const quad eq = host_dop::step<quad>(q, Sq);
      const double edd = host_dop::step<double>(q, Sd);
      int sk = sc.sk;
      regrade(Sn, sk, sc.ok);
      for (int c = 0; c < 3; ++c) {
        const int p = (c + axis) % 3;
        put(p, Sq[p], word(Sn[c], sc.se - exps(sk, c)), Sd[p]);
      }
      if ((double)eq > 2e-7) {
        const quad rq = host_dop::q_pow(eq, (quad)-0.125);
        rf.push_back(std::fabs((double)((quad)out.root8 / rq - 1)));
        rd.push_back(std::fabs((double)(host_dop::q_pow((quad)edd, (quad)-0.125) / rq - 1)));
        if (std::fabs((double)eq - 1.0) > 1e-3) wrong += out.accept != (eq <= 1);
      } else {
        wrong += 0.9 * out.root8 < 6.0 || !out.accept;  // growth is clamped at 6
      }
    } else if (form == 1) {
      int le, gl;
      if (!adjoint_scale(L, sc.ok, le, gl)) return 1;
      spin_words(L, le, gl, Lw);
      StageLocal<3> ks, ys;
      AdjMoments m;
      if (!dop_adjoint(ks, ys, sc, w[0], w[1], w[2], ga, wm, we, x, q.tx, q.h, pulse, Sw, Lw, m, gl)) {
        ++refused;
        continue;
      }
      host_adj::Case a{};
      for (int c = 0; c < 3; ++c) {
        a.o0[c] = q.o0[c];
        a.o1[c] = q.o1[c];
        a.o2[c] = q.o2[c];
        a.S[c] = q.S[c];
      }
      a.ga = q.ga; a.w = q.w; a.t0 = q.t0; a.tx = q.tx; a.h = q.h;
      quad lq[3], Mq[12];
      double lD[3], MD[12];
      host_adj::back<quad>(a, l, lq, Mq);
      host_adj::back<double>(a, l, lD, MD);
      const int E = sc.se + le + m.exp;
      for (int c = 0; c < 3; ++c) {
        const int p = (c + axis) % 3;
        put(p, lq[p], word(Lw[c], le - exps(gl, c)), lD[p]);
        put(3 + p, Mq[p], word(m.z0[c], E - m.e[c]), MD[p]);
        put(6 + p, Mq[3 + p], word(m.z1[c], E - m.e[c]), MD[3 + p]);
        put(9 + p, Mq[6 + p], word(m.z2[c], E - m.e[c]), MD[6 + p]);
      }
      const i64 pw[3] = {m.cz, m.sz, m.scz};
      for (int j = 0; j < 3; ++j)
        if (pulse) put(12 + j, Mq[9 + j], word(pw[j], E + 1 - m.e[sc.pz]), MD[9 + j]);
    } else {
      i64 y[3], e[3];
      if (!(form == 3 ? quat_step<true>(sc, w[0], w[1], w[2], ga, wm, we, x, q.tx, q.h, Sw, y, e)
                      : quat_step<false>(sc, w[0], w[1], w[2], ga, wm, we, x, q.tx, q.h, Sw, y, e))) {
        ++refused;
        continue;
      }
      host_quat::Case a{};
      for (int c = 0; c < 3; ++c) {
        a.o0[c] = q.o0[c];
        a.o1[c] = q.o1[c];
        a.o2[c] = q.o2[c];
        a.S[c] = q.S[c];
      }
      a.ga = q.ga; a.w = q.w; a.t0 = q.t0; a.tx = q.tx; a.h = q.h;
      quad wq[3], eq[3];
      double wd[3], eD[3];
      host_quat::step<quad>(a, wq, eq);
      host_quat::step<double>(a, wd, eD);
      for (int c = 0; c < 3; ++c) {
        const int p = (c + axis) % 3;
        put(p, wq[p], word(y[c], sc.se - exps(sc.sk, c)), wd[p]);
        put(3 + p, eq[p], word(e[c], sc.se - exps(sc.sk, c)), eD[p]);
      }
    }
    ++taken;
  }
  std::printf("taken %ld refused %ld wrong %ld judged %ld root8 %.4g %.4g", taken, refused, wrong, (long)rf.size(),
              host_dop::median(rf), host_dop::median(rd));
  const int parts = form == 0 ? 3 : (form == 1 ? (pulse ? 15 : 12) : 6);
  for (int j = 0; j < parts; ++j) std::printf("\n%d %.4g %.4g", j, ef[j], ed[j]);
  std::printf("\n");
  return 0;
}
