// integratorType 6: the noise spectrum of the field each particle sees.
//
// The reference (src/particle.cpp:746-824, src/integrator.cpp:724-743,
// src/floquet.cpp:25-156) integrates no spin for this type.  Along every
// trajectory segment it samples the noise field
//   x(t) = gamma (v x E / c^2 + grad(p) + testNoise(t)) / 2
// on the grid of multiples of the particle's step h and feeds it to a
// per-particle aggregator of 17 Goertzel recursions, one per frequency of the
// dressed-spin Floquet analysis (floquet_diagonalize: the eigenphase of the
// one-period propagator of gamma (B0 + pulse) gives the splitting dE, and the
// frequencies are k w + {-dE, 0, dE}).  Per frequency and field component the
// aggregator keeps the recursion's last two values s1, s2 and the Laplace
// term of the covariance diagonal; it restarts at every window.
//
// Here one warp serves kSpecGroup particles in two alternating phases.  First
// each of its lanes runs its own particle's trajectory for a few segments into
// shared memory; then the warp takes the particles one after another: 32 samples
// at a time, the noise field of one sample per lane, the recursions (17
// frequencies x 3 components) two per lane.
//
// What bounds it: the FP64 pipe.  A sample costs 12 FP64 instructions of the
// recursions, one for its time and 1/16 or so of the ~45 of its noise field,
// against ~160 when every lane evaluated every sample (three sines of a test
// noise of amplitude zero among them) and one lane held all three components of a
// frequency: 4,099 particles x 0.02 s took 92 ms.
//
// The noise field and the recursions use the
// reference's operations in its order without contraction, so a run without
// test noise matches the reference's aggregators bit for bit; with test noise
// the device's sin of w t enters.  What this file leaves to the caller: the
// reference's reduction of the per-particle covariances (its CPU loop nests
// the tree the wrong way round, src/particle.cpp:826-834, and its GPU path does
// not reduce) is replaced by a plain sum over particles (st_covariance_spectrum
// in st_api.cpp), and the Floquet master equation that turns the spectrum into
// b_end (src/integrator.cpp:790-890, Eigen's matrix exponential) is not built.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "st_device.cuh"
#include "st_engine.cuh"
#include "st_tableau.h"

namespace st {

// ---------------------------------------------------------------- host: Floquet frequencies
namespace {

struct HVec {
  double x, y, z;
};
struct HQuat {
  double w, x, y, z;
};
inline HVec hv(double x, double y, double z) { return {x, y, z}; }
inline HVec hadd(HVec a, HVec b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
inline HVec hscale(double s, HVec a) { return {a.x * s, a.y * s, a.z * s}; }
inline HVec hcross(HVec a, HVec b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
inline double hdot(HVec a, HVec b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// qMult (src/quaternion.cpp)
inline HQuat hqmul(HQuat a, HQuat b) {
  return {a.w * b.w - a.x * b.x - a.y * b.y - a.z * b.z, a.w * b.x + a.x * b.w + a.y * b.z - a.z * b.y,
          a.w * b.y + a.y * b.w + a.z * b.x - a.x * b.z, a.w * b.z + a.z * b.w + a.x * b.y - a.y * b.x};
}
// rodriguezQuat (src/quaternion.cpp:150-156): rotation by |k| dt about -k/|k|
inline HQuat hrot(HVec k, double dt) {
  const double angle = sqrt(k.x * k.x + k.y * k.y + k.z * k.z);
  HVec n = {k.x / angle, k.y / angle, k.z / angle};
  const double h = angle * dt;
  n = hscale(-sin(h / 2.0), n);
  return {cos(h / 2.0), n.x, n.y, n.z};
}

// findCrossTerm (src/integrator.cpp:63-70) for a particle at rest at the
// origin at t0: the field of the dressed spin (interpolate, :48-61, moves it
// only under gravity).
HVec cross_term(const st_options& o, double t, double t0) {
  HVec p = hv(0.0, 0.0, 0.0), v = hv(0.0, 0.0, 0.0);
  if (o.gravity) {
    const HVec a = hv(0.0, kGravity, 0.0);
    p = hadd(hadd(p, hscale(t - t0, v)), hscale(t - t0, hscale(t - t0, hscale(0.5, a))));
    v = hadd(v, hscale(t - t0, a));
  }
  const HVec Gx = hv(o.Gx.x, o.Gx.y, o.Gx.z), Gy = hv(o.Gy.x, o.Gy.y, o.Gy.z), Gz = hv(o.Gz.x, o.Gz.y, o.Gz.z);
  const HVec G = hv(hdot(p, Gx), hdot(p, Gy), hdot(p, Gz));
  const HVec pulse = hv(0.0, 0.0, o.a * cos(o.w * t));
  const HVec E = hv(o.E.x, o.E.y, o.E.z), B0 = hv(o.B0.x, o.B0.y, o.B0.z);
  const HVec B = hadd(hadd(hadd(pulse, B0), hscale(1.0 / kC2, hcross(v, E))), G);
  return hscale(o.gamma, B);
}

// sum_j c_j B_j with the five coefficients taken forwards or backwards
HVec exponent(const double c[5], bool rev, const HVec B[5]) {
  HVec s = hscale(c[rev ? 4 : 0], B[0]);
  for (int j = 1; j < 5; ++j) s = hadd(s, hscale(c[rev ? 4 - j : j], B[j]));
  return s;
}

// integrateHamiltonian (src/integrator.cpp:745-785): y = q1 q2 ... q11 y per
// CFET8 step of h over [t0, tf].
int hamiltonian(const st_options& o, double t0, double tf, HQuat& y, double h) {
  using namespace cfet;
  static const double G[6][5] = {{G11, G12, G13, G14, G15}, {G21, G22, G23, G24, G25}, {G31, G32, G33, G34, G35},
                                 {G41, G42, G43, G44, G45}, {G51, G52, G53, G54, G55}, {G61, G62, G63, G64, G65}};
  static const double X[5] = {X1, X2, X3, X4, X5};
  double t = t0;
  unsigned int nstep = 0;
  while (t < tf) {
    nstep++;
    if (nstep > o.nmax) return -2;
    const double rest = tf - t;
    if (h >= rest) h = rest;
    HVec B[5];
    for (int i = 0; i < 5; ++i) B[i] = cross_term(o, t + X[i] * h, t0);
    HQuat q[12];
    for (int r = 0; r < 5; ++r) q[11 - r] = hrot(exponent(G[r], true, B), h);  // q11 .. q7
    for (int r = 5; r >= 0; --r) q[r + 1] = hrot(exponent(G[r], false, B), h);  // q6 .. q1
    HQuat prod = hqmul(q[1], q[2]);
    for (int r = 3; r <= 11; ++r) prod = hqmul(prod, q[r]);
    y = hqmul(prod, y);
    t += h;
  }
  return 0;
}

}  // namespace

int floquet_frequencies(const st_options& o, double freq[kSpecFreqs], double* dt) {
  if (!(o.w != 0.0) || !std::isfinite(o.w)) return -1;  // no period: the reference's loop would not end
  const double t0 = 0.0, tf = (2 * M_PI) / o.w;
  const int n_prop = 100;
  HQuat y = {1.0, 0.0, 0.0, 0.0};
  for (int i = 0; i < n_prop; ++i) {
    const double t1 = t0 + (tf - t0) * i / n_prop;
    const double t2 = t0 + (tf - t0) * (i + 1) / n_prop;
    hamiltonian(o, t1, t2, y, 1e-6);
  }
  // qEigenval (src/quaternion.cpp:169-172) of the period's propagator
  const double ez = -sqrt(1.0 - y.w * y.w);
  const double ea = fabs(atan2(ez, y.w)) / (tf - t0);
  const double eb = -ea;
  const double deltaE = ea - eb;
  for (int k = 0; k <= 11 / 2; ++k)
    for (int i = -1; i < 2; ++i) {
      const int index = k * 3 + i;
      if (index >= 0) freq[index] = deltaE * i + k * o.w;
    }
  *dt = (tf - t0) / n_prop;
  return 0;
}

int build_spec_set(const st_options& o, SpecSet* q) {
  double f[kSpecFreqs], dt = 0.0;
  if (floquet_frequencies(o, f, &dt) != 0) return -1;
  for (int k = 0; k < kSpecFreqs; ++k) {
    q->freq[k] = f[k];
    // goertzel_stage_1 / _2 (src/floquet.cpp:25-38) evaluate these per sample
    const double angle = f[k] * dt;
    q->two_cos[k] = 2 * cos(angle);
    q->sin_a[k] = sin(angle);
  }
  q->fdt = dt;
  q->na[0] = o.noiseAmplitudes.x; q->na[1] = o.noiseAmplitudes.y; q->na[2] = o.noiseAmplitudes.z;
  q->nw[0] = o.noiseFrequencies.x; q->nw[1] = o.noiseFrequencies.y; q->nw[2] = o.noiseFrequencies.z;
  return 0;
}

// ---------------------------------------------------------------- device
// The noise field at t of a segment starting at (t0, p0, v0), halved:
// findNoiseTerm (src/integrator.cpp:72-80) in the reference's operation order.
__device__ __forceinline__ void noise_sample(const SetParams& P, const SpecSet& Q, const SegStart& s0, double t,
                                             double& xx, double& xy, double& xz) {
  const double d = __dsub_rn(t, s0.t);
  double px = __dadd_rn(s0.px, __dmul_rn(d, s0.vx));
  double py = __dadd_rn(s0.py, __dmul_rn(d, s0.vy));
  double pz = __dadd_rn(s0.pz, __dmul_rn(d, s0.vz));
  double vx = s0.vx, vy = s0.vy, vz = s0.vz;
  if (P.gravity) {
    px = __dadd_rn(px, __dmul_rn(d, __dmul_rn(d, __dmul_rn(0.0, 0.5))));
    py = __dadd_rn(py, __dmul_rn(d, __dmul_rn(d, __dmul_rn(kGravity, 0.5))));
    pz = __dadd_rn(pz, __dmul_rn(d, __dmul_rn(d, __dmul_rn(0.0, 0.5))));
    vx = __dadd_rn(vx, __dmul_rn(d, 0.0));
    vy = __dadd_rn(vy, __dmul_rn(d, kGravity));
    vz = __dadd_rn(vz, __dmul_rn(d, 0.0));
  }
  auto dot3 = [](double ax, double ay, double az, const double* g) {
    return __dadd_rn(__dadd_rn(__dmul_rn(ax, g[0]), __dmul_rn(ay, g[1])), __dmul_rn(az, g[2]));
  };
  const double gx = dot3(px, py, pz, P.Gx), gy = dot3(px, py, pz, P.Gy), gz = dot3(px, py, pz, P.Gz);
  const double cx = __dsub_rn(__dmul_rn(vy, P.Ez), __dmul_rn(vz, P.Ey));
  const double cy = __dsub_rn(__dmul_rn(vz, P.Ex), __dmul_rn(vx, P.Ez));
  const double cz = __dsub_rn(__dmul_rn(vx, P.Ey), __dmul_rn(vy, P.Ex));
  // no amplitude, no sine: 0 sin(w t) adds nothing
  double nx = 0.0, ny = 0.0, nz = 0.0;
  if (Q.na[0] != 0.0 || !isfinite(Q.nw[0])) nx = __dmul_rn(Q.na[0], sin(__dmul_rn(Q.nw[0], t)));
  if (Q.na[1] != 0.0 || !isfinite(Q.nw[1])) ny = __dmul_rn(Q.na[1], sin(__dmul_rn(Q.nw[1], t)));
  if (Q.na[2] != 0.0 || !isfinite(Q.nw[2])) nz = __dmul_rn(Q.na[2], sin(__dmul_rn(Q.nw[2], t)));
  const double bx = __dadd_rn(__dadd_rn(__dmul_rn(cx, P.inv_c2), gx), nx);
  const double by = __dadd_rn(__dadd_rn(__dmul_rn(cy, P.inv_c2), gy), ny);
  const double bz = __dadd_rn(__dadd_rn(__dmul_rn(cz, P.inv_c2), gz), nz);
  xx = __dmul_rn(__dmul_rn(bx, P.gamma), 0.5);  // a division by two, exactly
  xy = __dmul_rn(__dmul_rn(by, P.gamma), 0.5);
  xz = __dmul_rn(__dmul_rn(bz, P.gamma), 0.5);
}

constexpr int kSpecRec = 3 * kSpecFreqs;  // recursions of a particle: frequency k, component c at 3 k + c
constexpr int kSpecSegs = 12;              // segments per particle and trajectory phase
// Shared memory of a warp: segments (t0, p0, v0, t1), a batch of samples, the recursions'
// state (s1, s2, im) and sample counts of the group's particles.
struct SpecShared {
  double seg[kSpecGroup][kSpecSegs][8];
  double x[32][3];
  double acc[kSpecGroup][3][kSpecRec];
  long long ns[kSpecGroup];
};

// One window (window >= 0) or up to next_t (window < 0) of every particle of
// a spectrum context.  Trajectory, window bookkeeping and failure codes as
// the plain kernel (n_steps counts segments); S is not integrated.
template <bool GAS>
__global__ void __launch_bounds__(kSpecBlock) k_spectrum(RunArgs a, int window, double next_t, SpecArgs sp) {
  extern __shared__ double st_smem[];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  SpecShared& sh = reinterpret_cast<SpecShared*>(st_smem)[threadIdx.x >> 5];
  const int64_t first = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kSpecGroup;
  const int64_t i = first + lane;  // lanes past the group own no particle
  unsigned long long n_seg = 0;
  bool hit = false;
  const unsigned long long dl = run_deadline(a);
  const bool mine = lane < kSpecGroup && i < a.s.n;
  bool run = false;
  double tf = next_t, hs = 1.0;
  int set = 0;
  PState p;
  p.stop = true;
  if (mine) {
    set = a.s.set[i];
    const SetParams& P = a.sets[set];
    run = true;
    if (window >= 0) {
      run = window < P.nwin && a.s.w_done[i] == window;
      tf = ((double)window + 1.0) * P.ioutInt;
    }
    if (run) {
      p = load_state(a.s, i);
      hs = p.h;  // the sampling step (integrateSpectrum's h)
    }
  }
  for (int k = lane; k < kSpecGroup * 3 * kSpecRec; k += 32) (&sh.acc[0][0][0])[k] = 0.0;
  if (lane < kSpecGroup) sh.ns[lane] = 0;
  // this lane's recursions: lane and lane + 32 of the 51 (the second for lanes below 19)
  const int r0 = lane, r1 = lane + 32 < kSpecRec ? lane + 32 : lane;
  bool finished = !run || p.stop;
  unsigned int guard = 0;
  while (__any_sync(FULL, !finished)) {
    // ---- trajectories, one particle per lane
    int n = 0;
    if (!finished) {
      const SetParams& P = a.sets[set];
      while (n < kSpecSegs && !finished) {
        SegStart s0;
        finished = traj_event<false, GAS>(p, P, tf, s0);
        ++n_seg;
        if (p.fail == 0) {
          double* q = sh.seg[lane][n++];
          q[0] = s0.t;
          q[1] = s0.px; q[2] = s0.py; q[3] = s0.pz;
          q[4] = s0.vx; q[5] = s0.vy; q[6] = s0.vz;
          q[7] = p.t;
        }
        if (p.stop) {
          nan_fill(p);
          finished = true;
        }
        p.n_steps += 1;
      }
    }
    hit = __any_sync(FULL, past_deadline(dl));
    if (hit) break;
    __syncwarp();
    // ---- samples, one particle after another
    for (int g = 0; g < kSpecGroup; ++g) {
      const int ng = __shfl_sync(FULL, n, g);
      if (ng == 0) continue;
      const int sg = __shfl_sync(FULL, set, g);
      const double h = __shfl_sync(FULL, hs, g);
      const SetParams& P = a.sets[sg];
      const SpecSet& Q = sp.sets[sg];
      const double c2a = Q.two_cos[r0 / 3], sna = __dmul_rn(2.0, Q.sin_a[r0 / 3]);
      const double c2b = Q.two_cos[r1 / 3], snb = __dmul_rn(2.0, Q.sin_a[r1 / 3]);
      const int ca = r0 % 3, cb = r1 % 3;
      double s1a = sh.acc[g][0][r0], s2a = sh.acc[g][1][r0], ima = sh.acc[g][2][r0];
      double s1b = sh.acc[g][0][r1], s2b = sh.acc[g][1][r1], imb = sh.acc[g][2][r1];
      long long ns = 0;
      for (int k = 0; k < ng && !hit; ++k) {
        const double* q = sh.seg[g][k];
        const SegStart s0 = {q[0], q[1], q[2], q[3], q[4], q[5], q[6]};
        // integrateSpectrum (src/integrator.cpp:730-743): the samples on
        // the grid of multiples of h in (t0, t]
        double t = __dmul_rn(__dadd_rn(floor(__ddiv_rn(s0.t, h)), 1.0), h);
        const double nt = __dmul_rn(__dadd_rn(floor(__ddiv_rn(q[7], h)), 1.0), h);
        const double lim = __dsub_rn(nt, __ddiv_rn(h, 2.0));
        while (t < lim && !hit) {
          // up to 32 samples: their times one after another (each the sum before plus h, rounded)
          double mt = t;
          int cnt = 0;
          while (cnt < 32 && t < lim) {
            if (lane == cnt) mt = t;
            t = __dadd_rn(t, h);
            ++cnt;
          }
          if (lane < cnt) noise_sample(P, Q, s0, mt, sh.x[lane][0], sh.x[lane][1], sh.x[lane][2]);
          __syncwarp();
          for (int j = 0; j < cnt; ++j) {
            // goertzel_stage_1, goertzel_stage_2_vector's b and covMat::add_outer
            // (src/floquet.cpp:25-38, 107-120); 2 (sin s2 x) as (2 sin) s2 x, exactly
            const double xa = sh.x[j][ca], xb = sh.x[j][cb];
            const double na = __dsub_rn(__dadd_rn(xa, __dmul_rn(c2a, s1a)), s2a);
            s2a = s1a;
            s1a = na;
            ima = __dadd_rn(ima, __dmul_rn(__dmul_rn(sna, s2a), xa));
            const double nb = __dsub_rn(__dadd_rn(xb, __dmul_rn(c2b, s1b)), s2b);
            s2b = s1b;
            s1b = nb;
            imb = __dadd_rn(imb, __dmul_rn(__dmul_rn(snb, s2b), xb));
          }
          __syncwarp();
          ns += cnt;
          if (((++guard) & 127u) == 0u) hit = __any_sync(FULL, past_deadline(dl));
        }
      }
      sh.acc[g][0][r0] = s1a; sh.acc[g][1][r0] = s2a; sh.acc[g][2][r0] = ima;
      if (r1 != r0) {
        sh.acc[g][0][r1] = s1b; sh.acc[g][1][r1] = s2b; sh.acc[g][2][r1] = imb;
      }
      if (lane == 0) sh.ns[g] += ns;
      __syncwarp();
    }
    if (hit) break;
  }
  __syncwarp();
  if (!hit) {
    if (run) {
      store_state(a.s, i, p);
      if (window >= 0) a.s.w_done[i] = window + 1;
      sp.nsamp[i] = sh.ns[lane];
    }
    const unsigned ran = __ballot_sync(FULL, run);
    const int64_t n = a.s.n;
    for (int k = lane; k < kSpecGroup * 3 * kSpecRec; k += 32) {
      const int g = k % kSpecGroup, f = k / kSpecGroup;  // neighbouring lanes: neighbouring particles
      if (!(ran >> g & 1u)) continue;
      const int q = f / kSpecRec, r = f - q * kSpecRec;
      double* dst = q == 0 ? sp.s1 : (q == 1 ? sp.s2 : sp.im);
      dst[(int64_t)r * n + first + g] = sh.acc[g][q][r];
    }
  }
  if (hit && lane == 0) atomicExch(&a.status->deadline_hit, 1);
  if (a.count_work && n_seg) atomicAdd(&a.status->segments, n_seg);
}

// ---------------------------------------------------------------- results
// The aggregators ([(3 k + c) n + i]) per particle ([i][k][c]).
__global__ void k_spec_gather(const double* src, double* dst, int64_t n) {
  __shared__ double tile[32][33];
  const int64_t i0 = (int64_t)blockIdx.x * 32;
  const int r0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int r = r0 + k;
    const int64_t i = i0 + threadIdx.x;
    if (r < kSpecRec && i < n) tile[k][threadIdx.x] = src[(int64_t)r * n + i];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int64_t i = i0 + k;
    const int r = r0 + threadIdx.x;
    if (r < kSpecRec && i < n) dst[i * kSpecRec + r] = tile[threadIdx.x][k];
  }
}

// Covariance spectrum of particles [first, first + n_set): block k sums frequency k's
// 18 values over the particles, thread t those t, t + 256, ... in order, then a
// fixed tree.  goertzel_stage_2 (src/floquet.cpp:40-47): c = a + i b, variance = c c^dag,
// a = s1 - cos(w dt) s2, b = sin(w dt) s2; then the Laplace term on the diagonal
// (SpectrumAggregator::get_covariance_spectrum, :130-145).
constexpr int kCovBlock = 256;
__global__ void __launch_bounds__(kCovBlock) k_covariance(SpecArgs sp, int64_t n, int64_t first, int64_t n_set,
                                                          const double* cos_sin, double* out) {
  __shared__ double sh[kCovBlock];
  const int k = blockIdx.x;
  const double ca = cos_sin[2 * k], sa = cos_sin[2 * k + 1];
  double m[18];
  for (int q = 0; q < 18; ++q) m[q] = 0.0;
  for (int64_t j = threadIdx.x; j < n_set; j += kCovBlock) {
    const int64_t i = first + j;
    double re[3], imc[3], la[3];
    for (int q = 0; q < 3; ++q) {
      const double x1 = sp.s1[(int64_t)(3 * k + q) * n + i], x2 = sp.s2[(int64_t)(3 * k + q) * n + i];
      la[q] = sp.im[(int64_t)(3 * k + q) * n + i];
      re[q] = __dsub_rn(x1, __dmul_rn(ca, x2));
      imc[q] = __dmul_rn(sa, x2);
    }
    for (int r = 0; r < 3; ++r)
      for (int q = 0; q < 3; ++q) {  // c_r conj(c_q)
        m[(r * 3 + q) * 2] += __dadd_rn(__dmul_rn(re[r], re[q]), __dmul_rn(imc[r], imc[q]));
        m[(r * 3 + q) * 2 + 1] += __dsub_rn(__dmul_rn(imc[r], re[q]), __dmul_rn(re[r], imc[q]));
      }
    for (int r = 0; r < 3; ++r) m[(r * 3 + r) * 2 + 1] += -la[r];
  }
  for (int q = 0; q < 18; ++q) {
    __syncthreads();
    sh[threadIdx.x] = m[q];
    __syncthreads();
    for (int s = kCovBlock / 2; s > 0; s >>= 1) {
      if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[k * 18 + q] = sh[0];
  }
}

int launch_spec_gather(const double* src, double* dst, int64_t n, void* stream) {
  if (n <= 0) return 0;
  k_spec_gather<<<dim3((unsigned)((n + 31) / 32), (kSpecRec + 31) / 32), dim3(32, 8), 0, (cudaStream_t)stream>>>(src, dst, n);
  return (int)cudaGetLastError();
}
int launch_covariance(const SpecArgs& sp, int64_t n, int64_t first, int64_t n_set, const double* cos_sin, double* out,
                      void* stream) {
  k_covariance<<<kSpecFreqs, kCovBlock, 0, (cudaStream_t)stream>>>(sp, n, first, n_set, cos_sin, out);
  return (int)cudaGetLastError();
}

// Opt the kernels in to their shared memory (before any capture of a launch).
int spectrum_prepare() {
  const int sm = (int)(kSpecBlock / 32 * sizeof(SpecShared));
  cudaError_t e = cudaFuncSetAttribute(k_spectrum<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_spectrum<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  return (int)e;
}

int launch_spectrum(const RunArgs& a, int window, double next_t, const SpecArgs& sp, void* stream) {
  if (a.s.n == 0) return 0;
  const int64_t warps = (a.s.n + kSpecGroup - 1) / kSpecGroup;
  const unsigned grid = (unsigned)((warps * 32 + kSpecBlock - 1) / kSpecBlock);
  const size_t sm = kSpecBlock / 32 * sizeof(SpecShared);
  if (a.any_gas)
    k_spectrum<true><<<grid, kSpecBlock, sm, (cudaStream_t)stream>>>(a, window, next_t, sp);
  else
    k_spectrum<false><<<grid, kSpecBlock, sm, (cudaStream_t)stream>>>(a, window, next_t, sp);
  return (int)cudaGetLastError();
}

}  // namespace st
