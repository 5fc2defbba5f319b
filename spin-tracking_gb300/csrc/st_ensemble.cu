// Ensemble statistics of one parameter set at one snapshot, on the device:
// mean spin and polarisation, and the precession phase analysis of the
// reference's scripts (scripts/nedmSim.py:151-179 shiftDatapoints and
// benchmarks/CheckingFrequencyShiftFromEField.ipynb analyzeDataset):
//   phi = atan2(Sz, Sy) of every particle with failureState 0;
//   align: with `location` the left edge of the most populated of 1000
//          equal bins over [min phi, max phi] (numpy.histogram's binning),
//          phi <= location - pi gains 2 pi, phi >= location + pi loses 2 pi;
//   clip:  drop phi outside mean +- 5 std of the aligned set;
//   mean and population std of what is left, the mean wrapped to [-pi, pi];
//   frequency shift = wrap(mean - atan2(cos(w t), sin(w t))) / (2 pi t),
//          w = gamma |B0| sign(B0x).
// Also the mean and population std of the unwrapped phase atan2(Sz, Sy) +
// 2 pi turns over the same particles (no alignment needed).
// Sums are per-block partials combined in a fixed order by the block that
// finishes last, so the result is the same on every call.
//
// What bounds it: one atan2 per particle (some 60 FP64 instructions, 76 cycles
// of a sub-partition's pipe each: 0.12 ms for 524,288 particles) and the latency
// of six small launches.  The phase is computed once, by the first pass, and kept
// in a scratch array (eight passes that each recomputed it, and eight
// single-thread kernels between them, took 0.9 ms); every pass's last block also
// finishes it, so the next pass needs no launch in between.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <stdint.h>

#include "st_internal.h"

namespace st {

namespace {
constexpr int kEnsBlock = 256;
constexpr int kEnsBins = kEnsHistBins;
constexpr double kPi = 3.141592653589793;

struct EnsView {
  const double *t, *Sx, *Sy, *Sz;
  const int32_t *fail, *turns;
  int64_t first, n;
};

__device__ __forceinline__ double unwrapped(double phi, int turns) { return fma(2.0 * kPi, (double)turns, phi); }

// ctl slots: the ENS_* indices of st_internal.h

__device__ __forceinline__ bool ens_phi(const EnsView& v, int64_t i, double& phi) {
  if (v.fail[i] != 0) return false;
  phi = atan2(v.Sz[i], v.Sy[i]);
  return !isnan(phi);
}

// numpy's aligned value (both tests on the unshifted phase)
__device__ __forceinline__ double ens_align(double phi, double loc) {
  double p = phi;
  if (phi <= __dsub_rn(loc, kPi)) p = __dadd_rn(p, 2.0 * kPi);
  if (phi >= __dadd_rn(loc, kPi)) p = __dsub_rn(p, 2.0 * kPi);
  return p;
}

// numpy.histogram bin of x for `bins` equal bins over [e0, e1]
__device__ __forceinline__ int ens_bin(double x, double e0, double e1) {
  const double denom = __dsub_rn(e1, e0);
  const double f = __dmul_rn(__ddiv_rn(__dsub_rn(x, e0), denom), (double)kEnsBins);
  int k = (int)f;
  if (k >= kEnsBins) k = kEnsBins - 1;
  if (k < 0) k = 0;
  const double step = __ddiv_rn(denom, (double)kEnsBins);
  const double lo = __dadd_rn(__dmul_rn((double)k, step), e0);
  const double hi = (k + 1 == kEnsBins) ? e1 : __dadd_rn(__dmul_rn((double)(k + 1), step), e0);
  if (x < lo) --k;
  else if (x >= hi && k != kEnsBins - 1) ++k;
  return k;
}

constexpr int kEnsVals = 8;
// Sum (or minimum, maximum) of a value over the block, in thread 0 (fixed tree order).
__device__ double block_reduce(double* sh, double v, int op) {
  const int t = threadIdx.x;
  __syncthreads();
  sh[t] = v;
  __syncthreads();
  for (int s = kEnsBlock / 2; s > 0; s >>= 1) {
    if (t < s) sh[t] = op == 0 ? sh[t] + sh[t + s] : (op == 1 ? fmin(sh[t], sh[t + s]) : fmax(sh[t], sh[t + s]));
    __syncthreads();
  }
  return sh[0];
}

// Values of each pass's partials and how they combine (0 sum, 1 minimum, 2 maximum):
//   pass 0: count, sum S (3), min phi, max phi, sum of unwrapped phases, first particle counted
//   pass 1: squared deviations of the unwrapped phases (and the histogram)
//   pass 2, 4: count and sum of the aligned (4: clipped) phases
//   pass 3, 5: their squared deviations
__device__ __forceinline__ int ens_nvals(int pass) { return pass == 0 ? 8 : (pass == 2 || pass == 4 ? 2 : 1); }
__device__ __forceinline__ int ens_op(int pass, int q) { return pass == 0 ? (q == 4 || q == 7 ? 1 : (q == 5 ? 2 : 0)) : 0; }

// The last block of a pass combines the partials: thread t sums blocks t, t + 256, ...
// in order, then the block tree.
__device__ void ens_finish(const EnsView& v, int pass, double* sh, double* ctl, const double* part, int nblk,
                           const unsigned int* hist) {
  double r[kEnsVals];
  const int nv = ens_nvals(pass);
  for (int q = 0; q < nv; ++q) {
    const int op = ens_op(pass, q);
    double a = op == 0 ? 0.0 : (op == 1 ? INFINITY : -INFINITY);
    for (int b = threadIdx.x; b < nblk; b += kEnsBlock) {
      const double x = __ldcg(part + b * kEnsVals + q);
      a = op == 0 ? a + x : (op == 1 ? fmin(a, x) : fmax(a, x));
    }
    r[q] = block_reduce(sh, a, op);
  }
  if (pass == 1) {  // the most populated bin, the first of equals (numpy.argmax)
    unsigned long long best = 0;
    for (int k = threadIdx.x; k < kEnsBins; k += kEnsBlock) {
      const unsigned long long c = ((unsigned long long)__ldcg(hist + k) << 32) | (unsigned)(kEnsBins - k);
      if (c > best) best = c;
    }
    __syncthreads();
    unsigned long long* u = reinterpret_cast<unsigned long long*>(sh);
    u[threadIdx.x] = best;
    __syncthreads();
    for (int s = kEnsBlock / 2; s > 0; s >>= 1) {
      if ((int)threadIdx.x < s && u[threadIdx.x + s] > u[threadIdx.x]) u[threadIdx.x] = u[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      const int k = kEnsBins - (int)(unsigned)(u[0] & 0xffffffffull);
      const double e0 = ctl[ENS_EDGE0], e1 = ctl[ENS_EDGE1];
      ctl[ENS_LOC] = __dadd_rn(__dmul_rn((double)k, __ddiv_rn(__dsub_rn(e1, e0), (double)kEnsBins)), e0);
    }
  }
  if (threadIdx.x != 0) return;
  if (pass == 0) {
    ctl[ENS_COUNT] = r[0];
    ctl[ENS_SX] = r[1];
    ctl[ENS_SY] = r[2];
    ctl[ENS_SZ] = r[3];
    ctl[ENS_MIN] = r[4];
    ctl[ENS_MAX] = r[5];
    ctl[ENS_UMEAN] = r[6] / r[0];
    double e0 = r[4], e1 = r[5];
    if (e0 == e1) {
      e0 = e0 - 0.5;
      e1 = e1 + 0.5;
    }
    ctl[ENS_EDGE0] = e0;
    ctl[ENS_EDGE1] = e1;
    // time of the first particle that counts
    ctl[ENS_T] = r[7] < INFINITY ? v.t[v.first + (int64_t)r[7]] : __longlong_as_double(0x7ff8000000000000ll);
  } else if (pass == 1) {
    ctl[ENS_USTD] = sqrt(r[0] / ctl[ENS_COUNT]);
  } else if (pass == 2) {
    ctl[ENS_MEAN1] = r[1] / r[0];
  } else if (pass == 3) {
    ctl[ENS_STD1] = sqrt(r[0] / ctl[ENS_COUNT]);
  } else if (pass == 4) {
    ctl[ENS_KEPT] = r[0];
    ctl[ENS_MEAN2] = r[1] / r[0];
  } else {
    ctl[ENS_STD2] = sqrt(r[0] / ctl[ENS_KEPT]);
  }
}

// One pass; phi: scratch of n phases (NaN: the particle does not count), written by pass 0.
__global__ void __launch_bounds__(kEnsBlock) k_ens_pass(EnsView v, int pass, double* phis, double* ctl, double* part,
                                                        unsigned int* hist, unsigned int* done) {
  __shared__ double sh[kEnsBlock];
  __shared__ unsigned int hsh[kEnsBins];
  __shared__ bool last;
  const int64_t stride = (int64_t)gridDim.x * kEnsBlock;
  double acc[kEnsVals];
  for (int q = 0; q < kEnsVals; ++q) {
    const int op = ens_op(pass, q);
    acc[q] = op == 0 ? 0.0 : (op == 1 ? INFINITY : -INFINITY);
  }
  if (pass == 1)
    for (int k = threadIdx.x; k < kEnsBins; k += kEnsBlock) hsh[k] = 0u;
  __syncthreads();
  for (int64_t j = (int64_t)blockIdx.x * kEnsBlock + threadIdx.x; j < v.n; j += stride) {
    const int64_t i = v.first + j;
    if (pass == 0) {
      double phi;
      const bool ok = ens_phi(v, i, phi);
      phis[j] = ok ? phi : __longlong_as_double(0x7ff8000000000000ll);
      if (!ok) continue;
      acc[0] += 1.0;
      acc[1] += v.Sx[i];
      acc[2] += v.Sy[i];
      acc[3] += v.Sz[i];
      acc[4] = fmin(acc[4], phi);
      acc[5] = fmax(acc[5], phi);
      acc[6] += unwrapped(phi, v.turns[i]);
      acc[7] = fmin(acc[7], (double)j);
      continue;
    }
    const double phi = phis[j];
    if (isnan(phi)) continue;
    if (pass == 1) {
      atomicAdd(&hsh[ens_bin(phi, ctl[ENS_EDGE0], ctl[ENS_EDGE1])], 1u);
      const double d = unwrapped(phi, v.turns[i]) - ctl[ENS_UMEAN];
      acc[0] = fma(d, d, acc[0]);
    } else {
      const double p = ens_align(phi, ctl[ENS_LOC]);
      if (pass >= 4) {  // numpy: shifted < mean - std * 5, shifted > mean + std * 5
        const double w5 = __dmul_rn(ctl[ENS_STD1], 5.0);
        if (p < __dsub_rn(ctl[ENS_MEAN1], w5) || p > __dadd_rn(ctl[ENS_MEAN1], w5)) continue;
      }
      if (pass == 2 || pass == 4) {
        acc[0] += 1.0;
        acc[1] += p;
      } else {
        const double d = p - ((pass == 3) ? ctl[ENS_MEAN1] : ctl[ENS_MEAN2]);
        acc[0] = fma(d, d, acc[0]);
      }
    }
  }
  if (pass == 1) {
    __syncthreads();
    for (int k = threadIdx.x; k < kEnsBins; k += kEnsBlock)
      if (hsh[k]) atomicAdd(&hist[k], hsh[k]);
  }
  for (int q = 0; q < ens_nvals(pass); ++q) {
    const double r = block_reduce(sh, acc[q], ens_op(pass, q));
    if (threadIdx.x == 0) part[blockIdx.x * kEnsVals + q] = r;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(done + pass, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  ens_finish(v, pass, sh, ctl, part, gridDim.x, hist);
}
}  // namespace

// Run the passes for particles [first, first + n) of the given arrays; ctl
// receives ensemble_ctl_count() doubles (slots of the enum above); hist: the
// histogram and one counter per pass; phis: n doubles of scratch.
int ensemble_device(const double* t, const double* Sx, const double* Sy, const double* Sz, const int32_t* fail,
                    const int32_t* turns, int64_t first, int64_t n, double* ctl, double* part, unsigned int* hist,
                    double* phis, int max_blocks, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  EnsView v{t, Sx, Sy, Sz, fail, turns, first, n};
  const int nblk = (int)std::min<int64_t>(max_blocks, std::max<int64_t>(1, (n + kEnsBlock - 1) / kEnsBlock));
  cudaError_t e = cudaMemsetAsync(hist, 0, sizeof(unsigned int) * (kEnsBins + kEnsPasses), s);
  if (e != cudaSuccess) return (int)e;
  for (int pass = 0; pass < kEnsPasses; ++pass)
    k_ens_pass<<<nblk, kEnsBlock, 0, s>>>(v, pass, phis, ctl, part, hist, hist + kEnsBins);
  return (int)cudaGetLastError();
}

int ensemble_ctl_count() { return ENS_USTD + 1; }

// ---------------------------------------------------------------- phase
namespace {
__global__ void k_gather_phase(const double* Sy, const double* Sz, const int32_t* turns, int64_t n, double* dst) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = unwrapped(atan2(Sz[i], Sy[i]), turns[i]);
}
}  // namespace

namespace {
// Spins of n particles as a dense array of three doubles each.
__global__ void k_gather_spins(const double* Sx, const double* Sy, const double* Sz, int64_t n, double* dst) {
  __shared__ double sh[3 * 256];
  const int64_t base = (int64_t)blockIdx.x * 256, i = base + threadIdx.x;
  if (i < n) {  // stride 3: no two lanes of a half warp share a bank
    sh[3 * threadIdx.x] = Sx[i];
    sh[3 * threadIdx.x + 1] = Sy[i];
    sh[3 * threadIdx.x + 2] = Sz[i];
  }
  __syncthreads();
  const int64_t left = 3 * (n - base);
  for (int k = threadIdx.x; k < 3 * 256 && k < left; k += 256) dst[3 * base + k] = sh[k];
}
}  // namespace

// Coalesced on both sides through shared memory (three strided copies of 8-byte rows took
// 0.8 ms for 524,288 particles; the traffic of 25 MB takes 4 us).
int launch_gather_spins(const double* Sx, const double* Sy, const double* Sz, int64_t n, double* dst, void* stream) {
  if (n <= 0) return 0;
  k_gather_spins<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(Sx, Sy, Sz, n, dst);
  return (int)cudaGetLastError();
}

int launch_gather_phase(const double* Sy, const double* Sz, const int32_t* turns, int64_t n, double* dst,
                        void* stream) {
  if (n <= 0) return 0;
  k_gather_phase<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(Sy, Sz, turns, n, dst);
  return (int)cudaGetLastError();
}

}  // namespace st
