// Kernel templates of the window engine (the plain, flattened and
// trajectory-ahead kernels) and their device helpers.  Included by
// st_kernels.cu (instantiations for integrator types 0 and 1) and
// st_kernels_ext.cu (EXT: also types 2-5), which compile in parallel.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "st_device.cuh"

namespace st {

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Deadline armed for this run (0 = none); read once per thread.
__device__ __forceinline__ unsigned long long run_deadline(const RunArgs& a) {
  return a.deadline_armed ? *((volatile unsigned long long*)&a.status->deadline_ns) : 0ull;
}
__device__ __forceinline__ bool past_deadline(unsigned long long dl) { return dl != 0ull && globaltimer_ns() > dl; }

// Whether a set's integrator type integrates the spin in this instantiation:
// 0 DOP853, 1 RK45, and with EXT also 2-5; any other type tracks the
// trajectory only (src/particle.cpp:568-594 integrates nothing for it).
template <bool EXT>
__device__ __forceinline__ bool spin_on(int it) {
  return it == 0 || it == 1 || (EXT && it >= 2 && it <= 5);
}

// Start the integrator of the set's type over a segment.
template <bool EXT, bool FX>
__device__ __forceinline__ void spin_begin(Seg& g, const SetParams& P, double& Sx, double& Sy, double& Sz, double h) {
  if (P.integrator == 0)
    dop_begin<FX>(g, P, Sx, Sy, Sz, h);
  else if (!EXT || P.integrator == 1)
    rk45_begin(g, h);
  else
    ext_begin(g, h);
}

__device__ __forceinline__ void warp_add(unsigned long long* dst, unsigned long long v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, v);
}

__device__ __forceinline__ void nan_fill(PState& p) {
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  p.t = nan;
  p.px = p.py = p.pz = nan;
  p.vx = p.vy = p.vz = nan;
  p.Sx = p.Sy = p.Sz = nan;
}

__device__ __forceinline__ void write_snap(const RunArgs& a, int64_t i, int w, const PState& p) {
  if (a.snap == nullptr || w < a.w_begin || w >= a.w_end) return;
  char* b = a.snap + (size_t)(w - a.w_begin) * a.snap_layout.bytes;
  const size_t* o = a.snap_layout.off;
  reinterpret_cast<double*>(b + o[0])[i] = p.t;
  reinterpret_cast<double*>(b + o[1])[i] = p.px;
  reinterpret_cast<double*>(b + o[2])[i] = p.py;
  reinterpret_cast<double*>(b + o[3])[i] = p.pz;
  reinterpret_cast<double*>(b + o[4])[i] = p.vx;
  reinterpret_cast<double*>(b + o[5])[i] = p.vy;
  reinterpret_cast<double*>(b + o[6])[i] = p.vz;
  reinterpret_cast<double*>(b + o[7])[i] = p.Sx;
  reinterpret_cast<double*>(b + o[8])[i] = p.Sy;
  reinterpret_cast<double*>(b + o[9])[i] = p.Sz;
  reinterpret_cast<int32_t*>(b + o[10])[i] = p.fail;
  reinterpret_cast<uint64_t*>(b + o[11])[i] = p.n_coll;
  reinterpret_cast<uint64_t*>(b + o[12])[i] = p.n_bounce;
  reinterpret_cast<uint64_t*>(b + o[13])[i] = p.n_steps;
  reinterpret_cast<int32_t*>(b + o[14])[i] = p.turns;
}

// ------------------------------------------------------------------ plain
// The reference's per-particle window loop (src/particle.cpp:558-614) with
// nested segment and step loops.  Returns false if the deadline passed (the
// caller then discards the window's progress).
template <bool EXT>
__device__ __forceinline__ bool window_nested(PState& p, const SetParams& P, double tf, unsigned long long dl,
                                              unsigned long long& n_dop, unsigned long long& n_rk,
                                              unsigned long long& n_ext, unsigned long long& n_seg) {
  double tempH = p.h;
  bool finished = false;
  unsigned int guard = 0;
  Seg g;
  g.carry = false;
  while (!finished && !p.stop) {
    SegStart s0;
    finished = traj_event(p, P, tf, s0);
    ++n_seg;
    if (p.fail == 0) {
      int res = 0;
      if (spin_on<EXT>(P.integrator)) {
        seg_setup<kFixedPoint>(g, P, s0, p.t);
        if (P.integrator == 0) {
          dop_begin<kFixedPoint>(g, P, p.Sx, p.Sy, p.Sz, tempH);
          do {
            res = dop_attempt<kFixedPoint>(g, P, p.Sx, p.Sy, p.Sz);
            ++n_dop;
            if (((++guard) & 1023u) == 0u && past_deadline(dl)) return false;
          } while (res == 0);
        } else if (!EXT || P.integrator == 1) {
          rk45_begin(g, tempH);
          do {
            res = rk45_attempt<kFixedPoint>(g, P, p.Sx, p.Sy, p.Sz);
            ++n_rk;
            if (((++guard) & 1023u) == 0u && past_deadline(dl)) return false;
          } while (res == 0);
        } else {
          ext_begin(g, tempH);
          do {
            res = ext_attempt<kFixedPoint>(g, P, p.Sx, p.Sy, p.Sz);
            ++n_ext;
            if (((++guard) & 1023u) == 0u && past_deadline(dl)) return false;
          } while (res == 0);
        }
        tempH = g.h;
        p.turns += g.turns;
        if (res > 0) res = 0;
      }
      if (P.keep) p.h = tempH;
      if (res < 0) {
        p.stop = true;
        p.fail = res;
      }
    }
    if (p.stop) {
      nan_fill(p);
      g.carry = false;
    }
    p.n_steps += 1;
    if (((++guard) & 255u) == 0u && past_deadline(dl)) return false;
  }
  spin_settle<kFixedPoint>(g, P, p.Sx, p.Sy, p.Sz);
  return true;
}

// window >= 0: advance particles whose next window is `window` to its end
// ((window+1)*ioutInt of their set) and mark it done.  window < 0: advance
// every particle to next_t (runSimulation semantics, no window bookkeeping).
// EXT: also integrator types 2-5.
template <int BLOCK, bool EXT>
__global__ void __launch_bounds__(BLOCK) k_plain(RunArgs a, int window, double next_t) {
  const int lane = threadIdx.x & 31;
  const int64_t i = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * a.spread + lane;
  unsigned long long n_dop = 0, n_rk = 0, n_ext = 0, n_seg = 0;
  bool hit = false;
  const unsigned long long dl = run_deadline(a);
  if (lane < a.spread && i < a.s.n) {
    const SetParams& P = a.sets[a.s.set[i]];
    double tf = next_t;
    bool run = true;
    if (window >= 0) {
      run = window < P.nwin && a.s.w_done[i] == window;
      tf = ((double)window + 1.0) * P.ioutInt;
    }
    if (run) {
      PState p = load_state(a.s, i);
      if (window_nested<EXT>(p, P, tf, dl, n_dop, n_rk, n_ext, n_seg)) {
        store_state(a.s, i, p);
        if (window >= 0) a.s.w_done[i] = window + 1;
      } else {
        hit = true;
      }
    }
  }
  if (hit) atomicExch(&a.status->deadline_hit, 1);
  if (a.count_work) {
    warp_add(&a.status->dop_attempts, n_dop);
    warp_add(&a.status->rk45_attempts, n_rk);
    if (EXT) warp_add(&a.status->ext_attempts, n_ext);
    warp_add(&a.status->segments, n_seg);
  }
}

// ------------------------------------------------------------------ persistent
enum LaneMode { M_FETCH = 0, M_EVENT = 1, M_SEG = 2, M_WEND = 3, M_DONE = 4 };

template <int BLOCK, int MINB, bool EXT, bool FX>
__global__ void __launch_bounds__(BLOCK, MINB) k_persistent(RunArgs a) {
  int mode = (int)(threadIdx.x & 31) < a.spread ? M_FETCH : M_DONE;
  int64_t i = 0;
  const SetParams* P = a.sets;
  PState p;
  Seg g;
  g.carry = false;
  int w = 0, wlast = 0;
  double tf = 0.0, tempH = 0.0;
  bool finished = false, hit = false;
  unsigned long long n_dop = 0, n_rk = 0, n_ext = 0, n_seg = 0;
  unsigned int tick = 0;
  const unsigned long long dl = run_deadline(a);
  while (true) {
    // Phase A (divergent, short): bring this lane to a segment that needs
    // step attempts, or run out of work.
    while (mode != M_SEG && mode != M_DONE) {
      if (mode == M_FETCH) {
        const unsigned long long item = atomicAdd(&a.status->queue_head, 1ull);
        if (item >= (unsigned long long)a.nitems) {
          mode = M_DONE;
          break;
        }
        i = a.order ? a.order[item] : (int64_t)item;
        P = &a.sets[a.s.set[i]];
        w = a.s.w_done[i];
        wlast = min(a.w_end, P->nwin);
        if (w >= wlast) continue;
        p = load_state(a.s, i);
        tf = ((double)w + 1.0) * P->ioutInt;
        tempH = p.h;
        finished = false;
        mode = M_EVENT;
      }
      if (mode == M_EVENT) {
        if (p.stop) {
          mode = M_WEND;
        } else {
          SegStart s0;
          finished = traj_event(p, *P, tf, s0);
          ++n_seg;
          if (p.fail == 0 && spin_on<EXT>(P->integrator)) {
            seg_setup<FX>(g, *P, s0, p.t);
            spin_begin<EXT, FX>(g, *P, p.Sx, p.Sy, p.Sz, tempH);
            mode = M_SEG;
          } else {
            if (p.fail == 0 && P->keep) p.h = tempH;
            if (p.stop) {
              nan_fill(p);
              g.carry = false;
            }
            p.n_steps += 1;
            mode = (finished || p.stop) ? M_WEND : M_EVENT;
          }
          if (((++tick) & 255u) == 0u && past_deadline(dl)) {
            hit = true;
            mode = M_DONE;
            break;
          }
        }
      }
      if (mode == M_WEND) {
        spin_settle<FX>(g, *P, p.Sx, p.Sy, p.Sz);
        write_snap(a, i, w, p);
        ++w;
        store_state(a.s, i, p);  // every window end is a resumable checkpoint
        a.s.w_done[i] = w;
        if (w < wlast) {
          tf = ((double)w + 1.0) * P->ioutInt;
          tempH = p.h;
          finished = false;
          mode = M_EVENT;
        } else {
          mode = M_FETCH;
        }
      }
    }
    if (mode == M_DONE) break;
    // Phase B (converged): one step attempt for every lane.
    int r;
    if (P->integrator == 0) {
      r = dop_attempt<FX>(g, *P, p.Sx, p.Sy, p.Sz);
      ++n_dop;
    } else if (!EXT || P->integrator == 1) {
      r = rk45_attempt<FX>(g, *P, p.Sx, p.Sy, p.Sz);
      ++n_rk;
    } else {
      r = ext_attempt<FX>(g, *P, p.Sx, p.Sy, p.Sz);
      ++n_ext;
    }
    if (r != 0) {
      tempH = g.h;
      p.turns += g.turns;
      if (P->keep) p.h = tempH;
      if (r < 0) {
        p.stop = true;
        p.fail = r;
      }
      if (p.stop) {
        nan_fill(p);
        g.carry = false;
      }
      p.n_steps += 1;
      mode = (finished || p.stop) ? M_WEND : M_EVENT;
    }
    if (((++tick) & 255u) == 0u && past_deadline(dl)) {
      hit = true;
      break;
    }
  }
  if (hit) atomicExch(&a.status->deadline_hit, 1);
  if (a.count_work) {
    // lanes leave the loop at different times: aggregate with plain atomics
    if (n_dop) atomicAdd(&a.status->dop_attempts, n_dop);
    if (n_rk) atomicAdd(&a.status->rk45_attempts, n_rk);
    if (n_ext) atomicAdd(&a.status->ext_attempts, n_ext);
    if (n_seg) atomicAdd(&a.status->segments, n_seg);
  }
}

// ------------------------------------------------------------------ batched (trajectory ahead)
// The trajectory of a particle does not depend on its spin, so each lane runs
// its particles' trajectories ahead of the spin integration, into a ring of
// segment records in device memory.  A warp alternates two phases: the
// trajectory phase fills the rings of all its lanes (one event per lane and
// round), the spin phase integrates (one step attempt per lane and iteration)
// until lanes run dry.  A record carries the segment's time span and field
// polynomial (o0, o1), so starting a segment on the spin side is a ring pop.
//
// Why phases this long, and rings in memory: the instructions of either phase
// about fill what a sub-partition holds close by (~16 KB), and beyond that they
// arrive at 8 bytes per cycle and SM.  With 8-record rings in shared memory the
// two phases alternated every other attempt and half the time went into
// instruction supply (1,048,576 particles x 0.1 s: 398 ms with the trajectory
// in FP64, 463 ms with its faster but larger integer code).  A ring of 64 records is
// about 190 attempts.  The rings of a full grid (7.7 KB a lane, 14.9 with 128 records) exceed L2:
// 286 bytes of DRAM traffic per segment, 142 GB/s, 2% of the copy bandwidth.
//
// The trajectory side crosses window ends and goes on to its next particle, so
// rings never block there: at a window end it saves its state in one of
// kAheadSlots slots, from which the spin side writes the window's checkpoint
// and snapshot when it gets there.  So every window end is an exact, resumable
// checkpoint, and the main state holds nothing newer than the spin side's last
// finished window.
constexpr int kAheadSlots = 4;

struct alignas(16) SegRec {
  double t0, t1, o0[3], o1[3], o2[3];  // o2 only in fixed point (in doubles it is the set's)
#if !ST_GRAD_IS_LINEAR
  double p0[3], v0[3];
#endif
  int on, scale;  // the fixed-point field scale (SegScale), packed
  int flags, grade;    // (grade: the field's, SegScale::ok)
};
static_assert(!ST_GRAD_IS_LINEAR || sizeof(SegRec) == 112, "the memory figures given for the rings");
// SegRec::flags: window end reached, particle stopped, bounce, gas collision, field in fixed
// point, start of a new particle (its index in t0); bits 8-15 sanity failure code.
enum { R_FIN = 1, R_STOP = 2, R_WALL = 4, R_GAS = 8, R_FX = 16, R_FETCH = 32 };

// Trajectory fields of a particle's state.
struct alignas(16) TrajState {
  double t, px, py, pz, vx, vy, vz, next_gas, spare;
  uint64_t rx, ry, rz, rw;
  int marks, pad;  // last collision | wall << 8 | spare valid << 16
};
__device__ __forceinline__ TrajState traj_of(const PState& p) {
  return {p.t, p.px, p.py, p.pz, p.vx, p.vy, p.vz, p.next_gas, p.rng.spare, p.rng.x, p.rng.y, p.rng.z, p.rng.w,
          (int)(uint8_t)p.coll | (int)(uint8_t)p.wall << 8 | (p.rng.has ? 1 << 16 : 0), 0};
}
__device__ __forceinline__ void traj_into(PState& p, const TrajState& s) {
  p.t = s.t;
  p.px = s.px; p.py = s.py; p.pz = s.pz;
  p.vx = s.vx; p.vy = s.vy; p.vz = s.vz;
  p.next_gas = s.next_gas;
  p.rng.spare = s.spare;
  p.rng.x = s.rx; p.rng.y = s.ry; p.rng.z = s.rz; p.rng.w = s.rw;
  p.coll = (char)(s.marks & 0xff);
  p.wall = (char)((s.marks >> 8) & 0xff);
  p.rng.has = (s.marks >> 16) != 0;
}

// A lane's scratch: the trajectory side's state between phases, the window-end slots, the ring.
__host__ __device__ constexpr size_t ahead_lane_bytes(int q) {
  return (size_t)(1 + kAheadSlots) * sizeof(TrajState) + (size_t)q * sizeof(SegRec);
}

// ---- adjoint tape (TAPE instantiation only)
// Cursor of one particle's two tape chains.
struct TapeCursor {
  int sp, sf, gp, gf;  // step chain: last page and its records; segment chain likewise
  long long ns, ng;    // records counted (stored or not)
  bool ok;             // every record so far was stored
};

__device__ __forceinline__ void tape_open(TapeCursor& c) {
  c.sp = -1;
  c.sf = kTapeStepsPerPage;
  c.gp = -1;
  c.gf = kTapeSegsPerPage;
  c.ns = c.ng = 0;
  c.ok = true;
}

// Address of a chain's next record, or null once the pool has run out (the
// particle's tape is then incomplete and is rebuilt by a replay).
__device__ __forceinline__ double* tape_slot(const TapeArgs& t, int& page, int& fill, int per_page, int rec_d,
                                             bool& ok) {
  if (!ok) return nullptr;
  if (fill == per_page) {
    const unsigned long long np = atomicAdd(t.pool_head, 1ull);
    if (np >= (unsigned long long)t.pool_pages) {
      ok = false;
      return nullptr;
    }
    t.page_prev[np] = page;
    page = (int)np;
    fill = 0;
  }
  return t.pool + (size_t)page * kTapePageD + (size_t)(fill++) * rec_d;
}

__device__ __forceinline__ void tape_step(const TapeArgs& t, TapeCursor& c, double yx, double yy, double yz, double x,
                                          double hs) {
  ++c.ns;
  double* r = tape_slot(t, c.sp, c.sf, kTapeStepsPerPage, kTapeStepD, c.ok);
  if (r) {
    r[0] = yx; r[1] = yy; r[2] = yz; r[3] = x; r[4] = hs;
  }
}

__device__ __forceinline__ void tape_seg(const TapeArgs& t, TapeCursor& c, const SegStart& s0) {
  ++c.ng;
  double* r = tape_slot(t, c.gp, c.gf, kTapeSegsPerPage, kTapeSegD, c.ok);
  if (r) {
    r[0] = s0.t;
    r[1] = s0.px; r[2] = s0.py; r[3] = s0.pz;
    r[4] = s0.vx; r[5] = s0.vy; r[6] = s0.vz;
    r[7] = 0.0;
  }
}

// A particle's segment (trajectory side) or step (spin side) cursor at its
// fetch: a fresh chain, or (append) the chain the previous launch closed,
// continued.
__device__ __forceinline__ void tape_resume_segs(const TapeArgs& t, TapeCursor& c, int64_t i) {
  tape_open(c);
  if (!t.append) return;
  c.gp = t.seg_page[i];
  c.gf = c.gp < 0 ? kTapeSegsPerPage : t.seg_fill[i];
  c.ng = t.nsegs[i];
  c.ok = t.complete[i] != 0;
}
__device__ __forceinline__ void tape_resume_steps(const TapeArgs& t, TapeCursor& c, int64_t i) {
  tape_open(c);
  if (!t.append) return;
  c.sp = t.step_page[i];
  c.sf = c.sp < 0 ? kTapeStepsPerPage : t.step_fill[i];
  c.ns = t.nsteps[i];
}

// Close a chain.  The trajectory side runs ahead, so it closes a particle's
// segments first; the particle's tape is complete when both sides stored everything.
__device__ __forceinline__ void tape_close_segs(const TapeArgs& t, const TapeCursor& c, int64_t i) {
  t.seg_page[i] = c.gp;
  t.seg_fill[i] = c.gp < 0 ? 0 : c.gf;
  t.nsegs[i] = c.ng;
  t.complete[i] = c.ok ? 1 : 0;
}
__device__ __forceinline__ void tape_close_steps(const TapeArgs& t, const TapeCursor& c, int64_t i) {
  t.step_page[i] = c.sp;
  t.step_fill[i] = c.sp < 0 ? 0 : c.sf;
  t.nsteps[i] = c.ns;
  if (!c.ok) t.complete[i] = 0;
}

// View of state checkpoint k (same field layout as checkpoint 0, k * stride
// bytes on; the set indices are shared by every slot).
__device__ __forceinline__ DeviceState state_slot(const DeviceState& b, int64_t stride, int k) {
  DeviceState s = b;
  const int64_t o = stride * (int64_t)k;
#define ST_OFF(f) s.f = reinterpret_cast<decltype(s.f)>(reinterpret_cast<char*>(b.f) + o);
  ST_OFF(t) ST_OFF(px) ST_OFF(py) ST_OFF(pz) ST_OFF(vx) ST_OFF(vy) ST_OFF(vz) ST_OFF(Sx) ST_OFF(Sy) ST_OFF(Sz)
  ST_OFF(h) ST_OFF(next_gas) ST_OFF(rx) ST_OFF(ry) ST_OFF(rz) ST_OFF(rw) ST_OFF(rspare) ST_OFF(rhas) ST_OFF(fail)
  ST_OFF(n_coll) ST_OFF(n_bounce) ST_OFF(n_steps) ST_OFF(stop) ST_OFF(coll) ST_OFF(wall) ST_OFF(w_done)
  ST_OFF(turns)
#undef ST_OFF
  return s;
}

// A record's field scale in two words.
__device__ __forceinline__ int pack_exps(const fx::SegScale& s) { return (int)((unsigned)s.oe << 16) | (s.te & 0xffff); }
__device__ __forceinline__ fx::SegScale unpack_scale(int on, int exps, int grade) {
  fx::SegScale s;
  s.on = fx::bits_f32((uint32_t)on);
  s.oe = exps >> 16;
  s.te = (int)(short)(exps & 0xffff);
  s.se = 0;
  s.ok = grade;
  return s;
}

// One trajectory event of a lane into ring record r.  Returns its flags.
template <bool TAPE, bool GAS, bool EXT, bool FX>
__device__ __forceinline__ int produce_record(PState& tp, const SetParams& P, double tf, SegRec* r, EventDefer& dd,
                                              const TapeArgs& ta, TapeCursor& tc) {
  SegStart s0;
  tp.n_bounce = tp.n_coll = 0;
  const bool fin = traj_event<true, GAS>(tp, P, tf, s0, &dd);
  int flags = (fin ? R_FIN : 0) | (tp.stop ? R_STOP : 0) | (tp.n_bounce != 0 ? R_WALL : 0) | (tp.n_coll != 0 ? R_GAS : 0) |
              ((tp.fail & 0xff) << 8);
  r->t0 = s0.t;
  r->t1 = tp.t;
  if (spin_on<EXT>(P.integrator)) {
    SegPoly q;
    seg_poly<FX>(q, P, s0, tp.t);
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      r->o0[c] = q.o0[c];
      r->o1[c] = q.o1[c];
      if (FX) r->o2[c] = q.o2[c];
    }
#if !ST_GRAD_IS_LINEAR
    r->p0[0] = s0.px; r->p0[1] = s0.py; r->p0[2] = s0.pz;
    r->v0[0] = s0.vx; r->v0[1] = s0.vy; r->v0[2] = s0.vz;
#endif
    if (q.fx) {
      r->on = (int)fx::f32_bits(q.sc.on);
      r->scale = pack_exps(q.sc);
      r->grade = q.sc.ok;
      flags |= R_FX;
    }
  }
  // the segments the spin side integrates, in order
  if (TAPE && !tp.stop && tp.fail == 0) tape_seg(ta, tc, s0);
  r->flags = flags;
  return flags;
}

enum BatchedMode { B_FETCH = 0, B_NEED = 1, B_SEG = 2, B_WEND = 3, B_DONE = 4 };

// Diffuse reflections and Maxwell-Boltzmann gas collisions are deferred
// (traj_event<true>): a lane with one pending produces no further records
// until the warp computes the pending events together (deferred_events_warp),
// when defer_k lanes have one or nothing else can go on.
// starve: the spin phase ends when this many lanes have run dry (or every lane
// that could go on has).  keep: the trajectory phase goes on while this many
// lanes have room (or one is dry).
// TAPE: also write the adjoint tape (steps and segments of every particle)
// and state checkpoints at every ta.ckpt_every-th window end.
// GAS = false: the instantiation for launches without gas collisions.
// EXT: also integrator types 2-5.  FX: with fixed-point steps (seg_scale).
template <int BLOCK, int MINB, bool TAPE, bool GAS, bool EXT, bool FX>
__global__ void __launch_bounds__(BLOCK, MINB) k_batched(RunArgs a, int starve, int keep, int defer_k, TapeArgs ta) {
  extern __shared__ double st_smem[];
  // DOP853 stage derivatives
  char* stages = reinterpret_cast<char*>(st_smem);
  fx::StageSmem ks{reinterpret_cast<fx::Limb2*>(stages) + threadIdx.x,
                   reinterpret_cast<fx::Limb*>(stages + 12 * sizeof(fx::Limb2) * BLOCK) + threadIdx.x, BLOCK};
  const unsigned FULL = 0xffffffffu;
  const int QCAP = a.ahead_q;
  const int lane = threadIdx.x & 31;
  // (lanes without particles share the last one's scratch, and only ever read it)
  char* const mine = a.ahead + ((((size_t)blockIdx.x * BLOCK + threadIdx.x) >> 5) * a.spread + min(lane, a.spread - 1)) *
                                   ahead_lane_bytes(QCAP);
  TrajState* const slots = reinterpret_cast<TrajState*>(mine);  // [0]: between phases, [1 + k]: window ends
  SegRec* const ring = reinterpret_cast<SegRec*>(slots + 1 + kAheadSlots);
  // ---- trajectory side
  int64_t ti = 0;
  int tw = 0, twl = 0;
  bool t_run = false, t_done = lane >= a.spread, t_wend = false, t_stop = false;
  // ---- ring and window slots (records and slots in use)
  int qhead = 0, qcount = 0, whead = 0, wcount = 0, waiting = 0;  // waiting: particles in the ring
  // ---- spin side
  int mode = B_NEED;
  int64_t i = 0;
  const SetParams* P = a.sets;
  Seg g;
  g.carry = false;
  double Sx = 0.0, Sy = 0.0, Sz = 0.0, ph = 0.0, tempH = 0.0;
  uint64_t n_steps = 0, s_ncoll = 0, s_nbounce = 0;
  int s_fail = 0, turns = 0, w = 0, wlast = 0;
  bool s_stop = false, s_slot = false, cur_fin = false, skip = false;
  unsigned long long n_dop = 0, n_rk = 0, n_ext = 0, n_seg = 0;
  unsigned int tick = 0, dry = 0;
  bool hit = false;
  const unsigned long long dl = run_deadline(a);
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  TapeCursor tcg, tcs;  // segment chain (trajectory side), step chain (spin side)
  tape_open(tcg);
  tape_open(tcs);
  while (true) {
    // ================================================================ trajectory phase
    {
      PState tp;
      tp.stop = false;
      tp.fail = 0;
      tp.Sx = tp.Sy = tp.Sz = tp.h = 0.0;
      tp.turns = 0;
      tp.n_coll = tp.n_bounce = tp.n_steps = 0;
      traj_into(tp, slots[0]);
      const SetParams* tP = a.sets;
      double tf = 0.0;
      if (t_run) {
        tP = &a.sets[a.s.set[ti]];
        tf = ((double)tw + 1.0) * tP->ioutInt;
      }
      // A ring may hold many particles of few segments.  A lane takes them all while plenty wait; of
      // the last ones, only one beside the one that its spin side is on, so that no lane holds many
      // while others go without.
      const bool plenty = *((volatile unsigned long long*)&a.status->queue_head) +
                              4ull * gridDim.x * (BLOCK / 32) * a.spread <=
                          (unsigned long long)a.nitems;
      EventDefer dd;  // every field set: the warp's flush shuffles them from every lane
#pragma unroll
      for (int k = 0; k < 7; ++k) dd.x[k] = 0.0;
      dd.wall = 'x';
      dd.pending = false;
      dd.gas = false;
      dd.spare_first = false;
#pragma unroll 1
      for (int round = 0; round < (1 << 20); ++round) {
        // a finished window (or a stopped particle): its state into a slot, once the
        // last reflection's velocity is known
        if (t_wend && !dd.pending && wcount < kAheadSlots) {
          int k = whead + wcount;
          if (k >= kAheadSlots) k -= kAheadSlots;
          slots[1 + k] = traj_of(tp);
          ++wcount;
          t_wend = false;
          ++tw;
          if (t_stop || tw >= twl) {
            t_run = false;
            if (TAPE) tape_close_segs(ta, tcg, ti);
          } else {
            tf = ((double)tw + 1.0) * tP->ioutInt;
          }
          t_stop = false;
        }
        // the next particle
        if (!t_run && !t_done && qcount < QCAP && (plenty || waiting == 0)) {
          const unsigned long long item = atomicAdd(&a.status->queue_head, 1ull);
          if (item >= (unsigned long long)a.nitems) {
            t_done = true;
          } else {
            ti = a.order ? a.order[item] : (int64_t)item;
            tP = &a.sets[a.s.set[ti]];
            tw = a.s.w_done[ti];
            twl = min(a.w_end, tP->nwin);
            if (TAPE) tape_resume_segs(ta, tcg, ti);
            if (tw < twl) {
              int k = qhead + qcount;
              if (k >= QCAP) k -= QCAP;
              ring[k].t0 = __longlong_as_double((long long)ti);
              ring[k].flags = R_FETCH;
              ++qcount;
              ++waiting;
              tp = load_state(a.s, ti);
              t_run = !tp.stop;  // a particle that stopped before: the spin side carries it to the end
              tp.stop = false;
              tp.fail = 0;
              tf = ((double)tw + 1.0) * tP->ioutInt;
            }
            if (TAPE && !t_run) {
              tape_close_segs(ta, tcg, ti);
              if (tw >= twl) {  // nothing to run: its step chain as it was
                TapeCursor same;
                tape_resume_steps(ta, same, ti);
                tape_close_steps(ta, same, ti);
              }
            }
          }
        }
        const bool prod = t_run && !t_wend && !dd.pending && qcount < QCAP;
        const unsigned pm = __ballot_sync(FULL, prod);
        const unsigned defer_m = __ballot_sync(FULL, dd.pending);
        const bool more = prod || (!t_run && !t_done && qcount < QCAP && (plenty || waiting == 0)) || (t_wend && wcount < kAheadSlots);
        const unsigned mm = __ballot_sync(FULL, more);
        const bool leave = mm == 0u || (__popc(mm) < keep && !__any_sync(FULL, more && qcount == 0));
        if (defer_m != 0u && (__popc(defer_m) >= defer_k || pm == 0u || leave)) {
          deferred_events_warp<GAS>(tp, *tP, dd, defer_m, lane);
          continue;
        }
        if (leave) break;
        if (prod) {
          int k = qhead + qcount;
          if (k >= QCAP) k -= QCAP;
          const int flags = produce_record<TAPE, GAS, EXT, FX>(tp, *tP, tf, ring + k, dd, ta, tcg);
          ++qcount;
          ++n_seg;
          t_stop = (flags & R_STOP) != 0;
          t_wend = t_stop || (flags & R_FIN) != 0;
        }
        if (((++tick) & 255u) == 0u && __any_sync(FULL, past_deadline(dl))) {
          hit = true;
          break;
        }
      }
      if (lane < a.spread) slots[0] = traj_of(tp);
      if (hit) break;
    }
    // ================================================================ spin phase
    bool moved = false;
#pragma unroll 1
    while (true) {
      // ---- boundaries of this lane: pop records, window ends, particles
      bool starved = false;
#pragma unroll 1
      for (int guard = 0; guard < 8; ++guard) {
        if (mode == B_NEED) {
          if (qcount == 0) {
            if (t_done && !t_run)
              mode = B_DONE;
            else
              starved = true;
            break;
          }
          const SegRec* r = ring + qhead;
          qhead = (qhead + 1 == QCAP) ? 0 : qhead + 1;
          --qcount;
          moved = true;
          const int flags = r->flags;
          if (flags & R_FETCH) {
            --waiting;
            skip = false;
            i = (int64_t)__double_as_longlong(r->t0);
            P = &a.sets[a.s.set[i]];
            w = a.s.w_done[i];
            wlast = min(a.w_end, P->nwin);
            Sx = a.s.Sx[i]; Sy = a.s.Sy[i]; Sz = a.s.Sz[i];
            ph = tempH = a.s.h[i];
            n_steps = a.s.n_steps[i];
            s_ncoll = a.s.n_coll[i];
            s_nbounce = a.s.n_bounce[i];
            s_fail = a.s.fail[i];
            turns = a.s.turns[i];
            s_stop = a.s.stop[i] != 0;
            s_slot = false;
            if (TAPE) tape_resume_steps(ta, tcs, i);
            if (s_stop) mode = B_WEND;
            continue;
          }
          if (skip) {  // records past a stepper failure
            if (flags & (R_FIN | R_STOP)) {
              whead = (whead + 1 == kAheadSlots) ? 0 : whead + 1;
              --wcount;
            }
            continue;
          }
          if (flags & R_WALL) ++s_nbounce;
          if (flags & R_GAS) ++s_ncoll;
          cur_fin = (flags & R_FIN) != 0;
          const int code = (int)(signed char)((flags >> 8) & 0xff);
          if (code != 0 || (flags & R_STOP)) {  // without a code: a diffuse hit on an edge or corner
            if (code != 0) s_fail = code;
            s_stop = s_slot = true;
            Sx = Sy = Sz = nan;
            g.carry = false;
            n_steps += 1;
            mode = B_WEND;
          } else if (spin_on<EXT>(P->integrator)) {
            SegPoly q;
            q.fx = (flags & R_FX) != 0;
            if (FX) q.sc = unpack_scale(r->on, r->scale, r->grade);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              q.o0[c] = r->o0[c];
              q.o1[c] = r->o1[c];
              if (FX) q.o2[c] = r->o2[c];
            }
            seg_open<FX>(g, *P, q, r->t0, r->t1);
#if !ST_GRAD_IS_LINEAR
            g.p0x = r->p0[0]; g.p0y = r->p0[1]; g.p0z = r->p0[2];
            g.v0x = r->v0[0]; g.v0y = r->v0[1]; g.v0z = r->v0[2];
#endif
            spin_begin<EXT, FX>(g, *P, Sx, Sy, Sz, tempH);
            mode = B_SEG;
            break;
          } else {  // trajectory only: the segment completes at once
            n_steps += 1;
            if (cur_fin) {
              s_slot = true;
              mode = B_WEND;
            }
          }
        } else if (mode == B_WEND) {
          PState out;
          if (s_slot) {
            if (wcount == 0) {  // the trajectory side has not got round to it (slots were full)
              starved = true;
              break;
            }
            traj_into(out, slots[1 + whead]);
            whead = (whead + 1 == kAheadSlots) ? 0 : whead + 1;
            --wcount;
          } else {
            out = load_state(a.s, i);  // stopped: the trajectory fields stay (or become NaN)
          }
          spin_settle<FX>(g, *P, Sx, Sy, Sz);
          out.Sx = Sx; out.Sy = Sy; out.Sz = Sz;
          out.h = ph;
          out.turns = turns;
          out.n_steps = n_steps;
          out.n_coll = s_ncoll;
          out.n_bounce = s_nbounce;
          out.fail = s_fail;
          out.stop = s_stop;
          if (s_stop) nan_fill(out);
          s_slot = false;
          moved = true;
          write_snap(a, i, w, out);
          ++w;
          store_state(a.s, i, out);  // every window end is a resumable checkpoint
          a.s.w_done[i] = w;
          if (TAPE && ta.ckpt_every > 0 && w % ta.ckpt_every == 0 && w / ta.ckpt_every < ta.ckpt_count) {
            const DeviceState ck = state_slot(ta.ckpt, ta.ckpt_stride, w / ta.ckpt_every);
            store_state(ck, i, out);
            ck.w_done[i] = w;
          }
          if (TAPE && w >= wlast) tape_close_steps(ta, tcs, i);
          tempH = ph;
          mode = (w < wlast && s_stop) ? B_WEND : B_NEED;
        } else {
          break;  // B_SEG or B_DONE
        }
      }
      const unsigned seg_m = __ballot_sync(FULL, mode == B_SEG);
      const unsigned starved_m = __ballot_sync(FULL, starved);
      const unsigned busy_m = __ballot_sync(FULL, mode == B_NEED || mode == B_WEND);
      if (starved_m != 0u && (__popc(starved_m) >= starve || seg_m == 0u)) break;
      if (seg_m == 0u) {
        if (busy_m == 0u) break;  // every lane done
        continue;                 // lanes with more boundaries than one pass takes
      }
      moved = true;
      // ---- one step attempt for every lane with an open segment
      if (mode == B_SEG) {
        int r;
        if (P->integrator == 0) {
          double y0x = Sx, y0y = Sy, y0z = Sz;
          if (TAPE && FX && g.fx) dop_spin(g, *P, y0x, y0y, y0z);
          const double x0 = g.x;
          r = dop_attempt_v<FX>(fx::Lane3(), ks, g, *P, Sx, Sy, Sz);
          ++n_dop;
          if (TAPE && g.acc) tape_step(ta, tcs, y0x, y0y, y0z, x0, g.hu);
        } else if (!EXT || P->integrator == 1) {
          r = rk45_attempt<FX>(g, *P, Sx, Sy, Sz);
          ++n_rk;
        } else {
          const double y0x = Sx, y0y = Sy, y0z = Sz, x0 = g.x;
          r = ext_attempt<FX>(g, *P, Sx, Sy, Sz);
          ++n_ext;
          if (TAPE && g.acc) tape_step(ta, tcs, y0x, y0y, y0z, x0, g.hu);
        }
        if (r != 0) {
          tempH = g.h;
          turns += g.turns;
          if (P->keep) ph = tempH;
          if (r < 0) {
            s_fail = r;
            s_stop = true;
            Sx = Sy = Sz = nan;
            g.carry = false;
            if (t_run && ti == i) {  // the trajectory side is still on this particle: it goes to the next
              t_run = t_wend = t_stop = false;
              qcount = wcount = 0;
              if (TAPE) tape_close_segs(ta, tcg, i);
            } else {
              skip = true;
              if (cur_fin) {
                whead = (whead + 1 == kAheadSlots) ? 0 : whead + 1;
                --wcount;
              }
            }
          }
          n_steps += 1;
          s_slot = cur_fin && !s_stop;
          mode = (cur_fin || s_stop) ? B_WEND : B_NEED;
        }
      }
      if (((++tick) & 255u) == 0u && __any_sync(FULL, past_deadline(dl))) {
        hit = true;
        break;
      }
    }
    if (hit) break;
    if (__all_sync(FULL, mode == B_DONE)) break;
    // a starved lane always gets a record in the next trajectory phase; this bound only
    // protects the device from a logic error
    dry = __any_sync(FULL, moved) ? 0u : dry + 1u;
    if (dry > 1000000u) {
      hit = true;
      atomicExch(&a.status->pad, 1);
      break;
    }
  }
  if (hit) atomicExch(&a.status->deadline_hit, 1);
  if (a.count_work) {
    warp_add(&a.status->dop_attempts, n_dop);
    warp_add(&a.status->rk45_attempts, n_rk);
    if (EXT) warp_add(&a.status->ext_attempts, n_ext);
    warp_add(&a.status->segments, n_seg);
  }
}

// ------------------------------------------------------------------ EXT instantiations
// The adjoint's record pass: the trajectory-ahead kernel with its tape on, in
// one configuration.
constexpr int kTapeBlock = 64, kTapeQcap = 64;

// Defined in st_kernels_fp64.cu: the kernel of persistent variant v, and the record pass, for runs in
// which no set steps in fixed point.
const void* variant_fn_fp64(int v, bool gas);
const void* tape_fn_fp64(bool gas);
// Defined in st_kernels_ext.cu: the kernel of persistent variant v with
// integrator types 2-5, the record pass with them (gas-capable), and the plain
// kernel's launch with them.
const void* variant_fn_ext(int v);
const void* tape_fn_ext();
int launch_plain_ext(const RunArgs& a, int window, double next_t, int block, void* stream);

}  // namespace st
