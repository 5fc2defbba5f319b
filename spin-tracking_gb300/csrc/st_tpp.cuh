// Three lanes per particle (k_tpp3): the threads-per-particle axis of the
// launch variants.  Lanes 3g, 3g+1, 3g+2 of a warp share particle g (ten per
// warp; lanes 30 and 31 idle).  The three run the trajectory, the window
// bookkeeping and the step controller together (the same instructions on the
// same values), and split the DOP853 stage arithmetic by spin component: lane
// 3g + c keeps component c of the stage derivatives and gets the other two of
// a cross product by shuffles.  The arithmetic is the single-lane kernel's
// fixed-point code over another lane view, so results are bit-identical.  For
// DOP853 runs only: the host offers these variants to no run with RK45 sets.
// Flattened loop shape (k_persistent): a group fetches a particle, runs its
// events inline and attempts steps when its segment is open.
#pragma once

#include "st_engine.cuh"

namespace st {

// One spin component per lane of a group of three.
struct Lane1 {
  static constexpr int N = 1;
  unsigned mask;  // the group's three lanes
  int base;       // its first lane
  int c;          // this lane's component
  __device__ __forceinline__ fx::Limb get(fx::Limb v, int comp) const {
    return {__shfl_sync(mask, v.h, base + comp), __shfl_sync(mask, v.l, base + comp)};
  }
  __device__ __forceinline__ void cross(const fx::Limb y[1], const fx::Limb w[1], fx::Acc k[1]) const {
    const int a = c == 2 ? 0 : c + 1, b = c == 0 ? 2 : c - 1;
    const fx::Limb ya = get(y[0], a), yb = get(y[0], b), wa = get(w[0], a), wb = get(w[0], b);
    k[0] = {0, fx::kHalfLimb};
    fx::mac(k[0], ya, wb);
    fx::mac(k[0], yb, fx::neg(wa));
  }
  __device__ __forceinline__ void gather(const fx::i64 v[1], fx::i64 all[3]) const {
#pragma unroll
    for (int k = 0; k < 3; ++k) all[k] = __shfl_sync(mask, v[0], base + k);
  }
  __device__ __forceinline__ bool any(bool b) const { return __any_sync(mask, b) != 0; }
  __device__ __forceinline__ int comp(int) const { return c; }
  __device__ __forceinline__ void pick(fx::i64 x, fx::i64 y, fx::i64 z, fx::i64 v[1]) const {
    v[0] = c == 0 ? x : (c == 1 ? y : z);
  }
};

template <int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) k_tpp3(RunArgs a) {
  const int lane = threadIdx.x & 31;
  Lane1 G;
  G.base = (lane / 3) * 3;
  G.c = lane - G.base;
  G.mask = 7u << G.base;
  const bool lead = G.c == 0;
  int mode = lane < 30 ? M_FETCH : M_DONE;
  int64_t i = 0;
  const SetParams* P = a.sets;
  PState p;
  Seg g;
  g.carry = false;
  int w = 0, wlast = 0;
  double tf = 0.0, tempH = 0.0;
  bool finished = false, hit = false;
  unsigned long long n_dop = 0, n_seg = 0;
  unsigned int tick = 0;
  const unsigned long long dl = run_deadline(a);
  while (mode != M_DONE) {
    // the group's boundaries (the three lanes take the same path)
    while (mode != M_SEG && mode != M_DONE) {
      if (mode == M_FETCH) {
        unsigned long long item = 0;
        if (lead) item = atomicAdd(&a.status->queue_head, 1ull);
        item = __shfl_sync(G.mask, item, G.base);
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
          if (lead) ++n_seg;
          if (p.fail == 0 && spin_on<false>(P->integrator)) {
            seg_setup<true>(g, *P, s0, p.t);
            spin_begin<false, true>(g, *P, p.Sx, p.Sy, p.Sz, tempH);
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
          bool late = ((++tick) & 255u) == 0u && past_deadline(dl);
          late = __shfl_sync(G.mask, late, G.base);  // one decision per group
          if (late) {
            hit = true;
            mode = M_DONE;
            break;
          }
        }
      }
      if (mode == M_WEND) {
        spin_settle<true>(g, *P, p.Sx, p.Sy, p.Sz);
        if (lead) {
          write_snap(a, i, w, p);
          store_state(a.s, i, p);  // every window end is a resumable checkpoint
          a.s.w_done[i] = w + 1;
        }
        ++w;
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
    // one step attempt of the group's open segment
    int r;
    if (P->integrator == 0) {
      fx::StageLocal<1> ks;
      r = dop_attempt_v<true>(G, ks, g, *P, p.Sx, p.Sy, p.Sz);
      if (lead) ++n_dop;
    } else {
      // runs with RK45 sets do not get this kernel (the host leaves these
      // variants out for them); if one did, its particles stop with an error
      if (lead) atomicExch(&a.status->pad, 1);
      r = -1;
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
    bool late = ((++tick) & 255u) == 0u && past_deadline(dl);
    late = __shfl_sync(G.mask, late, G.base);
    if (late) {
      hit = true;
      break;
    }
  }
  if (hit && lead) atomicExch(&a.status->deadline_hit, 1);
  if (a.count_work) {
    if (n_dop) atomicAdd(&a.status->dop_attempts, n_dop);
    if (n_seg) atomicAdd(&a.status->segments, n_seg);
  }
}

}  // namespace st
