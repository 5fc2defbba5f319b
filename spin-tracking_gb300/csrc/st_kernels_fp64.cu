// The window engine's kernels for runs in which no set steps in fixed point (beta, or an absolute
// tolerance far below the relative one, or RK45): steps inlined in FP64.  What
// bounds them is the FP64 pipe, so one occupancy per family suffices: a variant with
// more blocks per SM takes the same kernel, and the three-lane variants, whose
// point is the fixed-point step, the flattened one.  Compiled as its own translation
// unit, in parallel with st_kernels.cu; builds with edited field hooks have these in the
// places of the others.
#include "st_engine.cuh"
#include "st_split.cuh"

namespace st {

#if ST_GRAD_IS_LINEAR && ST_PULSE_IS_Z_COS
template <bool GAS>
static const void* variant_fn_g(int v) {
  switch (v) {
    case 0: return reinterpret_cast<const void*>(&k_persistent<128, 1, false, false>);
    case 1:
    case 17: return reinterpret_cast<const void*>(&k_persistent<128, 2, false, false>);
    case 2:
    case 18: return reinterpret_cast<const void*>(&k_persistent<128, 3, false, false>);
    case 3: return reinterpret_cast<const void*>(&k_persistent<64, 4, false, false>);
    case 4: return reinterpret_cast<const void*>(&k_persistent<256, 1, false, false>);
    case 14: return reinterpret_cast<const void*>(&k_split<3, 1, 2, 8, GAS, 0, 0, false>);
    case 15: return reinterpret_cast<const void*>(&k_split<6, 2, 1, 8, GAS, 0, 0, false>);
#if ST_TRAJ_CORRECTLY_ROUNDED
    case 16: return reinterpret_cast<const void*>(&k_split<8, 4, 1, 8, GAS, 184, 136, false>);
#else
    case 16: return nullptr;  // ptxas 13.0 crashes on this instantiation with CUDA's inline log/sin/cos/acos
#endif
    case 19: return reinterpret_cast<const void*>(&k_batched<256, 1, false, GAS, false, false>);
    default: return reinterpret_cast<const void*>(&k_batched<64, 4, false, GAS, false, false>);
  }
}
const void* variant_fn_fp64(int v, bool gas) { return gas ? variant_fn_g<true>(v) : variant_fn_g<false>(v); }
const void* tape_fn_fp64(bool gas) {
  return gas ? reinterpret_cast<const void*>(&k_batched<kTapeBlock, 4, true, true, false, false>)
             : reinterpret_cast<const void*>(&k_batched<kTapeBlock, 4, true, false, false, false>);
}
#else
const void* variant_fn_fp64(int, bool) { return nullptr; }
const void* tape_fn_fp64(bool) { return nullptr; }
#endif

}  // namespace st
