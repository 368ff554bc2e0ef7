// Instantiation of the warp-specialised complex64 FP32 fused chain pass of three steps (gsb_group.cuh).
#include "gsb_group.cuh"
#include "gsb_pick.h"

namespace gsb {

template <> void *pick_group_ws_three<GSB_SLOTS>() { return (void *)k_group<float2, float, 3, 0, GSB_SLOTS, 2, true>; }

}  // namespace gsb
