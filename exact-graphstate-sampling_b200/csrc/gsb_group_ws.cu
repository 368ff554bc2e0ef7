// Instantiations of the warp-specialised complex64 FP32 fused chain passes (tiles of 2^9 classes or more,
// gsb_group.cuh): two steps here, three in gsb_group_ws3.cu, the sampling ones (a trailing step) in gsb_group_wst.cu.
#include "gsb_group.cuh"
#include "gsb_pick.h"

namespace gsb {

template <> void *pick_group_ws<GSB_SLOTS>(int d, int tr) {
    if (tr) return pick_group_ws_trailing<GSB_SLOTS>(d);
    return d == 3 ? pick_group_ws_three<GSB_SLOTS>() : (void *)k_group<float2, float, 2, 0, GSB_SLOTS, 2, true>;
}

}  // namespace gsb
