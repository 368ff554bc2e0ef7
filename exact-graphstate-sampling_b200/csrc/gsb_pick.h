// The complex64 FP32 and the complex128 fused-pass kernels are instantiated in translation units of their
// own, so the library's objects compile in parallel; these return their addresses for cudaLaunchKernel.
#pragma once

// Each is compiled twice, for launches of one item and (GSB_SLOTS = 1) of several.
#ifndef GSB_SLOTS
#define GSB_SLOTS 0
#endif

namespace gsb {

template <bool SLOTS> void *pick_group_f32(int d, int tr);   // two CTAs per SM, one barrier per tile (gsb_group_f32.cu)
template <bool SLOTS> void *pick_group_ws(int d, int tr);    // warp-specialised, tiles of 2^9 classes or more (gsb_group_ws.cu)
template <bool SLOTS> void *pick_group_ws_three();           // the same, three steps (gsb_group_ws3.cu)
template <bool SLOTS> void *pick_group_ws_trailing(int d);   // the same with a trailing step, tr = 1 (gsb_group_wst.cu)
template <bool SLOTS> void *pick_group3(int d, int tr);      // three CTAs per SM (gsb_group3.cu)
template <bool SLOTS> void *pick_group128(int d, int tr, bool ws);   // complex128 (gsb_group128.cu)

}  // namespace gsb
