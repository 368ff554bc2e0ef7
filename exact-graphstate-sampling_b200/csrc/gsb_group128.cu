// Instantiations of the complex128 fused passes (gsb_group.cuh): with a barrier per tile, and warp-specialised for chain
// passes with tiles of 2^8 classes or more (one class per step thread).
#include "gsb_group.cuh"
#include "gsb_pick.h"

namespace gsb {

template <> void *pick_group128<GSB_SLOTS>(int d, int tr, bool ws) {
    if (tr) return d == 2 ? (void *)k_group<double2, double, 2, 1, GSB_SLOTS> : (void *)k_group<double2, double, 1, 1, GSB_SLOTS>;
    if (ws) return d == 3 ? (void *)k_group<double2, double, 3, 0, GSB_SLOTS, 2, true> : (void *)k_group<double2, double, 2, 0, GSB_SLOTS, 2, true>;
    return d == 3 ? (void *)k_group<double2, double, 3, 0, GSB_SLOTS> : (void *)k_group<double2, double, 2, 0, GSB_SLOTS>;
}

}  // namespace gsb
