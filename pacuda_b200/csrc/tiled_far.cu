// The on-chip executor for launches with a plan of more than 65536 folded entries (many distinct pairs of
// scale and factor). Its kernels stand in a file of their own, which is loaded when such a plan first runs.
#include "../../include/pacman_recurrence.h"
#include "tiled.cuh"

namespace pacuda {
namespace {

template <class K> const void *far_of(bool abi) {
    return abi ? (const void *)run_tiled<K, true, true> : (const void *)run_tiled<K, false, true>;
}

}  // namespace

const void *tiled_far_kernel(int kernel, bool abi) {
    switch (kernel) {
    case PACMAN_RECURRENCE_KERNEL_F64: return far_of<KindF64>(abi);
    case PACMAN_RECURRENCE_KERNEL_MIXED: return far_of<KindMixed>(abi);
    case PACMAN_RECURRENCE_KERNEL_MIXED64: return far_of<KindMixed64>(abi);
    default: return far_of<KindDF64>(abi);
    }
}

}  // namespace pacuda
