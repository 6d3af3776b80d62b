// The scans of 4- and 1-byte elements (src/kernels/scalar/scan.rs:284-326, :424-439), as passes of
// fold_scan.cuh.
#include "fold_scan.cuh"

namespace vkc {

template <vkc_type T> static FoldScanMake int_scan(int fold, bool by) {
    switch (fold) {
    case F_ADD: return scan_of<T, F_ADD>(by);
    case F_MUL: return scan_of<T, F_MUL>(by);
    case F_MIN: return scan_of<T, F_MIN>(by);
    case F_MAX: return scan_of<T, F_MAX>(by);
    case F_AND: return scan_of<T, F_AND>(by);
    case F_OR: return scan_of<T, F_OR>(by);
    default: return scan_of<T, F_XOR>(by);
    }
}

FoldScanMake narrow_scan(vkc_type t, int fold, bool by) {
    if (t == VKC_F32) return fold == F_MIN ? scan_of<VKC_F32, F_MIN>(by) : scan_of<VKC_F32, F_MAX>(by);
    if (t == VKC_I32) return int_scan<VKC_I32>(fold, by);
    if (t == VKC_U8) return int_scan<VKC_U8>(fold, by);
    return fold == F_AND ? scan_of<VKC_BOOL, F_AND>(by)
           : fold == F_OR ? scan_of<VKC_BOOL, F_OR>(by) : scan_of<VKC_BOOL, F_XOR>(by);
}

}  // namespace vkc
