// The scans of 8-byte elements beside the i64 sums, which are k_scan.cu's (src/kernels/scalar/scan.rs:284-326,
// :424-439), as passes of fold_scan.cuh.
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

FoldScanMake wide_scan(vkc_type t, int fold, bool by) {
    if (t == VKC_F64) return fold == F_MIN ? scan_of<VKC_F64, F_MIN>(by) : scan_of<VKC_F64, F_MAX>(by);
    return t == VKC_U64 ? int_scan<VKC_U64>(fold, by) : int_scan<VKC_I64>(fold, by);
}

}  // namespace vkc
