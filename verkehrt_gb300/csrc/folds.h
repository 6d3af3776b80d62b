// The folds of the kernel families as types and words: their element widths, sum types and identities.
#pragma once

#include "vkc_internal.h"

namespace vkc {

typedef unsigned long long u64;

enum Fold { F_ADD = 0, F_MUL = 1, F_MIN = 2, F_MAX = 3, F_AND = 4, F_OR = 5, F_XOR = 6 };

__host__ __device__ constexpr int width_of(vkc_type t) {
    return t == VKC_F64 || t == VKC_I64 || t == VKC_U64 ? 8 : (t == VKC_F32 || t == VKC_I32 ? 4 : 1);
}
__host__ __device__ constexpr vkc_type sum_type(vkc_type t) {
    return t == VKC_I32 ? VKC_I64 : (t == VKC_U8 ? VKC_U64 : t);
}
__host__ __device__ constexpr bool is_float(vkc_type t) { return t == VKC_F64 || t == VKC_F32; }
__host__ __device__ constexpr bool is_signed_t(vkc_type t) { return t == VKC_I64 || t == VKC_I32; }

// Num::wrapping on the element type (elementwise.rs:386-400): truncate and widen back.
template <vkc_type T> __host__ __device__ constexpr u64 wrap(u64 v) {
    return T == VKC_I32 ? static_cast<u64>(static_cast<long long>(static_cast<int>(static_cast<unsigned>(v))))
           : (T == VKC_U8 || T == VKC_BOOL) ? (v & 0xffull) : v;
}

// scan.rs:99-120, :130-233 (identity): add/or/xor 0, mul 1, and all ones (bool: true), min the
// highest value (+inf), max the lowest (-inf).
template <vkc_type T, int F> __host__ __device__ constexpr u64 identity() {
    return F == F_ADD || F == F_OR || F == F_XOR ? 0ull
           : F == F_MUL ? 1ull
           : F == F_AND ? (T == VKC_BOOL ? 1ull : wrap<T>(~0ull))
           : F == F_MIN ? (T == VKC_F64 ? 0x7ff0000000000000ull
                           : T == VKC_F32 ? 0x7f800000ull
                           : T == VKC_I64 ? 0x7fffffffffffffffull
                           : T == VKC_I32 ? 0x7fffffffull
                           : T == VKC_U8 ? 0xffull : ~0ull)
                        : (T == VKC_F64 ? 0xfff0000000000000ull
                           : T == VKC_F32 ? 0xff800000ull
                           : T == VKC_I64 ? 0x8000000000000000ull
                           : T == VKC_I32 ? 0xffffffff80000000ull : 0ull);
}

// The scanner of scan_<fold>_T or scan_by_<fold>_T (k_scan_wide.cu, k_scan_narrow.cu).
struct ScannerImpl;
using FoldScanMake = ScannerImpl *(*)(vkc_ctx *);
FoldScanMake wide_scan(vkc_type t, int fold, bool by);    // 8-byte elements
FoldScanMake narrow_scan(vkc_type t, int fold, bool by);  // 4- and 1-byte elements

}  // namespace vkc
