// One rounded f64 add by integer steps, for the chains of dependent adds of the canonical order.
#pragma once

#include "kcommon.cuh"

namespace vkc {

constexpr unsigned long long MANT = 0xfffffffffffffull;
constexpr unsigned long long ONE52 = 1ull << 52;

__device__ __forceinline__ double as_f64(unsigned long long b) { return __longlong_as_double(static_cast<long long>(b)); }
__device__ __forceinline__ unsigned long long as_bits(double d) { return static_cast<unsigned long long>(__double_as_longlong(d)); }

// fl(s + x) on bits. When s is a positive normal in binade E >= -959, x is non-negative and below
// that binade and the sum stays in it, s = S u with u = 2^(E-52) and fl(s + x) = (S + RNE(x/u)) u
// with ties to the even S (the integer steps of seg_tf for one row); otherwise the FP64 add.
__device__ __forceinline__ unsigned long long add_bits(unsigned long long s, unsigned long long x) {
    const unsigned KE = static_cast<unsigned>(s >> 52);  // with the sign bit: a negative s is above 2047
    const unsigned ex = static_cast<unsigned>(x >> 52);  // likewise a negative x
    if (KE >= 64u && KE <= 2046u && ex < KE) {
        const unsigned k = min(KE - ex, 63u);  // zero and subnormal rows: k = 63, no increment
        const unsigned long long w = ((x & MANT) | ONE52) + (1ull << (k - 1));
        unsigned long long inc = w >> k;
        const unsigned long long S = (s & MANT) | ONE52;
        if ((w << (64 - k)) == 0) {  // exactly halfway: to the even neighbour
            inc -= 1;
            inc += (S + inc) & 1;
        }
        const unsigned long long S2 = S + inc;
        if (S2 < (ONE52 << 1)) return (static_cast<unsigned long long>(KE) << 52) | (S2 & MANT);
    }
    return as_bits(__dadd_rn(as_f64(s), as_f64(x)));
}

}  // namespace vkc
