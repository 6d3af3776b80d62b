// reduce_into_add_f64: per-bucket float sums. The reference has no float reduce_into (the gap
// is listed at src/kernels/scalar/scan.rs:408-415); its tier-2 design notes
// (docs/superpowers/specs/2026-10-31-verkehrt-tier2-design.md:171-172) give the candidate order
// this entry computes: rows below b = n - n % 16 go to stripe i mod 16 of their bucket, each
// stripe adds its rows in index order from +0.0, and the 16 stripes combine pairwise (+8, +4,
// +2, +1). The bucket's rows from b on then fold into the result in index order, the canonical
// sum's tail rule (reduce.rs:77-91, finish_lanes): under that reading the notes' property holds,
// with every key equal the bucket's sum has the bits of reduce_add_f64.
//
// Equivalently, out[k] is the canonical sum of the rows with every row of another bucket read as
// +0.0: a stripe starts at +0.0 and never holds -0.0 (a sum is -0.0 only when both terms are), so
// adding +0.0 leaves it unchanged. Three paths:
//  * very few buckets of many rows (rif_masks): that identity, per bucket: the masked rows, then
//    reduce_add_f64;
//  * otherwise the rows below b are sorted, stably, by (key, stripe), a 32-bit image whose radix
//    passes carry the values; each stripe of each bucket is then a contiguous chain that one thread
//    adds in index order, the sixteen of a bucket side by side, so that they combine by shuffles;
//    one thread folds the tail rows in order. Buckets with chains far longer than even keys give are
//    masked instead (rif_limit). (Until now an argsort, two gathers by its order and a
//    warp a chain whose 32 lanes all ran the chain: 4.36 ms against 0.72 for 33 M rows in 1024
//    buckets, 2.26 ms of it FP64 adds that 31 lanes repeated.)
//  * buckets so many that a table of their chains would dwarf the rows (rif_tables): the chains are
//    found by a scan over the sorted rows instead.
// Arguments and errors follow reduce_into_add_i64 (index.rs:194-222): the values' kind first,
// then the keys (checked_keys, index.rs:116-130), a length mismatch, the result's allocation.
#include <algorithm>
#include <vector>

#include "add_bits.cuh"
#include "radix.h"
#include "reduce_common.h"

namespace vkc {

vkc_status bucket_key_error(vkc_ctx *ctx, const long long *k, int64_t n, int64_t nb, bool *found);

// Measured: the masked path costs about 130 us a bucket and 7.2 us a bucket per million rows; the
// sorted one 100 us, 16 us per million rows and its longest chain at 40 ns a row, n / (16 nb) rows when
// the keys are even. Masked where that is less: up to 1 bucket of 2^17 rows, 4 of 2^20, 15 of 2^25.
static double rif_mask_us(int64_t n) { return 130.0 + 7.2e-6 * static_cast<double>(n); }
constexpr double RIF_CHAIN_US = 0.04;  // a row of a chain
static bool rif_masks(int64_t n, int64_t nb) {
    const double rows = static_cast<double>(n), k = static_cast<double>(nb);
    return k * rif_mask_us(n) < 100.0 + 16e-6 * rows + RIF_CHAIN_US * rows / (16.0 * k);
}
// Keys need not be even. A bucket with a chain of more rows than this is left out of the sorted path's
// first sums, which note it (RifHeavy): masked sums of such buckets follow where they take less than the
// longest chain, else the chains themselves. Twice the even chain, so that keys about even are summed at
// once; and rows that take as long as a bucket's masked sum. (2^25 rows, 95% of them in one of 16 / 1024
// buckets: 83.1 / 83.0 ms in chains, 0.95 / 0.88 ms so; 16 even ones 5.83 ms either way.)
static unsigned rif_limit(int64_t n, int64_t nb) {
    const double rows = std::max(rif_mask_us(n) / RIF_CHAIN_US, static_cast<double>(n) / (8.0 * static_cast<double>(nb)));
    return static_cast<unsigned>(std::min(rows, 4e9));
}
struct RifHeavy {
    static constexpr int MOST = 254;
    unsigned count, longest, bucket[MOST];  // all zero before the sums
};
// Images (key * 16 + stripe) of 32 bits, and a table of every chain no larger than a few rows' worth.
static bool rif_tables(int64_t n, int64_t nb) {
    return n < (int64_t(1) << 32) && nb <= (int64_t(1) << 28) && nb <= n + (int64_t(1) << 16);
}

// v[i] = x[i] for rows of bucket k, else +0.0.
__global__ void rif_mask_kernel(const long long *__restrict__ keys, const unsigned long long *__restrict__ x,
                                int64_t n, long long k, unsigned long long *__restrict__ v) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        v[i] = keys[i] == k ? x[i] : 0ull;
}

__global__ void rif_store_kernel(unsigned long long *out, int64_t k, unsigned long long bits) { out[k] = bits; }

// c[i] = key * 16 + stripe for the rows below b (keys are in range, below 2^59).
__global__ void rif_composite_kernel(const long long *__restrict__ keys, int64_t b, long long *__restrict__ c) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < b; i += stride)
        c[i] = keys[i] * 16 + (i & 15);
}

// heads[p] = 1 where a chain (one stripe of one bucket, in sorted order) starts.
__global__ void rif_heads_kernel(const long long *__restrict__ cs, int64_t b, unsigned *__restrict__ heads) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < b; p += stride)
        heads[p] = p == 0 || cs[p] != cs[p - 1];
}

// A warp per 32-row window of sorted positions: for each chain that starts in the window, in
// order, the warp reads the chain RIF_U x 32 rows at a time (all the loads in flight together;
// the rows of a chain are contiguous, so the lanes still in it are a prefix of each 32) and adds
// them in order from +0.0, every lane holding the same running sum; chain o (its ordinal among
// the heads) gets its composite key and sum. The window of the last row writes the number of
// chains.
constexpr int RIF_U = 8;
__global__ void __launch_bounds__(256) rif_chain_kernel(const long long *__restrict__ cs,
                                                        const unsigned long long *__restrict__ v, int64_t b,
                                                        const unsigned *__restrict__ heads,
                                                        const unsigned *__restrict__ ord,
                                                        long long *__restrict__ chain_key,
                                                        unsigned long long *__restrict__ chain_sum,
                                                        unsigned *__restrict__ nchains) {
    const int lane = threadIdx.x & 31;
    const int64_t p0 = (static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32;
    if (p0 >= b) return;
    const int64_t pl = p0 + lane;
    if (pl == b - 1) *nchains = ord[pl] + heads[pl];
    unsigned hm = __ballot_sync(FULL, pl < b && heads[pl] != 0);
    while (hm) {
        const int i = __ffs(hm) - 1;
        hm &= hm - 1;
        const int64_t p = p0 + i;
        const long long key = cs[p];
        double s = 0.0;
        for (int64_t q0 = p;; q0 += 32 * RIF_U) {
            bool in[RIF_U];
            double x[RIF_U];
#pragma unroll
            for (int u = 0; u < RIF_U; ++u) {
                const int64_t q = q0 + u * 32 + lane;
                in[u] = q < b && cs[q] == key;
                x[u] = q < b ? as_f64(v[q]) : 0.0;
            }
            bool more = true;
#pragma unroll
            for (int u = 0; u < RIF_U; ++u) {
                const unsigned m = __ballot_sync(FULL, in[u]);
                if (more) {
                    const int len = m == FULL ? 32 : __ffs(~m) - 1;
#pragma unroll 8
                    for (int j = 0; j < len; ++j) s = __dadd_rn(s, __shfl_sync(FULL, x[u], j));
                    more = len == 32;
                }
            }
            if (!more) break;
        }
        if (lane == 0) {
            chain_key[ord[p]] = key;
            chain_sum[ord[p]] = static_cast<unsigned long long>(__double_as_longlong(s));
        }
    }
}

// One thread per bucket that has chains: its stripes (+0.0 where a stripe has no rows) combine
// pairwise, +8, +4, +2, +1, into out[bucket].
__global__ void rif_combine_kernel(const long long *__restrict__ chain_key,
                                   const unsigned long long *__restrict__ chain_sum,
                                   const unsigned *__restrict__ nchains, unsigned long long *__restrict__ out) {
    const int64_t m = *nchains;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t o = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; o < m; o += stride) {
        const long long k = chain_key[o] >> 4;
        if (o > 0 && (chain_key[o - 1] >> 4) == k) continue;
        double s[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) s[j] = 0.0;
        for (int64_t o2 = o; o2 < m && (chain_key[o2] >> 4) == k; ++o2) s[chain_key[o2] & 15] = as_f64(chain_sum[o2]);
#pragma unroll
        for (int step = 8; step > 0; step >>= 1)
#pragma unroll
            for (int j = 0; j < step; ++j) s[j] = __dadd_rn(s[j], s[j + step]);
        out[k] = static_cast<unsigned long long>(__double_as_longlong(s[0]));
    }
}

// The rows from b on, fewer than 16, fold into their buckets in index order.
__global__ void rif_tail_kernel(const long long *__restrict__ keys, const unsigned long long *__restrict__ x,
                                int64_t b, int64_t n, uint64_t nb, unsigned long long *__restrict__ out) {
    for (int64_t i = b; i < n; ++i)
        if (static_cast<uint64_t>(keys[i]) < nb) out[keys[i]] = static_cast<unsigned long long>(__double_as_longlong(__dadd_rn(as_f64(out[keys[i]]), as_f64(x[i]))));
}

static vkc_status rif_tail(vkc_ctx *ctx, const long long *keys, const unsigned long long *x, int64_t b, int64_t n, int64_t nb,
                           unsigned long long *out) {
    if (b == n) return VKC_OK;
    rif_tail_kernel<<<1, 1, 0, ctx->stream>>>(keys, x, b, n, static_cast<uint64_t>(nb), out);
    return launched(ctx, "rif_tail");
}

// A whole entry of the table by name, on array arguments; the result array in *res.
static vkc_status call_whole(vkc_ctx *ctx, const char *name, std::initializer_list<const vkc_array *> arrays,
                             vkc_array **res) {
    const KernelDef *d = kernel_def(name);
    if (!d || !d->whole) return fail(ctx, VKC_USAGE, std::string("no entry ") + name);
    vkc_value in[4] = {};
    int k = 0;
    for (const vkc_array *a : arrays) {
        in[k].kind = VKC_VALUE_ARRAY;
        in[k].array = const_cast<vkc_array *>(a);
        ++k;
    }
    vkc_value out{};
    vkc_status st = d->whole(ctx, in, k, &out);
    *res = st ? nullptr : out.array;
    return st;
}

// ------------------------------------------------------------------ the sorted path

// Images of the rows below b (a row out of range gets image 0, so that no later kernel leaves its
// tables: the call fails), and the first key out of range among all n rows.
__global__ void __launch_bounds__(256) rif_images_kernel(const long long *__restrict__ keys, int64_t n, int64_t b, uint64_t nb,
                                                         unsigned *__restrict__ img, DevStatus *status) {
    constexpr int R = 4;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    unsigned long long bad = ~0ull;
    for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < n; i0 += R * stride) {
        unsigned long long k[R];
#pragma unroll
        for (int j = 0; j < R; ++j) k[j] = i0 + j * stride < n ? static_cast<unsigned long long>(__ldcs(keys + i0 + j * stride)) : 0ull;
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int64_t i = i0 + j * stride;
            if (i >= n) break;
            const bool ok = k[j] < nb;
            if (!ok && static_cast<unsigned long long>(i) < bad) bad = static_cast<unsigned long long>(i);
            if (i < b) img[i] = ok ? static_cast<unsigned>(k[j]) * 16u + static_cast<unsigned>(i & 15) : 0u;
        }
    }
    if (bad != ~0ull) atomicMin(&status->first_bad, bad);
}

// span[c] = the rows [x, y) of chain c among the sorted images (zeroed: empty chains).
__global__ void __launch_bounds__(256) rif_spans_kernel(const unsigned *__restrict__ img, int64_t b, uint2 *__restrict__ span) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x * 4;
    for (int64_t p = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 4; p < b; p += stride) {
        // b is a multiple of 16, so four images from p on are there.
        const uint4 q = *reinterpret_cast<const uint4 *>(img + p);
        const unsigned v[6] = {p ? img[p - 1] : ~q.x, q.x, q.y, q.z, q.w, p + 4 < b ? img[p + 4] : ~q.w};
#pragma unroll
        for (int j = 1; j < 5; ++j) {
            if (v[j] != v[j - 1]) span[v[j]].x = static_cast<unsigned>(p + j - 1);
            if (v[j] != v[j + 1]) span[v[j]].y = static_cast<unsigned>(p + j);
        }
    }
}

// Whether a bucket, whose sixteen chains lie in sixteen lanes from `lane` & 16 on, has a chain of more than
// `limit` rows; noted, and *flag set for the host, when `heavy` is given.
__device__ __forceinline__ bool rif_is_heavy(unsigned len, unsigned limit, int64_t bucket, RifHeavy *heavy, unsigned *flag) {
    unsigned most = len;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(FULL, most, o));
    if (most <= limit) return false;
    if (heavy && (threadIdx.x & 15) == 0) {
        const unsigned i = atomicAdd(&heavy->count, 1u);
        if (i < RifHeavy::MOST) heavy->bucket[i] = static_cast<unsigned>(bucket);
        atomicMax(&heavy->longest, most);
        *reinterpret_cast<volatile unsigned *>(flag) = 1u;
    }
    return true;
}

// One block per two buckets: a warp adds, one thread per chain, and a second warp copies the next
// RC_ROWS rows of each of the 32 chains into shared memory (each a coalesced run, RC_STAGES - 1
// stages ahead; by the adding warp itself the copies' issue took half as long again as the adds). A
// row of a chain costs 31 ns, the latency of an FP64 add. (add_bits, the adds as integer steps, took
// 110 ns: it pays where a chain's neighbours fill the pipe, not here.) With `heavy` the buckets with a
// chain beyond `limit` are noted there and left out.
constexpr int RC_ROWS = 32, RC_STAGES = 3, RC_PITCH = RC_ROWS + 1;

__global__ void __launch_bounds__(64) rif_sum_kernel(const uint2 *__restrict__ span, const unsigned long long *__restrict__ v,
                                                     int64_t nb, unsigned long long *__restrict__ out, unsigned limit,
                                                     RifHeavy *heavy, unsigned *flag) {
    __shared__ unsigned long long buf[RC_STAGES][32][RC_PITCH];
    const int lane = threadIdx.x & 31;
    const bool copies = threadIdx.x >= 32;
    for (int64_t pair = blockIdx.x; pair * 2 < nb; pair += gridDim.x) {
        const int64_t c = pair * 32 + lane;
        const uint2 s = c < nb * 16 ? span[c] : make_uint2(0u, 0u);
        const bool mine = !heavy || !rif_is_heavy(s.y - s.x, limit, c >> 4, copies ? nullptr : heavy, flag);
        const unsigned len = mine ? s.y - s.x : 0u, most = __reduce_max_sync(FULL, len);
        const int steps = static_cast<int>((static_cast<int64_t>(most) + RC_ROWS - 1) / RC_ROWS);
        auto issue = [&](int k) {
            if (k < steps) {
#pragma unroll 8
                for (int t = 0; t < 32; ++t) {
                    const unsigned first = __shfl_sync(FULL, s.x, t), n = __shfl_sync(FULL, len, t);
                    const unsigned r = static_cast<unsigned>(k) * RC_ROWS + lane;
                    if (r < n)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<unsigned>(
                                         __cvta_generic_to_shared(&buf[k % RC_STAGES][t][lane]))),
                                     "l"(v + first + r)
                                     : "memory");
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        if (copies)
            for (int k = 0; k < RC_STAGES - 1; ++k) issue(k);
        double acc = 0.0;
        for (int k = 0; k < steps; ++k) {
            if (copies) asm volatile("cp.async.wait_group %0;" ::"n"(RC_STAGES - 2) : "memory");
            __syncthreads();  // step k's rows have landed, and the buffer of step k - 1 is free
            if (copies) {
                issue(k + RC_STAGES - 1);
            } else {
                const unsigned done = static_cast<unsigned>(k) * RC_ROWS;
                const int rows = len > done ? static_cast<int>(min(len - done, static_cast<unsigned>(RC_ROWS))) : 0;
                const unsigned long long *x = buf[k % RC_STAGES][lane];
                int i = 0;
                for (; i + 8 <= rows; i += 8) {
                    double t[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) t[j] = as_f64(x[i + j]);
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc = __dadd_rn(acc, t[j]);
                }
                for (; i < rows; ++i) acc = __dadd_rn(acc, as_f64(x[i]));
            }
        }
        if (copies) asm volatile("cp.async.wait_group 0;" ::: "memory");
        // +8, +4, +2, +1 over the bucket's sixteen stripes.
        if (!copies) {
#pragma unroll
            for (int step = 8; step > 0; step >>= 1) {
                const double other = __shfl_down_sync(FULL, acc, step, 16);
                if ((lane & 15) < step) acc = __dadd_rn(acc, other);
            }
            if ((lane & 15) == 0 && c < nb * 16 && mine) out[c >> 4] = as_bits(acc);
        }
        __syncthreads();  // the buffers are free for the next pair
    }
}

// Many buckets of few rows: one thread per chain reads its rows itself, the chains of a warp lying
// side by side. (The staged form spends about 2 us a block on a pair of buckets however short: 2^20
// buckets of 2^20 rows took 883 us.)
constexpr int64_t RIF_SHORT_ROWS = 4;  // average rows of a chain below which this form runs
__global__ void __launch_bounds__(256) rif_short_kernel(const uint2 *__restrict__ span, const unsigned long long *__restrict__ v,
                                                        int64_t nb, unsigned long long *__restrict__ out, unsigned limit,
                                                        RifHeavy *heavy, unsigned *flag) {
    const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    uint2 s = c < nb * 16 ? span[c] : make_uint2(0u, 0u);
    const bool left_out = rif_is_heavy(s.y - s.x, limit, c >> 4, heavy, flag);
    if (left_out) s.y = s.x;
    double acc = 0.0;
    for (unsigned p = s.x; p < s.y; p += 4) {
        double t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) t[j] = p + j < s.y ? as_f64(v[p + j]) : 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j) acc = __dadd_rn(acc, t[j]);  // +0.0 changes no sum
    }
#pragma unroll
    for (int step = 8; step > 0; step >>= 1) {
        const double other = __shfl_down_sync(FULL, acc, step, 16);
        if ((threadIdx.x & 15) < step) acc = __dadd_rn(acc, other);
    }
    if ((threadIdx.x & 15) == 0 && c < nb * 16 && !left_out) out[c >> 4] = as_bits(acc);
}

// The masked path: for each of the buckets, reduce_add_f64 of the rows with the others read as +0.0.
static vkc_status rif_masked(vkc_ctx *ctx, const long long *keys, const unsigned long long *x, int64_t n,
                             const std::vector<unsigned> &buckets, unsigned long long *out) {
    vkc_array *v;
    vkc_status st = new_array(ctx, VKC_F64, n, false, &v);
    if (st) return st;
    const KernelDef *sum = kernel_def("reduce_add_f64");
    for (const unsigned k : buckets) {
        rif_mask_kernel<<<stream_grid(ctx, n, 256, 8, 4096), 256, 0, ctx->stream>>>(
            keys, x, n, k, static_cast<unsigned long long *>(v->data()));
        if ((st = launched(ctx, "rif_mask"))) break;
        ReducerImpl *r = sum->red(ctx);
        if (!r) {
            st = VKC_ALLOC;
            break;
        }
        Arg a{true, v, {}};
        vkc_scalar s{};
        st = r->update(ctx, &a, 1);
        if (!st) st = r->finish(ctx, &s);
        delete r;
        if (st) break;
        rif_store_kernel<<<1, 1, 0, ctx->stream>>>(out, k, s.bits);
        if ((st = launched(ctx, "rif_store"))) break;
    }
    vkc_array_release(v);
    return st;
}

// The sorted path and the rows from b on, waited for; *bad: some key is out of range (and no sum holds).
static vkc_status rif_sorted(vkc_ctx *ctx, const long long *keys, const unsigned long long *x, int64_t n, int64_t b,
                             int64_t nb, unsigned long long *out, bool *bad) {
    int passes = 1;  // of the image's bits: the largest is 16 nb - 1
    while (passes < 4 && ((16 * static_cast<uint64_t>(nb) - 1) >> (8 * passes))) ++passes;
    static const int shifts[4] = {0, 8, 16, 24};
    vkc_array *ia = nullptr, *ib = nullptr, *va = nullptr, *vb = nullptr, *ca = nullptr, *oa = nullptr, *sa = nullptr,
              *sp = nullptr;
    auto done = [&](vkc_status st) {
        for (vkc_array *a : {ia, ib, va, vb, ca, oa, sa, sp})
            if (a) vkc_array_release(a);
        return st;
    };
    int64_t cw, sw;
    radix_table_words(b, &cw, &sw);
    vkc_status st;
    void *h;
    if ((st = new_array(ctx, VKC_I32, b, false, &ia)) || (st = new_array(ctx, VKC_I32, b, false, &ib)) ||
        (st = new_array(ctx, VKC_F64, b, false, &va)) || (passes > 1 && (st = new_array(ctx, VKC_F64, b, false, &vb))) ||
        (st = new_array(ctx, VKC_I32, cw, false, &ca)) || (st = new_array(ctx, VKC_I32, cw, false, &oa)) ||
        (st = new_array(ctx, VKC_I32, sw, false, &sa)) ||
        (st = new_array(ctx, VKC_U64, 16 * nb + static_cast<int64_t>(sizeof(RifHeavy) / 8), true, &sp)) ||
        (st = pinned(ctx, sizeof(RifHeavy), &h)))
        return done(st);
    auto *first = static_cast<unsigned *>(ib->data());
    rif_images_kernel<<<stream_grid(ctx, n, 256, 8, 4096), 256, 0, ctx->stream>>>(keys, n, b, static_cast<uint64_t>(nb), first,
                                                                                  ctx->status);
    if ((st = launched(ctx, "rif_images"))) return done(st);
    const RadixTables t{static_cast<unsigned *>(ca->data()), static_cast<unsigned *>(oa->data()),
                        static_cast<unsigned *>(sa->data())};
    const RadixPairs<unsigned, unsigned long long> p{
        first, x, {static_cast<unsigned *>(ia->data()), first},
        {static_cast<unsigned long long *>(va->data()), vb ? static_cast<unsigned long long *>(vb->data()) : nullptr}};
    int at = 0;
    if ((st = radix_pairs(ctx, p, b, shifts, passes, t, &at))) return done(st);
    auto *span = static_cast<uint2 *>(sp->data());
    auto *heavy = reinterpret_cast<RifHeavy *>(span + 16 * nb);
    auto *flag = static_cast<unsigned *>(h);
    *flag = 0;
    const unsigned limit = rif_limit(n, nb);
    rif_spans_kernel<<<stream_grid(ctx, b / 4, 256, 8, 1024), 256, 0, ctx->stream>>>(p.img[at], b, span);
    // Every pair of buckets that fits a wave of resident blocks, then further ones by stride.
    const int pairs = static_cast<int>(std::min<int64_t>((nb + 1) / 2, static_cast<int64_t>(ctx->sms) * 8));
    if (b < RIF_SHORT_ROWS * 16 * nb)
        rif_short_kernel<<<static_cast<int>((16 * nb + 255) / 256), 256, 0, ctx->stream>>>(span, p.pay[at], nb, out, limit, heavy, flag);
    else
        rif_sum_kernel<<<pairs, 64, 0, ctx->stream>>>(span, p.pay[at], nb, out, limit, heavy, flag);
    if ((st = launched(ctx, "rif_sums"))) return done(st);
    if ((st = rif_tail(ctx, keys, x, b, n, nb, out))) return done(st);
    DevStatus ds;
    if ((st = read_status(ctx, &ds))) return done(st);
    *bad = ds.first_bad != ~0ull;
    if (*bad || !*flag) return done(VKC_OK);
    // Buckets with long chains: masked, the rows from b on among them, or their chains and then those rows.
    RifHeavy hv;
    VKC_CUDA(ctx, cudaMemcpyAsync(h, heavy, sizeof hv, cudaMemcpyDeviceToHost, ctx->stream));
    VKC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    memcpy(&hv, h, sizeof hv);
    if (hv.count <= RifHeavy::MOST && hv.count * rif_mask_us(n) < RIF_CHAIN_US * hv.longest) {
        st = rif_masked(ctx, keys, x, n, std::vector<unsigned>(hv.bucket, hv.bucket + hv.count), out);
        if (st != VKC_ALLOC) return done(st);
    }
    // (Every sum again: the others have their tail rows already.)
    rif_sum_kernel<<<pairs, 64, 0, ctx->stream>>>(span, p.pay[at], nb, out, 0u, nullptr, nullptr);
    if ((st = launched(ctx, "rif_sums"))) return done(st);
    if ((st = rif_tail(ctx, keys, x, b, n, nb, out))) return done(st);
    VKC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return done(VKC_OK);
}

// ------------------------------------------------------------------ the other paths

// Without a table of the chains, over the rows below b (b > 0).
static vkc_status rif_scanned(vkc_ctx *ctx, const vkc_array *keys, const vkc_array *vals, int64_t b,
                             unsigned long long *out) {
    vkc_array *c = nullptr, *perm = nullptr, *cs = nullptr, *v = nullptr, *heads = nullptr, *ord = nullptr,
              *sums = nullptr, *ckey = nullptr, *csum = nullptr;
    auto done = [&](vkc_status st) {
        for (vkc_array *a : {c, perm, cs, v, heads, ord, sums, ckey, csum})
            if (a) vkc_array_release(a);
        return st;
    };
    vkc_status st;
    if ((st = new_array(ctx, VKC_I64, b, false, &c))) return done(st);
    const int grid = stream_grid(ctx, b, 256, 8, 4096);
    rif_composite_kernel<<<grid, 256, 0, ctx->stream>>>(static_cast<const long long *>(keys->data()), b,
                                                        static_cast<long long *>(c->data()));
    if ((st = launched(ctx, "rif_composite"))) return done(st);
    if ((st = call_whole(ctx, "argsort_i64", {c}, &perm))) return done(st);
    if ((st = call_whole(ctx, "gather_i64", {c, perm}, &cs))) return done(st);
    if ((st = call_whole(ctx, "gather_f64", {vals, perm}, &v))) return done(st);
    const int64_t sw = scan_counts_sum_words(b);
    if ((st = new_array(ctx, VKC_I32, b, false, &heads)) || (st = new_array(ctx, VKC_I32, b, false, &ord)) ||
        (st = new_array(ctx, VKC_I32, sw + 1, false, &sums)) || (st = new_array(ctx, VKC_I64, b, false, &ckey)) ||
        (st = new_array(ctx, VKC_F64, b, false, &csum)))
        return done(st);
    auto *h = static_cast<unsigned *>(heads->data());
    auto *od = static_cast<unsigned *>(ord->data());
    auto *nchains = static_cast<unsigned *>(sums->data()) + sw;
    const auto *csp = static_cast<const long long *>(cs->data());
    rif_heads_kernel<<<grid, 256, 0, ctx->stream>>>(csp, b, h);
    scan_counts(ctx, h, b, static_cast<unsigned *>(sums->data()), od);
    rif_chain_kernel<<<static_cast<int>((b + 255) / 256), 256, 0, ctx->stream>>>(csp, static_cast<const unsigned long long *>(v->data()), b, h, od,
                                                    static_cast<long long *>(ckey->data()),
                                                    static_cast<unsigned long long *>(csum->data()), nchains);
    rif_combine_kernel<<<grid, 256, 0, ctx->stream>>>(static_cast<const long long *>(ckey->data()),
                                                      static_cast<const unsigned long long *>(csum->data()), nchains,
                                                      out);
    return done(launched(ctx, "rif_chains"));
}

static vkc_status reduce_into_add_f64(vkc_ctx *ctx, const vkc_value *args, int nargs, vkc_value *out) {
    vkc_status st;
    if (nargs != 3) return fail(ctx, VKC_RUNTIME, arity_error(3, nargs));
    if (!array_arg(ctx, args[1], VKC_F64, &st)) return st;
    int64_t nb;
    if (!array_arg(ctx, args[0], VKC_I64, &st) || !i64_arg(ctx, args[2], &nb, &st)) return st;
    if (nb < 0) return fail(ctx, VKC_RUNTIME, "negative bucket count " + std::to_string(nb));
    const vkc_array *keys = args[0].array, *vals = args[1].array;
    const int64_t n = keys->len;
    const auto *k = static_cast<const long long *>(keys->data());
    bool found;
    if (vals->len != n) {
        if ((st = bucket_key_error(ctx, k, n, nb, &found))) return st;
        return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(n) + " keys for " +
                                          std::to_string(vals->len) + " values");
    }
    vkc_array *o;
    st = new_array(ctx, VKC_F64, nb, true, &o);  // +0.0 in every bucket
    if (st) {
        std::string msg = ctx->err;
        vkc_status kst = bucket_key_error(ctx, k, n, nb, &found);
        if (kst) return kst;
        return fail(ctx, st, msg);
    }
    auto *ov = static_cast<unsigned long long *>(o->data());
    const auto *x = static_cast<const unsigned long long *>(vals->data());
    const int64_t b = n - n % 16;
    bool sorted = b > 0 && nb > 0 && !rif_masks(n, nb) && rif_tables(n, nb);
    if (sorted) {
        // The keys are checked with their images; an error is found once the sums are done.
        bool bad = false;
        st = rif_sorted(ctx, k, x, n, b, nb, ov, &bad);
        if (!st && bad) st = bucket_key_error(ctx, k, n, nb, &found);
        // Its table takes 128 bytes a bucket: without room for it, the chains by a scan.
        sorted = st != VKC_ALLOC;
        if (!sorted) VKC_CUDA(ctx, cudaMemsetAsync(ov, 0, static_cast<size_t>(nb) * 8, ctx->stream));
    }
    if (!sorted && !(st = bucket_key_error(ctx, k, n, nb, &found)) && n > 0) {
        if (rif_masks(n, nb)) {
            std::vector<unsigned> all(static_cast<size_t>(nb));
            for (int64_t i = 0; i < nb; ++i) all[static_cast<size_t>(i)] = static_cast<unsigned>(i);
            st = rif_masked(ctx, k, x, n, all, ov);
        } else {
            if (b > 0) st = rif_scanned(ctx, keys, vals, b, ov);
            if (!st) st = rif_tail(ctx, k, x, b, n, nb, ov);
        }
    }
    if (st) {
        vkc_array_release(o);
        return st;
    }
    out->kind = VKC_VALUE_ARRAY;
    out->array = o;
    return VKC_OK;
}

void register_reduce_into_f64(std::vector<KernelDef> &t) {
    // The i64 entry's inputs (keys, values, bucket count) and cost (index.rs:241-255).
    KernelDef d{"reduce_into_add_f64", VKC_WHOLE,
                {InSpec{IN_ARRAY, VKC_I64}, InSpec{IN_ARRAY, VKC_F64}, InSpec{IN_SCALAR, VKC_I64}}, true, VKC_F64, 32};
    d.whole = reduce_into_add_f64;
    t.push_back(d);
}

}  // namespace vkc
