// Batched execution of one planned statement over many arrays, and CUDA graphs of statement
// sequences: the device side of the reference executor's per-array loop (src/exec.rs:162-231,
// Strategy :77-91), which runs a statement once per array and so pays every kernel launch and
// host round trip once per array.
//
// A batch is a table of arrays in device memory (pointer, rows, first row in the batch's
// concatenation, index), ordered largest first so that the persistent kernels' tickets hand out
// the long arrays early. The batch entries only enqueue work on the context's stream: no host
// synchronisation, and no allocation once a batch's scratch exists, so a sequence of them can
// be captured in a CUDA graph (vkc_graph_begin / vkc_graph_end) and replayed.
//
//  * filter -> sum (vkc_batch_filter_sum_f64): one persistent kernel; a block takes an array and
//    compacts its survivors in row order chunk by chunk, feeding the whole blocks of 16 to the
//    reference's 16 lanes (lane j takes survivors j, j+16, ... below the last whole block of 16,
//    with IEEE adds in that order), combines the lanes +8, +4, +2, +1 and adds the tail
//    (src/kernels/scalar/reduce.rs:45-91): the bits of filter then reduce_add_f64.
//  * argsort (vkc_batch_argsort_i64): each array sorted for itself by stable radix passes over the key
//    digits given (all eight when none are), in tiles of one array each (radix.h, radix_segs). In
//    batches of short arrays (plan_segs) every row gets one image instead, its array's number above
//    the key digits, in 32 bits where they fit; the passes sort all rows by (array, key), and the last
//    one writes each array's positions to its output. Stability makes every output the array's
//    own argsort. (Key digits and number beyond 64 bits: the order by the keys first, then by the
//    arrays' numbers, found again from the positions.)
#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <numeric>
#include <type_traits>
#include <vector>

#include "lookback.cuh"
#include "radix.h"
#include "reduce_common.h"

namespace vkc {

struct BSeg {
    const void *ptr;
    int64_t n;
    int64_t base;   // first row of the array in the batch's concatenation (in index order)
    int64_t index;  // position of the array in the caller's list
};

// A batched argsort's outputs: the number of their batch, and the tables on the device that hold their rows'
// addresses.
struct BatchOuts {
    uint64_t serial = 0;
    DeviceMem outs;         // output pointers [n], index order
    DeviceMem segs;         // SortSeg[n] and each tile's array, when arrays are sorted for themselves
    bool captured = false;  // a graph holds the tables: kept until the batch is freed
};

}  // namespace vkc

struct vkc_batch {
    vkc_ctx *ctx = nullptr;
    uint64_t serial = 0;  // no other batch's, also after this one is freed
    vkc_type type = VKC_F64;
    std::vector<vkc_array *> arrays;  // retained, caller's order
    std::vector<vkc::BSeg> host;      // largest first
    int64_t total = 0;
    vkc::DeviceMem table;             // BSeg[n] on the device, largest first
    vkc::DeviceMem bases;             // int64 first rows [n + 1], index order (for the argsort)
    vkc::DeviceMem chunks;            // int64 [n + 1]: first concat chunk of each array, table order
    // Argsort scratch, made on first use.
    std::vector<vkc_array *> scratch;
    void *img[2] = {nullptr, nullptr};  // 64-bit images of `total` rows each
    unsigned *pos[2] = {nullptr, nullptr};
    unsigned *counts = nullptr, *offs = nullptr, *sums = nullptr;
    int seg_tiles = 0, seg_tile = 0;  // tiles of arrays sorted for themselves, or 0, and a tile's rows
    std::vector<std::unique_ptr<vkc::BatchOuts>> outs;  // the last few outputs' tables, and captured ones
};

namespace vkc {

// ------------------------------------------------------------------ filter -> sum

constexpr int BF_THREADS = 256;
constexpr int BF_WARPS = BF_THREADS / 32;
constexpr int BF_ROWS = 8;                        // rows per thread per chunk
constexpr int BF_CHUNK = BF_THREADS * BF_ROWS;    // 2048 rows

// One block per array, one read of its rows, by chunks: the survivors go side by side into shared memory
// behind the fewer than 16 that the chunk before left over, sixteen threads add the whole blocks of 16 to
// the lanes of the canonical order, and what is over at the end is its tail. The next chunk's rows are in
// flight meanwhile. (Counting the survivors first, to know the tail, and reading the rows eight to a thread
// took 316 us for 63 M rows in 4096 arrays, now about 100.)
template <bool POS>
__global__ void __launch_bounds__(BF_THREADS) batch_filter_sum_kernel(const BSeg *__restrict__ segs, int nseg,
                                                                     CmpRange r, unsigned long long *sums,
                                                                     unsigned *ticket) {
    __shared__ double s_keep[2][16 + BF_CHUNK];  // survivors in row order, a chunk in one, the next in the other
    __shared__ unsigned s_cnt[2][BF_ROWS * BF_WARPS];
    __shared__ int s_seg;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (;;) {
        if (t == 0) s_seg = static_cast<int>(atomicAdd(ticket, 1u));
        __syncthreads();
        const int sg = s_seg;
        if (sg >= nseg) break;
        const BSeg seg = segs[sg];
        const auto *x = static_cast<const unsigned long long *>(seg.ptr);
        double acc = 0.0;   // lane t (t < 16) of the canonical order
        unsigned over = 0;  // survivors left over by the chunk before, at the start of its other buffer
        int cur = 0;
        unsigned long long v[BF_ROWS], nv[BF_ROWS];
        auto load = [&](int64_t r0, unsigned long long (&to)[BF_ROWS]) {
#pragma unroll
            for (int j = 0; j < BF_ROWS; ++j) to[j] = r0 + j * BF_THREADS + t < seg.n ? __ldg(x + r0 + j * BF_THREADS + t) : 0ull;
        };
        load(0, v);
        for (int64_t r0 = 0; r0 < seg.n; r0 += BF_CHUNK, cur ^= 1) {
            unsigned keep = 0, votes[BF_ROWS];
#pragma unroll
            for (int j = 0; j < BF_ROWS; ++j) {
                const bool k = r0 + j * BF_THREADS + t < seg.n && in_range_t<POS>(r, v[j]);
                keep |= static_cast<unsigned>(k) << j;
                votes[j] = __ballot_sync(FULL, k);
                if (lane == 0) s_cnt[cur][j * BF_WARPS + w] = __popc(votes[j]);
            }
            load(r0 + BF_CHUNK, nv);
            __syncthreads();
            // The survivors before each step of each warp: entries 2 lane and 2 lane + 1 of the counts.
            static_assert(BF_ROWS * BF_WARPS == 64, "two counts a lane");
            const unsigned c0 = s_cnt[cur][2 * lane], c1 = s_cnt[cur][2 * lane + 1];
            unsigned inc = c0 + c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += y;
            }
            const unsigned total = over + __shfl_sync(FULL, inc, 31), before = over + inc - c0 - c1;
            double *keeps = s_keep[cur];
#pragma unroll
            for (int j = 0; j < BF_ROWS; ++j) {
                const int e = j * BF_WARPS + w;
                unsigned at = __shfl_sync(FULL, (w & 1) ? before + c0 : before, e >> 1);
                at += __popc(votes[j] & ((1u << lane) - 1u));
                if ((keep >> j) & 1u) keeps[at] = __longlong_as_double(static_cast<long long>(v[j]));
            }
            __syncthreads();
            const unsigned whole = total & ~15u;
            if (t < 16) {
                for (unsigned i = t; i < whole; i += 16) acc = __dadd_rn(acc, keeps[i]);
            } else if (w == 1 && lane < total - whole) {
                s_keep[cur ^ 1][lane] = keeps[whole + lane];
            }
            over = total - whole;
#pragma unroll
            for (int j = 0; j < BF_ROWS; ++j) v[j] = nv[j];
        }
        __syncthreads();
        if (w == 0) {
            // +8, +4, +2, +1 (lane j adds lane j + step), then the tail into lane 0.
#pragma unroll
            for (int step = 8; step > 0; step >>= 1) {
                const double other = __shfl_down_sync(FULL, acc, step);
                if (lane < step) acc = __dadd_rn(acc, other);
            }
            if (lane == 0) {
                for (unsigned j = 0; j < over; ++j) acc = __dadd_rn(acc, s_keep[cur][j]);
                sums[seg.index] = static_cast<unsigned long long>(__double_as_longlong(acc));
            }
        }
        __syncthreads();
    }
    // The last block resets the ticket for the next launch.
    __syncthreads();
    if (t == 0) {
        const unsigned prev = atomicAdd(ticket + 1, 1u);
        if (prev == gridDim.x - 1) {
            ticket[0] = 0;
            ticket[1] = 0;
        }
    }
}

// Counts of rows with x <cmp> c per array (length of filter), one block per array.
template <bool POS>
__global__ void __launch_bounds__(BF_THREADS) batch_count_kernel(const BSeg *__restrict__ segs, int nseg, CmpRange r,
                                                                long long *counts, unsigned *ticket) {
    __shared__ int s_seg;
    const int t = threadIdx.x;
    for (;;) {
        if (t == 0) s_seg = static_cast<int>(atomicAdd(ticket, 1u));
        __syncthreads();
        const int sg = s_seg;
        if (sg >= nseg) break;
        const BSeg seg = segs[sg];
        const auto *x = static_cast<const unsigned long long *>(seg.ptr);
        unsigned long long kc = 0;
        for (int64_t i = t; i < seg.n; i += BF_THREADS) kc += in_range_t<POS>(r, __ldg(x + i));
        unsigned long long k;
        block_exclusive_sum<unsigned long long>(kc, &k);
        if (t == 0) counts[seg.index] = static_cast<long long>(k);
        __syncthreads();
    }
    __syncthreads();
    if (t == 0) {
        const unsigned prev = atomicAdd(ticket + 1, 1u);
        if (prev == gridDim.x - 1) {
            ticket[0] = 0;
            ticket[1] = 0;
        }
    }
}

// dot_f64 per pair of arrays (x from xs, y from ys, same index and length), one block per pair:
// lane j (thread j < 16) adds fl(x*y) of rows j, j+16, ... below the last whole block of 16 in
// order, the lanes combine +8, +4, +2, +1, and the tail rows are added to lane 0 in order
// (src/kernels/scalar/fused.rs:73-106 with reduce.rs:45-91). The other threads stage the rows
// into shared memory ahead of the lanes. Meant for short arrays: a lane's chain is n/16 adds.
constexpr int BD_CHUNK = 4096;

__global__ void __launch_bounds__(BF_THREADS) batch_dot_kernel(const BSeg *__restrict__ xs, const BSeg *__restrict__ ys,
                                                              int nseg, unsigned long long *sums, unsigned *ticket) {
    __shared__ double s_p[BD_CHUNK];  // the chunk's products fl(x*y)
    __shared__ int s_seg;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (;;) {
        if (t == 0) s_seg = static_cast<int>(atomicAdd(ticket, 1u));
        __syncthreads();
        const int sg = s_seg;
        if (sg >= nseg) break;
        const BSeg sx = xs[sg];
        const BSeg sy = ys[sg];
        const auto *x = static_cast<const double *>(sx.ptr);
        const auto *y = static_cast<const double *>(sy.ptr);
        const int64_t n = sx.n, b = n - n % 16;
        double acc = 0.0;
        for (int64_t r0 = 0; r0 < n; r0 += BD_CHUNK) {
            const int rows = static_cast<int>(n - r0 < BD_CHUNK ? n - r0 : BD_CHUNK);
            for (int i = t; i < rows; i += BF_THREADS) s_p[i] = __dmul_rn(__ldg(x + r0 + i), __ldg(y + r0 + i));
            __syncthreads();
            if (t < 16) {
                // r0 is a multiple of 16, so row r0 + i belongs to lane i mod 16.
                for (int i = t; i < rows && r0 + i < b; i += 16) acc = __dadd_rn(acc, s_p[i]);
            }
            __syncthreads();
        }
        if (w == 0) {
#pragma unroll
            for (int step = 8; step > 0; step >>= 1) {
                const double other = __shfl_down_sync(FULL, acc, step);
                if (lane < step) acc = __dadd_rn(acc, other);
            }
            if (lane == 0) {
                for (int64_t i = b; i < n; ++i) acc = __dadd_rn(acc, __dmul_rn(__ldg(x + i), __ldg(y + i)));
                sums[sx.index] = static_cast<unsigned long long>(__double_as_longlong(acc));
            }
        }
        __syncthreads();
    }
    __syncthreads();
    if (t == 0) {
        const unsigned prev = atomicAdd(ticket + 1, 1u);
        if (prev == gridDim.x - 1) {
            ticket[0] = 0;
            ticket[1] = 0;
        }
    }
}

// ------------------------------------------------------------------ argsort

// Rows of one array per block of the image and concatenation kernels; chunks[] gives each array's
// first block, table order.
constexpr int BC_ROWS = 8192;

// The array (table order) that block c works on: the last one whose first block is <= c (an empty
// array has no block).
__device__ __forceinline__ int batch_chunk_array(const int64_t *__restrict__ chunks, int nseg, int64_t c) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (chunks[mid] <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The sort images: row i of array a gets (a << 8 digits) + the chosen digits of its key's
// sign-flipped image (NUMBER = false: the digits alone). One block per chunk: a search a block, not
// one a row, and 12 bytes moved a row (the former pass wrote 64-bit images and positions from a grid
// over the arrays: 326 us for 63 M rows).
template <class IMG, bool NUMBER>
__global__ void __launch_bounds__(256) batch_images_kernel(const BSeg *__restrict__ segs, int nseg,
                                                           const int64_t *__restrict__ chunks, BatchDigits d,
                                                           IMG *__restrict__ img) {
    const int64_t c = blockIdx.x;
    const int lo = batch_chunk_array(chunks, nseg, c);
    const BSeg seg = segs[lo];
    const int64_t r0 = (c - chunks[lo]) * BC_ROWS, r1 = min(seg.n, r0 + BC_ROWS);
    const auto *k = static_cast<const unsigned long long *>(seg.ptr);
    const IMG number = NUMBER ? static_cast<IMG>(static_cast<unsigned long long>(seg.index) << (8 * d.n)) : IMG(0);
#pragma unroll 8
    for (int64_t r = r0 + threadIdx.x; r < r1; r += 256) {
        const unsigned long long key = __ldcs(k + r) ^ 0x8000000000000000ull;
        unsigned long long im = 0;
        for (int j = 0; j < d.n; ++j) im |= ((key >> d.shift[j]) & 0xffull) << (8 * j);
        img[seg.base + r] = static_cast<IMG>(im) | number;
    }
}

// The number of the array each position belongs to (bases[nseg] = total).
__global__ void __launch_bounds__(256) batch_owner_kernel(const int64_t *__restrict__ bases, int nseg,
                                                          const unsigned *__restrict__ pos,
                                                          unsigned *__restrict__ number, int64_t total) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t p = pos[i];
        int lo = 0, hi = nseg - 1;  // the last array whose first row is <= p (arrays may be empty)
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (bases[mid] <= p) lo = mid;
            else hi = mid - 1;
        }
        number[i] = static_cast<unsigned>(lo);
    }
}

// ------------------------------------------------------------------ concatenation

// Batched statements whose kernel has no batched form (group_id, reduce_into, scans) run once
// over the concatenation of the batch's arrays, with an index column naming each row's array:
// a segmented statement keyed by that column gives every array's own result. One block per chunk.
template <int W>
__global__ void __launch_bounds__(256) batch_concat_kernel(const BSeg *__restrict__ segs, int nseg,
                                                           const int64_t *__restrict__ chunks, void *rows,
                                                           long long *index) {
    using U = typename std::conditional<W == 8, unsigned long long,
                                        typename std::conditional<W == 4, unsigned, unsigned char>::type>::type;
    const int64_t c = blockIdx.x;
    const int lo = batch_chunk_array(chunks, nseg, c);
    const BSeg seg = segs[lo];
    const int64_t r0 = (c - chunks[lo]) * BC_ROWS;
    const int64_t r1 = min(seg.n, r0 + BC_ROWS);
    const U *src = static_cast<const U *>(seg.ptr);
    U *dst = static_cast<U *>(rows) + seg.base;
#pragma unroll 8
    for (int64_t r = r0 + threadIdx.x; r < r1; r += 256) {
        dst[r] = __ldcs(src + r);
        if (index) index[seg.base + r] = seg.index;
    }
}

static bool capturing(vkc_ctx *ctx) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cs) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return cs != cudaStreamCaptureStatusNone;
}

}  // namespace vkc

using namespace vkc;

extern "C" VKC_API vkc_status vkc_batch_new(vkc_ctx *ctx, int n, vkc_array *const *arrays, vkc_batch **out) {
    if (!ctx || !out || n < 0 || (n > 0 && !arrays)) return VKC_USAGE;
    *out = nullptr;
    if (capturing(ctx)) return fail(ctx, VKC_USAGE, "vkc_batch_new during a stream capture");
    static std::atomic<uint64_t> serials{0};
    auto *b = new vkc_batch;
    b->ctx = ctx;
    b->serial = ++serials;
    b->type = n > 0 ? arrays[0]->type : VKC_F64;
    std::vector<int64_t> base(static_cast<size_t>(n) + 1, 0);
    for (int i = 0; i < n; ++i) {
        if (!arrays[i] || arrays[i]->type != b->type) {
            delete b;
            return fail(ctx, VKC_RUNTIME, "batch arrays must share one element type");
        }
        base[i + 1] = base[i] + arrays[i]->len;
    }
    b->total = base[n];
    for (int i = 0; i < n; ++i) {
        vkc_array_retain(arrays[i]);
        await_write(ctx, arrays[i]);  // batches are read and written on the context stream
        b->arrays.push_back(arrays[i]);
        b->host.push_back(BSeg{arrays[i]->data(), arrays[i]->len, base[i], i});
    }
    std::stable_sort(b->host.begin(), b->host.end(), [](const BSeg &a, const BSeg &c) { return a.n > c.n; });
    auto upload = [&](DeviceMem &m, const void *src, size_t bytes) -> vkc_status {
        if (!bytes) return VKC_OK;
        void *p = nullptr;
        VKC_CUDA(ctx, cudaMallocAsync(&p, bytes, ctx->stream));
        m.ptr = p;
        m.box = ctx->box;
        void *h;
        vkc_status st = pinned(ctx, bytes, &h);
        if (st) return st;
        VKC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        memcpy(h, src, bytes);
        VKC_CUDA(ctx, cudaMemcpyAsync(p, h, bytes, cudaMemcpyHostToDevice, ctx->stream));
        VKC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        return VKC_OK;
    };
    std::vector<int64_t> chunk(static_cast<size_t>(n) + 1, 0);
    for (int i = 0; i < n; ++i) chunk[i + 1] = chunk[i] + (b->host[i].n + BC_ROWS - 1) / BC_ROWS;
    vkc_status st = upload(b->table, b->host.data(), sizeof(BSeg) * b->host.size());
    if (!st) st = upload(b->bases, base.data(), sizeof(int64_t) * base.size());
    if (!st) st = upload(b->chunks, chunk.data(), sizeof(int64_t) * chunk.size());
    if (st) {
        vkc_batch_free(b);
        return st;
    }
    *out = b;
    return VKC_OK;
}

extern "C" VKC_API void vkc_batch_free(vkc_batch *b) {
    if (!b) return;
    for (vkc_array *a : b->arrays) vkc_array_release(a);
    for (vkc_array *a : b->scratch) vkc_array_release(a);
    delete b;
}

extern "C" VKC_API int vkc_batch_len(const vkc_batch *b) { return b ? static_cast<int>(b->arrays.size()) : 0; }

extern "C" VKC_API vkc_status vkc_batch_filter_sum_f64(vkc_ctx *ctx, vkc_batch *b, int cmp, double c,
                                                       vkc_array *sums) {
    if (!ctx || !b || !sums) return VKC_USAGE;
    if (b->type != VKC_F64) return fail(ctx, VKC_RUNTIME, "batch filter_sum: expected f64[] arrays");
    if (cmp < 0 || cmp > 5) return fail(ctx, VKC_USAGE, "batch filter_sum: comparison 0..5 (eq ne lt le gt ge)");
    const int n = static_cast<int>(b->host.size());
    if (sums->type != VKC_F64 || sums->len != n)
        return fail(ctx, VKC_RUNTIME, "batch filter_sum: the result array must be f64[" + std::to_string(n) + "]");
    if (n == 0) return VKC_OK;
    const CmpRange r = cmp_range(cmp, c);
    const int grid = std::min(n, ctx->sms * 8);
    await_write(ctx, sums);
    auto *out = static_cast<unsigned long long *>(sums->data());
    const auto *tab = static_cast<const BSeg *>(b->table.ptr);
    unsigned *ticket = ctx->counters + 4;  // two words, zero between launches
    if (pos_range(r)) batch_filter_sum_kernel<true><<<grid, BF_THREADS, 0, ctx->stream>>>(tab, n, r, out, ticket);
    else batch_filter_sum_kernel<false><<<grid, BF_THREADS, 0, ctx->stream>>>(tab, n, r, out, ticket);
    return launched(ctx, "batch_filter_sum");
}

extern "C" VKC_API vkc_status vkc_batch_count_f64(vkc_ctx *ctx, vkc_batch *b, int cmp, double c, vkc_array *counts) {
    if (!ctx || !b || !counts) return VKC_USAGE;
    if (b->type != VKC_F64) return fail(ctx, VKC_RUNTIME, "batch count: expected f64[] arrays");
    if (cmp < 0 || cmp > 5) return fail(ctx, VKC_USAGE, "batch count: comparison 0..5 (eq ne lt le gt ge)");
    const int n = static_cast<int>(b->host.size());
    if (counts->type != VKC_I64 || counts->len != n)
        return fail(ctx, VKC_RUNTIME, "batch count: the result array must be i64[" + std::to_string(n) + "]");
    if (n == 0) return VKC_OK;
    const CmpRange r = cmp_range(cmp, c);
    const int grid = std::min(n, ctx->sms * 8);
    await_write(ctx, counts);
    auto *out = static_cast<long long *>(counts->data());
    const auto *tab = static_cast<const BSeg *>(b->table.ptr);
    if (pos_range(r)) batch_count_kernel<true><<<grid, BF_THREADS, 0, ctx->stream>>>(tab, n, r, out, ctx->counters + 4);
    else batch_count_kernel<false><<<grid, BF_THREADS, 0, ctx->stream>>>(tab, n, r, out, ctx->counters + 4);
    return launched(ctx, "batch_count");
}

extern "C" VKC_API vkc_status vkc_batch_dot_f64(vkc_ctx *ctx, vkc_batch *xs, vkc_batch *ys, vkc_array *sums) {
    if (!ctx || !xs || !ys || !sums) return VKC_USAGE;
    if (xs->type != VKC_F64 || ys->type != VKC_F64) return fail(ctx, VKC_RUNTIME, "batch dot: expected f64[] arrays");
    const int n = static_cast<int>(xs->host.size());
    if (static_cast<int>(ys->host.size()) != n) return fail(ctx, VKC_RUNTIME, "batch dot: batches of different sizes");
    // Both tables are largest first with ties kept in index order, so equal lengths pair up.
    for (int i = 0; i < n; ++i)
        if (xs->arrays[i]->len != ys->arrays[i]->len)
            return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(xs->arrays[i]->len) + " vs " +
                                              std::to_string(ys->arrays[i]->len));
    if (sums->type != VKC_F64 || sums->len != n)
        return fail(ctx, VKC_RUNTIME, "batch dot: the result array must be f64[" + std::to_string(n) + "]");
    if (n == 0) return VKC_OK;
    const int grid = std::min(n, ctx->sms * 8);
    await_write(ctx, sums);
    batch_dot_kernel<<<grid, BF_THREADS, 0, ctx->stream>>>(static_cast<const BSeg *>(xs->table.ptr),
                                                           static_cast<const BSeg *>(ys->table.ptr), n,
                                                           static_cast<unsigned long long *>(sums->data()),
                                                           ctx->counters + 4);
    return launched(ctx, "batch_dot");
}

namespace vkc {

// Whether each array is sorted for itself, in how many tiles of how many rows. A pass for each key digit
// and none for the array's number, no images made before the first, one output array a tile; but a tile
// holds rows of one array, so that short arrays leave it mostly empty: from half-full tiles of 2048 rows on
// it is the faster way for any number of digits (4096 arrays of 1387 rows on average, 1 / 2 / 4 / 8 digits:
// 119 / 190 / 340 / 672 us a call against 227 / 285 / 437 / 731 with the number in the image; of 967 rows,
// 47% full, 8 digits 629 against 595). Tiles of 3072 rows are the better ones for longer arrays (4096 of
// 15.5 K rows, 2 digits: 866 us, 921 in 2048, 857 in 4096, 1663 with the number; of 2774 rows 267 and 250).
static void plan_segs(vkc_batch *b) {
    b->seg_tile = b->total >= 4096 * static_cast<int64_t>(b->host.size()) ? 3072 : 2048;
    int64_t tiles = 0;
    for (const BSeg &g : b->host) tiles += (g.n + b->seg_tile - 1) / b->seg_tile;
    b->seg_tiles = b->total >= tiles * (b->seg_tile / 2) ? static_cast<int>(tiles) : 0;
}

static vkc_status upload_table(vkc_ctx *ctx, DeviceMem &m, const void *src, size_t bytes) {
    void *h;
    m.box = ctx->box;
    VKC_CUDA(ctx, cudaMallocAsync(&m.ptr, bytes, ctx->stream));
    const vkc_status st = pinned(ctx, bytes, &h);
    if (st) return st;
    VKC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    memcpy(h, src, bytes);
    VKC_CUDA(ctx, cudaMemcpyAsync(m.ptr, h, bytes, cudaMemcpyHostToDevice, ctx->stream));
    VKC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return VKC_OK;
}

// The sort's scratch (it depends on the keys alone): all of it or none.
static vkc_status argsort_scratch(vkc_ctx *ctx, vkc_batch *keys) {
    const int64_t total = keys->total;
    int64_t cw, sw;
    radix_table_words(total, &cw, &sw);
    plan_segs(keys);
    if (keys->seg_tiles) {
        cw = std::max(cw, int64_t(256) * keys->seg_tiles);
        sw = std::max(sw, scan_counts_sum_words(cw));
    }
    vkc_array *a[7] = {};
    const vkc_type ty[7] = {VKC_U64, VKC_U64, VKC_I32, VKC_I32, VKC_I32, VKC_I32, VKC_I32};
    const int64_t len[7] = {total, total, total, total, cw, cw, sw};
    for (int i = 0; i < 7; ++i) {
        const vkc_status st = new_array(ctx, ty[i], len[i], false, &a[i]);
        if (st) {
            for (int j = 0; j < i; ++j) vkc_array_release(a[j]);
            return st;
        }
    }
    keys->scratch.assign(a, a + 7);
    keys->img[0] = a[0]->data();
    keys->img[1] = a[1]->data();
    keys->pos[0] = static_cast<unsigned *>(a[2]->data());
    keys->pos[1] = static_cast<unsigned *>(a[3]->data());
    keys->counts = static_cast<unsigned *>(a[4]->data());
    keys->offs = static_cast<unsigned *>(a[5]->data());
    keys->sums = static_cast<unsigned *>(a[6]->data());
    return VKC_OK;
}

// The tables of these outputs, made on their first use. Batches are told apart by their numbers (a batch's
// address may be another one's after it is freed), and a batch's arrays are the same all its life.
constexpr int BATCH_OUTS = 4;  // outputs whose tables are kept beside the captured ones
static vkc_status argsort_outs(vkc_ctx *ctx, vkc_batch *keys, const vkc_batch *outs, bool cap, const BatchOuts **found) {
    const size_t n = keys->arrays.size();
    for (auto &o : keys->outs) {
        if (o->serial != outs->serial) continue;
        o->captured = o->captured || cap;
        *found = o.get();
        return VKC_OK;
    }
    if (cap) return fail(ctx, VKC_USAGE, "batch argsort: make its first call before capturing");
    auto o = std::make_unique<BatchOuts>();
    o->serial = outs->serial;
    std::vector<void *> rows;
    for (const vkc_array *a : outs->arrays) rows.push_back(a->data());
    vkc_status st = upload_table(ctx, o->outs, rows.data(), sizeof(void *) * n);
    if (!st && keys->seg_tiles) {
        // The arrays in the concatenation's order, and each tile's array.
        std::vector<unsigned char> table(sizeof(SortSeg) * n + sizeof(int) * keys->seg_tiles);
        auto *segs = reinterpret_cast<SortSeg *>(table.data());
        int *tile = reinterpret_cast<int *>(segs + n);
        int64_t base = 0, t = 0;
        for (size_t i = 0; i < n; ++i) {
            const vkc_array *a = keys->arrays[i];
            segs[i] = SortSeg{static_cast<const unsigned long long *>(a->data()), static_cast<long long *>(rows[i]), base, a->len, t};
            for (int64_t j = 0; j < a->len; j += keys->seg_tile) tile[t++] = static_cast<int>(i);
            base += a->len;
        }
        st = upload_table(ctx, o->segs, table.data(), table.size());
    }
    if (st) return st;
    const auto old = std::find_if(keys->outs.begin(), keys->outs.end(), [](const auto &p) { return !p->captured; });
    if (std::count_if(keys->outs.begin(), keys->outs.end(), [](const auto &p) { return !p->captured; }) >= BATCH_OUTS)
        keys->outs.erase(old);
    keys->outs.push_back(std::move(o));
    *found = keys->outs.back().get();
    return VKC_OK;
}

}  // namespace vkc

extern "C" VKC_API vkc_status vkc_batch_argsort_i64(vkc_ctx *ctx, vkc_batch *keys, const vkc_batch *outs,
                                                    unsigned key_digits) {
    if (!ctx || !keys || !outs) return VKC_USAGE;
    if (keys->type != VKC_I64) return fail(ctx, VKC_RUNTIME, "batch argsort: expected i64[] keys");
    const int n = static_cast<int>(keys->arrays.size());
    if (outs->type != VKC_I64 || static_cast<int>(outs->arrays.size()) != n)
        return fail(ctx, VKC_RUNTIME, "batch argsort: outputs must be " + std::to_string(n) + " i64[] arrays");
    for (int i = 0; i < n; ++i)
        if (outs->arrays[i]->len != keys->arrays[i]->len)
            return fail(ctx, VKC_RUNTIME, "batch argsort: output " + std::to_string(i) + " has the wrong length");
    const int64_t total = keys->total;
    if (n == 0 || total == 0) return VKC_OK;
    for (int i = 0; i < n; ++i) await_write(ctx, outs->arrays[i]);
    if (total >= (int64_t(1) << 32)) return fail(ctx, VKC_USAGE, "batch argsort of 2^32 rows or more");
    const bool cap = capturing(ctx);
    vkc_status st;
    // Scratch and the outputs' tables: on first use, never during a capture.
    if (keys->scratch.empty()) {
        if (cap) return fail(ctx, VKC_USAGE, "batch argsort: make its first call before capturing");
        if ((st = argsort_scratch(ctx, keys))) return st;
    }
    const BatchOuts *to;
    if ((st = argsort_outs(ctx, keys, outs, cap, &to))) return st;
    if (n > 65536) return fail(ctx, VKC_USAGE, "batch argsort of more than 65536 arrays");
    const auto *tab = static_cast<const BSeg *>(keys->table.ptr);
    const auto *bases = static_cast<const int64_t *>(keys->bases.ptr);
    const auto *ch = static_cast<const int64_t *>(keys->chunks.ptr);
    int64_t nchunks = 0;
    for (const BSeg &g : keys->host) nchunks += (g.n + BC_ROWS - 1) / BC_ROWS;
    // Key digits: given, or all eight. Then the array's number, one or two digits.
    if (key_digits == 0) key_digits = 0xff;
    BatchDigits d{};
    for (int k = 0; k < 8; ++k)
        if ((key_digits >> k) & 1u) d.shift[d.n++] = 8 * k;
    d.run = d.shift[d.n - 1] - d.shift[0] == 8 * (d.n - 1);
    if (keys->seg_tiles) {
        const auto *segs = static_cast<const SortSeg *>(to->segs.ptr);
        return radix_segs(ctx, BatchSegs{segs, reinterpret_cast<const int *>(segs + n), keys->seg_tiles, keys->seg_tile, d}, keys->img,
                          keys->pos, total, RadixTables{keys->counts, keys->offs, keys->sums});
    }
    const int numbers = n > 256 ? 2 : 1, digits = d.n + numbers;
    int shifts[8];
    for (int k = 0; k < 8; ++k) shifts[k] = 8 * k;
    const RadixTables t{keys->counts, keys->offs, keys->sums};
    BatchOut batch{bases, static_cast<const unsigned long long *>(to->outs.ptr), 8 * d.n};
    const int blocks = static_cast<int>(nchunks);
    if (digits <= 4) {
        batch_images_kernel<unsigned, true><<<blocks, 256, 0, ctx->stream>>>(tab, n, ch, d, static_cast<unsigned *>(keys->img[1]));
        if ((st = launched(ctx, "batch_images"))) return st;
        return radix_batch(ctx, false, keys->img[1], keys->img, keys->pos, batch, total, shifts, digits, t);
    }
    auto *wide = static_cast<unsigned long long *>(keys->img[1]);
    if (digits <= 8) {
        batch_images_kernel<unsigned long long, true><<<blocks, 256, 0, ctx->stream>>>(tab, n, ch, d, wide);
        if ((st = launched(ctx, "batch_images"))) return st;
        return radix_batch(ctx, true, wide, keys->img, keys->pos, batch, total, shifts, digits, t);
    }
    batch_images_kernel<unsigned long long, false><<<blocks, 256, 0, ctx->stream>>>(tab, n, ch, d, wide);
    if ((st = launched(ctx, "batch_images"))) return st;
    if ((st = radix_batch_keys(ctx, wide, keys->img, keys->pos, total, shifts, d.n, t))) return st;
    const int at = (d.n - 1) & 1;
    auto *number = static_cast<unsigned *>(keys->img[1 - at]);
    batch_owner_kernel<<<stream_grid(ctx, total, 256, 8, 2048), 256, 0, ctx->stream>>>(bases, n, keys->pos[at], number, total);
    if ((st = launched(ctx, "batch_owner"))) return st;
    batch.index_shift = 0;
    return radix_batch_numbers(ctx, number, keys->pos[at], static_cast<unsigned *>(keys->img[at]), keys->pos[1 - at], batch,
                               total, numbers, t);
}

extern "C" VKC_API vkc_status vkc_batch_concat(vkc_ctx *ctx, vkc_batch *b, vkc_array **rows, vkc_array **index) {
    if (!ctx || !b || !rows) return VKC_USAGE;
    *rows = nullptr;
    if (index) *index = nullptr;
    vkc_status st;
    vkc_array *r = nullptr, *ix = nullptr;
    if ((st = new_array(ctx, b->type, b->total, false, &r))) return st;
    if (index && (st = new_array(ctx, VKC_I64, b->total, false, &ix))) {
        vkc_array_release(r);
        return st;
    }
    const int n = static_cast<int>(b->host.size());
    int64_t nchunks = 0;
    for (const BSeg &g : b->host) nchunks += (g.n + BC_ROWS - 1) / BC_ROWS;
    if (nchunks > 0) {
        const auto *tab = static_cast<const BSeg *>(b->table.ptr);
        const auto *ch = static_cast<const int64_t *>(b->chunks.ptr);
        long long *ip = ix ? static_cast<long long *>(ix->data()) : nullptr;
        const dim3 grid(static_cast<unsigned>(nchunks));
        switch (type_width(b->type)) {
        case 8: batch_concat_kernel<8><<<grid, 256, 0, ctx->stream>>>(tab, n, ch, r->data(), ip); break;
        case 4: batch_concat_kernel<4><<<grid, 256, 0, ctx->stream>>>(tab, n, ch, r->data(), ip); break;
        default: batch_concat_kernel<1><<<grid, 256, 0, ctx->stream>>>(tab, n, ch, r->data(), ip); break;
        }
        if ((st = launched(ctx, "batch_concat"))) {
            vkc_array_release(r);
            vkc_array_release(ix);
            return st;
        }
    }
    *rows = r;
    if (index) *index = ix;
    return VKC_OK;
}

// ------------------------------------------------------------------ CUDA graphs

struct vkc_graph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

extern "C" VKC_API vkc_status vkc_graph_begin(vkc_ctx *ctx) {
    if (!ctx) return VKC_USAGE;
    VKC_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    return VKC_OK;
}

extern "C" VKC_API vkc_status vkc_graph_end(vkc_ctx *ctx, vkc_graph **out) {
    if (!ctx || !out) return VKC_USAGE;
    *out = nullptr;
    auto *g = new vkc_graph;
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &g->graph);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&g->exec, g->graph, 0);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (g->graph) cudaGraphDestroy(g->graph);
        delete g;
        return fail(ctx, VKC_DEVICE, std::string("graph capture failed: ") + cudaGetErrorString(e));
    }
    *out = g;
    return VKC_OK;
}

extern "C" VKC_API vkc_status vkc_graph_launch(vkc_ctx *ctx, vkc_graph *g) {
    if (!ctx || !g) return VKC_USAGE;
    VKC_CUDA(ctx, cudaGraphLaunch(g->exec, ctx->stream));
    return VKC_OK;
}

extern "C" VKC_API void vkc_graph_free(vkc_graph *g) {
    if (!g) return;
    if (g->exec) cudaGraphExecDestroy(g->exec);
    if (g->graph) cudaGraphDestroy(g->graph);
    delete g;
}
