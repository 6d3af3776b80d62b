// argsort_T: the stable ascending positions of the rows (src/kernels/scalar/index.rs:159-173,
// src/kernels/scalar/index/radix.rs:126-259), for i64, u64, i32 and u8 keys; and the radix passes
// that the batched argsort and the float bucket sums use.
//
// LSD radix sort over 8-bit digits of (image, payload) pairs, as the reference does, restated for
// the GPU:
//  * the image of a key is its order-preserving unsigned value (radix.rs:58-61: the sign bit
//    flipped); one reduction finds the images' least and greatest value and the bits that vary.
//    The passes cover the bytes that vary (radix.rs:203-211: an equal digit leaves the order
//    unchanged), or, when those are fewer, the bytes of the image's distance from the least one
//    (signed keys of a small range vary in every byte, but not in their distance);
//  * each pass is reduce-then-scan over tiles of 256 x radix_items rows (the autotuner's table:
//    2048, 3072 or 4096 rows by size): `up` counts each tile's digits into a digit-major table, one
//    exclusive scan of that table gives every (digit, tile) its first output row, and `down` ranks
//    the tile's rows stably by digit and scatters them. The first pass reads the keys, the last
//    writes the positions as i64. (A single-pass lookback per digit was slower here: the lookback
//    of 256 digits per tile advances a few tiles per L2 round trip.)
//  * `down` finds the lanes of a warp that share a digit by a ballot per digit bit. (An atomic OR of
//    the lane's bit into the digit's shared word took a third of the instructions, 1.6 a row against
//    3.8, but twice the shared-memory wavefronts, and these then bound the pass: 101 us against 79
//    for 2^24 rows.)
// Stability makes the output the reference's; inputs of at most 2048 rows are sorted in one
// block by comparison (as the reference does below 1024 rows, radix.rs:140-151), inputs of at
// most 8192 rows by the same radix passes inside one block.
#include <algorithm>

#include "lookback.cuh"
#include "radix.h"
#include "reduce_common.h"

namespace vkc {

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RADIX = 256;

// Rows per thread of a pass (the autotuner's radix_items: 8, 12 or 16; even, as ranks are
// packed in pairs), the tile, and the resident blocks per SM that the down kernel's registers
// allow. PAIR: bytes of an image and its payload.
template <int ITEMS, int PAIR> struct RsShape {
    static_assert(ITEMS % 4 == 0, "ranks are packed two per word, images counted four at a time");
    static constexpr int TILE = RS_THREADS * ITEMS;
    static constexpr int MIN_BLOCKS = ITEMS >= 16 ? (PAIR == 8 ? 4 : 3) : (ITEMS >= 12 ? 4 : 5);
    // Dynamic shared memory of the down kernel: the tile's images and payloads sorted by digit.
    static constexpr size_t DOWN_SMEM = static_cast<size_t>(PAIR) * TILE;
};
constexpr int RS_MIN_TILE = RS_THREADS * 8;

// The keys of the first pass: the image of the key word k is (k ^ flip) - low, W bytes wide.
template <int W> struct KeyWord;
template <> struct KeyWord<8> { using T = unsigned long long; };
template <> struct KeyWord<4> { using T = unsigned; };
template <> struct KeyWord<1> { using T = unsigned char; };
struct KeySource {
    const void *keys;
    unsigned long long flip, low;
};
template <int W> __device__ __forceinline__ unsigned long long key_image(const KeySource &k, int64_t r) {
    using T = typename KeyWord<W>::T;
    return (static_cast<unsigned long long>(__ldcs(static_cast<const T *>(k.keys) + r)) ^ k.flip) - k.low;
}

// range[0..3]: the AND and the least (from all ones), the OR and the greatest (from zero) of the
// images.
template <int W>
__global__ void __launch_bounds__(256) rs_range_kernel(KeySource k, int64_t n, unsigned long long *range) {
    constexpr int R = 8;  // rows a thread loads together
    unsigned long long all = ~0ull, lo = ~0ull, any = 0, hi = 0;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < n; i0 += R * stride) {
        unsigned long long v[R];
#pragma unroll
        for (int j = 0; j < R; ++j) v[j] = key_image<W>(k, i0 + j * stride < n ? i0 + j * stride : i0);
#pragma unroll
        for (int j = 0; j < R; ++j) {
            all &= v[j];
            any |= v[j];
            lo = min(lo, v[j]);
            hi = max(hi, v[j]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        all &= __shfl_xor_sync(FULL, all, o);
        any |= __shfl_xor_sync(FULL, any, o);
        lo = min(lo, __shfl_xor_sync(FULL, lo, o));
        hi = max(hi, __shfl_xor_sync(FULL, hi, o));
    }
    __shared__ unsigned long long s[4][8];
    if ((threadIdx.x & 31) == 0) {
        const int w = threadIdx.x >> 5;
        s[0][w] = all;
        s[1][w] = lo;
        s[2][w] = any;
        s[3][w] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            all &= s[0][w];
            lo = min(lo, s[1][w]);
            any |= s[2][w];
            hi = max(hi, s[3][w]);
        }
        atomicAnd(range, all);
        atomicMin(range + 1, lo);
        atomicOr(range + 2, any);
        atomicMax(range + 3, hi);
    }
}

// Where a pass reads and writes. W (template): keys of W bytes with the row numbers as payloads
// (the first pass of a sort), or 0: images and payloads. OUT (template): images and payloads, the
// payloads alone as i64 rows (the last pass of an argsort), or each array's rows to its own output
// (the last pass of a batched argsort, whose images hold the array's number above `index_shift`).
enum RsOut { OUT_PAIRS = 0, OUT_ROWS = 1, OUT_BATCH = 2 };
template <class IMG, class PAY> struct RsArgs {
    KeySource k;
    const IMG *img_in;
    const PAY *pay_in;
    IMG *img_out;
    PAY *pay_out;
    long long *out;
    BatchOut batch;
    // SEG passes: the arrays, and each tile's; the digits of the images.
    const SortSeg *segs;
    const int *tile_seg;
    BatchDigits digits;
};

// What a block works on. SEG (template): every tile belongs to one array, whose rows are sorted among
// themselves: the counts lie array-major, in an array digit-major, so that their one exclusive scan gives
// each (array, digit, tile) its first row of the concatenation.
struct RsTile {
    int64_t row0, end;   // its rows
    int64_t at, stride;  // digit d's count is number at + d * stride
};
template <bool SEG, int TILE> __device__ __forceinline__ RsTile rs_tile(const SortSeg &seg, int64_t n, int tiles, int tile) {
    if constexpr (SEG) {
        const int64_t j = tile - seg.tile0, r = j * TILE;
        return RsTile{seg.base + r, min(seg.base + r + TILE, seg.base + seg.n), static_cast<int64_t>(RADIX) * seg.tile0 + j,
                      (seg.n + TILE - 1) / TILE};
    } else {
        const int64_t r = static_cast<int64_t>(tile) * TILE;
        return RsTile{r, min(r + TILE, n), tile, tiles};
    }
}
// The images of rows r0 + 32 j of array `seg` (those below `end`): the chosen digits of the key side by
// side, with `run` as many above the last one as the image holds, which no pass looks at. The loads are all
// in flight together (a choice of digits between them took the first pass from 580 to 300 us, 63 M rows).
template <int ITEMS, bool WHOLE, class IMG>
__device__ __forceinline__ void seg_images(const SortSeg &seg, const BatchDigits &d, int64_t r0, int64_t end, IMG (&img)[ITEMS]) {
    const unsigned long long *k = seg.keys + (r0 - seg.base);
    const int sh = d.shift[0];
    if (d.run) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j)
            img[j] = WHOLE || r0 + j * 32 < end ? static_cast<IMG>((__ldcs(k + j * 32) ^ 0x8000000000000000ull) >> sh) : IMG(0);
        return;
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const unsigned long long key = WHOLE || r0 + j * 32 < end ? __ldcs(k + j * 32) ^ 0x8000000000000000ull : 0ull;
        unsigned long long im = 0;
        for (int i = 0; i < d.n; ++i) im |= ((key >> d.shift[i]) & 0xffull) << (8 * i);
        img[j] = static_cast<IMG>(im);
    }
}

// Up: the digit counts of every tile, digit-major: counts[d * tiles + tile]. Shared-memory
// atomics into one histogram per warp (the order of the increments does not matter here). W: the
// first pass, from keys of W bytes; 0: from images.
template <int RS_ITEMS, int W, bool SEG, class IMG>
__global__ void __launch_bounds__(RS_THREADS) rs_up_kernel(KeySource k, const IMG *img_in, int64_t n,
                                                           int shift, int tiles, unsigned *counts,
                                                           const SortSeg *segs, const int *tile_seg, BatchDigits digits) {
    chain_enter();
    img_in = chained(img_in);
    k.keys = chained(k.keys);
    constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
    __shared__ unsigned s_cnt[RS_WARPS][RADIX];
    const int tile = blockIdx.x;
    const SortSeg seg = SEG ? segs[tile_seg[tile]] : SortSeg{};
    const RsTile tl = rs_tile<SEG, RS_TILE>(seg, n, tiles, tile);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < RS_WARPS * RADIX; i += RS_THREADS) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    const int64_t base = tl.row0 + static_cast<int64_t>(w) * (32 * RS_ITEMS);
    if (base + 32 * RS_ITEMS <= tl.end) {
        IMG img[RS_ITEMS];
        if constexpr (SEG && W != 0) {
            seg_images<RS_ITEMS, true>(seg, digits, base + lane, tl.end, img);
        } else if constexpr (SEG) {
#pragma unroll
            for (int j = 0; j < RS_ITEMS; ++j) img[j] = __ldcs(img_in + base + j * 32 + lane);
        } else if constexpr (W != 0) {
#pragma unroll
            for (int j = 0; j < RS_ITEMS; ++j) img[j] = static_cast<IMG>(key_image<W>(k, base + j * 32 + lane));
        } else {
            constexpr int V = 16 / sizeof(IMG);  // images of a 16-byte load (image buffers start aligned)
#pragma unroll
            for (int j = 0; j < RS_ITEMS / V; ++j) {
                const uint4 u = __ldcs(reinterpret_cast<const uint4 *>(img_in + base) + j * 32 + lane);
                if constexpr (V == 4) {
                    img[4 * j] = u.x;
                    img[4 * j + 1] = u.y;
                    img[4 * j + 2] = u.z;
                    img[4 * j + 3] = u.w;
                } else {
                    img[2 * j] = (static_cast<unsigned long long>(u.y) << 32) | u.x;
                    img[2 * j + 1] = (static_cast<unsigned long long>(u.w) << 32) | u.z;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < RS_ITEMS; ++j) atomicAdd(&s_cnt[w][static_cast<unsigned>(img[j] >> shift) & 0xffu], 1u);
    } else if constexpr (SEG) {
        IMG img[RS_ITEMS];
        if constexpr (W != 0) {
            seg_images<RS_ITEMS, false>(seg, digits, base + lane, tl.end, img);
        } else {
#pragma unroll
            for (int j = 0; j < RS_ITEMS; ++j) img[j] = base + j * 32 + lane < tl.end ? __ldcs(img_in + base + j * 32 + lane) : IMG(0);
        }
#pragma unroll
        for (int j = 0; j < RS_ITEMS; ++j)
            if (base + j * 32 + lane < tl.end) atomicAdd(&s_cnt[w][static_cast<unsigned>(img[j] >> shift) & 0xffu], 1u);
    } else {
        for (int j = 0; j < RS_ITEMS; ++j) {
            const int64_t r = base + j * 32 + lane;
            if (r < tl.end) {
                const IMG im = W == 0 ? img_in[r] : static_cast<IMG>(key_image<W ? W : 8>(k, r));
                atomicAdd(&s_cnt[w][static_cast<unsigned>(im >> shift) & 0xffu], 1u);
            }
        }
    }
    __syncthreads();
    const int d = threadIdx.x;  // RS_THREADS == RADIX
    unsigned total = 0;
#pragma unroll
    for (int ww = 0; ww < RS_WARPS; ++ww) total += s_cnt[ww][d];
    counts[tl.at + d * tl.stride] = total;
}

// The lanes of the warp whose 8-bit digit equals this lane's, among the lanes of `valid`: one
// ballot per digit bit, each lane keeping the lanes that agree with it on that bit.
__device__ __forceinline__ unsigned digit_peers(unsigned d, unsigned valid) {
    unsigned m = valid;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const unsigned bit = (d >> b) & 1u;
        const unsigned v = __ballot_sync(FULL, bit);
        m &= ~(v ^ (0u - bit));  // keep the lanes whose bit b equals this lane's
    }
    return m;
}

// Exclusive scan of `m` u32 counts (n < 2^32, so sums fit) in SCAN_CHUNK-element blocks:
// block sums, one block scanning the sums, then each block scanning its chunk from its base.
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_CHUNK = SCAN_THREADS * SCAN_ITEMS;

__global__ void __launch_bounds__(SCAN_THREADS) rs_scan_sums(const unsigned *c, int64_t m, unsigned *sums) {
    chain_enter();
    const int64_t b0 = static_cast<int64_t>(blockIdx.x) * SCAN_CHUNK;
    unsigned t = 0;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        const int64_t i = b0 + j * SCAN_THREADS + threadIdx.x;
        if (i < m) t += c[i];
    }
    unsigned total;
    block_exclusive_sum<unsigned>(t, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// One block: exclusive scan of `k` block sums in place.
__global__ void __launch_bounds__(1024) rs_scan_top(unsigned *sums, int k) {
    chain_enter();
    __shared__ unsigned carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b0 = 0; b0 < k; b0 += 1024) {
        const int i = b0 + threadIdx.x;
        const unsigned v = i < k ? sums[i] : 0u;
        unsigned total;
        const unsigned ex = block_exclusive_sum<unsigned>(v, &total);
        if (i < k) sums[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
}

// Thread t holds the chunk's rows t * SCAN_ITEMS .. + SCAN_ITEMS - 1 (contiguous), so a block
// exclusive sum of the thread totals orders them. VEC: both arrays start on 16-byte boundaries, so a
// thread's rows move as four 16-byte accesses (one word at a time, each warp access touched 32
// sectors: 17 us for 2.5 M counts).
template <bool VEC>
__global__ void __launch_bounds__(SCAN_THREADS) rs_scan_apply(const unsigned *c, int64_t m, const unsigned *sums, unsigned *out) {
    chain_enter();
    const int64_t b0 = static_cast<int64_t>(blockIdx.x) * SCAN_CHUNK + static_cast<int64_t>(threadIdx.x) * SCAN_ITEMS;
    const bool whole = VEC && b0 + SCAN_ITEMS <= m;
    unsigned v[SCAN_ITEMS], t = 0;
    if (whole) {
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS / 4; ++q) {
            const uint4 u = *reinterpret_cast<const uint4 *>(c + b0 + 4 * q);
            v[4 * q] = u.x;
            v[4 * q + 1] = u.y;
            v[4 * q + 2] = u.z;
            v[4 * q + 3] = u.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < SCAN_ITEMS; ++j) v[j] = b0 + j < m ? c[b0 + j] : 0u;
    }
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) t += v[j];
    unsigned total;
    unsigned run = sums[blockIdx.x] + block_exclusive_sum<unsigned>(t, &total);
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        const unsigned x = v[j];
        v[j] = run;
        run += x;
    }
    if (whole) {
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS / 4; ++q)
            *reinterpret_cast<uint4 *>(out + b0 + 4 * q) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    } else {
#pragma unroll
        for (int j = 0; j < SCAN_ITEMS; ++j)
            if (b0 + j < m) out[b0 + j] = v[j];
    }
}

// A short table in one block: every 16-byte unit of it in a register, the warps' sums of its eight pieces
// scanned by one warp. (A pass over up to 2^18 rows spends most of its time in launches: with the three
// kernels above a sort of 2^18 32-bit keys took about 135 us a call, then 105, and 84 since the passes'
// kernels are launched as a chain.)
constexpr int SCAN_ONE = 32768;
__global__ void __launch_bounds__(1024) rs_scan_one(const unsigned *c, int m, unsigned *out) {
    chain_enter();
    __shared__ unsigned s_sum[8 * 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint4 v[8];
    unsigned inc[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const int i = p * 4096 + static_cast<int>(threadIdx.x) * 4;
        v[p] = i < m ? *reinterpret_cast<const uint4 *>(c + i) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int p = 0; p < 8; ++p) inc[p] = v[p].x + v[p].y + v[p].z + v[p].w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            const unsigned y = __shfl_up_sync(FULL, inc[p], o);
            if (lane >= o) inc[p] += y;
        }
    }
    if (lane == 31) {
#pragma unroll
        for (int p = 0; p < 8; ++p) s_sum[p * 32 + w] = inc[p];
    }
    __syncthreads();
    if (w == 0) {
        unsigned q[8], sum = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            q[i] = s_sum[lane * 8 + i];
            sum += q[i];
        }
        unsigned before = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(FULL, before, o);
            if (lane >= o) before += y;
        }
        before -= sum;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            s_sum[lane * 8 + i] = before;
            before += q[i];
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const int i = p * 4096 + static_cast<int>(threadIdx.x) * 4;
        if (i >= m) break;
        const unsigned b = s_sum[p * 32 + w] + inc[p] - (v[p].x + v[p].y + v[p].z + v[p].w);
        *reinterpret_cast<uint4 *>(out + i) = make_uint4(b, b + v[p].x, b + v[p].x + v[p].y, b + v[p].x + v[p].y + v[p].z);
    }
}

// Exclusive scan of m u32 counts into out, with sum_words(m) words of scratch in `sums`
// (used by the partitioned gather as well as the passes below).
int64_t scan_counts_sum_words(int64_t m) { return (m + SCAN_CHUNK - 1) / SCAN_CHUNK; }
void scan_counts(vkc_ctx *ctx, const unsigned *c, int64_t m, unsigned *sums, unsigned *out) {
    const bool vec = ((reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    if (vec && m <= SCAN_ONE && m % 4 == 0) {
        launch_next(rs_scan_one, 1, 1024, 0, ctx->stream, c, static_cast<int>(m), out);
        return;
    }
    const int chunks = static_cast<int>(scan_counts_sum_words(m));
    launch_next(rs_scan_sums, chunks, SCAN_THREADS, 0, ctx->stream, c, m, sums);
    launch_next(rs_scan_top, 1, 1024, 0, ctx->stream, sums, chunks);
    if (vec)
        launch_next(rs_scan_apply<true>, chunks, SCAN_THREADS, 0, ctx->stream, c, m, sums, out);
    else
        launch_next(rs_scan_apply<false>, chunks, SCAN_THREADS, 0, ctx->stream, c, m, sums, out);
}

// Down: one pass over digit `shift` with the tile's first output row per digit in
// offsets[d * tiles + tile]. Bound by issue and by its shared-memory wavefronts: 40 M rows of 32-bit
// images take about 170 us (190 with two table lookups a row and three blocks an SM) against 95 us
// for the 640 MB moved.
struct __align__(16) RsShared {
    // Per warp and digit: the warp's rows of the digit so far; after the ranking, the first row of
    // the warp's rows of the digit in the sorted tile.
    unsigned short w[RS_WARPS][RADIX];
    unsigned excl[RADIX];  // the output row of sorted-tile row l is excl[d] + l
};

// The body of a down tile; WHOLE when every row of the tile is below n (all but the last
// tile), which drops the per-row bounds checks.
template <int RS_ITEMS, int W, int OUT, bool SEG, class IMG, class PAY, bool WHOLE>
__device__ __forceinline__ void rs_down_tile(const RsArgs<IMG, PAY> &a, const SortSeg &seg, const RsTile &tl, int shift,
                                             RsShared &sm, unsigned char *smem) {
    constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // Rows of this warp: warp-striped, row = base + j*32 + lane, so (j, lane) is row order.
    const int64_t base = tl.row0 + static_cast<int64_t>(w) * (32 * RS_ITEMS);
    IMG img[RS_ITEMS];
    PAY pay[W ? 1 : RS_ITEMS];
    unsigned rank2[RS_ITEMS / 2];  // two 16-bit ranks per word
    const unsigned lt = (1u << lane) - 1;
    if constexpr (SEG && W != 0) seg_images<RS_ITEMS, WHOLE>(seg, a.digits, base + lane, tl.end, img);
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        const int64_t r = base + j * 32 + lane;
        const bool in = WHOLE || r < tl.end;
        if constexpr (SEG && W != 0) {
        } else if constexpr (W != 0) {
            img[j] = in ? static_cast<IMG>(key_image<W>(a.k, r)) : IMG(0);
        } else {
            img[j] = in ? __ldcs(a.img_in + r) : IMG(0);
            pay[j] = in ? __ldcs(a.pay_in + r) : PAY(0);
        }
    }
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        const bool in = WHOLE || base + j * 32 + lane < tl.end;
        const unsigned d = static_cast<unsigned>(img[j] >> shift) & 0xffu;
        // Rank among this warp's earlier rows with the same digit.
        const unsigned peers = digit_peers(d, WHOLE ? FULL : __ballot_sync(FULL, in));
        const unsigned before = sm.w[w][d];
        __syncwarp();
        if (in) {
            const unsigned rk = before + __popc(peers & lt);
            rank2[j / 2] = (j & 1) ? (rank2[j / 2] | (rk << 16)) : rk;
            if ((peers & lt) == 0) sm.w[w][d] = static_cast<unsigned short>(before + __popc(peers));
        }
        __syncwarp();
    }
    __syncthreads();
    // Per digit: the digit's first row in the tile sorted by digit, and each warp's within it.
    {
        const int d = threadIdx.x;
        unsigned c[RS_WARPS], total = 0;
#pragma unroll
        for (int ww = 0; ww < RS_WARPS; ++ww) {
            c[ww] = sm.w[ww][d];
            total += c[ww];
        }
        unsigned tile_total;
        unsigned start = block_exclusive_sum<unsigned>(total, &tile_total);
        sm.excl[d] -= start;
#pragma unroll
        for (int ww = 0; ww < RS_WARPS; ++ww) {
            sm.w[ww][d] = static_cast<unsigned short>(start);
            start += c[ww];
        }
    }
    __syncthreads();
    // The tile sorted by digit (stable) in shared memory, then written out with consecutive
    // threads on consecutive rows of each digit's run, so the stores coalesce.
    PAY *s_pay = reinterpret_cast<PAY *>(smem);
    IMG *s_img = reinterpret_cast<IMG *>(smem + sizeof(PAY) * RS_TILE);
#pragma unroll
    for (int j = 0; j < RS_ITEMS; ++j) {
        if (WHOLE || base + j * 32 + lane < tl.end) {
            const unsigned l = sm.w[w][static_cast<unsigned>(img[j] >> shift) & 0xffu] +
                               ((rank2[j / 2] >> (16 * (j & 1))) & 0xffffu);
            s_img[l] = img[j];
            if constexpr (W != 0) s_pay[l] = static_cast<PAY>(base + j * 32 + lane - (SEG ? seg.base : 0));
            else s_pay[l] = pay[j];
        }
    }
    __syncthreads();
    long long *const out = seg.out - seg.base;
    auto put = [&](int l) {
        const IMG im = s_img[l];
        const unsigned dst = sm.excl[static_cast<unsigned>(im >> shift) & 0xffu] + static_cast<unsigned>(l);
        if constexpr (OUT == OUT_ROWS) {
            a.out[dst] = static_cast<long long>(s_pay[l]);
        } else if constexpr (OUT == OUT_BATCH && SEG) {
            out[dst] = static_cast<long long>(s_pay[l]);
        } else if constexpr (OUT == OUT_BATCH) {
            const unsigned i = static_cast<unsigned>(im >> a.batch.index_shift);
            const int64_t first = __ldg(a.batch.bases + i);
            reinterpret_cast<long long *>(__ldg(a.batch.outs + i))[dst - first] = static_cast<long long>(s_pay[l]) - first;
        } else {
            a.img_out[dst] = im;
            a.pay_out[dst] = s_pay[l];
        }
    };
    if (WHOLE) {
#pragma unroll
        for (int i = 0; i < RS_ITEMS; ++i) put(static_cast<int>(threadIdx.x) + i * RS_THREADS);
    } else {
        const int rows = static_cast<int>(tl.end - tl.row0);
        for (int l = threadIdx.x; l < rows; l += RS_THREADS) put(l);
    }
}

template <int RS_ITEMS, int W, int OUT, bool SEG, class IMG, class PAY>
__global__ void __launch_bounds__(RS_THREADS, (RsShape<RS_ITEMS, sizeof(IMG) + sizeof(PAY)>::MIN_BLOCKS))
    rs_down_kernel(RsArgs<IMG, PAY> a, int64_t n, int shift, int tiles, const unsigned *offsets) {
    chain_enter();
    a.img_in = chained(a.img_in);
    a.pay_in = chained(a.pay_in);
    a.k.keys = chained(a.k.keys);
    __shared__ RsShared sm;
    extern __shared__ __align__(16) unsigned char rs_smem[];
    const int tile = blockIdx.x;
    const SortSeg seg = SEG ? a.segs[a.tile_seg[tile]] : SortSeg{};
    const RsTile tl = rs_tile<SEG, RS_THREADS * RS_ITEMS>(seg, n, tiles, tile);
    for (int i = threadIdx.x; i < RS_WARPS * RADIX / 2; i += RS_THREADS) reinterpret_cast<unsigned *>(&sm.w[0][0])[i] = 0u;
    sm.excl[threadIdx.x] = offsets[tl.at + threadIdx.x * tl.stride];  // RS_THREADS == RADIX
    __syncthreads();
    if (tl.row0 + RS_THREADS * RS_ITEMS <= tl.end)
        rs_down_tile<RS_ITEMS, W, OUT, SEG, IMG, PAY, true>(a, seg, tl, shift, sm, rs_smem);
    else
        rs_down_tile<RS_ITEMS, W, OUT, SEG, IMG, PAY, false>(a, seg, tl, shift, sm, rs_smem);
}

// One pass in the tuned shape: up, the scan, down.
template <int ITEMS, int W, int OUT, class IMG, class PAY, bool SEG = false>
static void radix_pass_shape(vkc_ctx *ctx, const RsArgs<IMG, PAY> &a, int64_t n, int shift, const RadixTables &t, int seg_tiles = 0) {
    using S = RsShape<ITEMS, sizeof(IMG) + sizeof(PAY)>;
    static std::atomic<unsigned long long> configured{0};
    once_per_device(configured, ctx->device, [] {
        cudaFuncSetAttribute(rs_down_kernel<ITEMS, W, OUT, SEG, IMG, PAY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(S::DOWN_SMEM));
    });
    const int tiles = SEG ? seg_tiles : static_cast<int>((n + S::TILE - 1) / S::TILE);
    launch_next(rs_up_kernel<ITEMS, W, SEG, IMG>, tiles, RS_THREADS, 0, ctx->stream, a.k, a.img_in, n, shift, tiles, t.counts, a.segs,
                a.tile_seg, a.digits);
    scan_counts(ctx, t.counts, static_cast<int64_t>(RADIX) * tiles, t.sums, t.offs);
    launch_next(rs_down_kernel<ITEMS, W, OUT, SEG, IMG, PAY>, tiles, RS_THREADS, S::DOWN_SMEM, ctx->stream, a, n, shift, tiles, t.offs);
}
template <int W, int OUT, class IMG, class PAY>
static vkc_status radix_pass(vkc_ctx *ctx, const RsArgs<IMG, PAY> &a, int64_t n, int shift, const RadixTables &t) {
    switch (tune(ctx, TK_RADIX_ITEMS, n)) {
    case 8: radix_pass_shape<8, W, OUT, IMG, PAY>(ctx, a, n, shift, t); break;
    case 16: radix_pass_shape<16, W, OUT, IMG, PAY>(ctx, a, n, shift, t); break;
    default: radix_pass_shape<12, W, OUT, IMG, PAY>(ctx, a, n, shift, t); break;
    }
    return launched(ctx, "radix_pass");
}

// Words of the passes' tables for n rows: counts and offs each, and sums (for the smallest tile, so
// any tuned shape fits).
void radix_table_words(int64_t n, int64_t *count_words, int64_t *sum_words) {
    const int64_t tiles = (n + RS_MIN_TILE - 1) / RS_MIN_TILE;
    *count_words = static_cast<int64_t>(RADIX) * tiles;
    *sum_words = scan_counts_sum_words(*count_words);
}

template <class IMG, class PAY>
vkc_status radix_pairs(vkc_ctx *ctx, const RadixPairs<IMG, PAY> &p, int64_t n, const int *shifts, int passes,
                       const RadixTables &t, int *which) {
    int cur = 0;
    for (int i = 0; i < passes; ++i) {
        RsArgs<IMG, PAY> a{};
        a.img_in = i ? p.img[cur] : p.img_first;
        a.pay_in = i ? p.pay[cur] : p.pay_first;
        const int to = i ? 1 - cur : 0;
        a.img_out = p.img[to];
        a.pay_out = p.pay[to];
        const vkc_status st = radix_pass<0, OUT_PAIRS>(ctx, a, n, shifts[i], t);
        if (st) return st;
        cur = to;
    }
    *which = cur;
    return VKC_OK;
}
template vkc_status radix_pairs(vkc_ctx *, const RadixPairs<unsigned, unsigned long long> &, int64_t, const int *, int,
                                const RadixTables &, int *);

// The passes of an argsort: images from keys of W bytes, row numbers as payloads; the last pass
// writes OUT. img and pos hold two buffers of n rows each (the second is read only by three passes
// or more, the first only by two or more).
template <int W, int OUT, class IMG>
static vkc_status radix_argsort(vkc_ctx *ctx, const KeySource &k, IMG *const img[2], unsigned *const pos[2], long long *out,
                                const BatchOut &batch, int64_t n, const int *shifts, int passes, const RadixTables &t) {
    vkc_status st;
    int cur = 0;
    for (int i = 0; i < passes; ++i) {
        RsArgs<IMG, unsigned> a{};
        a.k = k;
        a.out = out;
        a.batch = batch;
        a.img_in = img[cur];
        a.pay_in = pos[cur];
        const int to = i ? 1 - cur : 0;
        a.img_out = img[to];
        a.pay_out = pos[to];
        const bool last = i == passes - 1;
        if (i == 0) st = last ? radix_pass<W, OUT>(ctx, a, n, shifts[i], t) : radix_pass<W, OUT_PAIRS>(ctx, a, n, shifts[i], t);
        else st = last ? radix_pass<0, OUT>(ctx, a, n, shifts[i], t) : radix_pass<0, OUT_PAIRS>(ctx, a, n, shifts[i], t);
        if (st) return st;
        cur = to;
    }
    return VKC_OK;
}

template <int ITEMS, class IMG>
static vkc_status segs_argsort(vkc_ctx *ctx, const BatchSegs &b, IMG *const img[2], unsigned *const pos[2], int64_t n,
                               const RadixTables &t) {
    int cur = 0;
    for (int i = 0; i < b.digits.n; ++i) {
        RsArgs<IMG, unsigned> a{};
        a.segs = b.segs;
        a.tile_seg = b.tile_seg;
        a.digits = b.digits;
        a.img_in = img[cur];
        a.pay_in = pos[cur];
        const int to = i ? 1 - cur : 0, shift = 8 * i;
        a.img_out = img[to];
        a.pay_out = pos[to];
        const bool last = i == b.digits.n - 1;
        if (i == 0 && last) radix_pass_shape<ITEMS, 8, OUT_BATCH, IMG, unsigned, true>(ctx, a, n, shift, t, b.tiles);
        else if (i == 0) radix_pass_shape<ITEMS, 8, OUT_PAIRS, IMG, unsigned, true>(ctx, a, n, shift, t, b.tiles);
        else if (last) radix_pass_shape<ITEMS, 0, OUT_BATCH, IMG, unsigned, true>(ctx, a, n, shift, t, b.tiles);
        else radix_pass_shape<ITEMS, 0, OUT_PAIRS, IMG, unsigned, true>(ctx, a, n, shift, t, b.tiles);
        const vkc_status st = launched(ctx, "radix_segs");
        if (st) return st;
        cur = to;
    }
    return VKC_OK;
}
vkc_status radix_segs(vkc_ctx *ctx, const BatchSegs &b, void *const img[2], unsigned *const pos[2], int64_t n,
                      const RadixTables &t) {
    if (b.digits.n > 4) {
        unsigned long long *w[2] = {static_cast<unsigned long long *>(img[0]), static_cast<unsigned long long *>(img[1])};
        return b.tile == RS_THREADS * 8 ? segs_argsort<8>(ctx, b, w, pos, n, t) : segs_argsort<12>(ctx, b, w, pos, n, t);
    }
    unsigned *w[2] = {static_cast<unsigned *>(img[0]), static_cast<unsigned *>(img[1])};
    return b.tile == RS_THREADS * 8 ? segs_argsort<8>(ctx, b, w, pos, n, t) : segs_argsort<12>(ctx, b, w, pos, n, t);
}

vkc_status radix_batch(vkc_ctx *ctx, bool wide, const void *images, void *const img[2], unsigned *const pos[2],
                       const BatchOut &batch, int64_t n, const int *shifts, int passes, const RadixTables &t) {
    const KeySource k{images, 0ull, 0ull};
    if (wide) {
        unsigned long long *b[2] = {static_cast<unsigned long long *>(img[0]), static_cast<unsigned long long *>(img[1])};
        return radix_argsort<8, OUT_BATCH, unsigned long long>(ctx, k, b, pos, nullptr, batch, n, shifts, passes, t);
    }
    unsigned *b[2] = {static_cast<unsigned *>(img[0]), static_cast<unsigned *>(img[1])};
    return radix_argsort<4, OUT_BATCH, unsigned>(ctx, k, b, pos, nullptr, batch, n, shifts, passes, t);
}

// The two halves of a batched argsort whose key digits and array number do not fit one image: the
// stable order by the 64-bit key images, then by the array numbers (images_n, payloads pay_n).
vkc_status radix_batch_keys(vkc_ctx *ctx, const void *images, void *const img[2], unsigned *const pos[2], int64_t n,
                            const int *shifts, int passes, const RadixTables &t) {
    unsigned long long *b[2] = {static_cast<unsigned long long *>(img[0]), static_cast<unsigned long long *>(img[1])};
    return radix_argsort<8, OUT_PAIRS, unsigned long long>(ctx, KeySource{images, 0ull, 0ull}, b, pos, nullptr, BatchOut{}, n,
                                                           shifts, passes, t);
}
vkc_status radix_batch_numbers(vkc_ctx *ctx, const unsigned *numbers, const unsigned *pay, unsigned *img_tmp,
                               unsigned *pay_tmp, const BatchOut &batch, int64_t n, int passes, const RadixTables &t) {
    RsArgs<unsigned, unsigned> a{};
    a.batch = batch;
    a.img_in = numbers;
    a.pay_in = pay;
    a.img_out = img_tmp;
    a.pay_out = pay_tmp;
    if (passes == 1) return radix_pass<0, OUT_BATCH>(ctx, a, n, 0, t);
    vkc_status st = radix_pass<0, OUT_PAIRS>(ctx, a, n, 0, t);
    if (st) return st;
    a.img_in = img_tmp;
    a.pay_in = pay_tmp;
    return radix_pass<0, OUT_BATCH>(ctx, a, n, 8, t);
}

__global__ void rs_iota_kernel(long long *out, int64_t n) {
    int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = i;
}

// Short inputs (the reference sorts up to 1024 rows by comparison, radix.rs:140-151): one
// block sorts (image, position) pairs in shared memory with a bitonic network. The pairs are
// distinct, so the order is total and the result is the stable order; padding pairs (all-ones
// image, position >= n) sort after every row.
constexpr int SMALL_SORT = 2048;

template <int W>
__global__ void __launch_bounds__(1024) small_argsort_kernel(KeySource key, int n, long long *__restrict__ out) {
    __shared__ unsigned long long s_img[SMALL_SORT];
    __shared__ unsigned s_pos[SMALL_SORT];
    int p = 1;
    while (p < n) p <<= 1;
    for (int i = threadIdx.x; i < p; i += blockDim.x) {
        s_img[i] = i < n ? key_image<W>(key, i) : ~0ull;
        s_pos[i] = static_cast<unsigned>(i);
    }
    __syncthreads();
    for (int k = 2; k <= p; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < p; i += blockDim.x) {
                const int l = i ^ j;
                if (l > i) {
                    const unsigned long long a = s_img[i], b = s_img[l];
                    const unsigned pa = s_pos[i], pb = s_pos[l];
                    const bool greater = a > b || (a == b && pa > pb);
                    if (greater == ((i & k) == 0)) {
                        s_img[i] = b;
                        s_img[l] = a;
                        s_pos[i] = pb;
                        s_pos[l] = pa;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = static_cast<long long>(s_pos[i]);
}

// Inputs of at most MID_SORT rows: one block of 1024 threads sorts (image, position) pairs in
// shared memory by the LSD passes of the active digits (the digits not equal in every row,
// found by a block-wide AND and OR of the images), each pass ranked stably as the down pass
// does (per warp, a ballot per digit bit; warp w holds rows 256w .. 256w + 255), one launch and
// no host synchronisation.
constexpr int MID_SORT = 8192;
constexpr int MID_THREADS = 1024, MID_ITEMS = MID_SORT / MID_THREADS, MID_WARPS = MID_THREADS / 32;
struct MidSmem {
    unsigned long long img[2][MID_SORT];
    unsigned short pos[2][MID_SORT];
    unsigned short wcnt[MID_WARPS][RADIX];  // per-warp digit counts, then offsets within the digit
    unsigned dstart[RADIX];                 // the digit's first row
    unsigned long long all_and[MID_WARPS], all_or[MID_WARPS];
};

template <int W>
__global__ void __launch_bounds__(MID_THREADS) mid_argsort_kernel(KeySource key, int n, long long *__restrict__ out) {
    extern __shared__ __align__(16) unsigned char mid_smem[];
    MidSmem &sm = *reinterpret_cast<MidSmem *>(mid_smem);
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    unsigned long long a = ~0ull, o = 0;
    for (int i = t; i < n; i += MID_THREADS) {
        const unsigned long long im = key_image<W>(key, i);
        sm.img[0][i] = im;
        sm.pos[0][i] = static_cast<unsigned short>(i);
        a &= im;
        o |= im;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a &= __shfl_xor_sync(FULL, a, off);
        o |= __shfl_xor_sync(FULL, o, off);
    }
    if (lane == 0) {
        sm.all_and[w] = a;
        sm.all_or[w] = o;
    }
    __syncthreads();
    a = ~0ull;
    o = 0;
#pragma unroll 4
    for (int k = 0; k < MID_WARPS; ++k) {
        a &= sm.all_and[k];
        o |= sm.all_or[k];
    }
    const unsigned long long varies = a ^ o;  // bits that differ between rows
    int cur = 0;
    const unsigned lt = (1u << lane) - 1;
    for (int shift = 0; shift < 64; shift += 8) {
        if (((varies >> shift) & 0xffu) == 0) continue;  // a constant digit leaves the order as it is
        for (int i = t; i < MID_WARPS * RADIX; i += MID_THREADS) (&sm.wcnt[0][0])[i] = 0;
        __syncthreads();
        unsigned long long img[MID_ITEMS];
        unsigned short pos[MID_ITEMS];
        unsigned rank2[MID_ITEMS / 2];
        const int base = w * (32 * MID_ITEMS);
#pragma unroll
        for (int j = 0; j < MID_ITEMS; ++j) {
            const int r = base + j * 32 + lane;
            img[j] = r < n ? sm.img[cur][r] : ~0ull;
            pos[j] = r < n ? sm.pos[cur][r] : 0;
        }
#pragma unroll
        for (int j = 0; j < MID_ITEMS; ++j) {
            const bool in = base + j * 32 + lane < n;
            const unsigned d = static_cast<unsigned>(img[j] >> shift) & 0xffu;
            const unsigned peers = digit_peers(d, __ballot_sync(FULL, in));
            const unsigned short before = sm.wcnt[w][d];
            __syncwarp();
            if (in) {
                const unsigned rk = before + __popc(peers & lt);
                rank2[j / 2] = (j & 1) ? (rank2[j / 2] | (rk << 16)) : rk;
                if ((peers & lt) == 0) sm.wcnt[w][d] = static_cast<unsigned short>(before + __popc(peers));
            }
            __syncwarp();
        }
        __syncthreads();
        // Per digit: the warps' offsets within it (threads 0..255), then the digits' first rows
        // (warp 0, eight digits a lane).
        unsigned total = 0;
        if (t < RADIX) {
#pragma unroll 4
            for (int ww = 0; ww < MID_WARPS; ++ww) {
                const unsigned c = sm.wcnt[ww][t];
                sm.wcnt[ww][t] = static_cast<unsigned short>(total);
                total += c;
            }
            sm.dstart[t] = total;
        }
        __syncthreads();
        if (t < 32) {
            unsigned v[8], run = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                v[k] = sm.dstart[8 * t + k];
                run += v[k];
            }
            unsigned x = run;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned y = __shfl_up_sync(FULL, x, off);
                if (lane >= off) x += y;
            }
            unsigned ex = x - run;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                sm.dstart[8 * t + k] = ex;
                ex += v[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < MID_ITEMS; ++j) {
            if (base + j * 32 + lane < n) {
                const unsigned d = static_cast<unsigned>(img[j] >> shift) & 0xffu;
                const unsigned l = sm.dstart[d] + sm.wcnt[w][d] + ((rank2[j / 2] >> (16 * (j & 1))) & 0xffffu);
                sm.img[cur ^ 1][l] = img[j];
                sm.pos[cur ^ 1][l] = pos[j];
            }
        }
        __syncthreads();
        cur ^= 1;
    }
    for (int i = t; i < n; i += MID_THREADS) out[i] = static_cast<long long>(sm.pos[cur][i]);
}

// index.rs:159-173 (ArgSort::run).
template <vkc_type T> static vkc_status argsort(vkc_ctx *ctx, const vkc_value *args, int nargs, vkc_value *out) {
    constexpr int W = T == VKC_I64 || T == VKC_U64 ? 8 : (T == VKC_I32 ? 4 : 1);
    vkc_status st;
    if (nargs != 1) return fail(ctx, VKC_RUNTIME, arity_error(1, nargs));
    if (!array_arg(ctx, args[0], T, &st)) return st;
    const vkc_array *xs = args[0].array;
    int64_t n = xs->len;
    if (n >= (int64_t(1) << 32))
        return fail(ctx, VKC_USAGE, "argsort of " + std::to_string(n) + " rows: at most 2^32 - 1 rows per call");
    vkc_array *o;
    if ((st = new_array(ctx, VKC_I64, n, false, &o))) return st;
    auto release = [&](vkc_status s) {
        vkc_array_release(o);
        return s;
    };
    auto finish = [&]() {
        out->kind = VKC_VALUE_ARRAY;
        out->array = o;
        return VKC_OK;
    };
    if (n == 0) return finish();
    KeySource key{xs->data(), T == VKC_I64 ? 1ull << 63 : (T == VKC_I32 ? 1ull << 31 : 0ull), 0ull};
    auto *oo = static_cast<long long *>(o->data());
    if (n <= SMALL_SORT) {
        small_argsort_kernel<W><<<1, 1024, 0, ctx->stream>>>(key, static_cast<int>(n), oo);
        if ((st = launched(ctx, "small_argsort"))) return release(st);
        return finish();
    }
    if (n <= MID_SORT) {
        static std::atomic<unsigned long long> configured{0};
        once_per_device(configured, ctx->device, [] {
            cudaFuncSetAttribute(mid_argsort_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(MidSmem)));
        });
        mid_argsort_kernel<W><<<1, MID_THREADS, sizeof(MidSmem), ctx->stream>>>(key, static_cast<int>(n), oo);
        if ((st = launched(ctx, "mid_argsort"))) return release(st);
        return finish();
    }
    // The images' range and varying bits.
    void *p, *h;
    if ((st = scratch(ctx, 4 * sizeof(unsigned long long), &p))) return release(st);
    auto *range = static_cast<unsigned long long *>(p);
    VKC_CUDA(ctx, cudaMemsetAsync(range, 0xff, 16, ctx->stream));
    VKC_CUDA(ctx, cudaMemsetAsync(range + 2, 0, 16, ctx->stream));
    rs_range_kernel<W><<<stream_grid(ctx, n, 256, 6, 16384), 256, 0, ctx->stream>>>(key, n, range);
    if ((st = launched(ctx, "rs_range"))) return release(st);
    if ((st = pinned(ctx, 32, &h))) return release(st);
    VKC_CUDA(ctx, cudaMemcpyAsync(h, range, 32, cudaMemcpyDeviceToHost, ctx->stream));
    VKC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const auto *r = static_cast<const unsigned long long *>(h);
    const unsigned long long varies = r[0] ^ r[2], spread = r[3] - r[1], least = r[1];
    int shifts[8], passes = 0, wide = 0;
    for (int b = 0; b < 8; ++b) {
        if ((varies >> (8 * b)) & 0xffu) shifts[passes++] = 8 * b;
        if (spread >> (8 * b)) ++wide;
    }
    if (wide < passes || (wide == passes && passes > 0 && spread >> 32 == 0 && shifts[passes - 1] >= 32)) {
        // Fewer bytes (or as many, in narrower images) in the distance from the least image.
        key.low = least;
        passes = wide;
        for (int b = 0; b < wide; ++b) shifts[b] = 8 * b;
    }
    if (passes == 0) {
        rs_iota_kernel<<<stream_grid(ctx, n, 256, 8, 2048), 256, 0, ctx->stream>>>(oo, n);
        if ((st = launched(ctx, "rs_iota"))) return release(st);
        return finish();
    }
    // Ping-pong buffers of (image, position), as radix.rs:224-232, and the passes' tables. When
    // every digit lies in the low 32 bits, the passes carry the image's low 32 bits: 16 bytes a
    // row per pass, not 24.
    vkc_array *ia = nullptr, *ib = nullptr, *pa = nullptr, *pb = nullptr, *ca = nullptr, *oa = nullptr, *sa = nullptr;
    auto cleanup = [&]() {
        for (vkc_array *a : {ia, ib, pa, pb, ca, oa, sa})
            if (a) vkc_array_release(a);
    };
    const bool narrow = W < 8 || shifts[passes - 1] < 32;
    const vkc_type img_type = narrow ? VKC_I32 : VKC_U64;
    int64_t cw, sw;
    radix_table_words(n, &cw, &sw);
    if ((passes > 1 && (new_array(ctx, img_type, n, false, &ia) || new_array(ctx, VKC_I32, n, false, &pa))) ||
        (passes > 2 && (new_array(ctx, img_type, n, false, &ib) || new_array(ctx, VKC_I32, n, false, &pb))) ||
        new_array(ctx, VKC_I32, cw, false, &ca) || new_array(ctx, VKC_I32, cw, false, &oa) ||
        new_array(ctx, VKC_I32, sw, false, &sa)) {
        cleanup();
        return release(fail(ctx, VKC_ALLOC, "cannot allocate argsort scratch for " + std::to_string(n) + " rows"));
    }
    auto words = [](vkc_array *a) { return a ? static_cast<unsigned *>(a->data()) : nullptr; };
    const RadixTables t{words(ca), words(oa), words(sa)};
    unsigned *pos[2] = {words(pa), words(pb)};
    if (narrow) {
        unsigned *img[2] = {words(ia), words(ib)};
        st = radix_argsort<W, OUT_ROWS, unsigned>(ctx, key, img, pos, oo, BatchOut{}, n, shifts, passes, t);
    } else if constexpr (W == 8) {
        unsigned long long *img[2] = {ia ? static_cast<unsigned long long *>(ia->data()) : nullptr,
                                      ib ? static_cast<unsigned long long *>(ib->data()) : nullptr};
        st = radix_argsort<8, OUT_ROWS, unsigned long long>(ctx, key, img, pos, oo, BatchOut{}, n, shifts, passes, t);
    }
    cleanup();
    return st ? release(st) : finish();
}

void register_sort(std::vector<KernelDef> &t) {
    // index.rs:241-255, :290-325: cost = key width + 8.
    struct S { vkc_type t; WholeFn f; };
    const S sorts[] = {{VKC_I64, argsort<VKC_I64>}, {VKC_U64, argsort<VKC_U64>}, {VKC_I32, argsort<VKC_I32>},
                       {VKC_U8, argsort<VKC_U8>}};
    for (const S &s : sorts) {
        KernelDef d{std::string("argsort_") + type_name(s.t), VKC_WHOLE, {InSpec{IN_ARRAY, s.t}}, true, VKC_I64,
                    static_cast<uint64_t>(type_width(s.t) + 8)};
        d.whole = s.f;
        t.push_back(d);
    }
}

}  // namespace vkc
