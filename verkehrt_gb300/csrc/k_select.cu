// Selections: filter_<cmp>_T, compress_T and where (src/kernels/scalar/select.rs:81-104,
// src/kernels/scalar/fused.rs:214-236).
//
// One persistent pass (tilepass.cuh): each tile is copied into shared memory by TMA, its survivor count
// goes to the decoupled lookback, its survivors are put side by side, and then written out at the tile's
// offset. The output is the rows in input order, so it does not depend on the
// tiling (select.rs:36-57 writes the same rows).
#include <cmath>

#include "reduce_common.h"
#include "tilepass.cuh"

namespace vkc {

constexpr int SEL_THREADS = 512;          // compute threads (+ 2 warps)
constexpr int SEL_TILE = 8192;                             // rows per tile (8-byte rows)
constexpr int SEL_SLICE = SEL_TILE / (SEL_THREADS / 32);   // rows per compute warp
constexpr int SEL_SLOTS = 3;                               // tile ring: 1 copy in flight
// (Filter tiles of 6144 rows in four slots, two copies in flight, were slower at 2^28: 0.56
// against 0.46 ms at 1% kept; a third more tiles meet the lookback rate.)
constexpr int SEL_WINDOW = 4;             // lookback: 32 * 4 tiles per step
constexpr int SEL_SMEM = 225 * 1024;      // of the slots and the output rows

enum SelKind { SEL_FILTER = 0, SEL_COMPRESS = 1, SEL_WHERE = 2 };

template <int W> struct Word;
template <> struct Word<8> { using T = unsigned long long; using S = long long; };
template <> struct Word<4> { using T = unsigned; using S = int; };
template <> struct Word<1> { using T = unsigned char; using S = signed char; };

// A filter's predicate on a row's bits b: (key(b) - lo <= span) != negate, unsigned. Integers are their
// own keys (of either sign: the difference wraps), floats their signed order keys (KEYED), or their bits
// where the range is one of non-negative keys: negative values and NaNs lie above every such range.
struct SelRange {
    unsigned long long lo, span;
    bool negate, keyed;
};

struct SelArgs {
    const void *x;          // values (filter, compress)
    const unsigned char *m; // mask (compress, where)
    SelRange r;             // filter predicate
    int64_t n;
    int64_t base;           // where: global row of row 0
    void *out;
    unsigned long long *total;  // survivor count of the launch
    unsigned long long *host;   // pinned: the count and the status word's timeout, written by the last block
    bool aligned;           // values and mask start on 16-byte boundaries
};

template <int W, bool KEYED> __device__ __forceinline__ bool sel_keep(const SelRange &r, typename Word<W>::T b) {
    using T = typename Word<W>::T;
    using S = typename Word<W>::S;
    const T k = KEYED ? static_cast<T>(b ^ (static_cast<T>(static_cast<S>(b) >> (8 * W - 1)) >> 1)) : b;
    return (static_cast<T>(k - static_cast<T>(r.lo)) <= static_cast<T>(r.span)) != r.negate;
}

// Nonzero bytes of a 32-bit word.
__device__ __forceinline__ unsigned nonzero_bytes(unsigned v) {
    const unsigned t = ~(((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v | 0x7f7f7f7fu);  // 0x80 per zero byte
    return 4u - __popc(t);
}

// A selection of 8-byte rows as a tile pass. A slot holds the tile's values and (compress) mask; the
// survivors are compacted into the values in place. A compute warp's slice is SEL_SLICE consecutive rows,
// read in steps of VV rows per lane, ranked with ballots, and copied out with consecutive lanes on
// consecutive rows. A filter's count keeps its ballots in the slot, so the stage touches
// only the steps and rows that survive. A tile that is not whole, or not 16-byte aligned, is
// read from global memory instead of the slot.
template <int KIND, bool KEYED> struct SelectPass {
    static constexpr int THREADS = SEL_THREADS;
    static constexpr bool ONE_READ = false;
    using R = CountRec;
    using V = unsigned long long;
    using T = unsigned long long;
    static constexpr int TILE = SEL_TILE;
    static constexpr int VAL_BYTES = 8 * SEL_TILE;
    static constexpr int MASK_BYTES = KIND == SEL_FILTER ? 0 : SEL_TILE;
    static constexpr int VK = KIND == SEL_FILTER ? 2 : 16;  // keys per lane per count step
    static constexpr int SK = SEL_SLICE / (32 * VK);
    static constexpr int BALLOT_BYTES = KIND == SEL_FILTER ? (SEL_THREADS / 32) * SK * 8 : 0;
    static constexpr int SLOT_BYTES = VAL_BYTES + MASK_BYTES + BALLOT_BYTES;
    static constexpr int SLOTS = SEL_SLOTS;
    static constexpr int OUT_BYTES = 0;  // behind the slots
    static constexpr int VV = 2;  // rows per lane per stage step
    static constexpr int SV = SEL_SLICE / (32 * VV);
    static_assert(SK >= 1 && SV >= 1, "a slice holds whole steps");
    static_assert(KIND != SEL_FILTER || SK <= 32, "one lane stores each step's ballots");
    using Staged = unsigned;  // survivors compacted in the warp's slice

    SelArgs a;

    __device__ bool whole(int tile) const {
        return a.aligned && static_cast<int64_t>(tile + 1) * SEL_TILE <= a.n;
    }
    __device__ unsigned bulk_bytes(int tile) const { return whole(tile) ? VAL_BYTES + MASK_BYTES : 0u; }
    __device__ void load(int tile, unsigned char *slot, unsigned long long *bar) const {
        const int64_t r0 = static_cast<int64_t>(tile) * SEL_TILE;
        bulk_load(slot, static_cast<const T *>(a.x) + r0, VAL_BYTES, bar);
        if (MASK_BYTES) bulk_load(slot + VAL_BYTES, a.m + r0, MASK_BYTES, bar);
    }
    __device__ bool keep_filter(unsigned long long v) const { return sel_keep<8, KEYED>(a.r, v); }

    // The slice's keys from `keys` (the slot, or global memory at the tile's first row).
    template <class K> __device__ unsigned count_keys(const K *keys, int64_t r0) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const int j = w * SEL_SLICE + lane * VK;  // row in the tile
        unsigned c = 0;
        if (KIND == SEL_FILTER) {
            ulonglong2 u[SK];
#pragma unroll
            for (int s = 0; s < SK; ++s) u[s] = *reinterpret_cast<const ulonglong2 *>(keys + j + s * 64);
#pragma unroll
            for (int s = 0; s < SK; ++s) c += keep_filter(u[s].x) + keep_filter(u[s].y);
        } else {
#pragma unroll
            for (int s = 0; s < SK; ++s) {
                const uint4 u = *reinterpret_cast<const uint4 *>(keys + j + s * 512);
                c += nonzero_bytes(u.x) + nonzero_bytes(u.y) + nonzero_bytes(u.z) + nonzero_bytes(u.w);
            }
        }
        return c;
    }

    // The filter's ballots of the warp's slice: step s, element e in [s].(x, y).
    __device__ uint2 *ballots(unsigned char *slot) const {
        return reinterpret_cast<uint2 *>(slot + VAL_BYTES + MASK_BYTES) + (threadIdx.x >> 5) * SK;
    }

    __device__ V count(int tile, unsigned char *slot) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const int64_t r0 = static_cast<int64_t>(tile) * SEL_TILE;
        unsigned c = 0;
        if (KIND == SEL_FILTER && whole(tile)) {
            const auto *k = reinterpret_cast<const unsigned long long *>(slot) + w * SEL_SLICE + lane * 2;
            uint2 *mb = ballots(slot);
            ulonglong2 u[SK];
#pragma unroll
            for (int s = 0; s < SK; ++s) u[s] = *reinterpret_cast<const ulonglong2 *>(k + s * 64);
#pragma unroll
            for (int s = 0; s < SK; ++s) {
                const unsigned m0 = __ballot_sync(FULL, keep_filter(u[s].x));
                const unsigned m1 = __ballot_sync(FULL, keep_filter(u[s].y));
                if (lane == s) mb[s] = make_uint2(m0, m1);
                c += __popc(m0) + __popc(m1);
            }
            return c;
        }
        if (whole(tile)) {
            c = KIND == SEL_FILTER ? count_keys(reinterpret_cast<const unsigned long long *>(slot), r0)
                                   : count_keys(slot + VAL_BYTES, r0);
        } else {
            // Row by row from global memory.
            for (int i = lane; i < SEL_SLICE; i += 32) {
                const int64_t r = r0 + w * SEL_SLICE + i;
                if (r >= a.n) break;
                if (KIND == SEL_FILTER) c += keep_filter(static_cast<const unsigned long long *>(a.x)[r]);
                else c += a.m[r] != 0;
            }
        }
        return warp_sum(c);
    }

    __device__ unsigned stage(int tile, unsigned char *slot) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const unsigned lt = (1u << lane) - 1;
        const int64_t r0 = static_cast<int64_t>(tile) * SEL_TILE;
        const bool sm = whole(tile);
        if (KIND == SEL_FILTER && sm) {
            // From the count's ballots: steps with no survivor are skipped, and a lane reads
            // its two rows only when one survives.
            unsigned long long *st = reinterpret_cast<unsigned long long *>(slot) + w * SEL_SLICE;
            const uint2 *mb = ballots(slot);
            unsigned total = 0;
            __syncwarp();
#pragma unroll 4
            for (int s = 0; s < SK; ++s) {
                const uint2 m = mb[s];
                if ((m.x | m.y) == 0) continue;
                const unsigned b = ((m.x >> lane) & 1u) | (((m.y >> lane) & 1u) << 1);
                ulonglong2 u = make_ulonglong2(0, 0);
                if (b) u = *reinterpret_cast<const ulonglong2 *>(st + s * 64 + lane * 2);
                unsigned q = total + __popc(m.x & lt) + __popc(m.y & lt);
                __syncwarp();  // the step is read before any of it is overwritten
                if (b & 1u) st[q++] = u.x;
                if (b & 2u) st[q] = u.y;
                total += __popc(m.x) + __popc(m.y);
            }
            return total;
        }
        T *st = reinterpret_cast<T *>(slot) + w * SEL_SLICE;  // in place
        unsigned total = 0;
#pragma unroll 2
        for (int s = 0; s < SV; ++s) {
            const int j = w * SEL_SLICE + s * (32 * VV) + lane * VV;  // row in the tile
            const int64_t i0 = r0 + j;
            T v[VV];
            unsigned bits = 0;
            if (sm) {
                const ulonglong2 u = *reinterpret_cast<const ulonglong2 *>(reinterpret_cast<const T *>(slot) + j);
                v[0] = u.x;
                v[1] = u.y;
                if (KIND != SEL_FILTER) {
                    const unsigned wd = *reinterpret_cast<const unsigned short *>(slot + VAL_BYTES + j);
                    bits = (wd & 0xffu ? 1u : 0u) | (wd & 0xff00u ? 2u : 0u);
                }
            } else {
#pragma unroll
                for (int k = 0; k < VV; ++k) {
                    const bool in = i0 + k < a.n;
                    v[k] = in ? static_cast<const T *>(a.x)[i0 + k] : T(0);
                    if (KIND != SEL_FILTER && in && a.m[i0 + k]) bits |= 1u << k;
                }
            }
            if (KIND == SEL_FILTER) {
#pragma unroll
                for (int k = 0; k < VV; ++k)
                    if ((sm || i0 + k < a.n) && keep_filter(v[k])) bits |= 1u << k;
            }
            // In-order ranks: the lanes before this one, element by element.
            unsigned before = 0, step_total = 0;
#pragma unroll
            for (int k = 0; k < VV; ++k) {
                const unsigned m = __ballot_sync(FULL, (bits >> k) & 1u);
                before += __popc(m & lt);
                step_total += __popc(m);
            }
            __syncwarp();  // the step is read before any of it is overwritten
            unsigned q = total + before;
#pragma unroll
            for (int k = 0; k < VV; ++k)
                if ((bits >> k) & 1u) {
                    st[q] = v[k];
                    ++q;
                }
            total += step_total;
        }
        return total;
    }

    __device__ void flush(int, V pre, unsigned total, unsigned char *slot) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const T *st = reinterpret_cast<const T *>(slot) + w * SEL_SLICE;
        __syncwarp();
        T *out = static_cast<T *>(a.out) + pre;
        // Pairs of rows as aligned 16-byte stores, after a single row when the output does
        // not start on a 16-byte boundary.
        const unsigned mis = (reinterpret_cast<uintptr_t>(out) & 15) ? 1u : 0u;
        const unsigned head = mis < total ? mis : total;
        if (head && lane == 0) out[0] = st[0];
        const unsigned pairs = (total - head) >> 1;
        for (unsigned i = lane; i < pairs; i += 32) {
            ulonglong2 u;
            u.x = st[head + 2 * i];
            u.y = st[head + 2 * i + 1];
            *reinterpret_cast<ulonglong2 *>(out + head + 2 * i) = u;
        }
        for (unsigned i = head + 2 * pairs + lane; i < total; i += 32) out[i] = st[i];
    }

    __device__ void last_tile(V inclusive) const { *a.total = inclusive; }
};

// `where`, and selections of 4- and 1-byte rows, as a tile pass. A compute warp's slice is ROWS steps of 32 consecutive rows, a row a lane:
// the count reads the values into registers (consecutive lanes on consecutive rows, every bank once) and
// keeps each step's vote in one of the lanes; the flush ranks the survivors by the votes, puts them side
// by side in the warp's output rows in shared memory, placed as the output is within 16 bytes, and sends
// the 16-byte units among them off as one bulk copy. Values and masks off the 16-byte grid are copied
// from the unit that holds their first row (of a slice, a row of the array it is cut from) up to a unit
// past their last, which the array must still hold. A tile that is not whole is read from global memory.
//
// Its instructions bound it, some 14 for 32 rows in the flush. Calls on 2^27 rows with 1 / 50 / 99% kept:
// `where` 259 / 323 / 589 us as a SelectPass of row numbers, now 174 / 172 / 210; a filter of a quarter of
// the f32 rows 474 (a mask of its own, then compress), now 190; compress_i32 of half 256, now 187.
// (Stored from the registers, without the output rows: where 179 / 210 / 227, f32 242. Votes and counts
// before each step from shared memory instead of shuffles: 199 / 196 / 210. 8-byte rows this way: filter
// 328 / 356 / 408 against SelectPass's 264 / 347 / 420, compress 372 / 402 / 435 against 272 / 331 / 407:
// there the lookback bounds it, and SelectPass's count publishes sooner. Off the 16-byte grid, where
// SelectPass reads row by row, a filter of half the rows 1538 there, 361 here; `where` 884 (calls of SelectPass),
// now 180.)
template <int KIND, int W, bool KEYED, int ROWS> struct RankPass {
    static constexpr int THREADS = SEL_THREADS;
    static constexpr bool ONE_READ = true;
    static constexpr int TILE = SEL_THREADS * ROWS;
    static constexpr int SLICE = 32 * ROWS;  // rows of a warp
    using R = CountRec;
    using V = unsigned long long;
    using T = typename Word<W>::T;
    using O = typename Word<KIND == SEL_WHERE ? 8 : W>::T;
    static constexpr int VAL_BYTES = KIND == SEL_WHERE ? 0 : W * TILE;
    static constexpr int MASK_BYTES = KIND == SEL_FILTER ? 0 : TILE;
    static constexpr int MASK_AT = VAL_BYTES ? VAL_BYTES + 16 : 0;
    static constexpr int SLOT_BYTES = MASK_AT + (MASK_BYTES ? MASK_BYTES + 16 : 0);
    // Output rows: of CHUNK steps at a time, in BUFS buffers a warp.
    static constexpr int CHUNK = KIND == SEL_WHERE && ROWS > 16 ? 8 : ROWS, BUFS = CHUNK < ROWS ? 2 : 1;
    static constexpr int UNIT = 16 / static_cast<int>(sizeof(O));  // rows of 16 bytes
    static constexpr int BUF_BYTES = (32 * CHUNK + UNIT) * static_cast<int>(sizeof(O));
    static constexpr int OUT_BYTES = BUFS * BUF_BYTES * (SEL_THREADS / 32);
    static constexpr int SLOTS = (SEL_SMEM - OUT_BYTES) / SLOT_BYTES < 8 ? (SEL_SMEM - OUT_BYTES) / SLOT_BYTES : 8;
    struct Staged {
        T v[KIND == SEL_WHERE ? 1 : ROWS];
        unsigned vote[(ROWS + 31) / 32];  // lane l: the votes of steps l, l + 32
    };

    SelArgs a;

    // Bytes of the first value, and mask byte, within their 16-byte units.
    __device__ unsigned x_off() const { return VAL_BYTES ? static_cast<unsigned>(reinterpret_cast<uintptr_t>(a.x) & 15) : 0u; }
    __device__ unsigned m_off() const { return MASK_BYTES ? static_cast<unsigned>(reinterpret_cast<uintptr_t>(a.m) & 15) : 0u; }
    __device__ bool whole(int tile) const { return static_cast<int64_t>(tile + 1) * TILE + (a.aligned ? 0 : 16) <= a.n; }
    __device__ unsigned bulk_bytes(int tile) const {
        return whole(tile) ? VAL_BYTES + (x_off() ? 16 : 0) + MASK_BYTES + (m_off() ? 16 : 0) : 0u;
    }
    __device__ void load(int tile, unsigned char *slot, unsigned long long *bar) const {
        const int64_t r0 = static_cast<int64_t>(tile) * TILE;
        const unsigned xo = x_off(), mo = m_off();
        if (VAL_BYTES) bulk_load(slot, static_cast<const unsigned char *>(a.x) + r0 * W - xo, VAL_BYTES + (xo ? 16 : 0), bar);
        if (MASK_BYTES) bulk_load(slot + MASK_AT, a.m + r0 - mo, MASK_BYTES + (mo ? 16 : 0), bar);
    }

    template <bool SLOT> __device__ __forceinline__ void vote_rows(const unsigned char *slot, int64_t r0, Staged &st) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const T *xs = reinterpret_cast<const T *>(slot + x_off());
        const unsigned char *ms = slot + MASK_AT + m_off();
#pragma unroll
        for (int g = 0; g < ROWS; ++g) {
            const int j = w * SLICE + g * 32 + lane;  // in the tile
            bool keep = SLOT || r0 + j < a.n;
            T v = 0;
            if constexpr (KIND != SEL_WHERE) {
                if (SLOT) v = xs[j];
                else if (keep) v = static_cast<const T *>(a.x)[r0 + j];
                st.v[g] = v;
            }
            if (KIND == SEL_FILTER) keep = keep && sel_keep<W, KEYED>(a.r, v);
            else if (SLOT) keep = ms[j] != 0;
            else if (keep) keep = a.m[r0 + j] != 0;
            const unsigned m = __ballot_sync(FULL, keep);
            if (lane == (g & 31)) st.vote[g >> 5] = m;
        }
    }

    __device__ __forceinline__ V count(int tile, const unsigned char *slot, Staged &st) const {
        const int64_t r0 = static_cast<int64_t>(tile) * TILE;
#pragma unroll
        for (int i = 0; i < (ROWS + 31) / 32; ++i) st.vote[i] = 0;
        if (whole(tile)) vote_rows<true>(slot, r0, st);
        else vote_rows<false>(slot, r0, st);
        unsigned c = 0;
#pragma unroll
        for (int i = 0; i < (ROWS + 31) / 32; ++i) c += __popc(st.vote[i]);
        return __reduce_add_sync(FULL, c);
    }

    __device__ __forceinline__ void flush(int tile, V pre, const Staged &st, unsigned char *rows) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const unsigned lt = (1u << lane) - 1u;
        const int64_t i0 = a.base + static_cast<int64_t>(tile) * TILE + w * SLICE + lane;
        O *out = static_cast<O *>(a.out) + pre;
#pragma unroll
        for (int c = 0; c < ROWS / CHUNK; ++c) {
            O *buf = reinterpret_cast<O *>(rows + (w * BUFS + c % BUFS) * BUF_BYTES);
            if (lane == 0) bulk_store_wait_read<BUFS - 1>();  // the copy out of this buffer
            __syncwarp();
            const unsigned mis = static_cast<unsigned>(reinterpret_cast<uintptr_t>(out) / sizeof(O)) % UNIT;
            O *at = buf + mis;
            unsigned total = 0;
#pragma unroll
            for (int g = c * CHUNK; g < (c + 1) * CHUNK; ++g) {
                const unsigned m = __shfl_sync(FULL, st.vote[g >> 5], g & 31);
                const unsigned q = total + __popc(m & lt);
                if ((m >> lane) & 1u) {
                    if constexpr (KIND == SEL_WHERE) at[q] = static_cast<O>(i0 + g * 32);
                    else at[q] = st.v[g];
                }
                total += __popc(m);
            }
            fence_proxy_async();
            __syncwarp();
            const unsigned head = min(total, (UNIT - mis) % UNIT), body = (total - head) / UNIT * UNIT;
            const unsigned rest = total - head - body;
            if (lane == 0 && body) bulk_store(out + head, at + head, body * sizeof(O));
            if (lane < head) out[lane] = at[lane];
            if (lane < rest) out[head + body + lane] = at[head + body + lane];
            out += total;
        }
    }
    // The copies are done before the block ends.
    __device__ void finish() const {
        if ((threadIdx.x & 31) == 0) bulk_store_wait();
    }
    __device__ void last_tile(V inclusive) const { *a.total = inclusive; }
};

template <class P>
__global__ void __launch_bounds__(SEL_THREADS + 64, 1) select_kernel(SelArgs a, int tiles, unsigned long long *recs,
                                                                     unsigned epoch, unsigned *counters,
                                                                     DevStatus *status) {
    P p{a};
    if (tile_pass<SEL_WINDOW>(p, recs, tiles, epoch, counters, status, 0ull) && threadIdx.x == 0) {
        a.host[0] = *a.total;
        a.host[1] = *reinterpret_cast<volatile unsigned *>(&status->timeout);
    }
}

// Few rows: one block, every row in a register (row 32 j + lane of warp w's slice in v[j]), ranked by
// ballots and one scan of the warps' counts. The tile pass takes 17 us for a thousand rows (its only
// tile is read row by row, and twice), this one about 3 (calls of 4096 rows 38 -> 19 us).
constexpr int SEL_SMALL_ITEMS = 16, SEL_SMALL = 1024 * SEL_SMALL_ITEMS;

template <int KIND, int W, bool KEYED>
__global__ void __launch_bounds__(1024) select_small_kernel(SelArgs a, DevStatus *status) {
    using T = typename Word<W>::T;
    using O = typename Word<KIND == SEL_WHERE ? 8 : W>::T;
    constexpr int I = SEL_SMALL_ITEMS;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, n = static_cast<int>(a.n);
    const int per = (n + 1023) / 1024 * 32;  // rows of a warp
    T v[KIND == SEL_WHERE ? 1 : I];
    unsigned m[I];
    unsigned char mb[KIND == SEL_FILTER ? 1 : I];
#pragma unroll
    for (int j = 0; j < I; ++j) {
        const int r = w * per + j * 32 + lane;
        const bool in = j * 32 < per && r < n;
        if (KIND != SEL_WHERE) v[j] = in ? static_cast<const T *>(a.x)[r] : T(0);
        if (KIND != SEL_FILTER) mb[j] = in ? a.m[r] : 0;
    }
    unsigned count = 0;
#pragma unroll
    for (int j = 0; j < I; ++j) {
        const bool in = j * 32 < per && w * per + j * 32 + lane < n;
        bool keep = false;
        if constexpr (KIND == SEL_FILTER) keep = in && sel_keep<W, KEYED>(a.r, v[j]);
        else keep = in && mb[j] != 0;
        m[j] = __ballot_sync(FULL, keep);
        count += __popc(m[j]);
    }
    __shared__ unsigned warp_count[32];
    if (lane == 0) warp_count[w] = count;
    __syncthreads();
    const unsigned mine = warp_count[lane];
    unsigned inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += y;
    }
    unsigned at = __shfl_sync(FULL, inc - mine, w);
    O *out = static_cast<O *>(a.out);
#pragma unroll
    for (int j = 0; j < I; ++j) {
        if ((m[j] >> lane) & 1u) {
            const unsigned q = at + __popc(m[j] & ((1u << lane) - 1u));
            if constexpr (KIND == SEL_WHERE) out[q] = static_cast<O>(a.base + w * per + j * 32 + lane);
            else out[q] = static_cast<O>(v[j]);
        }
        at += __popc(m[j]);
    }
    if (threadIdx.x == 31) {
        a.host[0] = inc;
        a.host[1] = *reinterpret_cast<volatile unsigned *>(&status->timeout);
    }
}

template <class P> static vkc_status launch_select(vkc_ctx *ctx, SelArgs &a) {
    const int tiles = static_cast<int>((a.n + P::TILE - 1) / P::TILE);
    vkc_status st;
    void *p;
    unsigned long long *recs;
    if ((st = scratch(ctx, 256, &p))) return st;
    if ((st = rec_arena(ctx, tiles, &recs))) return st;
    a.total = static_cast<unsigned long long *>(p);
    const unsigned epoch = next_epoch(ctx);
    constexpr size_t smem = static_cast<size_t>(P::SLOTS) * P::SLOT_BYTES + P::OUT_BYTES;
    auto *kernel = select_kernel<P>;
    static std::atomic<unsigned long long> configured{0};
    once_per_device(configured, ctx->device, [&] {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    });
    const int grid = tile_pass_grid(ctx, kernel, SEL_THREADS + 64, smem, tiles);
    kernel<<<grid, SEL_THREADS + 64, smem, ctx->stream>>>(a, tiles, recs, epoch, ctx->counters, ctx->status);
    return launched(ctx, "select");
}

template <int KIND, int W, bool KEYED>
static vkc_status run_select(vkc_ctx *ctx, SelArgs a, int64_t n, Builder *b) {
    if (n >= (int64_t(1) << 38)) return fail(ctx, VKC_USAGE, "selection of 2^38 rows or more");
    vkc_status st;
    void *at, *h;
    if ((st = b->reserve(n, &at))) return st;
    if ((st = pinned(ctx, 16, &h))) return st;
    a.out = at;
    a.host = static_cast<unsigned long long *>(h);
    a.aligned = (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.m) & 15) == 0;
    // Rows a thread: 16, or as many as fill a slot of 64 KB (a mask's, 32 KB) once each SM has two such
    // tiles. A tile's lookback takes some 5000 cycles while the memory is loaded, and tiles of fewer bytes
    // wait for it; before that more tiles keep more SMs at work (where of 20 M rows 89 us as 8192-row tiles,
    // 62 in these).
    constexpr int BIG = KIND == SEL_WHERE ? 64 : 32;
    if (n <= SEL_SMALL) {
        select_small_kernel<KIND, W, KEYED><<<1, 1024, 0, ctx->stream>>>(a, ctx->status);
        st = launched(ctx, "select_small");
    } else if constexpr (W == 8) {
        if (a.aligned) st = launch_select<SelectPass<KIND, KEYED>>(ctx, a);
        else st = launch_select<RankPass<KIND, 8, KEYED, 16>>(ctx, a);
    } else if (n >= int64_t(2) * ctx->sms * SEL_THREADS * BIG) {
        st = launch_select<RankPass<KIND, W, KEYED, BIG>>(ctx, a);
    } else {
        st = launch_select<RankPass<KIND, W, KEYED, 16>>(ctx, a);
    }
    if (st) return st;
    VKC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const unsigned long long k = a.host[0];
    if (a.host[1]) {  // a wait ran out, here or in work enqueued earlier: clear the status word
        DevStatus ds;
        if ((st = read_status(ctx, &ds))) return st;
    }
    // The count can only be at most the rows reserved; anything else is a broken launch.
    if (k > static_cast<unsigned long long>(n))
        return fail(ctx, VKC_DEVICE, "selection returned " + std::to_string(k) + " rows for " +
                                         std::to_string(n) + " input rows");
    b->len += static_cast<int64_t>(k);
    return VKC_OK;
}

static SelRange sel_range(long long lo, long long hi, bool negate, bool keyed) {
    if (lo > hi) return SelRange{0, ~0ull, !negate, false};  // empty
    if (keyed && lo >= 0 && !negate) keyed = false;
    return SelRange{static_cast<unsigned long long>(lo), static_cast<unsigned long long>(hi) - static_cast<unsigned long long>(lo), negate, keyed};
}

// x <cmp> c on f32 as a range of its order keys, as cmp_range makes one of f64's.
static SelRange f32_range(int cmp, unsigned bits) {
    auto key = [](unsigned b) { return static_cast<long long>(static_cast<int>((b >> 31) ? b ^ 0x7fffffffu : b)); };
    const long long inf = key(0x7f800000u), ninf = key(0xff800000u);
    if ((bits & 0x7fffffffu) > 0x7f800000u) return sel_range(1, 0, cmp == 1, true);
    const bool zero = (bits & 0x7fffffffu) == 0;
    const long long lo = zero ? key(0x80000000u) : key(bits), hi = zero ? key(0) : key(bits);  // -0 == +0
    switch (cmp) {
    case 0:
    case 1: return sel_range(lo, hi, cmp == 1, true);
    case 2: return sel_range(ninf, lo - 1, false, true);
    case 3: return sel_range(ninf, hi, false, true);
    case 4: return sel_range(hi + 1, inf, false, true);
    default: return sel_range(lo, inf, false, true);
    }
}

// x <cmp> c on integers from `min` to `max` (of u64: by the bits' order without the sign).
static SelRange int_range(int cmp, vkc_type t, unsigned long long bits) {
    // Values as keys whose signed order is theirs.
    const bool flip = t == VKC_U64;
    const unsigned long long top = 1ull << 63;
    const long long c = t == VKC_I32 ? static_cast<long long>(static_cast<int>(static_cast<unsigned>(bits)))
                                     : static_cast<long long>(flip ? bits ^ top : bits);
    const long long min = t == VKC_I32 ? INT32_MIN : INT64_MIN, max = t == VKC_I32 ? INT32_MAX : INT64_MAX;
    SelRange r;
    switch (cmp) {
    case 0:
    case 1: r = sel_range(c, c, cmp == 1, false); break;
    case 2: r = c == min ? sel_range(1, 0, false, false) : sel_range(min, c - 1, false, false); break;
    case 3: r = sel_range(min, c, false, false); break;
    case 4: r = c == max ? sel_range(1, 0, false, false) : sel_range(c + 1, max, false, false); break;
    default: r = sel_range(c, max, false, false); break;
    }
    if (flip && r.span != ~0ull) r.lo ^= top;
    return r;
}

// fused.rs:214-223 (filter_args) and :225-236.
template <vkc_type T, int C> static vkc_status filter_of(vkc_ctx *ctx, const Arg *args, int nargs, int64_t, Builder *b) {
    constexpr int W = T == VKC_F64 || T == VKC_I64 || T == VKC_U64 ? 8 : 4;
    vkc_status st;
    if (nargs != 2) return fail(ctx, VKC_RUNTIME, arity_error(2, nargs));
    if (!rows_arg(ctx, args[0], T, &st) || !splat_arg(ctx, args[1], T, &st)) return st;
    int64_t n = args[0].len();
    if (n == 0) return VKC_OK;
    SelArgs a{};
    a.x = args[0].a->data();
    a.n = n;
    if constexpr (T == VKC_F64 || T == VKC_F32) {
        if (T == VKC_F64) {
            const CmpRange r = cmp_range(C, args[1].f64());
            a.r = sel_range(r.lo, r.hi, r.negate != 0, true);
        } else {
            a.r = f32_range(C, static_cast<unsigned>(args[1].s.bits));
        }
        if (a.r.keyed) return run_select<SEL_FILTER, W, true>(ctx, a, n, b);
    } else {
        a.r = int_range(C, T, args[1].s.bits);
    }
    return run_select<SEL_FILTER, W, false>(ctx, a, n, b);
}

// select.rs:163-186 (compress_args): kinds, then equal row counts.
template <vkc_type T> static vkc_status compress(vkc_ctx *ctx, const Arg *args, int nargs, int64_t, Builder *b) {
    vkc_status st;
    if (nargs != 2) return fail(ctx, VKC_RUNTIME, arity_error(2, nargs));
    if (!rows_arg(ctx, args[0], T, &st) || !rows_arg(ctx, args[1], VKC_BOOL, &st)) return st;
    int64_t n = args[0].len();
    if (n != args[1].len())
        return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(n) + " values vs " +
                                          std::to_string(args[1].len()) + " mask rows");
    if (n == 0) return VKC_OK;
    SelArgs a{};
    a.x = args[0].a->data();
    a.m = static_cast<const unsigned char *>(args[1].a->data());
    a.n = n;
    switch (type_width(T)) {
    case 8: return run_select<SEL_COMPRESS, 8, false>(ctx, a, n, b);
    case 4: return run_select<SEL_COMPRESS, 4, false>(ctx, a, n, b);
    default: return run_select<SEL_COMPRESS, 1, false>(ctx, a, n, b);
    }
}

// select.rs:98-125 (where_append, check_row_indices): global rows base + i.
static vkc_status where_sel(vkc_ctx *ctx, const Arg *args, int nargs, int64_t base, Builder *b) {
    vkc_status st;
    if (nargs != 1) return fail(ctx, VKC_RUNTIME, arity_error(1, nargs));
    if (!rows_arg(ctx, args[0], VKC_BOOL, &st)) return st;
    int64_t n = args[0].len();
    if (base < 0 || n > INT64_MAX - base) return fail(ctx, VKC_RUNTIME, "row index fits in i64");
    if (n == 0) return VKC_OK;
    SelArgs a{};
    a.m = static_cast<const unsigned char *>(args[0].a->data());
    a.n = n;
    a.base = base;
    return run_select<SEL_WHERE, 1, false>(ctx, a, n, b);
}

template <vkc_type T> static SelectFn filter_of_cmp(int cmp) {
    const SelectFn fs[6] = {filter_of<T, 0>, filter_of<T, 1>, filter_of<T, 2>, filter_of<T, 3>, filter_of<T, 4>, filter_of<T, 5>};
    return fs[cmp];
}

SelectFn filter_fn(vkc_type t, int cmp) {
    switch (t) {
    case VKC_F64: return filter_of_cmp<VKC_F64>(cmp);
    case VKC_F32: return filter_of_cmp<VKC_F32>(cmp);
    case VKC_I64: return filter_of_cmp<VKC_I64>(cmp);
    case VKC_U64: return filter_of_cmp<VKC_U64>(cmp);
    default: return filter_of_cmp<VKC_I32>(cmp);
    }
}

void register_select(std::vector<KernelDef> &t) {
    static const char *names[6] = {"eq", "ne", "lt", "le", "gt", "ge"};
    InSpec xa{IN_ARRAY, VKC_F64}, xs{IN_SCALAR, VKC_F64};
    for (int c = 0; c < 6; ++c) {
        // fused.rs:307-318: cost 2 widths.
        KernelDef d{std::string("filter_") + names[c] + "_f64", VKC_SELECTION, {xa, xs}, true, VKC_F64, 16};
        d.sel = filter_fn(VKC_F64, c);
        t.push_back(d);
    }
    struct C { vkc_type t; SelectFn f; };
    const C comp[] = {{VKC_F64, compress<VKC_F64>}, {VKC_F32, compress<VKC_F32>},
                      {VKC_I64, compress<VKC_I64>}, {VKC_U64, compress<VKC_U64>},
                      {VKC_I32, compress<VKC_I32>}, {VKC_U8, compress<VKC_U8>},
                      {VKC_BOOL, compress<VKC_BOOL>}};
    for (const C &c : comp) {
        // select.rs:190-210: cost 2 widths + 1.
        KernelDef d{std::string("compress_") + type_name(c.t), VKC_SELECTION,
                    {InSpec{IN_ARRAY, c.t}, InSpec{IN_ARRAY, VKC_BOOL}}, true, c.t,
                    static_cast<uint64_t>(2 * type_width(c.t) + 1)};
        d.sel = c.f;
        t.push_back(d);
    }
    KernelDef d{"where", VKC_SELECTION, {InSpec{IN_ARRAY, VKC_BOOL}}, true, VKC_I64, 9};
    d.sel = where_sel;
    t.push_back(d);
}

}  // namespace vkc
