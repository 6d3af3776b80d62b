// Scans of every fold and element type (src/kernels/scalar/scan.rs:99-326) as one persistent pass over
// tiles (tilepass.cuh). Included by k_scan.cu (i64 sums), k_scan_wide.cu and k_scan_narrow.cu.
//
// scan.rs:248-282: row 0 and every row whose start flag is set lift their value, every other row steps
// the running value; state carries across updates. With the fold's identity as the state before the
// first row (step(identity, x) = lift(x)), out[i] is the fold of the state and the rows from the last
// start through i: an associative fold of (start, value) pairs, (s1, v1) then (s2, v2) =
// (s1 | s2, s2 ? v2 : v1 op v2).
#pragma once

#include <cstring>
#include <type_traits>

#include "folds.h"
#include "reduce_common.h"
#include "tilepass.cuh"

namespace vkc {

constexpr int SC_THREADS = 512;  // compute threads (+ 2 warps)
// The lookback's step: 32 tiles, one a lane. Wider ones find the prefix in one step too, but their polls,
// four records a lane, slow the copies they wait for: calls on 2^27 / 2^28 i64 rows plain with 4 records a
// lane 404 / 814 us, with 2 374 / 732, with 1 360 / 700; with segments 399 / 773, 395 / 753, 392 / 753.
constexpr int SC_WINDOW = 1;
constexpr int SC_SMEM = 224 * 1024;  // of the slots and the output rows

// The carried state of a scanner: the last output (as a word of the fold) and, of prev, whether any
// row was seen.
struct ScanState {
    u64 last;
    u64 seen;
};

// A fold on words: enc() makes a row's bits a word, dec() a word the output's bits. Sums are 8-byte
// words of the sum type, everything else words of the element's width (u8: 4 bytes). Float extremes fold
// the signed order keys of the values, so that a step is an integer comparison (a step of f64 values
// took two NaN tests and two comparisons on the FP64 pipe); a NaN is the key beyond the infinity that the
// fold tends to, and comes out as the canonical NaN.
template <vkc_type IT, int F> struct ScanOp {
    static constexpr vkc_type OT = F == F_ADD ? sum_type(IT) : IT;
    static constexpr int IW = width_of(IT), OW = width_of(OT);
    static constexpr bool FLT = is_float(IT);
    using X = typename std::conditional<IW == 8, u64, unsigned>::type;  // a row's bits
    using W = typename std::conditional<OW == 8, u64, unsigned>::type;
    using SW = typename std::conditional<OW == 8, long long, int>::type;
    static constexpr int SIGN = 8 * sizeof(W) - 1;

    __host__ __device__ static __forceinline__ W key(W b) { return b ^ (static_cast<W>(static_cast<SW>(b) >> SIGN) >> 1); }
    // The canonical NaN's bits; its key: above +inf's of a maximum, below -inf's of a minimum.
    static constexpr W QNAN = OW == 8 ? static_cast<W>(0x7ff8000000000000ull) : static_cast<W>(0x7fc00000u);
    static constexpr W NAN_KEY = F == F_MAX ? QNAN : static_cast<W>(~QNAN);
    __device__ static __forceinline__ bool nan(X b) {
        return IW == 8 ? (b & static_cast<X>(~(1ull << 63))) > static_cast<X>(0x7ff0000000000000ull)
                       : (b & 0x7fffffffu) > 0x7f800000u;
    }
    __device__ static __forceinline__ W enc(X b) {
        if (FLT) return nan(b) ? NAN_KEY : key(static_cast<W>(b));
        if (IT == VKC_I32 && F == F_ADD) return static_cast<W>(static_cast<long long>(static_cast<int>(b)));
        return static_cast<W>(b);
    }
    __device__ static __forceinline__ W dec(W k) {
        if (!FLT) return k;
        return F == F_MIN && k == NAN_KEY ? QNAN : key(k);
    }
    __host__ __device__ static __forceinline__ W ident() {
        constexpr u64 id = identity<OT, F>();
        return FLT ? key(static_cast<W>(id)) : static_cast<W>(id);
    }
    __device__ static __forceinline__ W op(W a, W b) {
        if (F == F_ADD) return a + b;
        if (F == F_MUL) return a * b;
        if (F == F_AND) return a & b;
        if (F == F_OR) return a | b;
        if (F == F_XOR) return a ^ b;
        const bool less = FLT || is_signed_t(IT) ? static_cast<SW>(a) < static_cast<SW>(b) : a < b;
        return less == (F == F_MIN) ? a : b;
    }
};

__device__ __forceinline__ ulonglong2 ld_relaxed128(const ulonglong2 *p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed128(ulonglong2 *p, ulonglong2 v) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(v.x), "l"(v.y) : "memory");
}

// A segmented partial: the fold since the last start, and whether a segment starts inside it.
template <class W> struct SegOf {
    W v;
    unsigned start;
};

// Lookback record of a segmented partial in two words, each carrying the epoch and the state: the start
// flag and the high half of the value in one, the low half in the other. Each word is read or
// written whole, so a record read in the middle of its update from aggregate to inclusive
// shows two states and is polled again.
template <class Op> struct SegRec {
    using V = SegOf<typename Op::W>;
    using W = ulonglong2;
    __device__ static V ident() { return V{Op::ident(), 0u}; }
    __device__ static V op(V a, V b) { return V{b.start ? b.v : Op::op(a.v, b.v), a.start | b.start}; }
    __device__ static W make(unsigned ep, unsigned state, V v) {
        const u64 tag = (static_cast<u64>(ep & 0xffffffu) << 40) | (static_cast<u64>(state) << 38);
        const u64 b = v.v;
        return W{tag | (static_cast<u64>(v.start & 1u) << 37) | (b >> 32), tag | (b & 0xffffffffull)};
    }
    __device__ static bool ready(W w, unsigned ep) {
        const u64 e = ep & 0xffffffu;
        return (w.x >> 40) == e && (w.y >> 40) == e && ((w.x >> 38) & 3u) == ((w.y >> 38) & 3u);
    }
    __device__ static unsigned state(W w) { return static_cast<unsigned>(w.x >> 38) & 3u; }
    __device__ static V value(W w) {
        return V{static_cast<typename Op::W>(((w.x & 0xffffffffull) << 32) | (w.y & 0xffffffffull)),
                 static_cast<unsigned>(w.x >> 37) & 1u};
    }
    __device__ static W load(const W *p) { return ld_relaxed128(p); }
    __device__ static void store(W *p, W w) { st_relaxed128(p, w); }
    __device__ static V shfl_up(V v, int o) {
        return V{__shfl_up_sync(FULL, v.v, o), __shfl_up_sync(FULL, v.start, o)};
    }
    __device__ static V shfl(V v, int src) { return V{__shfl_sync(FULL, v.v, src), __shfl_sync(FULL, v.start, src)}; }
    __device__ static V shfl_down(V v, int o) {
        return V{__shfl_down_sync(FULL, v.v, o), __shfl_down_sync(FULL, v.start, o)};
    }
};

// The pass. A compute warp's slice is SLICE consecutive rows, read in STEPS steps of 32 * VEC rows; in a
// step lane l holds rows VEC l .. VEC l + VEC - 1 (32 bytes of the wider of its input and output), so row
// order is (step, lane, item). The count scans the slice from its own start in registers, where it stays
// until the tile's prefix is known: the slot is read once and never written. What the prefix still has to
// reach are the slice's rows before its first start. (Counted first, then scanned in
// place with the starts beside the values and stored from there, the slot was read three times and written
// once, and the segmented scan was bound by its instructions: calls on 2^27 i64 rows took 403 us plain
// and 584 with segments, the other types' reduce, scan and apply kernels 1.1 to 2.6 ms. Now 360,
// 392, i32 sums 347, f64 extremes 410 plain and 543 with segments, f32 199, u8 158; 2.15 GB take 317 us at
// the copy's rate. Evict-first hints on the loads and stores change nothing.)
//
// Segments need no flags beside the values in the warp's scan: with the lanes that hold a start as a
// ballot, lane l takes what comes from o lanes below as long as that is not below the last such lane at
// or before l. A tile that is not whole, or not aligned, is read from global memory instead of the slot.
template <vkc_type IT, int F, bool BY> struct ScanPass {
    using Op = ScanOp<IT, F>;
    using X = typename Op::X;
    using W = typename Op::W;
    static constexpr int IW = Op::IW, OW = Op::OW;
    static constexpr int THREADS = SC_THREADS;
    // 8192 rows a tile, 16384 of 4-byte words (a slot of 64 KB at most): a lookback takes about
    // 5000 cycles while the memory is loaded, and shorter tiles wait for it (2^27 f32 rows in tiles of 8192:
    // 376 us a call, now 202; i64 rows in tiles of 4096, two blocks a SM: 745 us).
    static constexpr int TILE = (OW == 8 ? 16 : 32) * SC_THREADS;
    static constexpr int SLICE = TILE / (SC_THREADS / 32);  // rows per warp
    static constexpr int VEC = IW > 1 || OW > 1 ? 32 / (IW > OW ? IW : OW) : 16;  // rows per lane per step
    static constexpr int STEPS = SLICE / (32 * VEC);
    static constexpr int VAL_BYTES = IW * TILE;
    static constexpr int SLOT_BYTES = VAL_BYTES + (BY ? TILE : 0);
    static constexpr int OUT_BYTES = OW * TILE;
    static constexpr int SLOTS = (SC_SMEM - OUT_BYTES) / SLOT_BYTES < 8 ? (SC_SMEM - OUT_BYTES) / SLOT_BYTES : 8;
    static constexpr bool ONE_READ = true;
    using R = SegRec<Op>;
    using V = typename R::V;
    struct Staged {
        W v[STEPS][VEC];
        int first;  // the slice's rows before its first start
        bool raw;   // of this lane's rows, a NaN may start a segment
    };

    const void *x;
    const unsigned char *starts;
    void *out;
    int64_t n;
    bool aligned;      // x and starts (16 bytes) aligned: whole tiles go by TMA
    bool out_aligned;  // out too (16 bytes): whole slices leave by TMA

    __device__ bool whole(int tile) const { return aligned && static_cast<int64_t>(tile + 1) * TILE <= n; }
    __device__ unsigned bulk_bytes(int tile) const { return whole(tile) ? SLOT_BYTES : 0u; }
    __device__ void load(int tile, unsigned char *slot, unsigned long long *bar) const {
        const int64_t r0 = static_cast<int64_t>(tile) * TILE;
        bulk_load(slot, static_cast<const unsigned char *>(x) + r0 * IW, VAL_BYTES, bar);
        if (BY) bulk_load(slot + VAL_BYTES, starts + r0, TILE, bar);
    }
    __device__ __forceinline__ X row(int64_t i) const {
        if constexpr (IW == 8) return static_cast<const u64 *>(x)[i];
        else if constexpr (IW == 4) return static_cast<const unsigned *>(x)[i];
        else return static_cast<const unsigned char *>(x)[i];
    }

    // The rows of the slice as words, and their starts (bit k of f[s]: row k of step s). Rows past the end
    // are identities. Of a lane's 32 bytes every other four lanes read the second half first: read in
    // order, the halves of eight lanes fell on half of the banks.
    __device__ __forceinline__ void load_rows(bool sm, const unsigned char *slot, int64_t r0, W (&v)[STEPS][VEC],
                                              unsigned (&f)[STEPS], bool &raw) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        if (sm) {
#pragma unroll
            for (int s = 0; s < STEPS; ++s) {
                const int j = w * SLICE + (s * 32 + lane) * VEC;
                unsigned q[VEC * IW / 4];
                const unsigned char *p = slot + IW * j;
                if constexpr (VEC * IW == 32) {
                    const int odd = (lane >> 2) & 1;
                    const uint4 a = reinterpret_cast<const uint4 *>(p)[odd], b = reinterpret_cast<const uint4 *>(p)[odd ^ 1];
                    const uint4 lo = odd ? b : a, hi = odd ? a : b;
                    q[0] = lo.x, q[1] = lo.y, q[2] = lo.z, q[3] = lo.w, q[4] = hi.x, q[5] = hi.y, q[6] = hi.z, q[7] = hi.w;
                } else if constexpr (VEC * IW == 16) {
                    const uint4 a = *reinterpret_cast<const uint4 *>(p);
                    q[0] = a.x, q[1] = a.y, q[2] = a.z, q[3] = a.w;
                } else {
                    static_assert(VEC * IW == 4, "u8 rows of 8-byte sums");
                    q[0] = *reinterpret_cast<const unsigned *>(p);
                }
                f[s] = 0;
                bool any = false;  // a NaN among the lane's rows
                if (BY) {
#pragma unroll
                    for (int c = 0; c < VEC / 4; ++c) {
                        const unsigned m = *reinterpret_cast<const unsigned *>(slot + VAL_BYTES + j + 4 * c);
                        const unsigned h = ((((m & 0x7f7f7f7fu) + 0x7f7f7f7fu) | m) & 0x80808080u) >> 7;
                        f[s] |= ((h * 0x10204080u) >> 28) << (4 * c);  // bits 0, 8, 16 and 24 side by side
                    }
                }
#pragma unroll
                for (int k = 0; k < VEC; ++k) {
                    X b;
                    if constexpr (IW == 8) b = q[2 * k] | static_cast<X>(q[2 * k + 1]) << 32;
                    else if constexpr (IW == 4) b = q[k];
                    else b = (q[k / 4] >> (8 * (k & 3))) & 0xffu;
                    v[s][k] = Op::enc(b);
                    if (BY && Op::FLT) any = any || Op::nan(b);
                }
                if (BY && Op::FLT) raw = raw || (any && f[s] != 0);
            }
        } else {
#pragma unroll
            for (int s = 0; s < STEPS; ++s) {
                const int64_t i0 = r0 + w * SLICE + (s * 32 + lane) * VEC;
                f[s] = 0;
#pragma unroll
                for (int k = 0; k < VEC; ++k) {
                    const bool in = i0 + k < n;
                    const X b = in ? row(i0 + k) : X(0);
                    v[s][k] = in ? Op::enc(b) : Op::ident();
                    if (BY && in && starts[i0 + k]) {
                        f[s] |= 1u << k;
                        if (Op::FLT) raw = raw || Op::nan(b);
                    }
                }
            }
        }
    }

    // The steps' scans are independent until the carry, and run side by side.
    __device__ __forceinline__ V count(int tile, const unsigned char *slot, Staged &st) const {
        const int lane = threadIdx.x & 31;
        st.first = SLICE;
        st.raw = false;
        unsigned f[STEPS], heads[STEPS];
        W inc[STEPS];
        int reach[STEPS];
        load_rows(whole(tile), slot, static_cast<int64_t>(tile) * TILE, st.v, f, st.raw);
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
#pragma unroll
            for (int k = 1; k < VEC; ++k)
                if (!BY || !((f[s] >> k) & 1u)) st.v[s][k] = Op::op(st.v[s][k - 1], st.v[s][k]);
            inc[s] = st.v[s][VEC - 1];
            heads[s] = BY ? __ballot_sync(FULL, f[s] != 0) : 0u;
            const unsigned upto = heads[s] & (0xffffffffu >> (31 - lane));  // at or before this lane
            reach[s] = upto ? lane - (31 - __clz(upto)) : lane;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (int s = 0; s < STEPS; ++s) {
                const W y = __shfl_up_sync(FULL, inc[s], o);
                if (o <= reach[s]) inc[s] = Op::op(y, inc[s]);
            }
        }
        W carry = Op::ident();  // the slice so far
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            W ex = __shfl_up_sync(FULL, inc[s], 1);  // before this lane's rows, since the last start
            if (lane == 0) ex = carry;
            else if (!(heads[s] & ((1u << lane) - 1u))) ex = Op::op(carry, ex);
#pragma unroll
            for (int k = 0; k < VEC; ++k)
                if (!BY || !(f[s] & ((2u << k) - 1u))) st.v[s][k] = Op::op(ex, st.v[s][k]);
            const W end = __shfl_sync(FULL, inc[s], 31);
            if (BY && heads[s] && st.first == SLICE) {
                const int src = __ffs(heads[s]) - 1;
                st.first = (s * 32 + src) * VEC + __ffs(__shfl_sync(FULL, f[s], src)) - 1;
            }
            carry = heads[s] ? end : Op::op(carry, end);
        }
        return V{carry, st.first < SLICE ? 1u : 0u};
    }

    __device__ __forceinline__ void store(int64_t i, W v) const {
        if constexpr (OW == 8) static_cast<u64 *>(out)[i] = v;
        else if constexpr (OW == 4) static_cast<unsigned *>(out)[i] = v;
        else static_cast<unsigned char *>(out)[i] = static_cast<unsigned char>(v);
    }

    // A whole slice goes by way of the block's output rows in shared memory and a bulk copy, which leaves
    // the warp free for the next tile's count (stored from the registers, a flush of 64 KB held it for
    // 2260 of the 7150 cycles of a tile of i64 sums).
    __device__ __forceinline__ void flush(int tile, V pre, const Staged &st, unsigned char *rows) const {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const int64_t s0 = static_cast<int64_t>(tile) * TILE + w * SLICE;
        const bool bulk = out_aligned && s0 + SLICE <= n;
        unsigned char *mine = rows + w * SLICE * OW;
        if (bulk) {
            if (lane == 0) bulk_store_wait_read();  // the slice before has left them
            __syncwarp();
        }
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            const int q = (s * 32 + lane) * VEC;  // in the slice
            W e[VEC];
#pragma unroll
            for (int k = 0; k < VEC; ++k)
                e[k] = Op::dec(!BY || q + k < st.first ? Op::op(pre.v, st.v[s][k]) : st.v[s][k]);
            // A segment's first row is lifted as it is, a NaN with its payload.
            if (BY && Op::FLT && st.raw) {
#pragma unroll
                for (int k = 0; k < VEC; ++k) {
                    if (s0 + q + k >= n || !starts[s0 + q + k]) continue;
                    const X b = row(s0 + q + k);
                    if (Op::nan(b)) e[k] = static_cast<W>(b);
                }
            }
            if (bulk) {
                unsigned u[VEC * OW / 4];
#pragma unroll
                for (int k = 0; k < VEC; ++k) {
                    if constexpr (OW == 8) {
                        u[2 * k] = static_cast<unsigned>(e[k]), u[2 * k + 1] = static_cast<unsigned>(e[k] >> 32);
                    } else if constexpr (OW == 4) {
                        u[k] = e[k];
                    } else {
                        if (k % 4 == 0) u[k / 4] = 0;
                        u[k / 4] |= (e[k] & 0xffu) << (8 * (k & 3));
                    }
                }
                auto *p = reinterpret_cast<uint4 *>(mine + q * OW);
                const uint4 lo = make_uint4(u[0], u[1], u[2], u[3]);
                if constexpr (VEC * OW == 32) {
                    const uint4 hi = make_uint4(u[4], u[5], u[6], u[7]);
                    const int odd = (lane >> 2) & 1;
                    p[odd] = odd ? hi : lo;
                    p[odd ^ 1] = odd ? lo : hi;
                } else {
                    *p = lo;
                }
            } else {
#pragma unroll
                for (int k = 0; k < VEC; ++k)
                    if (s0 + q + k < n) store(s0 + q + k, e[k]);
            }
        }
        if (bulk) {
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) bulk_store(static_cast<unsigned char *>(out) + s0 * OW, mine, SLICE * OW);
        }
    }
    // The copies are done before the block ends.
    __device__ void finish() const {
        if ((threadIdx.x & 31) == 0) bulk_store_wait();
    }

    __device__ void last_tile(V) const {}
};

template <vkc_type IT, int F, bool BY>
__global__ void __launch_bounds__(SC_THREADS + 64, 1)
    scan_kernel(const void *x, const unsigned char *starts, void *out, int64_t n, bool aligned, bool out_aligned, int tiles,
                ulonglong2 *recs, unsigned epoch, bool fresh, ScanState *state, unsigned *counters, DevStatus *status) {
    using P = ScanPass<IT, F, BY>;
    using Op = typename P::Op;
    // The carried state (none in a first update) is read once, before this block publishes
    // anything; the block that finishes last rewrites it, after every block has read it.
    const typename Op::W carried = fresh ? Op::ident() : static_cast<typename Op::W>(state->last);
    const P p{x, starts, out, n, aligned, out_aligned};
    // The last row's output, the last tile's inclusive value, is the carried state.
    if (tile_pass<SC_WINDOW>(p, recs, tiles, epoch, counters, status, typename P::V{carried, 0u}) && threadIdx.x == 0)
        state->last = P::R::value(ld_relaxed128(rec_at<typename P::R>(recs, tiles - 1))).v;
}

template <vkc_type IT, int F> constexpr int scan_tiles(int64_t n) {
    constexpr int64_t rows = ScanPass<IT, F, false>::TILE;
    return static_cast<int>((n + rows - 1) / rows);
}

// Launches a scan on `stream` with the tile records at `recs` (REC_STRIDE bytes per tile).
template <vkc_type IT, int F, bool BY>
void launch_scan(int device, int sms, cudaStream_t stream, const void *x, const unsigned char *s, void *o, int64_t n,
                 int tiles, ulonglong2 *recs, unsigned epoch, bool fresh, ScanState *state, unsigned *counters,
                 DevStatus *status) {
    using P = ScanPass<IT, F, BY>;
    const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(s)) & 15) == 0;
    const bool out_aligned = (reinterpret_cast<uintptr_t>(o) & 15) == 0;
    constexpr size_t smem = static_cast<size_t>(P::SLOTS) * P::SLOT_BYTES + P::OUT_BYTES;
    static std::atomic<unsigned long long> configured{0};
    once_per_device(configured, device, [] {
        cudaFuncSetAttribute(scan_kernel<IT, F, BY>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    });
    const int grid = sms < tiles ? sms : tiles;  // one block a SM, for its shared memory
    scan_kernel<IT, F, BY><<<grid, SC_THREADS + 64, smem, stream>>>(x, s, o, n, aligned, out_aligned, tiles, recs, epoch,
                                                                    fresh, state, counters, status);
}

template <vkc_type IT, int F, bool BY> struct ScanImpl : ScannerImpl {
    ScanState *state = nullptr;  // uninitialised until the first update (fresh) or begin
    bool fresh = true;
    DeviceMem mem;  // owns `state`
    vkc_status begin(vkc_ctx *ctx) override {
        fresh = false;
        reducer_fill_kernel<<<1, 64, 0, ctx->stream>>>(&state->last, 1, Words4{{static_cast<u64>(ScanOp<IT, F>::ident())}});
        return launched(ctx, "scan_begin");
    }
    // scan.rs:228-282 (tile_rows): arity, kinds, then destination rows.
    vkc_status update(vkc_ctx *ctx, const Arg *args, int nargs, vkc_array *out) override {
        vkc_status st;
        const int want = BY ? 2 : 1;
        if (nargs != want) return fail(ctx, VKC_RUNTIME, arity_error(want, nargs));
        if (!rows_arg(ctx, args[0], IT, &st)) return st;
        if (BY && !rows_arg(ctx, args[1], VKC_BOOL, &st)) return st;
        if (out->type != ScanOp<IT, F>::OT) return fail(ctx, VKC_RUNTIME, "bad destination");
        const int64_t n = args[0].len();
        if (out->len != n || (BY && args[1].len() != n))
            return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(n) + " rows for a destination of " +
                                              std::to_string(out->len) + " rows");
        if (n == 0) return VKC_OK;
        const int tiles = scan_tiles<IT, F>(n);
        ulonglong2 *recs;
        if ((st = rec_arena(ctx, tiles, &recs))) return st;
        launch_scan<IT, F, BY>(ctx->device, ctx->sms, ctx->stream, args[0].a->data(),
                               BY ? args[1].ptr<unsigned char>() : nullptr, out->data(), n, tiles, recs, next_epoch(ctx),
                               fresh, state, ctx->counters, ctx->status);
        fresh = false;
        return launched(ctx, "scan");
    }
};

// CAPTURED: whether a scan may begin in a stream capture.
template <vkc_type IT, int F, bool BY, bool CAPTURED> ScannerImpl *make_scan(vkc_ctx *ctx) {
    auto *s = new ScanImpl<IT, F, BY>;
    bool captured;
    if (state_block(ctx, sizeof(ScanState), &s->mem, &captured) || (captured && !CAPTURED)) {
        delete s;
        return nullptr;
    }
    s->state = static_cast<ScanState *>(s->mem.ptr);
    return s;
}

template <vkc_type IT, int F> FoldScanMake scan_of(bool by) {
    return by ? make_scan<IT, F, true, false> : make_scan<IT, F, false, false>;
}

}  // namespace vkc
