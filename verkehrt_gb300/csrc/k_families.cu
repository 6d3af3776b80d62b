// The kernel families on every element type: the entries of the reference's registry that the
// specialised files (f64 sums, f64/i64 extremes, i64 scans and buckets, i64 sort and group ids)
// do not hold.
//
//   reductions  reduce_add/mul/min/max_T, reduce_and/or/xor_T, argmin/argmax_T, any, all
//               (src/kernels/scalar/reduce.rs:331-726)
//   fused       dot/sumsq/count_<cmp>/condsum_<cmp> on f32, i64, u64, i32, and the entries of
//               filter_<cmp> (k_select.cu's) (src/kernels/scalar/fused.rs:73-379)
//   scans       scan_<fold>_T, scan_by_<fold>_T (their entries; the passes are fold_scan.cuh's),
//               reduce_into_<fold>_T, prev_T
//               (src/kernels/scalar/scan.rs:16-439)
//   whole       group_id_T, group_id2_A_B (group.rs:259-363),
//               fill_T, same_len_T (construct.rs:49-120), slice_T (index.rs:240-258)
//
// Values travel as 64-bit words: i32 sign-extended, u8 and bool zero-extended, f32 as its 32
// bits. Every fold except the canonical float sum and product is order-free (wrapping integer
// arithmetic, the 754-2019 minimum/maximum, bit operations), so those reductions are a plain
// grid fold. The canonical order of a float
// product is sixteen chains of dependent IEEE multiplies: one block stages the rows in shared
// memory while sixteen threads run the chains (the float sums have exact parallel paths, in
// k_canon.cu and k_canon32.cu).
#include <climits>
#include <cstring>

#include "folds.h"
#include "kcommon.cuh"
#include "reduce_common.h"

namespace vkc {

vkc_status bucket_key_error(vkc_ctx *ctx, const long long *k, int64_t n, int64_t nb, bool *found);
// The canonical f32 sums (k_canon32.cu).
ReducerImpl *make_canon32_sum(vkc_ctx *ctx);
ReducerImpl *make_canon32_dot(vkc_ctx *ctx);
ReducerImpl *make_canon32_sumsq(vkc_ctx *ctx);
ReducerImpl *make_canon32_cond(vkc_ctx *ctx, int cmp);

namespace {

const char *FOLD_NAMES[7] = {"add", "mul", "min", "max", "and", "or", "xor"};
const char *CMP_NAME[6] = {"eq", "ne", "lt", "le", "gt", "ge"};

// Element load and store as words.
template <vkc_type T> __device__ __forceinline__ u64 ld_word(const void *p, int64_t i) {
    if (width_of(T) == 8) return static_cast<const u64 *>(p)[i];
    if (T == VKC_F32) return static_cast<const unsigned *>(p)[i];
    if (T == VKC_I32) return static_cast<u64>(static_cast<long long>(static_cast<const int *>(p)[i]));
    return static_cast<const unsigned char *>(p)[i];
}
template <int W> __device__ __forceinline__ void st_word(void *p, int64_t i, u64 v) {
    if (W == 8) static_cast<u64 *>(p)[i] = v;
    else if (W == 4) static_cast<unsigned *>(p)[i] = static_cast<unsigned>(v);
    else static_cast<unsigned char *>(p)[i] = static_cast<unsigned char>(v);
}

__device__ __forceinline__ bool nan64(u64 b) { return (b & ~(1ull << 63)) > 0x7ff0000000000000ull; }
__device__ __forceinline__ bool nan32(u64 b) { return (b & 0x7fffffffull) > 0x7f800000ull; }
template <vkc_type T> __device__ __forceinline__ bool is_nan(u64 w) {
    return T == VKC_F64 ? nan64(w) : (T == VKC_F32 ? nan32(w) : false);
}

// elementwise.rs:413-440: min2/max2 (NaN propagates, -0 below +0); Ord on integers.
template <vkc_type T, bool MAX> __device__ __forceinline__ u64 ext2(u64 a, u64 b) {
    if (T == VKC_F64) {
        if (nan64(a) || nan64(b)) return 0x7ff8000000000000ull;
        const double x = __longlong_as_double(static_cast<long long>(a)), y = __longlong_as_double(static_cast<long long>(b));
        if (x == y) return ((a >> 63) != 0) == !MAX ? a : b;
        return (MAX ? x > y : x < y) ? a : b;
    }
    if (T == VKC_F32) {
        if (nan32(a) || nan32(b)) return 0x7fc00000ull;
        const float x = __uint_as_float(static_cast<unsigned>(a)), y = __uint_as_float(static_cast<unsigned>(b));
        if (x == y) return ((a >> 31) & 1u) == (MAX ? 0u : 1u) ? a : b;
        return (MAX ? x > y : x < y) ? a : b;
    }
    if (is_signed_t(T)) {
        const long long x = static_cast<long long>(a), y = static_cast<long long>(b);
        return (MAX ? x >= y : x <= y) ? a : b;
    }
    return (MAX ? a >= b : a <= b) ? a : b;
}

// One step of fold F (scan.rs:130-233 ScanOp::step, the reductions' Accum steps): the
// accumulator of add is in the sum type.
template <vkc_type T, int F> __device__ __forceinline__ u64 step(u64 acc, u64 x) {
    if (F == F_ADD) return acc + x;
    if (F == F_MUL) return wrap<T>(acc * x);
    if (F == F_MIN) return ext2<T, false>(acc, x);
    if (F == F_MAX) return ext2<T, true>(acc, x);
    if (F == F_AND) return acc & x;
    if (F == F_OR) return acc | x;
    return acc ^ x;
}

// fused.rs:41-54: the comparison of the single-op kernels (IEEE for floats: NaN is unordered).
template <vkc_type T> __device__ __forceinline__ bool cmp_test(int cmp, u64 a, u64 b) {
    bool lt, eq, unord = false;
    if (T == VKC_F64) {
        const double x = __longlong_as_double(static_cast<long long>(a)), y = __longlong_as_double(static_cast<long long>(b));
        unord = x != x || y != y;
        lt = x < y;
        eq = x == y;
    } else if (T == VKC_F32) {
        const float x = __uint_as_float(static_cast<unsigned>(a)), y = __uint_as_float(static_cast<unsigned>(b));
        unord = x != x || y != y;
        lt = x < y;
        eq = x == y;
    } else if (is_signed_t(T)) {
        lt = static_cast<long long>(a) < static_cast<long long>(b);
        eq = a == b;
    } else {
        lt = a < b;
        eq = a == b;
    }
    if (unord) return cmp == 1;
    switch (cmp) {
    case 0: return eq;
    case 1: return !eq;
    case 2: return lt;
    case 3: return lt || eq;
    case 4: return !lt && !eq;
    default: return !lt;
    }
}

// Num::mul on the element type: one IEEE multiply (no contraction) or a wrapping product.
template <vkc_type T> __device__ __forceinline__ u64 mul_t(u64 a, u64 b) {
    if (T == VKC_F64)
        return static_cast<u64>(__double_as_longlong(__dmul_rn(__longlong_as_double(static_cast<long long>(a)),
                                                               __longlong_as_double(static_cast<long long>(b)))));
    if (T == VKC_F32)
        return __float_as_uint(__fmul_rn(__uint_as_float(static_cast<unsigned>(a)), __uint_as_float(static_cast<unsigned>(b))));
    return wrap<T>(a * b);
}

// Row values of the folds (fused.rs:73-212): the row itself, x*y, x*x, (x <cmp> c ? x : e),
// the predicate as 0/1, or a bool byte as 0/1.
enum Row { R_PLAIN = 0, R_DOT = 1, R_SUMSQ = 2, R_COND = 3, R_PRED = 4 };
struct RowArgs {
    const void *x;
    const void *y;
    int cmp;
    u64 c, e;
};
template <vkc_type T, int ROW> __device__ __forceinline__ u64 row_value(const RowArgs &a, u64 v, u64 y) {
    if (ROW == R_DOT) return mul_t<T>(v, y);
    if (ROW == R_SUMSQ) return mul_t<T>(v, v);
    if (ROW == R_COND) return cmp_test<T>(a.cmp, v, a.c) ? v : a.e;
    if (ROW == R_PRED) return cmp_test<T>(a.cmp, v, a.c) ? 1ull : 0ull;
    return v;
}

template <vkc_type T, int ROW> __device__ __forceinline__ u64 row_at(const RowArgs &a, int64_t i) {
    return row_value<T, ROW>(a, ld_word<T>(a.x, i), ROW == R_DOT ? ld_word<T>(a.y, i) : 0ull);
}

// Element k of a 16-byte unit, as a word.
template <vkc_type T> __device__ __forceinline__ u64 unit_word(const uint4 &q, int k) {
    const unsigned w[4] = {q.x, q.y, q.z, q.w};
    if (width_of(T) == 8) return w[2 * k] | static_cast<u64>(w[2 * k + 1]) << 32;
    if (T == VKC_F32) return w[k];
    if (T == VKC_I32) return static_cast<u64>(static_cast<long long>(static_cast<int>(w[k])));
    return (w[k >> 2] >> (8 * (k & 3))) & 0xffu;
}

// Rows before the first 16-byte unit of `p`, at most n.
template <vkc_type T> __device__ __forceinline__ int64_t unit_head(const void *p, int64_t n) {
    const int64_t h = static_cast<int64_t>((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / width_of(T);
    return h < n ? h : n;
}

// ------------------------------------------------------------------ order-free folds

// Every block folds its rows (grid-stride, four 16-byte loads in flight per thread; the rows outside
// the 16-byte grid, and all of a dot product whose columns lie differently on it, one by one), the warps
// and the block combine (the fold is commutative), and the last block to finish folds the block
// partials into the reducer's state word. (Loads of one element,
// 2^26 rows: reduce_max_i32 316 us a call, now 75, reduce_add_i32 317 and 56, dot_i32 230 and 91, count_gt_f32
// 217 and 58.)
template <vkc_type T, int F, int ROW>
__global__ void __launch_bounds__(256) fam_fold_kernel(RowArgs a, int64_t n, u64 *partials, unsigned *done, bool fresh, u64 *state,
                                                       u64 *host) {
    constexpr vkc_type AT = ROW == R_PRED ? VKC_U64 : T;  // predicate counts add as u64
    u64 acc = identity<AT, F>();
    const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    constexpr int E = 16 / width_of(T);  // rows of a unit
    constexpr int U = ROW == R_DOT ? 2 : 4;
    const bool alike = ROW != R_DOT || ((reinterpret_cast<uintptr_t>(a.x) ^ reinterpret_cast<uintptr_t>(a.y)) & 15) == 0;
    const int64_t head = alike ? unit_head<T>(a.x, n) : n;
    const int64_t units = (n - head) / E;
    const auto *x = reinterpret_cast<const uint4 *>(static_cast<const unsigned char *>(a.x) + head * width_of(T));
    const auto *y = reinterpret_cast<const uint4 *>(static_cast<const unsigned char *>(a.y) + head * width_of(T));
    auto unit = [&](const uint4 &p, const uint4 &q) {
#pragma unroll
        for (int k = 0; k < E; ++k)
            acc = step<AT, F>(acc, row_value<T, ROW>(a, unit_word<T>(p, k), ROW == R_DOT ? unit_word<T>(q, k) : 0ull));
    };
    int64_t i = tid;
    for (; i + (U - 1) * stride < units; i += U * stride) {
        uint4 p[U], q[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            p[u] = __ldcs(x + i + u * stride);
            q[u] = ROW == R_DOT ? __ldcs(y + i + u * stride) : uint4{};
        }
#pragma unroll
        for (int u = 0; u < U; ++u) unit(p[u], q[u]);
    }
    for (; i < units; i += stride) unit(x[i], ROW == R_DOT ? y[i] : uint4{});
    for (int64_t r = tid; r < head; r += stride) acc = step<AT, F>(acc, row_at<T, ROW>(a, r));
    for (int64_t r = head + units * E + tid; r < n; r += stride) acc = step<AT, F>(acc, row_at<T, ROW>(a, r));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = step<AT, F>(acc, __shfl_xor_sync(FULL, acc, o));
    __shared__ u64 ws[8];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        u64 s = ws[0];
        for (int w = 1; w < 8; ++w) s = step<AT, F>(s, ws[w]);
        partials[blockIdx.x] = s;
    }
    if (last_block(done) && threadIdx.x < 32) {
        u64 s = identity<AT, F>();
        for (unsigned b = threadIdx.x; b < gridDim.x; b += 32) s = step<AT, F>(s, partials[b]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = step<AT, F>(s, __shfl_xor_sync(FULL, s, o));
        if (threadIdx.x == 0) {
            if (!fresh) s = step<AT, F>(state[0], s);
            state[0] = s;
            state[2] = 1;  // rows seen
            if (host) {
                host[0] = s;
                host[2] = 1;
            }
        }
    }
}

// argmin/argmax (reduce.rs:417-468): the first NaN's row, else the first row of the extreme
// (-0 below +0). Each row is the pair (h, row) with h = 0 for a NaN, else the order key (argmin)
// or its complement (argmax); the result is the least pair. Non-NaN keys of floats are never 0.
template <vkc_type T> __device__ __forceinline__ u64 order_key(u64 w) {
    if (T == VKC_F64) return (w >> 63) ? ~w : (w | (1ull << 63));
    if (T == VKC_F32) return ((w >> 31) & 1u) ? (~w & 0xffffffffull) : (w | 0x80000000ull);
    if (is_signed_t(T)) return w ^ (1ull << 63);
    return w;
}
template <vkc_type T, bool MAX> __device__ __forceinline__ u64 arg_key(u64 w) {
    if (is_nan<T>(w)) return 0;
    return MAX ? ~order_key<T>(w) : order_key<T>(w);
}
__device__ __forceinline__ void arg_better(u64 &h, u64 &r, u64 h2, u64 r2) {
    if (h2 < h || (h2 == h && r2 < r)) {
        h = h2;
        r = r2;
    }
}

template <vkc_type T, bool MAX>
__global__ void __launch_bounds__(256) fam_arg_kernel(const void *x, int64_t n, u64 base, ulonglong2 *partials,
                                                      unsigned *done, bool fresh, u64 *state, u64 *host) {
    u64 h = ~0ull, r = ~0ull;
    const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    // Four 16-byte loads in flight a thread, as in the folds; a thread's units come in row order, so that a
    // strict comparison keeps the first row, as a position (unit of the thread, element) until the end.
    constexpr int E = 16 / width_of(T);
    const int64_t head = unit_head<T>(x, n), units = (n - head) / E;
    const auto *xu = reinterpret_cast<const uint4 *>(static_cast<const unsigned char *>(x) + head * width_of(T));
    int64_t at = -1;  // the best's unit
    unsigned k_at = 0;
    auto unit = [&](const uint4 &p, int64_t u) {
        const u64 before = h;
        if (at < 0) at = u;  // element 0 unless another is better (all may have the key ~0)
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const u64 key = arg_key<T, MAX>(unit_word<T>(p, k));
            if (key < h) {
                h = key;
                k_at = k;
            }
        }
        if (h != before) at = u;
    };
    int64_t i = tid;
    for (; i + 3 * stride < units; i += 4 * stride) {
        uint4 p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = __ldcs(xu + i + u * stride);
#pragma unroll
        for (int u = 0; u < 4; ++u) unit(p[u], i + u * stride);
    }
    for (; i < units; i += stride) unit(xu[i], i);
    if (at >= 0) r = base + static_cast<u64>(head + at * E + k_at);
    auto one = [&](int64_t q) { arg_better(h, r, arg_key<T, MAX>(ld_word<T>(x, q)), base + static_cast<u64>(q)); };
    for (int64_t q = tid; q < head; q += stride) one(q);
    for (int64_t q = head + units * E + tid; q < n; q += stride) one(q);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) arg_better(h, r, __shfl_xor_sync(FULL, h, o), __shfl_xor_sync(FULL, r, o));
    __shared__ u64 wh[8], wr[8];
    if ((threadIdx.x & 31) == 0) {
        wh[threadIdx.x >> 5] = h;
        wr[threadIdx.x >> 5] = r;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) arg_better(h, r, wh[w], wr[w]);
        partials[blockIdx.x] = make_ulonglong2(h, r);
    }
    if (last_block(done) && threadIdx.x < 32) {
        u64 bh = ~0ull, br = ~0ull;
        for (unsigned b = threadIdx.x; b < gridDim.x; b += 32) arg_better(bh, br, partials[b].x, partials[b].y);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) arg_better(bh, br, __shfl_xor_sync(FULL, bh, o), __shfl_xor_sync(FULL, br, o));
        if (threadIdx.x == 0) {
            if (!fresh) arg_better(bh, br, state[0], state[1]);
            state[0] = bh;
            state[1] = br;
            state[2] = 1;
            if (host) {
                host[0] = bh;
                host[1] = br;
                host[2] = 1;
            }
        }
    }
}

// The result word as a scalar of type t.
vkc_scalar word_scalar(vkc_type t, u64 w) {
    vkc_scalar s;
    s.type = t;
    s.bits = width_of(t) == 8 ? w : (width_of(t) == 4 ? (w & 0xffffffffull) : (w & 0xffull));
    return s;
}

// A scalar argument of type t as a word (i32 sign-extended).
u64 scalar_word(vkc_type t, const vkc_scalar &s) {
    if (t == VKC_I32) return static_cast<u64>(static_cast<long long>(static_cast<int>(static_cast<unsigned>(s.bits))));
    if (width_of(t) == 4) return s.bits & 0xffffffffull;
    if (width_of(t) == 1) return s.bits & 0xffull;
    return s.bits;
}

// Reducers of the order-free folds. State: [0] the folded word (argmin/argmax: [0] key, [1] row), [2]
// whether any row was seen.
// `base` counts the rows of earlier updates.
struct FamReducer : DevReducer {
    vkc_type in, out;
    int fold;      // F_*, or -1 argmin, -2 argmax
    int row;       // R_*
    int nargs_want;
    int cmp = 0;
    bool empty_error = false;  // min/max/argmin/argmax of no rows fail
    const char *what = "";
    u64 base = 0;
    u64 empty = ~0ull;  // the word of no rows: the result, or argmin/argmax's key
    using Launch = void (*)(vkc_ctx *, const RowArgs &, int64_t, int, void *, u64, bool, u64 *, u64 *);
    Launch launch = nullptr;

    vkc_status clear(vkc_ctx *ctx) override { return fill(ctx, 3, empty, ~0ull, 0); }
    vkc_status update(vkc_ctx *ctx, const Arg *args, int nargs) override {
        vkc_status st;
        if (nargs != nargs_want) return fail(ctx, VKC_RUNTIME, arity_error(nargs_want, nargs));
        if (!rows_arg(ctx, args[0], in, &st)) return st;
        RowArgs a{args[0].a->data(), nullptr, cmp, 0, 0};
        if (row == R_DOT) {
            if (!rows_arg(ctx, args[1], in, &st)) return st;
            if (args[0].len() != args[1].len())
                return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(args[0].len()) + " vs " +
                                                  std::to_string(args[1].len()));
            a.y = args[1].a->data();
        } else if (row == R_COND || row == R_PRED) {
            for (int i = 1; i < nargs; ++i)
                if (!splat_arg(ctx, args[i], in, &st)) return st;
            a.c = scalar_word(in, args[1].s);
            if (row == R_COND) a.e = scalar_word(in, args[2].s);
        }
        const int64_t n = args[0].len();
        if (n == 0) return VKC_OK;
        const int grid = stream_grid(ctx, n, 256, tune(ctx, TK_STREAM_BLOCKS, n), 4096);
        void *part;
        if ((st = scratch(ctx, 16 * static_cast<size_t>(grid), &part))) return st;
        launch(ctx, a, n, grid, part, base, fresh, static_cast<u64 *>(state), static_cast<u64 *>(slot(ctx)));
        updated(ctx);
        base += static_cast<u64>(n);
        return launched(ctx, "family_fold");
    }
    vkc_status finish(vkc_ctx *ctx, vkc_scalar *out_s) override {
        u64 h[3] = {empty, 0, 0};
        vkc_status st = fresh ? VKC_OK : result(ctx, h, sizeof h);
        if (st) return st;
        if (empty_error && !h[2]) return fail(ctx, VKC_RUNTIME, std::string(what) + " of an empty array");
        *out_s = fold < 0 ? scalar_i64(static_cast<int64_t>(h[1])) : word_scalar(out, h[0]);
        return VKC_OK;
    }
    vkc_status finish_into(vkc_ctx *ctx, void *dst) override {
        if (empty_error && base == 0) return fail(ctx, VKC_RUNTIME, std::string(what) + " of an empty array");
        const vkc_status st = fresh ? fill(ctx, 1, empty) : VKC_OK;
        if (st) return st;
        // Words are little-endian: the result type's bytes are the word's low bytes.
        return fold < 0 ? copy_out(ctx, dst, 8, 8) : copy_out(ctx, dst, static_cast<size_t>(width_of(out)));
    }
};

template <vkc_type T, int F, int ROW>
void launch_fold(vkc_ctx *ctx, const RowArgs &a, int64_t n, int grid, void *part, u64, bool fresh, u64 *state, u64 *host) {
    fam_fold_kernel<T, F, ROW><<<grid, 256, 0, ctx->stream>>>(a, n, static_cast<u64 *>(part), ctx->counters + 1, fresh, state, host);
}
template <vkc_type T, bool MAX>
void launch_arg(vkc_ctx *ctx, const RowArgs &a, int64_t n, int grid, void *part, u64 base, bool fresh, u64 *state, u64 *host) {
    fam_arg_kernel<T, MAX><<<grid, 256, 0, ctx->stream>>>(a.x, n, base, static_cast<ulonglong2 *>(part),
                                                          ctx->counters + 1, fresh, state, host);
}

template <vkc_type T, int F, int ROW, int NARGS>
ReducerImpl *make_fold(vkc_ctx *ctx, vkc_type out, int cmp, bool empty_error, const char *what) {
    auto *r = new FamReducer;
    if (r->alloc(ctx, 24)) {
        delete r;
        return nullptr;
    }
    r->in = T;
    r->out = out;
    r->fold = F;
    r->row = ROW;
    r->nargs_want = NARGS;
    r->cmp = cmp;
    r->empty_error = empty_error;
    r->what = what;
    r->launch = launch_fold<T, F, ROW>;
    r->empty = identity<ROW == R_PRED ? VKC_U64 : T, F>();
    return r;
}

template <vkc_type T, bool MAX> ReducerImpl *make_arg(vkc_ctx *ctx) {
    auto *r = new FamReducer;
    if (r->alloc(ctx, 24)) {
        delete r;
        return nullptr;
    }
    r->in = T;
    r->out = VKC_I64;
    r->fold = MAX ? -2 : -1;
    r->row = R_PLAIN;
    r->nargs_want = 1;
    r->empty_error = true;
    r->what = MAX ? "argmax" : "argmin";
    r->launch = launch_arg<T, MAX>;
    return r;
}

// ------------------------------------------------------------------ canonical float products
//
// reduce.rs:45-91: lane j multiplies rows 16b + j in order from 1; then the lanes 8, 4, 2 and 1
// apart; then the tail. One block: warps 1..7 stage chunk k + 1 (FC_ROWS rows, as row values)
// in shared memory while the first sixteen threads of warp 0 run their lane chains over chunk k.
constexpr int FC_BLOCKS = 128;               // 16-row blocks per chunk
constexpr int FC_ROWS = FC_BLOCKS * 16;      // rows per chunk

template <vkc_type T> __global__ void __launch_bounds__(256) fam_chain_kernel(const void *x, int64_t nb, u64 *lanes) {
    __shared__ u64 buf[2][FC_ROWS];
    const int t = threadIdx.x;
    const int64_t chunks = (nb + FC_BLOCKS - 1) / FC_BLOCKS;
    auto stage = [&](int64_t k, int first, int step) {
        const int64_t r0 = k * FC_ROWS, rows = min(static_cast<int64_t>(FC_ROWS), nb * 16 - r0);
        for (int i = first; i < rows; i += step) buf[k & 1][i] = ld_word<T>(x, r0 + i);
    };
    u64 s = t < 16 ? lanes[t] : 0ull;
    if (chunks > 0) stage(0, t, 256);
    __syncthreads();
    for (int64_t k = 0; k < chunks; ++k) {
        if (t >= 32) {
            if (k + 1 < chunks) stage(k + 1, t - 32, 224);
        } else if (t < 16) {
            const int blocks = static_cast<int>(min(static_cast<int64_t>(FC_BLOCKS), nb - k * FC_BLOCKS));
            const u64 *b = buf[k & 1];
            for (int i = 0; i < blocks; ++i) s = mul_t<T>(s, b[i * 16 + t]);
        }
        __syncthreads();
    }
    if (t < 16) lanes[t] = s;
}

// The tail rows (fewer than 16), kept until finish.
template <vkc_type T> __global__ void fam_chain_tail(const void *x, int64_t first, int rest, u64 *tail) {
    if (static_cast<int>(threadIdx.x) < rest) tail[threadIdx.x] = ld_word<T>(x, first + threadIdx.x);
}

// reduce.rs:77-91 (finish_lanes).
template <vkc_type T> __global__ void fam_chain_finish(u64 *st, int tail_len, u64 *host) {
    u64 acc[16];
    for (int j = 0; j < 16; ++j) acc[j] = st[j];
    for (int s = 8; s > 0; s >>= 1)
        for (int j = 0; j < s; ++j) acc[j] = mul_t<T>(acc[j], acc[j + s]);
    u64 r = acc[0];
    for (int j = 0; j < tail_len; ++j) r = mul_t<T>(r, st[16 + j]);
    st[32] = r;
    if (host) *host = r;
}

// CanonicalAcc (reduce.rs:253-323) on the device. State: [0..15] lanes, [16..31] tail, [32] result.
template <vkc_type T> struct ChainReducer : DevReducer {
    int tail_len = 0;

    vkc_status clear(vkc_ctx *) override { return VKC_OK; }  // made with its state

    vkc_status update(vkc_ctx *ctx, const Arg *args, int nargs) override {
        vkc_status st;
        if (nargs != 1) return fail(ctx, VKC_RUNTIME, arity_error(1, nargs));
        if (!rows_arg(ctx, args[0], T, &st)) return st;
        const int64_t n = args[0].len();
        if (tail_len != 0) return fail(ctx, VKC_RUNTIME, "canonical update after a partial block");
        const void *x = args[0].a->data();
        auto *s = static_cast<u64 *>(state);
        const int64_t nb = n / 16;
        const int rest = static_cast<int>(n % 16);
        if (nb > 0) fam_chain_kernel<T><<<1, 256, 0, ctx->stream>>>(x, nb, s);
        if (rest > 0) fam_chain_tail<T><<<1, 16, 0, ctx->stream>>>(x, nb * 16, rest, s + 16);
        tail_len = rest;
        return launched(ctx, "family_chain");
    }
    vkc_status combine(vkc_ctx *ctx) {
        fam_chain_finish<T><<<1, 1, 0, ctx->stream>>>(static_cast<u64 *>(state), tail_len, static_cast<u64 *>(slot(ctx)));
        updated(ctx);
        return launched(ctx, "family_chain_finish");
    }
    vkc_status finish(vkc_ctx *ctx, vkc_scalar *out) override {
        vkc_status st = combine(ctx);
        if (st) return st;
        u64 r = 0;
        if ((st = result(ctx, &r, 8, 32 * 8))) return st;
        *out = word_scalar(T, r);
        return VKC_OK;
    }
    vkc_status finish_into(vkc_ctx *ctx, void *dst) override {
        const vkc_status st = combine(ctx);
        return st ? st : copy_out(ctx, dst, static_cast<size_t>(width_of(T)), 32 * 8);
    }
};

template <vkc_type T> ReducerImpl *make_product(vkc_ctx *ctx) {
    auto *r = new ChainReducer<T>;
    const u64 one = T == VKC_F64 ? 0x3ff0000000000000ull : 0x3f800000ull;
    if (r->alloc(ctx, 33 * 8) || r->fill(ctx, 33, one, one, one, one)) {
        delete r;
        return nullptr;
    }
    return r;
}

// ------------------------------------------------------------------ prev

// prev_T (scan.rs:16-73): out[0] is the fill on the first update, else the last row of the
// previous update; out[i] = x[i - 1]. carry: [0] last row, [1] seen.
template <int W>
__global__ void fam_prev_kernel(const void *x, void *out, int64_t n, u64 fill, const u64 *carry) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        u64 v;
        if (i == 0) v = carry[1] ? carry[0] : fill;
        else if (W == 8) v = static_cast<const u64 *>(x)[i - 1];
        else if (W == 4) v = static_cast<const unsigned *>(x)[i - 1];
        else v = static_cast<const unsigned char *>(x)[i - 1];
        st_word<W>(out, i, v);
    }
}
template <int W> __global__ void fam_prev_carry(const void *x, int64_t n, u64 *carry) {
    carry[0] = W == 8 ? static_cast<const u64 *>(x)[n - 1]
                      : (W == 4 ? static_cast<const unsigned *>(x)[n - 1] : static_cast<const unsigned char *>(x)[n - 1]);
    carry[1] = 1;
}

struct FamPrev : ScannerImpl {
    vkc_type t;
    u64 *carry = nullptr;
    DeviceMem mem;
    vkc_status update(vkc_ctx *ctx, const Arg *args, int nargs, vkc_array *o) override {
        vkc_status st;
        if (nargs != 2) return fail(ctx, VKC_RUNTIME, arity_error(2, nargs));
        if (!rows_arg(ctx, args[0], t, &st) || !splat_arg(ctx, args[1], t, &st)) return st;
        const int64_t n = args[0].len();
        if (o->len != n)
            return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(n) + " rows for a destination of " +
                                              std::to_string(o->len) + " rows");
        if (n == 0) return VKC_OK;
        const int grid = stream_grid(ctx, n, 256, 8, 2048);
        const void *x = args[0].a->data();
        const u64 fill = args[1].s.bits;
        switch (width_of(t)) {
        case 8:
            fam_prev_kernel<8><<<grid, 256, 0, ctx->stream>>>(x, o->data(), n, fill, carry);
            fam_prev_carry<8><<<1, 1, 0, ctx->stream>>>(x, n, carry);
            break;
        case 4:
            fam_prev_kernel<4><<<grid, 256, 0, ctx->stream>>>(x, o->data(), n, fill, carry);
            fam_prev_carry<4><<<1, 1, 0, ctx->stream>>>(x, n, carry);
            break;
        default:
            fam_prev_kernel<1><<<grid, 256, 0, ctx->stream>>>(x, o->data(), n, fill, carry);
            fam_prev_carry<1><<<1, 1, 0, ctx->stream>>>(x, n, carry);
            break;
        }
        return launched(ctx, "family_prev");
    }
};

template <vkc_type T> ScannerImpl *make_prev_fam(vkc_ctx *ctx) {
    auto *s = new FamPrev;
    s->t = T;
    if (cudaMallocAsync(reinterpret_cast<void **>(&s->carry), 16, ctx->stream) != cudaSuccess ||
        cudaMemsetAsync(s->carry, 0, 16, ctx->stream) != cudaSuccess) {
        cudaGetLastError();
        delete s;
        return nullptr;
    }
    s->mem.ptr = s->carry;
    s->mem.box = ctx->box;
    return s;
}

// ------------------------------------------------------------------ reduce_into

// Each bucket word starts at the fold's identity; rows step their bucket with an atomic of the
// fold (a compare-and-swap loop for products and float extremes), then the words narrow to
// the output type. The fold is order-free, so the result is the reference's sequential one.
template <vkc_type IT, vkc_type OT, int F>
__device__ __forceinline__ void bucket_step(u64 *p, u64 v) {
    if (F == F_ADD) atomicAdd(p, v);
    else if (F == F_AND) atomicAnd(p, v);
    else if (F == F_OR) atomicOr(p, v);
    else if (F == F_XOR) atomicXor(p, v);
    else if ((F == F_MIN || F == F_MAX) && is_signed_t(IT)) {
        if (F == F_MIN) atomicMin(reinterpret_cast<long long *>(p), static_cast<long long>(v));
        else atomicMax(reinterpret_cast<long long *>(p), static_cast<long long>(v));
    } else if ((F == F_MIN || F == F_MAX) && !is_float(IT)) {
        if (F == F_MIN) atomicMin(p, v);
        else atomicMax(p, v);
    } else {
        u64 old = *reinterpret_cast<volatile u64 *>(p);
        for (;;) {
            const u64 want = F == F_MUL ? wrap<IT>(old * v) : step<IT, F>(old, v);
            if (want == old) break;
            const u64 seen = atomicCAS(p, old, want);
            if (seen == old) break;
            old = seen;
        }
    }
}

template <vkc_type OT, int F> __global__ void fam_bucket_init(u64 *w, int64_t nb) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nb; i += stride)
        w[i] = identity<OT, F>();
}

template <vkc_type IT, vkc_type OT, int F>
__global__ void __launch_bounds__(256) fam_bucket_kernel(const long long *keys, const void *vals, int64_t n, u64 *w) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        bucket_step<IT, OT, F>(w + keys[i], ld_word<IT>(vals, i));
}

template <int W> __global__ void fam_narrow(const u64 *w, void *out, int64_t nb) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nb; i += stride)
        st_word<W>(out, i, w[i]);
}

// index.rs:194-222 (ReduceInto): the values' kind, then checked_keys (:116-130: the keys' kind,
// the count, a negative count, the first key out of range), then the lengths, then the result.
template <vkc_type IT, int F>
vkc_status reduce_into_fam(vkc_ctx *ctx, const vkc_value *args, int nargs, vkc_value *out) {
    constexpr vkc_type OT = F == F_ADD ? sum_type(IT) : IT;
    vkc_status st;
    if (nargs != 3) return fail(ctx, VKC_RUNTIME, arity_error(3, nargs));
    if (!array_arg(ctx, args[1], IT, &st)) return st;
    int64_t nb;
    if (!array_arg(ctx, args[0], VKC_I64, &st) || !i64_arg(ctx, args[2], &nb, &st)) return st;
    if (nb < 0) return fail(ctx, VKC_RUNTIME, "negative bucket count " + std::to_string(nb));
    const vkc_array *keys = args[0].array, *vals = args[1].array;
    const int64_t n = keys->len;
    const auto *k = static_cast<const long long *>(keys->data());
    bool found;
    if ((st = bucket_key_error(ctx, k, n, nb, &found)) || found) return st;
    if (vals->len != n)
        return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(n) + " keys for " + std::to_string(vals->len) +
                                          " values");
    vkc_array *o;
    if ((st = new_array(ctx, OT, nb, false, &o))) return st;
    if (nb > 0) {
        u64 *w = static_cast<u64 *>(o->data());
        vkc_array *tmp = nullptr;
        if (width_of(OT) != 8) {
            if ((st = new_array(ctx, VKC_U64, nb, false, &tmp))) {
                vkc_array_release(o);
                return st;
            }
            w = static_cast<u64 *>(tmp->data());
        }
        const int g0 = stream_grid(ctx, nb, 256, 8, 2048);
        fam_bucket_init<OT, F><<<g0, 256, 0, ctx->stream>>>(w, nb);
        if (n > 0) {
            const int g = stream_grid(ctx, n, 256, 8, 2048);
            fam_bucket_kernel<IT, OT, F><<<g, 256, 0, ctx->stream>>>(k, vals->data(), n, w);
        }
        if (tmp) {
            if (width_of(OT) == 4) fam_narrow<4><<<g0, 256, 0, ctx->stream>>>(w, o->data(), nb);
            else fam_narrow<1><<<g0, 256, 0, ctx->stream>>>(w, o->data(), nb);
            vkc_array_release(tmp);
        }
        if ((st = launched(ctx, "family_reduce_into"))) {
            vkc_array_release(o);
            return st;
        }
    }
    out->kind = VKC_VALUE_ARRAY;
    out->array = o;
    return VKC_OK;
}

// ------------------------------------------------------------------ whole kernels

// Widens keys to i64 for the i64 group ids (any one-to-one image serves).
template <vkc_type T>
__global__ void fam_widen_kernel(const void *x, int64_t n, long long *o) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        o[i] = static_cast<long long>(ld_word<T>(x, i));
    }
}

template <vkc_type T> vkc_status widen(vkc_ctx *ctx, const vkc_array *a, vkc_array **out) {
    vkc_status st;
    if ((st = new_array(ctx, VKC_I64, a->len, false, out))) return st;
    if (a->len > 0) {
        const int g = stream_grid(ctx, a->len, 256, 8, 2048);
        fam_widen_kernel<T><<<g, 256, 0, ctx->stream>>>(a->data(), a->len, static_cast<long long *>((*out)->data()));
        if ((st = launched(ctx, "family_widen"))) {
            vkc_array_release(*out);
            return st;
        }
    }
    return VKC_OK;
}

// group_id_T (group.rs:259-274): ids by first occurrence depend only on which rows are equal.
template <vkc_type T> vkc_status group_id_fam(vkc_ctx *ctx, const vkc_value *args, int nargs, vkc_value *out) {
    vkc_status st;
    if (nargs != 1) return fail(ctx, VKC_RUNTIME, arity_error(1, nargs));
    if (!array_arg(ctx, args[0], T, &st)) return st;
    vkc_array *w;
    if ((st = widen<T>(ctx, args[0].array, &w))) return st;
    static const KernelDef *d = kernel_def("group_id_i64");
    vkc_value a{};
    a.kind = VKC_VALUE_ARRAY;
    a.array = w;
    st = d->whole(ctx, &a, 1, out);
    vkc_array_release(w);
    return st;
}

// group_id2_A_B (group.rs:276-299): both columns' kinds, then the lengths, as the reference.
template <vkc_type A, vkc_type B> vkc_status group_id2_fam(vkc_ctx *ctx, const vkc_value *args, int nargs, vkc_value *out) {
    vkc_status st;
    if (nargs != 2) return fail(ctx, VKC_RUNTIME, arity_error(2, nargs));
    if (!array_arg(ctx, args[0], A, &st) || !array_arg(ctx, args[1], B, &st)) return st;
    if (args[0].array->len != args[1].array->len)
        return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(args[0].array->len) + " vs " +
                                          std::to_string(args[1].array->len));
    vkc_array *wa, *wb;
    if ((st = widen<A>(ctx, args[0].array, &wa))) return st;
    if ((st = widen<B>(ctx, args[1].array, &wb))) {
        vkc_array_release(wa);
        return st;
    }
    static const KernelDef *d = kernel_def("group_id2_i64_i64");
    vkc_value a[2]{};
    a[0].kind = a[1].kind = VKC_VALUE_ARRAY;
    a[0].array = wa;
    a[1].array = wb;
    st = d->whole(ctx, a, 2, out);
    vkc_array_release(wa);
    vkc_array_release(wb);
    return st;
}

// fill_T (construct.rs:49-61): n copies of v; "negative length" for n < 0, the value's type,
// then the size.
template <int W> __global__ void fam_fill_kernel(void *o, int64_t n, u64 v) {
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) st_word<W>(o, i, v);
}

template <vkc_type T> vkc_status fill_fam(vkc_ctx *ctx, const vkc_value *args, int nargs, vkc_value *out) {
    vkc_status st;
    if (nargs != 2) return fail(ctx, VKC_RUNTIME, arity_error(2, nargs));
    int64_t n;
    if (!i64_arg(ctx, args[0], &n, &st)) return st;
    if (n < 0) return fail(ctx, VKC_RUNTIME, "negative length " + std::to_string(n));
    if (args[1].kind != VKC_VALUE_SCALAR || args[1].scalar.type != T)
        return fail(ctx, VKC_RUNTIME, std::string("expected ") + type_name(T) + ", got " + value_type_name(args[1]));
    vkc_array *o;
    if ((st = new_array(ctx, T, n, false, &o))) return st;
    if (n > 0) {
        const int g = stream_grid(ctx, n, 256, 8, 4096);
        const u64 v = args[1].scalar.bits;
        switch (width_of(T)) {
        case 8: fam_fill_kernel<8><<<g, 256, 0, ctx->stream>>>(o->data(), n, v); break;
        case 4: fam_fill_kernel<4><<<g, 256, 0, ctx->stream>>>(o->data(), n, v); break;
        default: fam_fill_kernel<1><<<g, 256, 0, ctx->stream>>>(o->data(), n, v); break;
        }
        if ((st = launched(ctx, "family_fill"))) {
            vkc_array_release(o);
            return st;
        }
    }
    out->kind = VKC_VALUE_ARRAY;
    out->array = o;
    return VKC_OK;
}

// slice_T (index.rs:240-258): a view of rows start..end, or "slice s..e out of range for length n".
template <vkc_type T> vkc_status slice_fam(vkc_ctx *ctx, const vkc_value *args, int nargs, vkc_value *out) {
    vkc_status st;
    if (nargs != 3) return fail(ctx, VKC_RUNTIME, arity_error(3, nargs));
    if (!array_arg(ctx, args[0], T, &st)) return st;
    int64_t s, e;
    if (!i64_arg(ctx, args[1], &s, &st) || !i64_arg(ctx, args[2], &e, &st)) return st;
    const int64_t len = args[0].array->len;
    if (s < 0 || e < 0 || s > e || e > len)
        return fail(ctx, VKC_RUNTIME, "slice " + std::to_string(s) + ".." + std::to_string(e) +
                                          " out of range for length " + std::to_string(len));
    vkc_array *v;
    if ((st = vkc_array_slice(ctx, args[0].array, s, e - s, &v))) return st;
    out->kind = VKC_VALUE_ARRAY;
    out->array = v;
    return VKC_OK;
}

// same_len_T (construct.rs:108-120): the array itself when its length is n.
template <vkc_type T> vkc_status same_len_fam(vkc_ctx *ctx, const vkc_value *args, int nargs, vkc_value *out) {
    vkc_status st;
    if (nargs != 2) return fail(ctx, VKC_RUNTIME, arity_error(2, nargs));
    if (!array_arg(ctx, args[0], T, &st)) return st;
    int64_t n;
    if (!i64_arg(ctx, args[1], &n, &st)) return st;
    const int64_t len = args[0].array->len;
    if (len != n) return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(len) + " vs " + std::to_string(n));
    vkc_array_retain(args[0].array);
    out->kind = VKC_VALUE_ARRAY;
    out->array = args[0].array;
    return VKC_OK;
}

// ------------------------------------------------------------------ registration helpers

InSpec arr(vkc_type t) { return InSpec{IN_ARRAY, t}; }
InSpec sca(vkc_type t) { return InSpec{IN_SCALAR, t}; }

void add_red(std::vector<KernelDef> &t, const std::string &name, std::vector<InSpec> in, vkc_type out, uint64_t cost,
             ReducerMake make) {
    KernelDef d{name, VKC_REDUCTION, std::move(in), false, out, cost};
    d.red = make;
    t.push_back(d);
}
void add_whole(std::vector<KernelDef> &t, const std::string &name, std::vector<InSpec> in, vkc_type out, uint64_t cost,
               WholeFn f, bool out_array = true) {
    KernelDef d{name, VKC_WHOLE, std::move(in), out_array, out, cost};
    d.whole = f;
    t.push_back(d);
}
void add_scan(std::vector<KernelDef> &t, const std::string &name, std::vector<InSpec> in, vkc_type out, uint64_t cost,
              ScanMake make) {
    KernelDef d{name, VKC_SCAN, std::move(in), true, out, cost};
    d.scan = make;
    t.push_back(d);
}

bool has(const std::vector<KernelDef> &t, const std::string &name) {
    for (const KernelDef &d : t)
        if (d.name == name) return true;
    return false;
}

// Reductions of one numeric type (reduce.rs:664-686): add (sum type), mul, min, max, argmin,
// argmax, each with cost = the input width.
template <vkc_type T> void reg_numeric(std::vector<KernelDef> &t) {
    const std::string n = type_name(T);
    const uint64_t w = width_of(T);
    if (T == VKC_F32) {
        add_red(t, "reduce_add_" + n, {arr(T)}, T, w, make_canon32_sum);
        add_red(t, "reduce_mul_" + n, {arr(T)}, T, w, make_product<VKC_F32>);
    } else {
        add_red(t, "reduce_add_" + n, {arr(T)}, sum_type(T), w,
                [](vkc_ctx *c) { return make_fold<T, F_ADD, R_PLAIN, 1>(c, sum_type(T), 0, false, ""); });
        add_red(t, "reduce_mul_" + n, {arr(T)}, T, w,
                [](vkc_ctx *c) { return make_fold<T, F_MUL, R_PLAIN, 1>(c, T, 0, false, ""); });
    }
    add_red(t, "reduce_min_" + n, {arr(T)}, T, w,
            [](vkc_ctx *c) { return make_fold<T, F_MIN, R_PLAIN, 1>(c, T, 0, true, "reduce_min"); });
    add_red(t, "reduce_max_" + n, {arr(T)}, T, w,
            [](vkc_ctx *c) { return make_fold<T, F_MAX, R_PLAIN, 1>(c, T, 0, true, "reduce_max"); });
    add_red(t, "argmin_" + n, {arr(T)}, VKC_I64, w, make_arg<T, false>);
    add_red(t, "argmax_" + n, {arr(T)}, VKC_I64, w, make_arg<T, true>);
}

// Bit folds (reduce.rs:688-702, :704-712 for bool).
template <vkc_type T> void reg_bits(std::vector<KernelDef> &t) {
    const std::string n = type_name(T);
    const uint64_t w = width_of(T);
    add_red(t, "reduce_and_" + n, {arr(T)}, T, w, [](vkc_ctx *c) { return make_fold<T, F_AND, R_PLAIN, 1>(c, T, 0, false, ""); });
    add_red(t, "reduce_or_" + n, {arr(T)}, T, w, [](vkc_ctx *c) { return make_fold<T, F_OR, R_PLAIN, 1>(c, T, 0, false, ""); });
    add_red(t, "reduce_xor_" + n, {arr(T)}, T, w, [](vkc_ctx *c) { return make_fold<T, F_XOR, R_PLAIN, 1>(c, T, 0, false, ""); });
}

// Fused kernels of one type (fused.rs:290-371): dot (2 widths), sumsq (1), count_<cmp> (1),
// filter_<cmp> (2), condsum_<cmp> (1); sums in the sum type.
template <vkc_type T, int C> void reg_cmp(std::vector<KernelDef> &t) {
    const std::string n = type_name(T), c = CMP_NAME[C];
    const uint64_t w = width_of(T);
    static_assert(T != VKC_F64, "the f64 entries are k_reduce.cu's, k_select.cu's and k_canon.cu's");
    add_red(t, "count_" + c + "_" + n, {arr(T), sca(T)}, VKC_I64, w,
            [](vkc_ctx *x) { return make_fold<T, F_ADD, R_PRED, 2>(x, VKC_I64, C, false, ""); });
    KernelDef f{"filter_" + c + "_" + n, VKC_SELECTION, {arr(T), sca(T)}, true, T, 2 * w};
    f.sel = filter_fn(T, C);
    t.push_back(f);
    if (T == VKC_F32)
        add_red(t, "condsum_" + c + "_" + n, {arr(T), sca(T), sca(T)}, T, w,
                [](vkc_ctx *x) { return make_canon32_cond(x, C); });
    else
        add_red(t, "condsum_" + c + "_" + n, {arr(T), sca(T), sca(T)}, sum_type(T), w,
                [](vkc_ctx *x) { return make_fold<T, F_ADD, R_COND, 3>(x, sum_type(T), C, false, ""); });
}

template <vkc_type T> void reg_fused(std::vector<KernelDef> &t) {
    const std::string n = type_name(T);
    const uint64_t w = width_of(T);
    if (T == VKC_F32) {
        add_red(t, "dot_" + n, {arr(T), arr(T)}, T, 2 * w, make_canon32_dot);
        add_red(t, "sumsq_" + n, {arr(T)}, T, w, make_canon32_sumsq);
    } else {
        add_red(t, "dot_" + n, {arr(T), arr(T)}, sum_type(T), 2 * w,
                [](vkc_ctx *c) { return make_fold<T, F_ADD, R_DOT, 2>(c, sum_type(T), 0, false, ""); });
        add_red(t, "sumsq_" + n, {arr(T)}, sum_type(T), w,
                [](vkc_ctx *c) { return make_fold<T, F_ADD, R_SUMSQ, 1>(c, sum_type(T), 0, false, ""); });
    }
    reg_cmp<T, 0>(t);
    reg_cmp<T, 1>(t);
    reg_cmp<T, 2>(t);
    reg_cmp<T, 3>(t);
    reg_cmp<T, 4>(t);
    reg_cmp<T, 5>(t);
}

template <vkc_type T> ScanMake scan_make(int fold, bool by) {
    return width_of(T) == 8 ? wide_scan(T, fold, by) : narrow_scan(T, fold, by);
}

// scan_<f>_T, scan_by_<f>_T, reduce_into_<f>_T (scan.rs:330-385): costs in+out widths, +1 for
// scan_by, 8 + in + 2 out for reduce_into.
template <vkc_type T, int F> void reg_fold(std::vector<KernelDef> &t) {
    constexpr vkc_type OT = F == F_ADD ? sum_type(T) : T;
    const std::string n = std::string(FOLD_NAMES[F]) + "_" + type_name(T);
    const uint64_t cost = width_of(T) + width_of(OT);
    if (!has(t, "scan_" + n)) add_scan(t, "scan_" + n, {arr(T)}, OT, cost, scan_make<T>(F, false));
    if (!has(t, "scan_by_" + n)) add_scan(t, "scan_by_" + n, {arr(T), arr(VKC_BOOL)}, OT, cost + 1, scan_make<T>(F, true));
    if (!has(t, "reduce_into_" + n))
        add_whole(t, "reduce_into_" + n, {arr(VKC_I64), arr(T), sca(VKC_I64)}, OT, 8 + width_of(T) + 2 * width_of(OT),
                  reduce_into_fam<T, F>);
}

template <vkc_type T> void reg_int_folds(std::vector<KernelDef> &t) {
    reg_fold<T, F_ADD>(t);
    reg_fold<T, F_MUL>(t);
    reg_fold<T, F_MIN>(t);
    reg_fold<T, F_MAX>(t);
    reg_fold<T, F_AND>(t);
    reg_fold<T, F_OR>(t);
    reg_fold<T, F_XOR>(t);
}

template <vkc_type T> void reg_prev(std::vector<KernelDef> &t) {
    const std::string n = std::string("prev_") + type_name(T);
    if (!has(t, n)) add_scan(t, n, {arr(T), sca(T)}, T, 2 * width_of(T), make_prev_fam<T>);
}

template <vkc_type T> void reg_whole_of(std::vector<KernelDef> &t) {
    const std::string n = type_name(T);
    const uint64_t w = width_of(T);
    add_whole(t, "fill_" + n, {sca(VKC_I64), sca(T)}, T, w, fill_fam<T>);
    add_whole(t, "slice_" + n, {arr(T), sca(VKC_I64), sca(VKC_I64)}, T, 0, slice_fam<T>);
    add_whole(t, "same_len_" + n, {arr(T), sca(VKC_I64)}, T, 0, same_len_fam<T>);
}

template <vkc_type A> void reg_group2(std::vector<KernelDef> &t) {
    const vkc_type bs[4] = {VKC_I64, VKC_U64, VKC_I32, VKC_U8};
    const WholeFn fs[4] = {group_id2_fam<A, VKC_I64>, group_id2_fam<A, VKC_U64>, group_id2_fam<A, VKC_I32>,
                           group_id2_fam<A, VKC_U8>};
    for (int i = 0; i < 4; ++i) {
        const std::string n = std::string("group_id2_") + type_name(A) + "_" + type_name(bs[i]);
        if (!has(t, n)) add_whole(t, n, {arr(A), arr(bs[i])}, VKC_I64, width_of(A) + width_of(bs[i]) + 8, fs[i]);
    }
}

}  // namespace

void register_families(std::vector<KernelDef> &t) {
    // reduce.rs:714-726
    reg_numeric<VKC_F32>(t);
    reg_numeric<VKC_I32>(t);
    reg_numeric<VKC_U8>(t);
    reg_numeric<VKC_U64>(t);
    add_red(t, "reduce_mul_f64", {arr(VKC_F64)}, VKC_F64, 8,
            make_product<VKC_F64>);
    add_red(t, "reduce_mul_i64", {arr(VKC_I64)}, VKC_I64, 8,
            [](vkc_ctx *c) { return make_fold<VKC_I64, F_MUL, R_PLAIN, 1>(c, VKC_I64, 0, false, ""); });
    reg_bits<VKC_I64>(t);
    reg_bits<VKC_I32>(t);
    reg_bits<VKC_U8>(t);
    reg_bits<VKC_U64>(t);
    add_red(t, "reduce_and_bool", {arr(VKC_BOOL)}, VKC_BOOL, 1,
            [](vkc_ctx *c) { return make_fold<VKC_BOOL, F_AND, R_PLAIN, 1>(c, VKC_BOOL, 0, false, ""); });
    add_red(t, "reduce_or_bool", {arr(VKC_BOOL)}, VKC_BOOL, 1,
            [](vkc_ctx *c) { return make_fold<VKC_BOOL, F_OR, R_PLAIN, 1>(c, VKC_BOOL, 0, false, ""); });
    add_red(t, "reduce_xor_bool", {arr(VKC_BOOL)}, VKC_BOOL, 1,
            [](vkc_ctx *c) { return make_fold<VKC_BOOL, F_XOR, R_PLAIN, 1>(c, VKC_BOOL, 0, false, ""); });
    add_red(t, "any", {arr(VKC_BOOL)}, VKC_BOOL, 1,
            [](vkc_ctx *c) { return make_fold<VKC_BOOL, F_OR, R_PLAIN, 1>(c, VKC_BOOL, 0, false, ""); });
    add_red(t, "all", {arr(VKC_BOOL)}, VKC_BOOL, 1,
            [](vkc_ctx *c) { return make_fold<VKC_BOOL, F_AND, R_PLAIN, 1>(c, VKC_BOOL, 0, false, ""); });
    // fused.rs:373-379
    reg_fused<VKC_F32>(t);
    reg_fused<VKC_I64>(t);
    reg_fused<VKC_U64>(t);
    reg_fused<VKC_I32>(t);
    // scan.rs:424-439
    reg_int_folds<VKC_I64>(t);
    reg_int_folds<VKC_U64>(t);
    reg_int_folds<VKC_I32>(t);
    reg_int_folds<VKC_U8>(t);
    reg_fold<VKC_F64, F_MIN>(t);
    reg_fold<VKC_F64, F_MAX>(t);
    reg_fold<VKC_F32, F_MIN>(t);
    reg_fold<VKC_F32, F_MAX>(t);
    reg_fold<VKC_BOOL, F_AND>(t);
    reg_fold<VKC_BOOL, F_OR>(t);
    reg_fold<VKC_BOOL, F_XOR>(t);
    reg_prev<VKC_F64>(t);
    reg_prev<VKC_F32>(t);
    reg_prev<VKC_U64>(t);
    reg_prev<VKC_I32>(t);
    reg_prev<VKC_U8>(t);
    reg_prev<VKC_BOOL>(t);
    // index.rs:290-325, group.rs:352-363, construct.rs:214-270
    add_whole(t, "group_id_u64", {arr(VKC_U64)}, VKC_I64, 16, group_id_fam<VKC_U64>);
    add_whole(t, "group_id_i32", {arr(VKC_I32)}, VKC_I64, 12, group_id_fam<VKC_I32>);
    add_whole(t, "group_id_u8", {arr(VKC_U8)}, VKC_I64, 9, group_id_fam<VKC_U8>);
    reg_group2<VKC_I64>(t);
    reg_group2<VKC_U64>(t);
    reg_group2<VKC_I32>(t);
    reg_group2<VKC_U8>(t);
    reg_whole_of<VKC_F64>(t);
    reg_whole_of<VKC_F32>(t);
    reg_whole_of<VKC_I64>(t);
    reg_whole_of<VKC_U64>(t);
    reg_whole_of<VKC_I32>(t);
    reg_whole_of<VKC_U8>(t);
    reg_whole_of<VKC_BOOL>(t);
}

}  // namespace vkc
