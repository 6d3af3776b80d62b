// The canonical f32 sums: reduce_add_f32, dot_f32, sumsq_f32 and condsum_<cmp>_f32, bit for bit the
// reference's order at every length (src/kernels/scalar/reduce.rs:45-91, :253-323;
// src/kernels/scalar/fused.rs:73-212): lane j (0..15) starts at +0.0 and adds rows j, j+16, ... one
// after another, the lanes combine +8, +4, +2, +1, and the tail rows fold into lane 0.
//
// A lane is a chain of n/16 dependent rounded adds, 4.4 cycles each at best. It is cut into tiles of 512 rows
// a lane that run in parallel, each as a function of the state it starts from. While the state
// stays in one binade [2^E, 2^(E+1)) with ulp u, s = S u and fl(s + x) = (S + RNE(x / u)) u, where
// a tie goes to the even S: the step depends on S by its parity alone. So the effect of a run of
// rows is known from two starts, one even and one odd: the run's adds are executed, as IEEE adds,
// from 1.5 * 2^E and from the next float, and the run moves any state of that binade by the same
// number of ulps, as long as no partial sum leaves the binade (from the lowest and highest one,
// kept as offsets). FP32 adds run at full rate here, so a row costs about six instructions and the
// passes are bound by memory: a tile's function needs no integer arithmetic on the rows and holds
// for rows and states of either sign (a negative state's magnitude moves by the mirrored adds).
//
//   C1  the approximate lane sums of every tile (float), one read;
//   C2  per lane their exclusive prefix from the lane's state: the binade each tile starts in;
//   C3  each tile's function in that binade, the second read (from L2 up to about 2^25 rows);
//   C4  the composed functions of 32 tiles that share a binade;
//   C5  per lane, the walk from the exact state: 32-tile chunks and tiles while their functions
//       apply, and the other tiles (binade crossings, a wrong estimate, special values) from their
//       rows by one warp, sixteen rows a thread, the rows of a thread whose run does not apply
//       added one by one. An estimate that is off costs time in the walk, never exactness.
//
// Measured on GB300 (a call alone) against one block that staged the rows and ran the sixteen chains:
// reduce_add_f32 of 2^20 rows 88 us (956), 2^24 rows 123 us (16.6 ms), 2^26 rows 212 us (147 ms);
// dot_f32 of 2^26 rows 336 us (157 ms), of which the two reads take 160.
#include "kcommon.cuh"
#include "reduce_common.h"

namespace vkc {

namespace {

constexpr int C32_THREADS = 256;
constexpr int C32_RUN = 8;                             // 16-row blocks per thread of a tile pass
constexpr int C32_BLOCKS = C32_THREADS / 4 * C32_RUN;  // 512 blocks (rows of a lane) per tile
constexpr int C32_CHUNK = 32;                          // tiles per chunk
constexpr unsigned C32_NONE = 0;  // no binade (codes of states are sign and exponent, never 0 or 255)
constexpr int C32_TOP = 1 << 24;

enum Row32 { R32_SUM = 0, R32_DOT = 1, R32_SUMSQ = 2, R32_COND = 3 };

struct Args32 {
    const float *x;
    const float *y;
    int cmp;
    float c, e;
};

__device__ __forceinline__ bool test32(int cmp, float x, float c) {
    switch (cmp) {
    case 0: return x == c;
    case 1: return x != c;
    case 2: return x < c;
    case 3: return x <= c;
    case 4: return x > c;
    default: return x >= c;
    }
}

// The row value fed to the lane (fused.rs:77-203): one IEEE multiply, never contracted.
template <int OP> __device__ __forceinline__ float value32(const Args32 &a, float x, float y) {
    if (OP == R32_DOT) return __fmul_rn(x, y);
    if (OP == R32_SUMSQ) return __fmul_rn(x, x);
    if (OP == R32_COND) return test32(a.cmp, x, a.c) ? x : a.e;
    return x;
}

// The effect of a run of rows on a state of one binade: the magnitude's move in ulps from an even
// (d0) and an odd (d1) start, a bound of the highest state on the way (mx) and of the lowest one within
// the parts that may move it down (mn; NO_FALL32 when there is none).
//
// The lowest state has to stay an ulp above 2^E whatever rose before it: a sum that rounds to 2^E may lie
// below it, on the finer grid. (A run up by k ulps and one down by k, composed, end where they began.)
struct Run32 {
    int d0, d1, mn, mx;
};
constexpr int NO_FALL32 = 1 << 30;  // no composed move reaches 2^29 (c32_runs): sums with it do not wrap
constexpr Run32 STILL32{0, 0, NO_FALL32, 0};

__device__ __forceinline__ Run32 then32(Run32 a, Run32 b) {
    return Run32{a.d0 + ((a.d0 & 1) ? b.d1 : b.d0), a.d1 + ((a.d1 & 1) ? b.d0 : b.d1),
                 min(a.mn, min(a.d0, a.d1) + b.mn), max(a.mx, max(a.d0, a.d1) + b.mx)};
}
__device__ __forceinline__ Run32 shfl_up32(Run32 v, int o) {
    return Run32{__shfl_up_sync(FULL, v.d0, o), __shfl_up_sync(FULL, v.d1, o), __shfl_up_sync(FULL, v.mn, o),
                 __shfl_up_sync(FULL, v.mx, o)};
}
__device__ __forceinline__ Run32 shfl_down32(Run32 v, int o) {
    return Run32{__shfl_down_sync(FULL, v.d0, o), __shfl_down_sync(FULL, v.d1, o), __shfl_down_sync(FULL, v.mn, o),
                 __shfl_down_sync(FULL, v.mx, o)};
}

// The code of a state: its sign and exponent bits. A usable one is a normal with a finite binade
// above it (so 1.5 * 2^E and 2^(E+1) are floats).
__device__ __forceinline__ unsigned code32(float s) {
    const unsigned c = __float_as_uint(s) >> 23, e = c & 0xffu;
    return e >= 1u && e <= 253u ? c : C32_NONE;
}

// Starts of the two runs of a binade, as magnitudes (rounding to nearest even is symmetric, so a
// negative state takes the rows with their signs flipped), and the magnitudes between which a run
// keeps its offsets exact: a partial sum that rounds to at least 2^E + 2 u and at most 2^(E+1) - 3 u
// has its exact value inside the binade, and so has the odd run's, at most one ulp further off.
struct Start32 {
    float even, odd, lo, hi;
};
__device__ __forceinline__ Start32 start32(unsigned code) {
    const unsigned e = (code & 0xffu) << 23;
    return Start32{__uint_as_float(e | 0x400000u), __uint_as_float(e | 0x400001u), __uint_as_float(e | 2u),
                   __uint_as_float(e | 0x7ffffdu)};
}

// The run of N row values from both starts. False (and no move) when it leaves the binade or
// meets a NaN.
template <int N> __device__ __forceinline__ bool run32(const float (&v)[N], unsigned code, Run32 *out) {
    const Start32 st = start32(code);
    const unsigned flip = (code >> 8) << 31;
    float a = st.even, b = st.odd, lo = a, hi = a;
    unsigned down = 0;  // sign bit: some row moves the magnitude down
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const unsigned bits = __float_as_uint(v[i]) ^ flip;
        down |= bits;
        a = __fadd_rn(a, __uint_as_float(bits));
        b = __fadd_rn(b, __uint_as_float(bits));
        lo = fminf(lo, a);
        hi = fmaxf(hi, a);
    }
    const int base = __float_as_int(st.even);
    const bool ok = lo >= st.lo && hi <= st.hi && a >= st.lo && b >= st.lo;
    // Offsets of the odd run differ from the even run's by at most one.
    *out = ok ? Run32{__float_as_int(a) - base, __float_as_int(b) - base - 1,
                      (down >> 31) ? __float_as_int(lo) - base - 1 : NO_FALL32, __float_as_int(hi) - base + 1}
              : STILL32;
    return ok;
}

// Applies f to state s, known to be of f's binade: false when a state on the way could leave it. Rows
// that move the magnitude down keep every state above 2^E by an ulp, so that no exact sum falls into the
// finer grid below.
__device__ __forceinline__ bool apply32(float s, Run32 f, float *out) {
    const int bits = __float_as_int(s), S = (bits & 0x7fffff) | 0x800000;
    if (S + f.mx >= C32_TOP || S + f.mn <= C32_TOP / 2) return false;
    *out = __int_as_float(bits + ((S & 1) ? f.d1 : f.d0));
    return true;
}

// The reducer's state on the device.
struct State32 {
    float lanes[16];
    float tail[16];
    float result;
    float pad;
};

struct Work32 {
    float *apx;        // [16][T] approximate lane sums
    unsigned *code;    // [16][T] binade of each tile's function (C2: the estimate, C3: NONE if it has none)
    Run32 *run;        // [16][T]
    unsigned *ccode;   // [16][C] chunks
    Run32 *crun;       // [16][C]
};

// The thread's run of a tile: blocks C32_RUN * (t >> 2) .. of lanes 4 (t & 3) .. + 3. Rows past the
// last whole block read as +0.0, which moves no state.
template <int OP, bool ALIGNED, bool LAST>
__device__ __forceinline__ void load32(const Args32 &a, int64_t nb, int tile, float (&v)[4][C32_RUN]) {
    const int64_t b0 = static_cast<int64_t>(tile) * C32_BLOCKS + (threadIdx.x >> 2) * C32_RUN;
    const int q = (threadIdx.x & 3) * 4;
    float4 x[C32_RUN], y[C32_RUN];
    auto get = [&](const float *p) {
        if (ALIGNED) return LAST ? __ldcs(reinterpret_cast<const float4 *>(p)) : __ldg(reinterpret_cast<const float4 *>(p));
        return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
    };
#pragma unroll
    for (int i = 0; i < C32_RUN; ++i) {
        x[i] = y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (b0 + i < nb) {
            x[i] = get(a.x + (b0 + i) * 16 + q);
            if (OP == R32_DOT) y[i] = get(a.y + (b0 + i) * 16 + q);
        }
    }
#pragma unroll
    for (int i = 0; i < C32_RUN; ++i) {
        const bool in = b0 + i < nb;
        v[0][i] = in ? value32<OP>(a, x[i].x, y[i].x) : 0.f;
        v[1][i] = in ? value32<OP>(a, x[i].y, y[i].y) : 0.f;
        v[2][i] = in ? value32<OP>(a, x[i].z, y[i].z) : 0.f;
        v[3][i] = in ? value32<OP>(a, x[i].w, y[i].w) : 0.f;
    }
}

// C1. Bound by the read.
template <int OP, bool ALIGNED>
__global__ void __launch_bounds__(C32_THREADS) c32_sums(Args32 a, int64_t nb, int T, Work32 wk) {
    chain_enter();
    __shared__ float part[C32_THREADS / 32][16];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float v[4][C32_RUN];
    load32<OP, ALIGNED, false>(a, nb, blockIdx.x, v);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < C32_RUN; ++i) s += v[h][i];
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) s += __shfl_xor_sync(FULL, s, o);
        if (lane < 4) part[w][lane * 4 + h] = s;
    }
    __syncthreads();
    if (threadIdx.x < 16) {
        float s = 0.f;
        for (int i = 0; i < C32_THREADS / 32; ++i) s += part[i][threadIdx.x];
        wk.apx[static_cast<int64_t>(threadIdx.x) * T + blockIdx.x] = s;
    }
}

// C2: one block per lane; a thread takes a run of consecutive tiles.
__global__ void __launch_bounds__(1024) c32_binades(int T, Work32 wk, const State32 *state) {
    chain_enter();
    __shared__ double warp_tot[32];
    const int L = blockIdx.x, t = threadIdx.x, lane = t & 31, w = t >> 5;
    const float *apx = wk.apx + static_cast<int64_t>(L) * T;
    unsigned *code = wk.code + static_cast<int64_t>(L) * T;
    const int per = (T + 1023) / 1024, k0 = min(T, t * per), k1 = min(T, k0 + per);
    double mine = 0.0;
    for (int k = k0; k < k1; ++k) mine += static_cast<double>(apx[k]);
    double inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_tot[w] = inc;
    __syncthreads();
    double run = static_cast<double>(state->lanes[L]) + inc - mine;
    for (int i = 0; i < w; ++i) run += warp_tot[i];
    for (int k = k0; k < k1; ++k) {
        code[k] = code32(static_cast<float>(run));
        run += static_cast<double>(apx[k]);
    }
}

// C3: a tile's functions. The eight threads of a warp that hold the same lanes compose theirs by
// shuffles (eight runs in row order, the low threads first), then the eight warps' through shared
// memory. Runs that only move up and meet no tie (d0 == d1) compose by adding.
template <int OP, bool ALIGNED>
__global__ void __launch_bounds__(C32_THREADS) c32_runs(Args32 a, int64_t nb, int T, Work32 wk) {
    chain_enter();
    __shared__ Run32 part[C32_THREADS / 32][16];
    __shared__ unsigned bad[C32_THREADS / 32];
    __shared__ unsigned s_code[16];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, tile = blockIdx.x;
    if (threadIdx.x < 16) s_code[threadIdx.x] = wk.code[static_cast<int64_t>(threadIdx.x) * T + tile];
    float v[4][C32_RUN];
    load32<OP, ALIGNED, true>(a, nb, tile, v);
    __syncthreads();
    Run32 f[4];
    unsigned fails = 0;  // bit h: lane 4 (t & 3) + h has no function here
    bool simple = true;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        const unsigned code = s_code[(lane & 3) * 4 + h];
        f[h] = STILL32;
        if (code == C32_NONE || !run32<C32_RUN>(v[h], code, &f[h])) fails |= 1u << h;
        simple = simple && f[h].d0 == f[h].d1 && f[h].mn == NO_FALL32 && f[h].mx == f[h].d0 + 1;
    }
    if (__all_sync(FULL, simple)) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            int d = f[h].d0;
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) d += __shfl_xor_sync(FULL, d, o);
            f[h] = Run32{d, d, NO_FALL32, d + 1};
        }
    } else {
#pragma unroll
        for (int h = 0; h < 4; ++h)
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                const Run32 g = shfl_down32(f[h], o);
                if (lane + o < 32) f[h] = then32(f[h], g);  // threads 0..3 end with all eight, in order
            }
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) fails |= __shfl_xor_sync(FULL, fails, o);
    if (lane < 4) {
#pragma unroll
        for (int h = 0; h < 4; ++h) part[w][lane * 4 + h] = f[h];
    }
    const unsigned all = (__shfl_sync(FULL, fails, 0) & 15u) | ((__shfl_sync(FULL, fails, 1) & 15u) << 4) |
                         ((__shfl_sync(FULL, fails, 2) & 15u) << 8) | ((__shfl_sync(FULL, fails, 3) & 15u) << 12);
    if (lane == 0) bad[w] = all;
    __syncthreads();
    if (threadIdx.x < 16) {
        const int L = threadIdx.x;
        Run32 r = part[0][L];
        unsigned no = bad[0];
        for (int i = 1; i < C32_THREADS / 32; ++i) {
            r = then32(r, part[i][L]);
            no |= bad[i];
        }
        // Sums of 64 runs of fewer than 2^23 ulps each stay below 2^30; what moves further than a
        // binade never applies.
        const bool ok = !((no >> L) & 1u) && r.mx < C32_TOP && r.mn > -C32_TOP;
        const int64_t at = static_cast<int64_t>(L) * T + tile;
        if (!ok) wk.code[at] = C32_NONE;
        wk.run[at] = r;
    }
}

// C4: one warp per lane and chunk.
__global__ void __launch_bounds__(256) c32_chunks(int T, int C, Work32 wk) {
    chain_enter();
    const int lane = threadIdx.x & 31;
    const int64_t g = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (g >= static_cast<int64_t>(16) * C) return;
    const int L = static_cast<int>(g / C), k = static_cast<int>(g % C), tile = k * C32_CHUNK + lane;
    const int64_t at = static_cast<int64_t>(L) * T + tile;
    const unsigned first = wk.code[static_cast<int64_t>(L) * T + k * C32_CHUNK];
    Run32 f = STILL32;
    bool ok = first != C32_NONE;
    if (tile < T) {
        ok = ok && wk.code[at] == first;
        if (ok) f = wk.run[at];
    }
    ok = __all_sync(FULL, ok);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Run32 h = shfl_down32(f, o);
        if (lane + o < 32) f = then32(f, h);
    }
    if (lane == 0) {
        const int64_t c = static_cast<int64_t>(L) * C + k;
        wk.ccode[c] = ok && f.mx < C32_TOP && f.mn > -C32_TOP ? first : C32_NONE;
        wk.crun[c] = f;
    }
}

// Ordered inclusive composition over the warp, then the number of leading threads whose prefix
// applies to s (all of the state's binade); *s becomes the state after them.
__device__ __forceinline__ int advance32(Run32 f, bool usable, float *s) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Run32 g = shfl_up32(f, o);
        if (lane >= o) f = then32(g, f);
    }
    float r = *s;
    const bool ok = usable && apply32(*s, f, &r);
    const unsigned no = __ballot_sync(FULL, !ok);
    const int m = no ? __ffs(no) - 1 : 32;
    if (m > 0) *s = __shfl_sync(FULL, r, m - 1);
    return m;
}

// C5's shared copies: the lane's chunk functions, the tile functions of chunks without one, and the
// rows of the tiles that are likely to be resolved (no function, or the last before another binade).
constexpr int W32_CHUNKS = 1024, W32_MIXED = 32, W32_TILES = 24;
struct Walk32 {
    Run32 crun[W32_CHUNKS];
    Run32 run[W32_MIXED][C32_CHUNK];
    float rows[W32_TILES][C32_BLOCKS];
    unsigned ccode[W32_CHUNKS];
    unsigned code[W32_MIXED][C32_CHUNK];
    short mixed_of[W32_CHUNKS];
    int chunk_of[W32_MIXED];
    int tile_of[W32_TILES];
    short rows_of[W32_MIXED][C32_CHUNK];
    alignas(16) float chain[C32_BLOCKS];
    int nmixed, ntiles;
};

constexpr int R32_ROWS = C32_BLOCKS / 32;  // rows per thread of a resolved tile

template <int OP> __device__ __forceinline__ float row_of(const Args32 &a, int64_t nb, int64_t b, int L) {
    if (b >= nb) return 0.f;
    return value32<OP>(a, __ldg(a.x + b * 16 + L), OP == R32_DOT ? __ldg(a.y + b * 16 + L) : 0.f);
}

// The rows of threads `first` on (sixteen each, of the whole warp in v) added one after another.
__device__ __forceinline__ float chain_rows(float (&buf)[C32_BLOCKS], const float (&v)[R32_ROWS], int first, float s) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < R32_ROWS; i += 4)
        *reinterpret_cast<float4 *>(&buf[(threadIdx.x & 31) * R32_ROWS + i]) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    __syncwarp();
    for (int r = first * R32_ROWS; r < C32_BLOCKS; r += R32_ROWS) {
        float4 x[R32_ROWS / 4];
#pragma unroll
        for (int i = 0; i < R32_ROWS / 4; ++i) x[i] = *reinterpret_cast<const float4 *>(&buf[r + 4 * i]);
#pragma unroll
        for (int i = 0; i < R32_ROWS / 4; ++i)
            s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, x[i].x), x[i].y), x[i].z), x[i].w);
    }
    return s;
}

// A thread whose rows no run carries costs a failed run, a composition and its sixteen adds, some 800
// cycles, where a chain adds the sixteen rows in 70. So after this many of them the rest of the tile is a
// chain, and sooner in the tiles after one that was. (Lanes whose rows leave their binade all the time took
// 26,000 cycles a tile: reduce_add_f32 of 2^20 rows that alternate between about -1e6 and 1e6 1690 us a call, now
// 377, one block of sixteen chains 920; of 2^17 such rows 290 / 86 / 149.)
constexpr int W32_FAILS = 2;

template <int OP>
__global__ void __launch_bounds__(256) c32_walk(Args32 a, int64_t nb, int T, int C, Work32 wk, State32 *state) {
    chain_enter();
    extern __shared__ __align__(16) unsigned char walk32_smem[];
    Walk32 &sm = *reinterpret_cast<Walk32 *>(walk32_smem);
    const int L = blockIdx.x, t = threadIdx.x;
    const unsigned *gcode = wk.code + static_cast<int64_t>(L) * T;
    const Run32 *grun = wk.run + static_cast<int64_t>(L) * T;
    const unsigned *gccode = wk.ccode + static_cast<int64_t>(L) * C;
    const Run32 *gcrun = wk.crun + static_cast<int64_t>(L) * C;
    if (t == 0) sm.nmixed = sm.ntiles = 0;
    __syncthreads();
    for (int c = t; c < min(C, W32_CHUNKS); c += 256) {
        const unsigned k = gccode[c];
        sm.ccode[c] = k;
        sm.crun[c] = gcrun[c];
        short slot = -1;
        // Without a function, or followed by a chunk of another binade: the sum may cross in its last tiles.
        if (k == C32_NONE || (c + 1 < C && gccode[c + 1] != k)) {
            const int m = atomicAdd(&sm.nmixed, 1);
            if (m < W32_MIXED) {
                slot = static_cast<short>(m);
                sm.chunk_of[m] = c;
            }
        }
        sm.mixed_of[c] = slot;
    }
    __syncthreads();
    for (int i = t; i < min(sm.nmixed, W32_MIXED) * C32_CHUNK; i += 256) {
        const int m = i / C32_CHUNK, j = i % C32_CHUNK, tile = sm.chunk_of[m] * C32_CHUNK + j;
        const unsigned k = tile < T ? gcode[tile] : C32_NONE;
        sm.code[m][j] = k;
        if (tile < T) sm.run[m][j] = grun[tile];
        short slot = -1;
        if (tile < T && (k == C32_NONE || (tile + 1 < T && gcode[tile + 1] != k))) {
            const int q = atomicAdd(&sm.ntiles, 1);
            if (q < W32_TILES) {
                slot = static_cast<short>(q);
                sm.tile_of[q] = tile;
            }
        }
        sm.rows_of[m][j] = slot;
    }
    __syncthreads();
    for (int i = t; i < min(sm.ntiles, W32_TILES) * C32_BLOCKS; i += 256) {
        const int q = i / C32_BLOCKS, r = i % C32_BLOCKS;
        // Row r of thread r / R32_ROWS, stored row-major over the threads (no bank conflicts).
        sm.rows[q][(r % R32_ROWS) * 32 + r / R32_ROWS] =
            row_of<OP>(a, nb, static_cast<int64_t>(sm.tile_of[q]) * C32_BLOCKS + r, L);
    }
    __syncthreads();
    if (t >= 32) return;

    const int lane = t;
    float s = state->lanes[L];
    int ahead = -1;  // the tile whose rows `next` holds
    float next[R32_ROWS];
    int tile = 0, chained = 0;  // chained: resolved tiles in a row that ended as chains
    while (tile < T && s == s) {  // a NaN stays one
        const unsigned code = code32(s);
        int c = tile / C32_CHUNK;
        if (code != C32_NONE && tile % C32_CHUNK == 0) {
            const int k = c + lane;
            unsigned kc = C32_NONE;
            Run32 f = STILL32;
            if (k < C) {
                kc = k < W32_CHUNKS ? sm.ccode[k] : gccode[k];
                if (kc == code) f = k < W32_CHUNKS ? sm.crun[k] : gcrun[k];
            }
            const int m = __shfl_sync(FULL, kc == code, 0) ? advance32(f, kc == code, &s) : 0;
            if (m > 0) {
                chained = 0;
                c += m;
                tile = c * C32_CHUNK;
                if (m == 32 || tile >= T) continue;  // else the chunk that ended the run, tile by tile
            }
        }
        const int slot = c < W32_CHUNKS ? sm.mixed_of[c] : -1;
        int j0 = tile % C32_CHUNK;
        if (code != C32_NONE) {
            const int j = j0 + lane, k = tile + lane;
            unsigned kc = C32_NONE;
            Run32 f = STILL32;
            if (j < C32_CHUNK && k < T) {
                kc = slot >= 0 ? sm.code[slot][j] : gcode[k];
                if (kc == code) f = slot >= 0 ? sm.run[slot][j] : grun[k];
            }
            const int m = __shfl_sync(FULL, kc == code, 0) ? advance32(f, kc == code, &s) : 0;
            if (m > 0) {
                chained = 0;
                tile += m;
                j0 += m;
                if (j0 >= C32_CHUNK || tile >= T) continue;  // else the tile that ended the run
            }
        }
        // The tile's rows, sixteen a thread.
        float v[R32_ROWS];
        const int held = slot >= 0 ? sm.rows_of[slot][j0] : -1;
        const int64_t b0 = static_cast<int64_t>(tile) * C32_BLOCKS + lane * R32_ROWS;
        if (held >= 0) {
#pragma unroll
            for (int i = 0; i < R32_ROWS; ++i) v[i] = sm.rows[held][i * 32 + lane];
        } else {
#pragma unroll
            for (int i = 0; i < R32_ROWS; ++i) v[i] = ahead == tile ? next[i] : row_of<OP>(a, nb, b0 + i, L);
            ahead = tile + 1;  // resolved tiles come in runs: the next one's rows are on their way
            if (ahead < T) {
#pragma unroll
                for (int i = 0; i < R32_ROWS; ++i) next[i] = row_of<OP>(a, nb, b0 + C32_BLOCKS + i, L);
            }
        }
        if (isinf(s)) {  // stays so, unless it meets the other infinity or a NaN
            bool ends = false;
#pragma unroll
            for (int i = 0; i < R32_ROWS; ++i) ends = ends || v[i] != v[i] || v[i] == -s;
            if (__any_sync(FULL, ends)) s = __int_as_float(0x7fc00000);
            ++tile;
            continue;
        }
        unsigned live = 0;  // threads with a row that is not a zero: the others move no state
        {
            unsigned any = 0;
#pragma unroll
            for (int i = 0; i < R32_ROWS; ++i) any |= __float_as_uint(v[i]) << 1;
            live = __ballot_sync(FULL, any != 0);
        }
        int fails = W32_FAILS - chained;
        for (int done = 0; done < 32;) {
            const unsigned now = code32(s), rest = live & (FULL << done);
            if (rest == 0) break;
            done = __ffs(rest) - 1;
            if (fails <= 0) {
                s = chain_rows(sm.chain, v, done, s);
                break;
            }
            if (now != C32_NONE) {
                Run32 f = STILL32;
                const bool ok = lane < done || run32<R32_ROWS>(v, now, &f);
                const int m = advance32(f, ok, &s);
                if (m > done) {
                    done = m;
                    continue;
                }
            }
            float r = s;
            if (lane == done) {
#pragma unroll
                for (int i = 0; i < R32_ROWS; ++i) r = __fadd_rn(r, v[i]);
            }
            s = __shfl_sync(FULL, r, done);
            ++done;
            --fails;
        }
        chained = fails <= 0 ? min(chained + 1, W32_FAILS) : 0;
        ++tile;
    }
    if (lane == 0) state->lanes[L] = s;
}

// Short inputs: the sixteen chains themselves, one block. The other warps stage the row values in
// shared memory, chunk after chunk, while sixteen threads add (4.4 cycles a row of a lane). With
// `result` the same launch combines the lanes and folds the tail in (finish_lanes).
constexpr int S32_BLOCKS = 512;           // 16-row blocks per staged chunk (32 KB)
// Up to 2^16 rows the chains themselves, else the tile passes: the chains take about 0.3 ns a row,
// the passes' five launches about 75 us up to a few million rows.
constexpr int64_t C32_SEQ_BLOCKS = 4096;

template <int OP>
__global__ void __launch_bounds__(512) c32_chain(Args32 a, int nb, int rest, bool fresh, State32 *state, float *result) {
    extern __shared__ __align__(16) float chain32[];
    __shared__ float s_tail[16];
    const int t = threadIdx.x, chunks = (nb + S32_BLOCKS - 1) / S32_BLOCKS;
    auto stage = [&](int k, int first, int step) {
        const int r0 = k * S32_BLOCKS * 16, rows = min(S32_BLOCKS * 16, nb * 16 - r0);
        float *to = chain32 + (k & 1) * (S32_BLOCKS * 16);
#pragma unroll 8
        for (int i = first; i < rows; i += step)
            to[i] = value32<OP>(a, __ldg(a.x + r0 + i), OP == R32_DOT ? __ldg(a.y + r0 + i) : 0.f);
    };
    float s = t < 16 && !fresh ? state->lanes[t] : 0.f;
    if (t < rest)
        s_tail[t] = value32<OP>(a, a.x[static_cast<int64_t>(nb) * 16 + t], OP == R32_DOT ? a.y[static_cast<int64_t>(nb) * 16 + t] : 0.f);
    if (chunks > 0) stage(0, t, 512);
    __syncthreads();
    for (int k = 0; k < chunks; ++k) {
        if (t >= 32) {
            if (k + 1 < chunks) stage(k + 1, t - 32, 480);
        } else if (t < 16) {
            const int blocks = min(S32_BLOCKS, nb - k * S32_BLOCKS);
            const float *b = chain32 + (k & 1) * (S32_BLOCKS * 16) + t;
            int i = 0;
            for (; i + 16 <= blocks; i += 16) {
                float v[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) v[u] = b[(i + u) * 16];
#pragma unroll
                for (int u = 0; u < 16; ++u) s = __fadd_rn(s, v[u]);
            }
            for (; i < blocks; ++i) s = __fadd_rn(s, b[i * 16]);
        }
        __syncthreads();
    }
    if (!result) {
        if (t < 16) state->lanes[t] = s;
        if (t < rest) state->tail[t] = s_tail[t];
        return;
    }
    if (t >= 32) return;
#pragma unroll
    for (int step = 8; step > 0; step >>= 1) {
        const float other = __shfl_down_sync(FULL, s, step);
        if (t < step) s = __fadd_rn(s, other);
    }
    if (t == 0) {
        for (int i = 0; i < rest; ++i) s = __fadd_rn(s, s_tail[i]);
        *result = s;
    }
}

// The rest rows (fewer than 16), kept as row values until finish.
template <int OP> __global__ void c32_tail(Args32 a, int64_t first, int rest, State32 *state) {
    chain_enter();
    const int j = threadIdx.x;
    if (j < rest) state->tail[j] = value32<OP>(a, a.x[first + j], OP == R32_DOT ? a.y[first + j] : 0.f);
}

// reduce.rs:77-91 (finish_lanes).
__global__ void c32_finish(State32 *state, int tail_len, float *host) {
    chain_enter();
    float acc[16];
    for (int j = 0; j < 16; ++j) acc[j] = state->lanes[j];
    for (int step = 8; step > 0; step >>= 1)
        for (int j = 0; j < step; ++j) acc[j] = __fadd_rn(acc[j], acc[j + step]);
    float r = acc[0];
    for (int j = 0; j < tail_len; ++j) r = __fadd_rn(r, state->tail[j]);
    state->result = r;
    if (host) *host = r;
}

size_t layout32(int T, int C, char *b, Work32 *wk) {
    auto up = [](size_t v) { return (v + 255) & ~size_t(255); };
    const size_t t16 = static_cast<size_t>(T) * 16, c16 = static_cast<size_t>(C) * 16;
    const size_t o_run = 0, o_crun = up(t16 * sizeof(Run32)), o_apx = o_crun + up(c16 * sizeof(Run32)),
                 o_code = o_apx + up(t16 * 4), o_ccode = o_code + up(t16 * 4);
    if (b)
        *wk = Work32{reinterpret_cast<float *>(b + o_apx), reinterpret_cast<unsigned *>(b + o_code),
                     reinterpret_cast<Run32 *>(b + o_run), reinterpret_cast<unsigned *>(b + o_ccode),
                     reinterpret_cast<Run32 *>(b + o_crun)};
    return o_ccode + up(c16 * 4);
}

template <int OP>
vkc_status launch_chain32(vkc_ctx *ctx, const Args32 &a, int nb, int rest, bool fresh, State32 *state, float *result) {
    constexpr size_t smem = 2 * S32_BLOCKS * 16 * sizeof(float);
    static std::atomic<unsigned long long> configured{0};
    once_per_device(configured, ctx->device, [] {
        cudaFuncSetAttribute(c32_chain<OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    });
    c32_chain<OP><<<1, 512, smem, ctx->stream>>>(a, nb, rest, fresh, state, result);
    return launched(ctx, "canon32_chain");
}

template <int OP> vkc_status launch_canon32(vkc_ctx *ctx, const Args32 &a, int64_t nb, State32 *state) {
    vkc_status st;
    const int64_t T64 = (nb + C32_BLOCKS - 1) / C32_BLOCKS;
    if (T64 > (int64_t(1) << 26)) return fail(ctx, VKC_USAGE, "array too long for one update");
    const int T = static_cast<int>(T64), C = (T + C32_CHUNK - 1) / C32_CHUNK;
    void *p;
    if ((st = scratch(ctx, layout32(T, C, nullptr, nullptr), &p))) return st;
    Work32 wk;
    layout32(T, C, static_cast<char *>(p), &wk);
    const bool aligned = (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 &&
                         (OP != R32_DOT || (reinterpret_cast<uintptr_t>(a.y) & 15) == 0);
    static std::atomic<unsigned long long> configured{0};
    once_per_device(configured, ctx->device, [] {
        cudaFuncSetAttribute(c32_walk<OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(Walk32)));
    });
    if (aligned) c32_sums<OP, true><<<T, C32_THREADS, 0, ctx->stream>>>(a, nb, T, wk);
    else c32_sums<OP, false><<<T, C32_THREADS, 0, ctx->stream>>>(a, nb, T, wk);
    if ((st = launched(ctx, "canon32_sums"))) return st;
    launch_next(c32_binades, 16, 1024, 0, ctx->stream, T, wk, state);
    if ((st = launched(ctx, "canon32_binades"))) return st;
    if (aligned) launch_next(c32_runs<OP, true>, T, C32_THREADS, 0, ctx->stream, a, nb, T, wk);
    else launch_next(c32_runs<OP, false>, T, C32_THREADS, 0, ctx->stream, a, nb, T, wk);
    if ((st = launched(ctx, "canon32_runs"))) return st;
    launch_next(c32_chunks, static_cast<unsigned>((static_cast<int64_t>(16) * C + 7) / 8), 256, 0, ctx->stream, T, C, wk);
    if ((st = launched(ctx, "canon32_chunks"))) return st;
    launch_next(c32_walk<OP>, 16, 256, sizeof(Walk32), ctx->stream, a, nb, T, C, wk, state);
    return launched(ctx, "canon32_walk");
}

float splat32(const Arg &a) {
    const unsigned b = static_cast<unsigned>(a.s.bits);
    float f;
    memcpy(&f, &b, 4);
    return f;
}

// CanonicalAcc over f32 rows (reduce.rs:253-323).
template <int OP> struct Canon32Reducer : DevReducer {
    int cmp = 0;
    int tail_len = 0;

    vkc_status take(vkc_ctx *ctx, const Arg *args, int nargs, Args32 *out) {
        vkc_status st;
        constexpr int want = OP == R32_DOT ? 2 : (OP == R32_COND ? 3 : 1);
        if (nargs != want) return fail(ctx, VKC_RUNTIME, arity_error(want, nargs));
        if (!rows_arg(ctx, args[0], VKC_F32, &st)) return st;
        Args32 &a = *out;
        a = Args32{args[0].ptr<float>(), nullptr, cmp, 0.f, 0.f};
        if (OP == R32_DOT) {
            if (!rows_arg(ctx, args[1], VKC_F32, &st)) return st;
            if (args[0].len() != args[1].len())
                return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(args[0].len()) + " vs " +
                                                  std::to_string(args[1].len()));
            a.y = args[1].ptr<float>();
        } else if (OP == R32_COND) {
            if (!splat_arg(ctx, args[1], VKC_F32, &st) || !splat_arg(ctx, args[2], VKC_F32, &st)) return st;
            a.c = splat32(args[1]);
            a.e = splat32(args[2]);
        }
        // reduce.rs:297-303: rows may only follow whole blocks.
        if (tail_len != 0) return fail(ctx, VKC_RUNTIME, "canonical update after a partial block");
        return VKC_OK;
    }
    vkc_status update(vkc_ctx *ctx, const Arg *args, int nargs) override {
        Args32 a;
        vkc_status st = take(ctx, args, nargs, &a);
        if (st) return st;
        const int64_t n = args[0].len(), nb = n / 16;
        const int rest = static_cast<int>(n % 16);
        auto *s = static_cast<State32 *>(state);
        if (n == 0) return VKC_OK;
        if (nb <= C32_SEQ_BLOCKS) {
            st = launch_chain32<OP>(ctx, a, static_cast<int>(nb), rest, fresh, s, nullptr);
        } else {
            if (fresh && (st = zero(ctx))) return st;
            st = launch_canon32<OP>(ctx, a, nb, s);
            if (!st && rest > 0) {
                launch_next(c32_tail<OP>, 1, 16, 0, ctx->stream, a, nb * 16, rest, s);
                st = launched(ctx, "canon32_tail");
            }
        }
        updated(ctx);
        tail_len = rest;
        return st;
    }
    vkc_status read(vkc_ctx *ctx, vkc_scalar *out) {
        unsigned b = 0;
        const vkc_status st = result(ctx, &b, 4, offsetof(State32, result));
        out->type = VKC_F32;
        out->bits = b;
        return st;
    }
    vkc_status once(vkc_ctx *ctx, const Arg *args, int nargs, vkc_scalar *out, void *dst, bool *done) override {
        *done = args[0].rows && args[0].len() / 16 <= C32_SEQ_BLOCKS;
        if (!*done) return VKC_OK;
        Args32 a;
        vkc_status st = take(ctx, args, nargs, &a);
        if (st) return st;
        const int64_t n = args[0].len();
        auto *s = static_cast<State32 *>(state);
        if (!dst && !(dst = slot(ctx))) dst = &s->result;
        auto *to = static_cast<float *>(dst);
        st = launch_chain32<OP>(ctx, a, static_cast<int>(n / 16), static_cast<int>(n % 16), fresh, s, to);
        updated(ctx);
        return st || !out ? st : read(ctx, out);
    }
    vkc_status combine(vkc_ctx *ctx) {
        vkc_status st;
        if (fresh && (st = zero(ctx))) return st;
        launch_next(c32_finish, 1, 1, 0, ctx->stream, static_cast<State32 *>(state), tail_len, static_cast<float *>(slot(ctx)));
        updated(ctx);
        return launched(ctx, "canon32_finish");
    }
    vkc_status finish(vkc_ctx *ctx, vkc_scalar *out) override {
        const vkc_status st = combine(ctx);
        return st ? st : read(ctx, out);
    }
    vkc_status finish_into(vkc_ctx *ctx, void *dst) override {
        const vkc_status st = combine(ctx);
        return st ? st : copy_out(ctx, dst, 4, offsetof(State32, result));
    }
};

template <int OP> ReducerImpl *make32(vkc_ctx *ctx, int cmp) {
    auto *r = new Canon32Reducer<OP>;
    if (r->alloc(ctx, sizeof(State32))) {
        delete r;
        return nullptr;
    }
    r->cmp = cmp;
    return r;
}

}  // namespace

ReducerImpl *make_canon32_sum(vkc_ctx *ctx) { return make32<R32_SUM>(ctx, 0); }
ReducerImpl *make_canon32_dot(vkc_ctx *ctx) { return make32<R32_DOT>(ctx, 0); }
ReducerImpl *make_canon32_sumsq(vkc_ctx *ctx) { return make32<R32_SUMSQ>(ctx, 0); }
ReducerImpl *make_canon32_cond(vkc_ctx *ctx, int cmp) { return make32<R32_COND>(ctx, cmp); }

}  // namespace vkc
