// Scans: scan_add_i64 and scan_by_add_i64 (src/kernels/scalar/scan.rs:284-326) as passes of
// fold_scan.cuh, plus prev_i64 (scan.rs:16-48) and the allocation-free scan.
#include <mutex>

#include "fold_scan.cuh"

namespace vkc {

// ------------------------------------------------------------------ prev

__global__ void prev_kernel(const unsigned long long *__restrict__ x, unsigned long long *__restrict__ out,
                            int64_t n, unsigned long long fill, const ScanState *state) {
    int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        out[i] = i == 0 ? (state->seen ? state->last : fill) : __ldcs(x + i - 1);
}

__global__ void prev_carry(const unsigned long long *x, int64_t n, ScanState *state) {
    state->last = x[n - 1];
    state->seen = 1;
}

// scan.rs:16-48 (Prev): row 0 is the fill on the first update, else the previous update's
// last row.
struct PrevImpl : ScannerImpl {
    ScanState *state = nullptr;
    DeviceMem mem;  // owns `state`
    vkc_status update(vkc_ctx *ctx, const Arg *args, int nargs, vkc_array *out) override {
        vkc_status st;
        if (nargs != 2) return fail(ctx, VKC_RUNTIME, arity_error(2, nargs));
        if (!rows_arg(ctx, args[0], VKC_I64, &st) || !splat_arg(ctx, args[1], VKC_I64, &st)) return st;
        int64_t n = args[0].len();
        if (out->len != n)
            return fail(ctx, VKC_RUNTIME, "length mismatch: " + std::to_string(n) +
                                              " rows for a destination of " + std::to_string(out->len) +
                                              " rows");
        if (n == 0) return VKC_OK;
        const auto *x = args[0].ptr<unsigned long long>();
        int grid = stream_grid(ctx, n, 256, 8, 2048);
        prev_kernel<<<grid, 256, 0, ctx->stream>>>(x, static_cast<unsigned long long *>(out->data()), n,
                                                  args[1].s.bits, state);
        if ((st = launched(ctx, "prev"))) return st;
        prev_carry<<<1, 1, 0, ctx->stream>>>(x, n, state);
        return launched(ctx, "prev_carry");
    }
};

static ScannerImpl *make_prev(vkc_ctx *ctx) {
    auto *s = new PrevImpl;
    bool captured;
    if (state_block(ctx, sizeof(ScanState), &s->mem, &captured)) {
        delete s;
        return nullptr;
    }
    s->state = static_cast<ScanState *>(s->mem.ptr);
    if (cudaMemsetAsync(s->state, 0, sizeof(ScanState), ctx->stream) != cudaSuccess) {
        cudaGetLastError();
        delete s;
        return nullptr;
    }
    return s;
}

void register_scan(std::vector<KernelDef> &t) {
    InSpec ia{IN_ARRAY, VKC_I64};
    // scan.rs:336-352: cost = input + output width (+1 for the starts byte).
    KernelDef d{"scan_add_i64", VKC_SCAN, {ia}, true, VKC_I64, 16};
    d.scan = make_scan<VKC_I64, F_ADD, false, true>;
    t.push_back(d);
    d = KernelDef{"scan_by_add_i64", VKC_SCAN, {ia, InSpec{IN_ARRAY, VKC_BOOL}}, true, VKC_I64, 17};
    d.scan = make_scan<VKC_I64, F_ADD, true, true>;
    t.push_back(d);
    d = KernelDef{"prev_i64", VKC_SCAN, {ia, InSpec{IN_SCALAR, VKC_I64}}, true, VKC_I64, 16};
    d.scan = make_prev;
    t.push_back(d);
}

}  // namespace vkc

// ------------------------------------------------------------------ allocation-free scan_add_i64
//
// vkc_scan_add_i64_noalloc: scan_add_i64 for callers that cannot allocate device memory. An
// embedding host that hands this library only its own buffers (an interpreter's arena or a
// memory pool with a fixed budget), or a serving loop that must not take the allocator's lock
// or latency while it answers a request, cannot use the entries above, which take their
// lookback scratch from a context arena that grows with cudaMallocAsync. This entry needs no
// context and allocates nothing: the lookback records live in the file-scope array below, whose
// address is looked up once per device. Every call shares the array and finds it as the last
// call left it, so each call clears the words that must start at zero (the ticket counters,
// the tile records, the carried state and the status). Calls that overlap on the GPU race on the
// array: issue them on one stream, or wait for one to finish before the next starts.
namespace vkc {

// Header (ticket counters, status, carried state), then one lookback record per tile, REC_STRIDE
// (128) bytes apart. 4 MiB and 512 bytes hold the 32,768 tiles of 2^28 rows.
constexpr int64_t NOALLOC_MAX_ROWS = int64_t(1) << 28;
constexpr int64_t NOALLOC_MAX_TILES = scan_tiles<VKC_I64, F_ADD>(NOALLOC_MAX_ROWS);
constexpr size_t NOALLOC_HEADER = 512;
constexpr size_t NOALLOC_BYTES = NOALLOC_HEADER + NOALLOC_MAX_TILES * REC_STRIDE;

static __device__ __align__(256) unsigned char g_scan_scratch[NOALLOC_BYTES];

constexpr int NOALLOC_MAX_DEVICES = 64;
static std::mutex g_noalloc_mu;
static unsigned char *g_noalloc_ptr[NOALLOC_MAX_DEVICES];
static int g_noalloc_sms[NOALLOC_MAX_DEVICES];

static void noalloc_msg(char *err, size_t err_len, const std::string &msg) {
    if (err && err_len) {
        size_t k = msg.size() < err_len - 1 ? msg.size() : err_len - 1;
        memcpy(err, msg.data(), k);
        err[k] = 0;
    }
}

}  // namespace vkc

extern "C" vkc_status vkc_scan_add_i64_noalloc(int device, const int64_t *in, int64_t *out, int64_t n,
                                               void *stream, char *err, size_t err_len) {
    using namespace vkc;
    noalloc_msg(err, err_len, "");
    if (n < 0 || n > NOALLOC_MAX_ROWS) {
        noalloc_msg(err, err_len, "vkc_scan_add_i64_noalloc: " + std::to_string(n) +
                                      " rows is more than its maximum of 268435456 rows (2^28)");
        return VKC_USAGE;
    }
    if (device < 0 || device >= NOALLOC_MAX_DEVICES) {
        noalloc_msg(err, err_len, "vkc_scan_add_i64_noalloc: device " + std::to_string(device) +
                                      " is out of range");
        return VKC_USAGE;
    }
    if (n == 0) return VKC_OK;
    if (!in || !out) {
        noalloc_msg(err, err_len, "vkc_scan_add_i64_noalloc: `in` and `out` must be device pointers, got NULL");
        return VKC_USAGE;
    }
    // Pointers the GPU cannot address as device memory of `device` (host memory, another
    // device's buffers) would fault the kernel: reject them before anything is launched.
    for (const void *p : {static_cast<const void *>(in), static_cast<const void *>(out)}) {
        cudaPointerAttributes at{};
        cudaError_t pe = cudaPointerGetAttributes(&at, p);
        if (pe != cudaSuccess) cudaGetLastError();
        bool ok = pe == cudaSuccess && (at.type == cudaMemoryTypeManaged ||
                                        (at.type == cudaMemoryTypeDevice && at.device == device));
        if (!ok) {
            noalloc_msg(err, err_len, "vkc_scan_add_i64_noalloc: `in` and `out` must be device or managed "
                                      "memory of device " + std::to_string(device));
            return VKC_USAGE;
        }
    }
    int prev = 0;
    if (cudaGetDevice(&prev) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        noalloc_msg(err, err_len, "vkc_scan_add_i64_noalloc: cannot make device " + std::to_string(device) +
                                      " current");
        return VKC_DEVICE;
    }
    auto done = [&](vkc_status st, const std::string &msg) {
        if (st != VKC_OK) noalloc_msg(err, err_len, msg);
        cudaSetDevice(prev);
        return st;
    };
    unsigned char *base;
    int sms;
    {
        // Set-up, once per device: the device address of the scratch array. On the first call on
        // a device this runs inside that call.
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_ptr[device]) {
            void *p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_scan_scratch);
            if (e != cudaSuccess || !p) {
                cudaGetLastError();
                return done(VKC_DEVICE, std::string("vkc_scan_add_i64_noalloc: cudaGetSymbolAddress failed: ") +
                                            cudaGetErrorString(e));
            }
            int sms = 0;
            e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
            if (e != cudaSuccess || sms < 1) {
                cudaGetLastError();
                return done(VKC_DEVICE, std::string("vkc_scan_add_i64_noalloc: cannot read the SM count: ") +
                                            cudaGetErrorString(e));
            }
            g_noalloc_sms[device] = sms;
            g_noalloc_ptr[device] = static_cast<unsigned char *>(p);
        }
        base = g_noalloc_ptr[device];
        sms = g_noalloc_sms[device];
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int tiles = scan_tiles<VKC_I64, F_ADD>(n);
    unsigned *counters = reinterpret_cast<unsigned *>(base);
    DevStatus *status = reinterpret_cast<DevStatus *>(base + 256);
    ScanState *state = reinterpret_cast<ScanState *>(base + 256 + sizeof(DevStatus));
    auto *recs = reinterpret_cast<ulonglong2 *>(base + NOALLOC_HEADER);
    // The header and the records of this call's tiles start at zero; with clean records one
    // epoch value serves every call.
    cudaError_t e = cudaMemsetAsync(base, 0, NOALLOC_HEADER, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(recs, 0, static_cast<size_t>(tiles) * REC_STRIDE, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return done(VKC_DEVICE, std::string("vkc_scan_add_i64_noalloc: ") + cudaGetErrorString(e));
    }
    launch_scan<VKC_I64, F_ADD, false>(device, sms, s, in, nullptr, out, n, tiles, recs, 1u, true, state, counters, status);
    e = cudaGetLastError();
    if (e != cudaSuccess) return done(VKC_DEVICE, std::string("vkc_scan_add_i64_noalloc: ") + cudaGetErrorString(e));
    // Synchronous, like the other entries: read the status word into host memory.
    DevStatus hs{};
    e = cudaMemcpyAsync(&hs, status, sizeof hs, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return done(VKC_DEVICE, std::string("vkc_scan_add_i64_noalloc: ") + cudaGetErrorString(e));
    }
    if (hs.timeout) return done(VKC_TIMEOUT, "vkc_scan_add_i64_noalloc: a device-side wait gave up");
    return done(VKC_OK, "");
}
