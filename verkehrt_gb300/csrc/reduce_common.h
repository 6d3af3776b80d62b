// Reducer plumbing shared by k_reduce.cu and k_canon.cu.
#pragma once

#include <cstring>

#include "kcommon.cuh"
#include "registry.h"

namespace vkc {

// Up to four 8-byte words that a fill repeats over a reducer's state.
struct Words4 {
    unsigned long long w[4];
};

// Word i of the state gets w.w[i < 4 ? i : 3].
static __global__ void reducer_fill_kernel(unsigned long long *p, int n, Words4 w) {
    const int i = threadIdx.x;
    if (i < n) p[i] = w.w[i < 4 ? i : 3];
}

// A reducer whose running state is a small device buffer owned by the reducer, uninitialised until
// the first update (`fresh`: its kernels then read no state, which saves a launch to clear it) or begin.
// The kernel that ends an update also writes the state's result words to a pinned slot, so that
// finish only waits for the stream: a call of a few rows costs one launch and one wait (a cleared
// state, a device-to-host copy and the pool's allocation and release around it made count_gt_f64 of
// 4096 rows take 31 us a call, now 20). Without a slot finish copies: where the result goes to a device
// address, where all slots are taken, and once an update was captured, whose replays write no slot.
struct DevReducer : ReducerImpl {
    void *state = nullptr;
    size_t bytes = 0;
    DeviceMem mem;  // gives `state` back on the context's stream, even after the context closed
    void *host = nullptr;  // the slot, from the first update that writes one
    bool copies = false;   // no update writes the slot from here on
    bool captured = false, lasts = false;  // made in a capture; used by later calls too (begin)
    bool fresh = true;
    cudaStream_t used = nullptr;  // the stream of the updates since the last result was read
    // The slot of a reducer dropped without finish may still be written: by the stream `used`.
    ~DevReducer() override {
        if (host) mem.box->give_slot(host, used);
    }
    // Where an update that is about to be launched writes its result, or nullptr.
    void *slot(vkc_ctx *ctx) {
        if (copies) return nullptr;
        copies = lasts ? stream_capturing(ctx->stream) : captured;
        if (!copies && !host) {
            host = mem.box->take_slot(ctx->stream);
            copies = !host;
        }
        return copies ? nullptr : host;
    }
    // After an update's launch.
    void updated(vkc_ctx *ctx) {
        fresh = false;
        used = ctx->stream;
    }
    vkc_status alloc(vkc_ctx *ctx, size_t n) {
        bytes = n;
        const vkc_status st = state_block(ctx, n, &mem, &captured);
        state = mem.ptr;
        return st;
    }
    vkc_status begin(vkc_ctx *ctx) override {
        lasts = true;
        fresh = false;
        return clear(ctx);
    }
    // The state of no rows.
    virtual vkc_status clear(vkc_ctx *ctx) { return zero(ctx); }
    void into_device() override { copies = true; }
    // The state's n bytes zeroed (before a first update whose kernels read it).
    vkc_status zero(vkc_ctx *ctx) {
        VKC_CUDA(ctx, cudaMemsetAsync(state, 0, bytes, ctx->stream));
        return VKC_OK;
    }
    // The state's first n words set on the device (a launch, so it can be captured): word i
    // gets w_i for i < 3, the rest w3.
    vkc_status fill(vkc_ctx *ctx, int n, unsigned long long w0, unsigned long long w1 = 0,
                    unsigned long long w2 = 0, unsigned long long w3 = 0) {
        reducer_fill_kernel<<<1, 64, 0, ctx->stream>>>(static_cast<unsigned long long *>(state), n,
                                                       Words4{{w0, w1, w2, w3}});
        return launched(ctx, "reducer_fill");
    }
    // What the updates left in the slot, once the stream is done; or the state's n bytes from byte `at`,
    // where those words lie in it.
    vkc_status result(vkc_ctx *ctx, void *h, size_t n, size_t at = 0) {
        if (copies || !host) return download(ctx, h, n, at);
        VKC_CUDA(ctx, cudaStreamSynchronize(used));
        used = nullptr;
        memcpy(h, host, n);
        return VKC_OK;
    }
    // n bytes of the state from byte `at` to the device address dst, on the context's stream.
    vkc_status copy_out(vkc_ctx *ctx, void *dst, size_t n, size_t at = 0) {
        VKC_CUDA(ctx, cudaMemcpyAsync(dst, static_cast<const char *>(state) + at, n,
                                      cudaMemcpyDeviceToDevice, ctx->stream));
        return VKC_OK;
    }
    vkc_status download(vkc_ctx *ctx, void *h, size_t n, size_t at = 0) {
        void *p;
        vkc_status st = pinned(ctx, n, &p);
        if (st) return st;
        VKC_CUDA(ctx, cudaMemcpyAsync(p, static_cast<char *>(state) + at, n,
                                      cudaMemcpyDeviceToHost, ctx->stream));
        VKC_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        memcpy(h, p, n);
        return VKC_OK;
    }
};

CmpRange cmp_range(int cmp, double c);
void register_canon(std::vector<KernelDef> &t);

}  // namespace vkc
