// Large copies between pageable host arrays and the device.
//
// cudaMemcpy from or to pageable memory goes through one driver thread and, into a fresh array, that thread's
// page faults: 2.5-4 GB/s here for results of 20-100 MB, several times the kernels that make them.  These
// copies are cut into slots of pinned memory that a few threads fill and empty side by side, each thread with
// two slots, so that its copy to the device or back overlaps its memcpy; the copies themselves are issued on the
// context's stream.  Arrays below kHostioMin, and pinned arrays, take one plain copy.
#include <string.h>

#include <thread>

#include "common.cuh"
#include "kernels.cuh"

static constexpr size_t kSlot = (size_t)1 << 20;
static constexpr size_t kHostioMin = (size_t)2 << 20;
static constexpr int kMaxThreads = 8;

struct exm_hostio {
    char *p = nullptr;   // 2 kMaxThreads slots of pinned memory
    cudaEvent_t ev[2 * kMaxThreads] = {};
};

void exm_hostio_release(exm_ctx *ctx)
{
    exm_hostio *h = ctx->hostio;
    if (!h) return;
    for (cudaEvent_t e : h->ev)
        if (e) {
            cudaEventSynchronize(e);   // a copy from its slot may still be in flight
            cudaEventDestroy(e);
        }
    if (h->p) cudaFreeHost(h->p);
    delete h;
    ctx->hostio = nullptr;
}

static exm_hostio *hostio(exm_ctx *ctx)
{
    if (!ctx->hostio) {
        exm_hostio *h = new exm_hostio();
        ctx->hostio = h;
        cudaError_t e = cudaMallocHost((void **)&h->p, 2 * kMaxThreads * kSlot);
        for (cudaEvent_t &v : h->ev)
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            exm_hostio_release(ctx);
        }
    }
    return ctx->hostio;   // null: no pinned memory to be had, plain copies
}

static bool pageable(const void *p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return true;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

// one thread's share of a copy: slots 2 t and 2 t + 1, pieces t, t + n, t + 2 n, ...
static cudaError_t share(exm_ctx *ctx, exm_hostio *h, char *host, char *dev, size_t bytes, bool to_device, int t, int n)
{
    cudaError_t e = cudaSetDevice(ctx->dev);
    const size_t pieces = (bytes + kSlot - 1) / kSlot;
    auto len = [&](size_t c) { return std::min(kSlot, bytes - c * kSlot); };
    auto slot = [&](int k) { return h->p + (size_t)(2 * t + k) * kSlot; };
    auto fetch = [&](size_t c, int k) {
        if (e == cudaSuccess) e = cudaEventSynchronize(h->ev[2 * t + k]);   // the slot's last copy
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(slot(k), dev + c * kSlot, len(c), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaEventRecord(h->ev[2 * t + k], ctx->stream);
    };
    int k = 0;
    if (!to_device && (size_t)t < pieces) fetch(t, 0);
    for (size_t c = t; c < pieces && e == cudaSuccess; c += n, k ^= 1) {
        if (to_device) {
            e = cudaEventSynchronize(h->ev[2 * t + k]);
            if (e != cudaSuccess) break;
            memcpy(slot(k), host + c * kSlot, len(c));
            e = cudaMemcpyAsync(dev + c * kSlot, slot(k), len(c), cudaMemcpyHostToDevice, ctx->stream);
            if (e == cudaSuccess) e = cudaEventRecord(h->ev[2 * t + k], ctx->stream);
        } else {
            if (c + n < pieces) fetch(c + n, k ^ 1);
            if (e == cudaSuccess) e = cudaEventSynchronize(h->ev[2 * t + k]);
            if (e == cudaSuccess) memcpy(host + c * kSlot, slot(k), len(c));
        }
    }
    return e;
}

static void copy(exm_ctx *ctx, char *host, char *dev, size_t bytes, bool to_device)
{
    exm_hostio *h = (bytes >= kHostioMin && pageable(host)) ? hostio(ctx) : nullptr;
    if (!h) {
        if (to_device)
            EXM_CUDA(cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, ctx->stream));
        else
            EXM_CUDA(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, ctx->stream));
        return;
    }
    const size_t pieces = (bytes + kSlot - 1) / kSlot;
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
    const int n = (int)std::min<size_t>(std::min<size_t>(kMaxThreads, cores), pieces);
    cudaError_t res[kMaxThreads];
    std::thread th[kMaxThreads];
    bool started[kMaxThreads] = {};
    for (int t = 1; t < n; ++t) {
        try {
            th[t] = std::thread([=, &res]() { res[t] = share(ctx, h, host, dev, bytes, to_device, t, n); });
            started[t] = true;
        } catch (const std::exception &) {   // no thread to be had: this one takes the share as well
        }
    }
    res[0] = share(ctx, h, host, dev, bytes, to_device, 0, n);
    for (int t = 1; t < n; ++t) {
        if (started[t])
            th[t].join();
        else
            res[t] = share(ctx, h, host, dev, bytes, to_device, t, n);
    }
    for (int t = 0; t < n; ++t) EXM_CUDA(res[t]);
}

// device -> host on the context's stream; the host array holds the data when the stream is synchronised
void exm_copy_out(exm_ctx *ctx, void *host, const void *dev, size_t bytes) { copy(ctx, (char *)host, (char *)dev, bytes, false); }

// host -> device on the context's stream; the host array is free again when the stream is synchronised
void exm_copy_in(exm_ctx *ctx, void *dev, const void *host, size_t bytes) { copy(ctx, (char *)host, (char *)dev, bytes, true); }
