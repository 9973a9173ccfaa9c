// Scratch of the layouts that are built on the device once per graph.
#pragma once
#include "gs_internal.cuh"

#include <algorithm>
#include <vector>

namespace {

inline uint32_t grid_for(uint64_t n, const gs_ctx* ctx) {
    const uint64_t b = (n + 255) / 256;
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(b, gs_grid_size(ctx, 16)));
}

inline int bits_for(uint64_t n) {   // bits that hold 0 .. n - 1, at least 1
    int b = 1;
    while ((1ull << b) < n) ++b;
    return b;
}

// Device buffers of a build: carved from one block (a cudaMalloc and a
// cudaFree per buffer took 10 of 18 ms at 24 M entries), freed together when
// the build ends; a buffer that no longer fits gets a block of its own.
struct Temps {
    gs_ctx* ctx;
    std::vector<void*> all;
    char* top = nullptr;
    char* end = nullptr;
    explicit Temps(gs_ctx* c) : ctx(c) {}
    ~Temps() {
        cudaStreamSynchronize(ctx->stream);
        for (void* p : all) gs_dev_free(p);
    }
    gs_status reserve(uint64_t bytes) {
        GS_TRY(gs_dev_alloc(ctx, (void**)&top, bytes));
        all.push_back(top);
        end = top + bytes;
        return GS_OK;
    }
    // Buffers to come are carved from [p, p + bytes), which holds nothing needed.
    void reuse(void* p, uint64_t bytes) {
        if (bytes <= (uint64_t)(end - top)) return;
        top = (char*)p;
        end = top + (bytes & ~255ull);
    }
    template <class T>
    gs_status get(T** out, uint64_t n) {
        const uint64_t bytes = (std::max<uint64_t>(1, n) * sizeof(T) + 255) & ~255ull;
        if (bytes <= (uint64_t)(end - top)) {
            *out = (T*)top;
            top += bytes;
            return GS_OK;
        }
        GS_TRY(gs_dev_alloc(ctx, (void**)out, bytes));
        all.push_back(*out);
        return GS_OK;
    }
};

// cub call in two steps: size, then work, with scratch from T that the next
// buffer (in stream order) may overwrite.
template <class F>
gs_status cub_run(Temps& T, const char* what, F call) {
    size_t bytes = 0;
    GS_CHECK_CUDA(T.ctx, call(nullptr, bytes));
    char *mark = T.top, *mark_end = T.end, *tmp = nullptr;
    GS_TRY(T.get(&tmp, bytes));
    cudaError_t e = call(tmp, bytes);
    T.ctx->launches++;
    if (e != cudaSuccess) return gs_cuda_fail(T.ctx, e, what);
    if (T.end == mark_end) T.top = mark;
    return GS_OK;
}

template <class T>
gs_status to_host(gs_ctx* ctx, T* dst, const T* src, uint64_t n) {
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(dst, src, n * sizeof(T), cudaMemcpyDeviceToHost, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return GS_OK;
}

}  // namespace
