// The L2-blocked sweep orders of a resident graph (sm_100a), made on the
// device at their first use.
//
// Tiles are grouped into blocks of `block` x `block` windows (row-major inside
// a block), so the vertex state that the tiles in flight touch (2 `block`
// windows) stays in L2.  Runs are short (one tile row, <= kBlockRunUnits units,
// one per warp of a CTA) so the CTAs in flight work inside one or two blocks.
// Used by the sweeps whose per-record state is large (WCC, k-core, batches,
// serving: kBlockWindows; multi-source BFS with 16-byte vertex state may pick
// kBlockWindowsSmall); their results do not depend on the order.
//
// The unit table is sorted by block with a radix sort (stable: file order
// inside a block), and the runs are read off it: a run starts every
// kBlockRunUnits units after the first of a (block, row).  Sorting and cutting
// on the host instead took 30 of the 35 ms of a first WCC or k-core at
// Kronecker 25 (470 K units); this takes under 1 ms.
#include "gs_internal.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>

namespace {

inline uint32_t grid_for(uint64_t n, const gs_ctx* ctx) {
    const uint64_t b = (n + 255) / 256;
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(b, gs_grid_size(ctx, 16)));
}

struct MaxOp {
    __host__ __device__ uint32_t operator()(uint32_t a, uint32_t b) const { return a > b ? a : b; }
};

__global__ void block_key_kernel(const gs_unit* __restrict__ units, uint32_t n, uint32_t block, int col_bits,
                                 uint32_t* __restrict__ key, uint32_t* __restrict__ idx) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += nth) {
        const uint32_t rc = units[u].rc;
        key[u] = (((rc >> 16) / block) << col_bits) | ((rc & 0xFFFFu) / block);
        idx[u] = u;
    }
}

// The units in block order; first[i] = i where a (block, row) starts, else 0.
__global__ void block_units_kernel(const gs_unit* __restrict__ units, const uint32_t* __restrict__ idx,
                                   const uint32_t* __restrict__ key, uint32_t n, gs_unit* __restrict__ out,
                                   uint32_t* __restrict__ first) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth) {
        const gs_unit u = units[idx[i]];
        out[i] = u;
        const bool starts = i > 0 && (key[i] != key[i - 1] || units[idx[i - 1]].rc >> 16 != u.rc >> 16);
        first[i] = starts ? i : 0u;
    }
}

// is_run[i]: a run starts at unit i; is_run[n] = 0.
__global__ void block_flag_kernel(const uint32_t* __restrict__ first, uint32_t n, uint32_t* __restrict__ is_run) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += nth)
        is_run[i] = i < n && (i - first[i]) % kBlockRunUnits == 0;
}

__global__ void block_runs_kernel(const gs_unit* __restrict__ units, const uint32_t* __restrict__ first,
                                  const uint32_t* __restrict__ run, uint32_t n, gs_tile_run* __restrict__ out) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth) {
        if (run[i + 1] == run[i]) continue;   // no run starts here
        uint32_t e = i + 1;
        while (e < n && e < i + kBlockRunUnits && first[e] == first[i]) ++e;
        out[run[i]] = gs_tile_run{units[i].rec_beg, units[e - 1].rec_beg + units[e - 1].n, 0, 0, i, e};
    }
}

gs_status blocked_order(gs_graph* g, uint32_t block, uint64_t* R_out, gs_tile_run** runs_out, gs_unit** units_out) {
    gs_ctx* ctx = g->ctx;
    cudaStream_t q = ctx->stream;
    const uint32_t U = (uint32_t)g->U;
    GS_TRY(gs_graph_alloc(g, (void**)units_out, std::max<uint64_t>(1, U) * sizeof(gs_unit)));
    uint32_t n_runs = 0;
    if (U) {
        int col_bits = 1;
        while ((1u << col_bits) < g->nw / block + 1) ++col_bits;
        size_t sort_b = 0, scan_b = 0, sum_b = 0;
        uint32_t* none = nullptr;
        GS_CHECK_CUDA(ctx, cub::DeviceRadixSort::SortPairs(nullptr, sort_b, none, none, none, none, U, 0, 2 * col_bits, q));
        GS_CHECK_CUDA(ctx, cub::DeviceScan::InclusiveScan(nullptr, scan_b, none, none, MaxOp(), U, q));
        GS_CHECK_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, sum_b, none, none, U + 1, q));
        const size_t cub_b = (std::max({sort_b, scan_b, sum_b}) + 255) & ~(size_t)255;
        const uint64_t u4 = ((uint64_t)U + 64) & ~63ull;   // U + 1 at least
        char* tmp = nullptr;
        const size_t tmp_b = cub_b + u4 * 4 * 6;
        GS_TRY(gs_pool_get(ctx, tmp_b, (void**)&tmp));
        uint32_t *key0 = (uint32_t*)(tmp + cub_b), *key1 = key0 + u4, *idx0 = key1 + u4, *idx1 = idx0 + u4,
                 *first = idx1 + u4, *run = first + u4;
        const uint32_t grid = grid_for(U, ctx);
        block_key_kernel<<<grid, 256, 0, q>>>(g->d_units, U, block, col_bits, key0, idx0);
        cudaError_t e = cub::DeviceRadixSort::SortPairs(tmp, sort_b, key0, key1, idx0, idx1, U, 0, 2 * col_bits, q);
        if (e == cudaSuccess) {
            block_units_kernel<<<grid, 256, 0, q>>>(g->d_units, idx1, key1, U, *units_out, first);
            e = cub::DeviceScan::InclusiveScan(tmp, scan_b, first, first, MaxOp(), U, q);
        }
        if (e == cudaSuccess) {
            block_flag_kernel<<<grid, 256, 0, q>>>(first, U, run);
            e = cub::DeviceScan::ExclusiveSum(tmp, sum_b, run, run, U + 1, q);
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->h_scalars, run + U, 4, cudaMemcpyDeviceToHost, q);
        if (e == cudaSuccess) e = cudaStreamSynchronize(q);
        n_runs = *(const uint32_t*)ctx->h_scalars;
        gs_status st = e == cudaSuccess ? gs_graph_alloc(g, (void**)runs_out, n_runs * sizeof(gs_tile_run))
                                        : gs_cuda_fail(ctx, e, "blocked order");
        if (st == GS_OK) {
            block_runs_kernel<<<grid, 256, 0, q>>>(*units_out, first, run, U, *runs_out);
            e = cudaGetLastError();
        }
        ctx->launches += 7;
        // wait: a server reads the order, and takes blocks of the pool, on streams of its own
        const cudaError_t w = cudaStreamSynchronize(q);
        if (e == cudaSuccess) e = w;
        if (e != cudaSuccess && st == GS_OK) st = gs_cuda_fail(ctx, e, "blocked order");
        gs_pool_put(ctx, tmp, tmp_b);
        if (st != GS_OK) return st;
    } else {
        GS_TRY(gs_graph_alloc(g, (void**)runs_out, sizeof(gs_tile_run)));
    }
    *R_out = n_runs;
    return GS_OK;
}

}  // namespace

gs_status gs_ensure_blocked(gs_graph* g) {
    if (g->stream || g->blocked_built) return GS_OK;
    const gs_status st = blocked_order(g, kBlockWindows, &g->R_blk, &g->d_runs_blk, &g->d_units_blk);
    if (st != GS_OK) {
        gs_graph_release(g, g->d_runs_blk);
        gs_graph_release(g, g->d_units_blk);
        g->d_runs_blk = nullptr;
        g->d_units_blk = nullptr;
        return st;
    }
    g->blocked_built = true;
    return GS_OK;
}

gs_status gs_ensure_blocked_small(gs_graph* g) {
    if (g->stream || g->blocked2_built) return GS_OK;
    const gs_status st = blocked_order(g, kBlockWindowsSmall, &g->R_blk2, &g->d_runs_blk2, &g->d_units_blk2);
    if (st != GS_OK) {
        gs_graph_release(g, g->d_runs_blk2);
        gs_graph_release(g, g->d_units_blk2);
        g->d_runs_blk2 = nullptr;
        g->d_units_blk2 = nullptr;
        return st;
    }
    g->blocked2_built = true;
    return GS_OK;
}
