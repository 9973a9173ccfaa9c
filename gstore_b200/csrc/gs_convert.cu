// In-memory converter "-c 1" on the device (grid::pre_grid + grid::proc_grid,
// gstore.cpp:1245-1458): edge pairs -> .start offsets, .grid records and
// .degree counts, as a resident graph.
//
//  1. count:   per non-self-loop edge, order (min, max) for the half grid,
//              find its tile, count it, count both endpoint degrees
//              (out-degree only for the directed grid) — gstore.cpp:1270-1312
//  2. scan:    exclusive prefix sum of the tile counts -> .start (:1316-1324)
//  3. scatter: each edge takes the next slot of its tile (:1403-1447)
//  4. sort:    records inside each tile are sorted by value (v1, then v0).
//              The reference leaves them in thread order, so any in-tile
//              order is a valid .grid; a sorted one is deterministic and lets
//              a warp's consecutive records touch neighbouring state words.
#include "gs_internal.cuh"

#include <cub/device/device_scan.cuh>
#include <cub/device/device_segmented_sort.cuh>

namespace {

__device__ __forceinline__ uint64_t dev_calc_index_half(uint64_t i, uint64_t j, uint64_t pc) {
    return ((i * ((pc << 1) - i - 1)) >> 1) + j;
}

// .start index of the tile holding (a, b), a <= b for the half grid.
__device__ __forceinline__ uint64_t tile_of(uint64_t a, uint64_t b, uint64_t p, int directed) {
    const uint64_t gi = a >> kGroupBits, gj = b >> kGroupBits;
    const uint64_t si = (a >> kTileBits) & 255, sj = (b >> kTileBits) & 255;
    if (directed) return ((gi * p + gj) << 16) + si * 256 + sj;
    if (gi == gj)
        return ((dev_calc_index_half(gi, gi, p) - gi) << 16) + ((gi * 257) << 7) +
               dev_calc_index_half(si, sj, 256);
    return ((dev_calc_index_half(gi, gj, p) - gi - 1) << 16) + (((gi + 1) * 257) << 7) + si * 256 + sj;
}

__global__ void count_kernel(const uint2* __restrict__ pairs, uint64_t n, uint64_t V, uint64_t p,
                             int directed, unsigned long long* __restrict__ counts, int32_t* __restrict__ deg,
                             int* bad) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t k = tid; k < n; k += nth) {
        const uint2 e = pairs[k];
        if (e.x == e.y) continue;  // is_self_loop
        if (e.x >= V || e.y >= V) {
            *bad = 1;
            continue;
        }
        uint64_t a = e.x, b = e.y;
        if (!directed && a > b) {
            a = e.y;
            b = e.x;
        }
        atomicAdd(counts + tile_of(a, b, p, directed), 1ull);
        atomicAdd(deg + e.x, 1);
        if (!directed) atomicAdd(deg + e.y, 1);
    }
}

__global__ void scatter_kernel(const uint2* __restrict__ pairs, uint64_t n, uint64_t p, int directed,
                               const uint64_t* __restrict__ start, unsigned int* __restrict__ cursor,
                               uint32_t* __restrict__ rec) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t k = tid; k < n; k += nth) {
        const uint2 e = pairs[k];
        if (e.x == e.y) continue;
        uint64_t a = e.x, b = e.y;
        if (!directed && a > b) {
            a = e.y;
            b = e.x;
        }
        const uint64_t t = tile_of(a, b, p, directed);
        const unsigned slot = atomicAdd(cursor + t, 1u);
        rec[start[t] + slot] = (uint32_t)(a & 0xFFFF) | ((uint32_t)(b & 0xFFFF) << 16);
    }
}

// The conversion of graphs of one tile group (V <= 2^24): the edges are split
// into buckets -- a tile, or 2^bits slices of a tile by the high bits of v1 --
// whose counters fit one CTA's shared memory, and the buckets are sorted.
// Buckets in order are tiles in file order, and a tile's sorted slices in order
// are the sorted tile.
//   * Counters in global memory, one per tile, take tens of thousands of
//     atomics on the same few addresses, and slots taken one by one scatter
//     single records.  Here a CTA takes a stretch of the edges, counts it in
//     shared memory and gets each bucket's slots in one piece, so that its
//     records of a bucket lie side by side.
//   * A segmented sort gives a segment to a CTA, which needs four passes over
//     memory for one that does not fit its shared memory: 1.7 ms for the three
//     tiles of 0.8 M edges over 100,003 vertices.  Slices are small (about
//     1,024 records and more) and many.
//   * But not for their own sake: the 2,080 tiles of Kronecker 22 cut into
//     33,280 slices took 1.82 ms to scatter (shorter stretches) and 2.50 to
//     sort instead of 0.98 and 2.13.
// 67 M edges of Kronecker 22, ms: count 1.60 -> 0.94, scatter 1.89 -> 0.81, sort
// 2.14 as before; 0.8 M edges over 100,003 vertices, all of it: 2.67 -> 0.48.  What
// is left of the count are the two random degree atomics per edge (~180 G/s).
constexpr uint32_t kMaxBuckets = 49152;        // 192 KB of counters
constexpr uint64_t kEnoughBuckets = 2048;      // no more slices from here on (at most 2^12 of one tile)
constexpr uint64_t kBucketRecords = 1024;      // records a slice should have on average
constexpr uint64_t kBucketMinEdges = 1u << 14; // fewer: the counters' clearing and reading costs more than it saves
constexpr int kBucketThreads = 1024;

struct Buckets {
    uint32_t nw;     // tiles per side that hold vertices
    int directed, bits;
    uint32_t n;      // buckets
};

__host__ __device__ __forceinline__ uint32_t bucket_tile(uint32_t i, uint32_t j, const Buckets& B) {
    return B.directed ? i * B.nw + j : i * (2 * B.nw - i + 1) / 2 + (j - i);   // file order
}
__device__ __forceinline__ uint32_t bucket_of(uint32_t a, uint32_t b, const Buckets& B) {
    return (bucket_tile(a >> kTileBits, b >> kTileBits, B) << B.bits) | ((b & 0xFFFFu) >> (kTileBits - B.bits));
}

// A CTA counts the stretch of `per` edges that it will scatter.  Table: its
// counts go to counts[t * gridDim + CTA], else they are added to counts[t].
template <bool Table>
__global__ void __launch_bounds__(kBucketThreads, 1)
    bucket_count_kernel(const uint2* __restrict__ pairs, uint64_t n, uint64_t per, uint64_t V, const Buckets B,
                        uint32_t* __restrict__ counts, int32_t* __restrict__ deg, int* bad) {
    extern __shared__ uint32_t s_count[];
    for (uint32_t t = threadIdx.x; t < B.n; t += kBucketThreads) s_count[t] = 0;
    __syncthreads();
    const uint64_t lo = blockIdx.x * per, hi = lo + per < n ? lo + per : n;
    for (uint64_t k = lo + threadIdx.x; k < hi; k += 4 * kBucketThreads) {
        uint2 e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            e[j] = k + j * kBucketThreads < hi ? __ldcs(pairs + k + j * kBucketThreads) : make_uint2(0, 0);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (e[j].x == e[j].y) continue;  // is_self_loop
            if (e[j].x >= V || e[j].y >= V) {
                *bad = 1;
                continue;
            }
            const bool swap = !B.directed && e[j].x > e[j].y;
            atomicAdd(s_count + bucket_of(swap ? e[j].y : e[j].x, swap ? e[j].x : e[j].y, B), 1u);
            atomicAdd(deg + e[j].x, 1);
            if (!B.directed) atomicAdd(deg + e[j].y, 1);
        }
    }
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < B.n; t += kBucketThreads) {
        if (Table) counts[(uint64_t)t * gridDim.x + blockIdx.x] = s_count[t];
        else if (s_count[t]) atomicAdd(counts + t, s_count[t]);
    }
}

// starts[t] = the scanned table's entry of bucket t's first stretch.
__global__ void bucket_table_start_kernel(const uint32_t* __restrict__ table, uint32_t n_buckets, uint32_t stretches,
                                          uint32_t* __restrict__ starts) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t <= n_buckets; t += nth)
        starts[t] = table[(uint64_t)t * stretches];
}

// cursor: the buckets' starts, and on return their ends; Table: the scanned
// table of counts, which has every stretch's slots.
template <bool Table>
__global__ void __launch_bounds__(kBucketThreads, 1)
    bucket_scatter_kernel(const uint2* __restrict__ pairs, uint64_t n, uint64_t per, const Buckets B,
                          uint32_t* __restrict__ cursor, uint32_t* __restrict__ rec) {
    extern __shared__ uint32_t s_slot[];
    const uint64_t lo = (uint64_t)blockIdx.x * per, hi = lo + per < n ? lo + per : n;
    auto each = [&](auto fn) {
        for (uint64_t k = lo + threadIdx.x; k < hi; k += 4 * kBucketThreads) {
            uint2 e[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) e[j] = k + j * kBucketThreads < hi ? pairs[k + j * kBucketThreads] : make_uint2(0, 0);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (e[j].x == e[j].y) continue;
                const bool swap = !B.directed && e[j].x > e[j].y;
                const uint32_t a = swap ? e[j].y : e[j].x, b = swap ? e[j].x : e[j].y;
                fn(bucket_of(a, b, B), (a & 0xFFFFu) | (b << 16));
            }
        }
    };
    if (Table) {
        for (uint32_t t = threadIdx.x; t < B.n; t += kBucketThreads) s_slot[t] = cursor[(uint64_t)t * gridDim.x + blockIdx.x];
    } else {
        for (uint32_t t = threadIdx.x; t < B.n; t += kBucketThreads) s_slot[t] = 0;
        __syncthreads();
        each([&](uint32_t t, uint32_t) { atomicAdd(s_slot + t, 1u); });
        __syncthreads();
        for (uint32_t t = threadIdx.x; t < B.n; t += kBucketThreads)
            if (const uint32_t c = s_slot[t]) s_slot[t] = atomicAdd(cursor + t, c);
    }
    __syncthreads();
    each([&](uint32_t t, uint32_t r) { rec[atomicAdd(s_slot + t, 1u)] = r; });
}

// .start of the one group's 256 x 256 tiles from the buckets' starts
// (start[n] = total); tiles beyond the vertices are empty.
__global__ void bucket_start_kernel(const uint32_t* __restrict__ bucket_start, const Buckets B, uint64_t T,
                                    uint64_t* __restrict__ start) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < kGroupTiles * kGroupTiles; k += nth) {
        const uint32_t i = k / kGroupTiles, j = k % kGroupTiles;
        if (k == 0) start[T] = bucket_start[B.n];
        if (!B.directed && j < i) continue;
        const uint64_t t = B.directed ? k : dev_calc_index_half(i, j, kGroupTiles);
        uint32_t at = B.n;
        if (i < B.nw && j < B.nw) at = bucket_tile(i, j, B) << B.bits;
        else if (i + 1 < B.nw) at = bucket_tile(i + 1, B.directed ? 0 : i + 1, B) << B.bits;   // the next row
        start[t] = bucket_start[at];
    }
}

__global__ void rebase_offsets_kernel(const uint64_t* __restrict__ start, uint64_t t0, uint64_t n,
                                      int* __restrict__ out) {
    const uint64_t base = start[t0];
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = (int)(start[t0 + i] - base);
}

// Flags a tile whose records are not in ascending order (a warp per unit;
// a unit's first record is compared with the last one of the previous unit
// when both lie in the same tile).
__global__ void tiles_unsorted_kernel(const gs_unit* __restrict__ units, uint64_t n_units,
                                      const uint32_t* __restrict__ rec, int* flag) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t u = warp; u < n_units; u += n_warps) {
        const gs_unit un = units[u];
        const bool joined = u > 0 && units[u - 1].rc == un.rc && units[u - 1].rec_beg + units[u - 1].n == un.rec_beg;
        bool bad = false;
        for (uint32_t k = lane; k < un.n; k += 32) {
            const uint64_t e = un.rec_beg + k;
            if ((k > 0 || joined) && rec[e] < rec[e - 1]) bad = true;
        }
        if (__any_sync(0xFFFFFFFFu, bad) && lane == 0) atomicExch(flag, 1);
    }
}

}  // namespace

gs_status gs_order_tiles(gs_graph* g, bool* sorted_now) {
    gs_ctx* ctx = g->ctx;
    *sorted_now = false;
    if (!g->d_rec || g->E < 2 || g->U == 0) return GS_OK;
    int* d_flag = (int*)ctx->d_scalars;
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(d_flag, 0, sizeof(int), ctx->stream));
    tiles_unsorted_kernel<<<gs_grid_size(ctx, 8), 256, 0, ctx->stream>>>(g->d_units, g->U, g->d_rec, d_flag);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    int h_flag = 0;
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(&h_flag, d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (!h_flag) return GS_OK;
    GS_TRY(gs_sort_tiles(ctx, g->d_tile_off, g->T, g->d_rec, g->E));
    *sorted_now = true;
    return GS_OK;
}

// Sorts the records of every tile (segments = tiles of `start`) from d_rec
// into d_out.
static gs_status sort_tiles_into(gs_ctx* ctx, const uint64_t* d_start, uint64_t n_tiles, uint32_t* d_rec,
                                 uint64_t n_rec, uint32_t* d_out) {
    std::vector<uint64_t> h(n_tiles + 1);
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(h.data(), d_start, (n_tiles + 1) * 8, cudaMemcpyDeviceToHost, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    // chunks of whole tiles with at most 2^30 records and 2^24 tiles each
    const uint64_t kMaxRec = 1ull << 30, kMaxTiles = 1ull << 24;
    int* d_off = nullptr;
    void* d_tmp = nullptr;
    size_t tmp_bytes = 0;
    const size_t off_bytes = (std::min(n_tiles, kMaxTiles) + 1) * sizeof(int);
    gs_status st = gs_pool_get(ctx, off_bytes, (void**)&d_off);
    uint64_t t0 = 0;
    while (st == GS_OK && t0 < n_tiles) {
        uint64_t t1 = t0;
        while (t1 < n_tiles && t1 - t0 < kMaxTiles && h[t1 + 1] - h[t0] <= kMaxRec) ++t1;
        if (t1 == t0) {
            st = gs_fail(ctx, GS_ERR_FORMAT, "a tile holds more than 2^30 records");
            break;
        }
        const uint64_t nr = h[t1] - h[t0];
        if (nr > 1) {
            rebase_offsets_kernel<<<256, 256, 0, ctx->stream>>>(d_start, t0, t1 - t0, d_off);
            ctx->launches++;
            size_t need = 0;
            cudaError_t e = cub::DeviceSegmentedSort::SortKeys(nullptr, need, d_rec + h[t0], d_out + h[t0], (int)nr,
                                                               (int)(t1 - t0), d_off, d_off + 1, ctx->stream);
            if (e == cudaSuccess && need > tmp_bytes) {
                gs_pool_put(ctx, d_tmp, tmp_bytes);
                d_tmp = nullptr;
                tmp_bytes = need;
                st = gs_pool_get(ctx, tmp_bytes, &d_tmp);
            }
            if (e == cudaSuccess && st == GS_OK)
                e = cub::DeviceSegmentedSort::SortKeys(d_tmp, need, d_rec + h[t0], d_out + h[t0], (int)nr,
                                                       (int)(t1 - t0), d_off, d_off + 1, ctx->stream);
            if (e != cudaSuccess && st == GS_OK) st = gs_cuda_fail(ctx, e, "segmented sort");
            ctx->launches++;
        } else if (nr == 1) {
            cudaError_t e = cudaMemcpyAsync(d_out + h[t0], d_rec + h[t0], 4, cudaMemcpyDeviceToDevice, ctx->stream);
            if (e != cudaSuccess) st = gs_cuda_fail(ctx, e, "copy");
        }
        t0 = t1;
    }
    // (pooled scratch is reused in stream order)
    gs_pool_put(ctx, d_off, off_bytes);
    gs_pool_put(ctx, d_tmp, tmp_bytes);
    return st;
}

// The same in place.
gs_status gs_sort_tiles(gs_ctx* ctx, const uint64_t* d_start, uint64_t n_tiles, uint32_t* d_rec, uint64_t n_rec) {
    if (n_rec < 2 || n_tiles == 0) return GS_OK;
    uint32_t* d_out = nullptr;
    GS_TRY(gs_pool_get(ctx, n_rec * 4, (void**)&d_out));
    gs_status st = sort_tiles_into(ctx, d_start, n_tiles, d_rec, n_rec, d_out);
    if (st == GS_OK) {
        cudaError_t e = cudaMemcpyAsync(d_rec, d_out, n_rec * 4, cudaMemcpyDeviceToDevice, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) st = gs_cuda_fail(ctx, e, "copy sorted records");
    } else {
        cudaStreamSynchronize(ctx->stream);
    }
    gs_pool_put(ctx, d_out, n_rec * 4);
    return st;
}


// Scratch of a conversion goes back to the context's pool (a conversion made
// seven cudaMalloc / cudaFree pairs, 3 of the 12 ms of Kronecker 22 and up to
// 0.7 s when the driver is slow), blocks over 1 GiB to the driver.
static void scratch_put(gs_ctx* ctx, void* p, size_t bytes) {
    if (bytes > (1ull << 30)) gs_dev_free(p);
    else gs_pool_put(ctx, p, bytes);
}

struct gs_converted {
    uint64_t* d_start = nullptr;
    int32_t* d_degree = nullptr;
    uint32_t* d_rec = nullptr;   // n_rec + kRecPad records, the padding zero
    uint64_t n_start = 0, n_rec = 0, V = 0;
    size_t rec_bytes() const { return (n_rec + kRecPad) * 4; }
};

static void converted_put(gs_ctx* ctx, gs_converted& c, bool rec) {
    scratch_put(ctx, c.d_start, c.n_start * 8);
    scratch_put(ctx, c.d_degree, std::max<uint64_t>(c.V, 1) * 4);
    if (rec) scratch_put(ctx, c.d_rec, c.rec_bytes());
}

// The two ways to fill c.d_start and c.d_rec; c.d_degree and *d_bad are zero,
// the count pass has been launched.
// The stretches of edges that a CTA counts and scatters, and whether their
// counts are kept as a table that is scanned as a whole, so that the scatter
// need not count again (Kronecker 22: 0.98 -> 0.81 ms; the table's scan 0.01):
// while it is small against the edges.
struct Stretches {
    uint64_t per;
    uint32_t n;
    bool table;
    Stretches(const gs_ctx* ctx, uint64_t n_pairs, const Buckets& B)
        : per(std::max<uint64_t>(4 * kBucketThreads, (n_pairs + 2 * ctx->num_sms - 1) / (2 * ctx->num_sms))),
          n((uint32_t)((n_pairs + per - 1) / per)),
          table((uint64_t)B.n * n <= n_pairs / 16) {}
    uint64_t counts(const Buckets& B) const { return table ? (uint64_t)B.n * n + 1 : B.n; }
};

// d_bucket: the buckets' starts, then the table or the cursors.
static gs_status fill_buckets(gs_ctx* ctx, const uint2* pairs, uint64_t n_pairs, const Buckets& B, const Stretches& S,
                              uint32_t* d_bucket, const int* d_bad, gs_converted& c) {
    cudaStream_t q = ctx->stream;
    uint32_t* d_cursor = d_bucket + B.n + 1;
    uint32_t* const d_scan = S.table ? d_cursor : d_bucket;
    const int n_scan = (int)(S.table ? S.counts(B) : B.n + 1);
    size_t scan_bytes = 0, sort_bytes = 0;
    GS_CHECK_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, d_scan, d_scan, n_scan, q));
    char* d_tmp = nullptr;
    GS_TRY(gs_pool_get(ctx, scan_bytes, (void**)&d_tmp));
    cudaError_t e = cub::DeviceScan::ExclusiveSum(d_tmp, scan_bytes, d_scan, d_scan, n_scan, q);
    scratch_put(ctx, d_tmp, scan_bytes);
    GS_CHECK_CUDA(ctx, e);
    if (S.table) {
        bucket_table_start_kernel<<<64, 256, 0, q>>>(d_cursor, B.n, S.n, d_bucket);
        GS_CHECK_CUDA(ctx, cudaGetLastError());
        ctx->launches++;
    } else {
        GS_CHECK_CUDA(ctx, cudaMemcpyAsync(d_cursor, d_bucket, (size_t)B.n * 4, cudaMemcpyDeviceToDevice, q));
    }
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars, d_bucket + B.n, 4, cudaMemcpyDeviceToHost, q));
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars + 1, d_bad, sizeof(int), cudaMemcpyDeviceToHost, q));
    bucket_start_kernel<<<64, 256, 0, q>>>(d_bucket, B, c.n_start - 1, c.d_start);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    GS_CHECK_CUDA(ctx, cudaStreamSynchronize(q));
    if (*(const int*)(ctx->h_scalars + 1))
        return gs_fail(ctx, GS_ERR_FORMAT, "an edge endpoint is >= the vertex count");
    c.n_rec = *(const uint32_t*)ctx->h_scalars;
    GS_TRY(gs_pool_get(ctx, c.rec_bytes(), (void**)&c.d_rec));
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(c.d_rec + c.n_rec, 0, kRecPad * 4, q));
    if (c.n_rec == 0) return GS_OK;
    uint32_t* d_raw = nullptr;   // the records before the sort
    GS_TRY(gs_pool_get(ctx, c.rec_bytes(), (void**)&d_raw));
    if (S.table)
        bucket_scatter_kernel<true><<<S.n, kBucketThreads, (size_t)B.n * 4, q>>>(pairs, n_pairs, S.per, B, d_cursor, d_raw);
    else
        bucket_scatter_kernel<false><<<S.n, kBucketThreads, (size_t)B.n * 4, q>>>(pairs, n_pairs, S.per, B, d_cursor, d_raw);
    e = cudaGetLastError();
    const int* seg = (const int*)d_bucket;   // n_rec <= 2^30
    if (e == cudaSuccess)
        e = cub::DeviceSegmentedSort::SortKeys(nullptr, sort_bytes, d_raw, c.d_rec, (int)c.n_rec, (int)B.n, seg, seg + 1, q);
    gs_status st = e == cudaSuccess ? gs_pool_get(ctx, sort_bytes, (void**)&d_tmp) : GS_OK;
    if (e == cudaSuccess && st == GS_OK) {
        e = cub::DeviceSegmentedSort::SortKeys(d_tmp, sort_bytes, d_raw, c.d_rec, (int)c.n_rec, (int)B.n, seg, seg + 1, q);
        scratch_put(ctx, d_tmp, sort_bytes);
    }
    ctx->launches += 4;
    scratch_put(ctx, d_raw, c.rec_bytes());
    return e == cudaSuccess ? st : gs_cuda_fail(ctx, e, "converter");
}

static gs_status fill_tiles(gs_ctx* ctx, const uint2* pairs, uint64_t n_pairs, uint64_t p, int directed,
                            uint32_t blocks, const int* d_bad, gs_converted& c) {
    cudaStream_t q = ctx->stream;
    const uint64_t T = c.n_start - 1;
    // cub's scratch, then the slot cursors
    size_t scan_bytes = 0;
    GS_CHECK_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, c.d_start, c.d_start, c.n_start, q));
    const size_t cursor_at = (scan_bytes + 255) & ~(size_t)255, tmp_bytes = cursor_at + T * 4;
    char* d_tmp = nullptr;
    GS_TRY(gs_pool_get(ctx, tmp_bytes, (void**)&d_tmp));
    unsigned int* d_cursor = (unsigned int*)(d_tmp + cursor_at);
    const gs_status st = [&]() -> gs_status {
        GS_CHECK_CUDA(ctx, cub::DeviceScan::ExclusiveSum(d_tmp, scan_bytes, c.d_start, c.d_start, c.n_start, q));
        GS_CHECK_CUDA(ctx, cudaMemsetAsync(d_cursor, 0, T * 4, q));
        GS_CHECK_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars, c.d_start + T, 8, cudaMemcpyDeviceToHost, q));
        GS_CHECK_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars + 1, d_bad, sizeof(int), cudaMemcpyDeviceToHost, q));
        GS_CHECK_CUDA(ctx, cudaStreamSynchronize(q));
        if (*(const int*)(ctx->h_scalars + 1))
            return gs_fail(ctx, GS_ERR_FORMAT, "an edge endpoint is >= the vertex count");
        c.n_rec = ctx->h_scalars[0];
        GS_TRY(gs_pool_get(ctx, c.rec_bytes(), (void**)&c.d_rec));
        GS_CHECK_CUDA(ctx, cudaMemsetAsync(c.d_rec + c.n_rec, 0, kRecPad * 4, q));
        if (c.n_rec == 0) return GS_OK;
        uint32_t* d_raw = nullptr;   // the records before the sort
        GS_TRY(gs_pool_get(ctx, c.rec_bytes(), (void**)&d_raw));
        scatter_kernel<<<blocks, 256, 0, q>>>(pairs, n_pairs, p, directed, c.d_start, d_cursor, d_raw);
        cudaError_t e = cudaGetLastError();
        ctx->launches++;
        gs_status sorted = GS_OK;
        if (e == cudaSuccess && c.n_rec == 1) e = cudaMemcpyAsync(c.d_rec, d_raw, 4, cudaMemcpyDeviceToDevice, q);
        else if (e == cudaSuccess) sorted = sort_tiles_into(ctx, c.d_start, T, d_raw, c.n_rec, c.d_rec);
        scratch_put(ctx, d_raw, c.rec_bytes());
        return e == cudaSuccess ? sorted : gs_cuda_fail(ctx, e, "converter");
    }();
    scratch_put(ctx, d_tmp, tmp_bytes);
    return st;
}

static gs_status convert_launch(gs_ctx* ctx, const uint32_t* d_pairs, uint64_t n_pairs, uint64_t V, int directed,
                                gs_converted& c) {
    uint32_t p, ps;
    uint64_t T;
    gs_geometry_of(V, directed, &p, &ps, &T);
    cudaStream_t q = ctx->stream;
    int* d_bad = (int*)ctx->d_scalars;
    const uint2* pairs = reinterpret_cast<const uint2*>(d_pairs);
    const uint32_t blocks = (uint32_t)std::max<uint64_t>(
        1, std::min<uint64_t>((n_pairs + 255) / 256, gs_grid_size(ctx, 16)));
    c.V = V;
    c.n_start = T + 1;
    GS_TRY(gs_pool_get(ctx, c.n_start * 8, (void**)&c.d_start));
    GS_TRY(gs_pool_get(ctx, std::max<uint64_t>(V, 1) * 4, (void**)&c.d_degree));
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(c.d_degree, 0, V * 4, q));
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(d_bad, 0, sizeof(int), q));
    // buckets: the tiles that hold vertices, sliced while a slice keeps
    // kBucketRecords records and the counters fit
    Buckets B{(uint32_t)((V + 0xFFFF) >> kTileBits), directed, 0, 0};
    const uint64_t tiles = directed ? (uint64_t)B.nw * B.nw : (uint64_t)B.nw * (B.nw + 1) / 2;
    if (p == 1 && tiles <= kMaxBuckets && n_pairs >= kBucketMinEdges && n_pairs <= (1ull << 30)) {
        while (tiles << B.bits < kEnoughBuckets && n_pairs >> (B.bits + 1) >= tiles * kBucketRecords) ++B.bits;
        B.n = (uint32_t)(tiles << B.bits);
        const Stretches S(ctx, n_pairs, B);
        auto* const count = S.table ? &bucket_count_kernel<true> : &bucket_count_kernel<false>;
        GS_CHECK_CUDA(ctx, gs_smem_limit_once<bucket_count_kernel<true>>(ctx->device, (int)(kMaxBuckets * 4)));
        GS_CHECK_CUDA(ctx, gs_smem_limit_once<bucket_count_kernel<false>>(ctx->device, (int)(kMaxBuckets * 4)));
        GS_CHECK_CUDA(ctx, gs_smem_limit_once<bucket_scatter_kernel<true>>(ctx->device, (int)(kMaxBuckets * 4)));
        GS_CHECK_CUDA(ctx, gs_smem_limit_once<bucket_scatter_kernel<false>>(ctx->device, (int)(kMaxBuckets * 4)));
        const size_t bucket_bytes = ((size_t)B.n + 1 + S.counts(B)) * 4;   // starts, and the table or cursors
        uint32_t* d_bucket = nullptr;
        GS_TRY(gs_pool_get(ctx, bucket_bytes, (void**)&d_bucket));
        uint32_t* const d_count = S.table ? d_bucket + B.n + 1 : d_bucket;
        // (the table needs a zero behind it only, the counts are added to)
        cudaError_t e = S.table ? cudaMemsetAsync(d_count + (uint64_t)B.n * S.n, 0, 4, q)
                                : cudaMemsetAsync(d_count, 0, ((size_t)B.n + 1) * 4, q);
        if (e == cudaSuccess) {
            count<<<S.n, kBucketThreads, (size_t)B.n * 4, q>>>(pairs, n_pairs, S.per, V, B, d_count, c.d_degree, d_bad);
            ctx->launches++;
            e = cudaGetLastError();
        }
        const gs_status st = e == cudaSuccess ? fill_buckets(ctx, pairs, n_pairs, B, S, d_bucket, d_bad, c)
                                              : gs_cuda_fail(ctx, e, "converter");
        scratch_put(ctx, d_bucket, bucket_bytes);
        return st;
    }
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(c.d_start, 0, c.n_start * 8, q));
    if (n_pairs) {
        count_kernel<<<blocks, 256, 0, q>>>(pairs, n_pairs, V, p, directed, (unsigned long long*)c.d_start, c.d_degree,
                                            d_bad);
        GS_CHECK_CUDA(ctx, cudaGetLastError());
        ctx->launches++;
    }
    return fill_tiles(ctx, pairs, n_pairs, p, directed, blocks, d_bad, c);
}

extern "C" gs_status gs_convert(gs_ctx* ctx, const uint32_t* pairs, uint64_t n_pairs, int is_device,
                                uint64_t V, gs_graph** out) {
    if (!ctx || !out || (n_pairs && !pairs) || V == 0 || V > (1ull << 32)) return GS_ERR_ARG;
    *out = nullptr;
    const uint32_t* d_pairs = pairs;
    uint32_t* d_copy = nullptr;
    if (!is_device && n_pairs) {
        GS_TRY(gs_pool_get(ctx, n_pairs * 8, (void**)&d_copy));
        cudaError_t e = cudaMemcpyAsync(d_copy, pairs, n_pairs * 8, cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) {
            scratch_put(ctx, d_copy, n_pairs * 8);
            return gs_cuda_fail(ctx, e, "copy pairs");
        }
        d_pairs = d_copy;
    }
    gs_converted c;
    gs_status st = convert_launch(ctx, d_pairs, n_pairs, V, ctx->directed, c);
    // a conversion that fails may leave kernels that read the pairs and the
    // scratch: both are given back below (one that succeeds waits further on)
    if (st != GS_OK) cudaStreamSynchronize(ctx->stream);
    if (d_copy) scratch_put(ctx, d_copy, n_pairs * 8);
    if (st != GS_OK) {
        converted_put(ctx, c, true);
        return st;
    }
    st = gs_graph_adopt(ctx, V, c.d_start, c.n_start, c.d_rec, c.n_rec, c.d_degree, out);
    if (st == GS_OK) (*out)->degree_from_records = true;
    converted_put(ctx, c, false);
    return st;
}
