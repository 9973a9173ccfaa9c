// PageRank sweep over row lists (sm_100a): pagerank_onepart (pr.cpp:119-154)
// for a resident graph, pulled instead of pushed.
//
// Per record (v0, v1) the reference does
//     rank[v1] += prior[v0];   rank[v0] += prior[v1]   (the second: half grid)
// A layout built once per graph lists, for every destination, the sources
// that push into it; a sweep reads the list (4 bytes per entry, streamed once)
// and gathers prior[source].  What bounds it is the gather: an SM looks up one
// 128-byte line of its L1 per clock, so 32 scattered lanes cost 32 clocks
// (~280 G gathers/s over the chip at best, L2 or L1 hit alike), while 32
// scattered shared-memory words cost about 3.2 (measured).  Hence:
//
//   * sources are numbered by falling number of pushes, and x is permuted
//     into that order at the start of a sweep.  In a graph with hubs the
//     first kRlPanel sources (128 KB of x) make up 72 / 36 / 25 % of the
//     entries at Kronecker scale 20 / 24 / 26;
//   * panel 0 (the first kRlPanel sources) is staged in shared memory by
//     every CTA of the main group; a source beyond it is read through L2.
//     Entries of long rows that fall into one of the next panels are split
//     off into row segments of their own, which a few CTAs sweep with that
//     panel staged instead: their gathers stay in shared memory too;
//   * rows are cut into segments of at most kRlSegMax entries and sorted by
//     length; 32 segments of (nearly) equal length make a slice, stored
//     transposed so that lane l reads 16 bytes (four entries) of segment l and
//     a warp 512 consecutive bytes.  A lane sums its segment in registers; no
//     shuffles, one `red` to y per segment (neighbouring segments of one row
//     are joined first, so a hub does not serialise on its own sum).
//
// The panel's size: a gather in flight holds a line of L1, and what is not
// shared memory is L1.  224 KB panels left 28 KB of L1, ~220 gathers in
// flight, and ran at a third of the lookup rate: 1,880 us per iteration at
// Kronecker 24 against 1,097 with 128 KB panels (96 KB: 1,146, 160 KB: 1,100;
// 16 panels each; 1,032-1,080 with 64).
//
// Per iteration against propagation blocking (gs_pr_blocked.cu: 12.5 bytes
// moved per entry, a shared-memory atomic per run of destinations): Kronecker
// 20 / 24 / 26, edge factor 16: 79 / 1,027 / 5,900 us against 146 / 1,862 /
// 8,010; the layout keeps 4.4 bytes per entry instead of 12.5.  Without hubs
// (uniform random, 3 M vertices, 24 M entries) 153 against 100: rl_worth.
// At Kronecker 23 the pull reads 28 % of its entries' sources through L2 and
// its L1 runs at 70 % of its peak; of DRAM it needs about a third.
#include "gs_internal.cuh"
#include "gs_temps.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <vector>

namespace {

constexpr uint32_t kRlPanel = 32768;      // sources per panel (a multiple of 2^kSortSkip)
constexpr int kSortSkip = 13;             // source bits the entry sort leaves alone
constexpr uint32_t kRlSegMax = 256;       // longest row segment
constexpr uint32_t kRlPanelRow = 8;       // entries of a row in a panel that are worth a segment of their own
constexpr uint32_t kRlHeavy = 256;        // rows from this length on are split by panel
constexpr int kRlThreads = 1024;
constexpr uint32_t kRlWarps = kRlThreads / 32;
constexpr uint32_t kGroups = 3 + kRlMaxPanels;   // heavy cold, light, heavy hot, then panels 1..
constexpr uint64_t kRlPanelMin = 1ull << 19;     // entries of long rows that make a panel worth staging
constexpr uint32_t kRlTopRows = 256;             // longest rows, whose sums are kept in 64 bits
constexpr uint64_t kRlL2Sources = 1ull << 24;    // sources whose x (64 MB) stays in L2
constexpr long long kWaitLimit = 1ll << 24;
static_assert(kRlPanel % (1u << kSortSkip) == 0, "a panel boundary must survive the entry sort");

struct RlArgs {
    const uint4* ent;
    const uint32_t* row;
    const uint8_t* n4;
    const gs_rl_unit* units;
    const float* x;          // permuted
    float* y;
    uint32_t n_src, n_panels;
    uint32_t unit_beg[kRlMaxPanels + 1];
    uint32_t home_beg[kRlMaxPanels + 1];
    double* top_sum;         // [n_top]
    uint32_t n_top;
    unsigned int* tick;      // [kRlMaxPanels] next unit of each panel, then CTAs finished; zero at launch and after it
    int* error;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool wait_bar(unsigned long long* bar, uint32_t parity) {
    const uint32_t a = smem_u32(bar);
    for (long long i = 0; i < kWaitLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__global__ void rl_permute_kernel(const float* __restrict__ x, const uint32_t* __restrict__ src, uint32_t n,
                                  float* __restrict__ out) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth) out[i] = __ldg(x + src[i]);
}

// An entry is a word index of the staged panel (kRlPanel itself: a zero, the
// padding), or, in panel 0's units, one more than the source's position.
__global__ void __launch_bounds__(kRlThreads, 1) rl_pull_kernel(const RlArgs a) {
    extern __shared__ __align__(128) float xs[];   // kRlPanel staged words, then the padding's zero
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int s_go;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        xs[kRlPanel] = 0.f;
    }
    uint32_t home = 0;
    while (home + 1 < a.n_panels && blockIdx.x >= a.home_beg[home + 1]) ++home;
    const float* xg = a.x - 1;
    auto at = [&](uint32_t i) -> float { return i <= kRlPanel ? xs[i] : __ldg(xg + i); };
    uint32_t parity = 0;
    // the CTA's own panel first, then any panel with units for all its warps
    for (uint32_t j = 0; j < a.n_panels; ++j) {
        const uint32_t p = home + j < a.n_panels ? home + j : home + j - a.n_panels;
        const uint32_t u0 = a.unit_beg[p], nu = a.unit_beg[p + 1] - u0;
        __syncthreads();   // every thread is done with the previous panel and has read s_go
        if (tid == 0) {
            const unsigned drawn = *(volatile unsigned int*)(a.tick + p);
            s_go = drawn + (j ? kRlWarps : 1u) <= nu;
            if (s_go) {
                const uint32_t first = p * kRlPanel;
                const uint32_t n = min(kRlPanel, a.n_src - first);
                const uint32_t bytes = ((n + 3) & ~3u) * 4;   // x is padded to a multiple of 4
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&bar)), "r"(bytes)
                             : "memory");
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        smem_u32(xs)),
                    "l"(a.x + first), "r"(bytes), "r"(smem_u32(&bar))
                    : "memory");
            }
        }
        __syncthreads();
        if (!s_go) continue;   // uniform
        const bool got = wait_bar(&bar, parity);
        parity ^= 1;
        if (!__syncthreads_and(got)) {
            // the copy is late: flag it and give it one more bounded wait, so
            // that the CTA does not leave with its copy still in flight
            if (tid == 0) {
                atomicExch(a.error, 1);
                wait_bar(&bar, parity ^ 1);
            }
            break;   // uniform
        }
        while (true) {
            uint32_t u = 0;
            if (lane == 0) u = atomicAdd(a.tick + p, 1u);
            u = __shfl_sync(0xFFFFFFFFu, u, 0);
            if (u >= nu) break;
            const gs_rl_unit d = a.units[u0 + u];
            const uint4* e = a.ent + (uint64_t)d.off * 32 + lane;
            const uint32_t myn = lane < d.n_slices ? a.n4[d.slice + lane] : 0u;
            const uint32_t* rows = a.row + (uint64_t)d.slice * 32 + lane;
            // the unit's entries are one stream, read two steps ahead across
            // its slices
            const uint4 z = make_uint4(0, 0, 0, 0);
            uint4 q0 = __ldcs(e), q1 = d.steps > 1 ? __ldcs(e + 32) : z;
            uint32_t t = 2;
            uint32_t r_next = rows[0];
            for (uint32_t s = 0; s < d.n_slices; ++s) {
                const uint32_t r = r_next;
                if (s + 1 < d.n_slices) r_next = rows[32 * (s + 1)];
                float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
                uint32_t k = __shfl_sync(0xFFFFFFFFu, myn, s);
                for (; k >= 2; k -= 2) {   // eight gathers in flight
                    const uint4 q = q0, w = q1;
                    if (t < d.steps) q0 = __ldcs(e + 32 * t);
                    if (t + 1 < d.steps) q1 = __ldcs(e + 32 * (t + 1));
                    t += 2;
                    const float v0 = at(q.x), v1 = at(q.y), v2 = at(q.z), v3 = at(q.w);
                    const float w0 = at(w.x), w1 = at(w.y), w2 = at(w.z), w3 = at(w.w);
                    s0 += v0 + w0;
                    s1 += v1 + w1;
                    s2 += v2 + w2;
                    s3 += v3 + w3;
                }
                if (k) {
                    const uint4 q = q0;
                    q0 = q1;
                    if (t < d.steps) q1 = __ldcs(e + 32 * t);
                    ++t;
                    s0 += at(q.x);
                    s1 += at(q.y);
                    s2 += at(q.z);
                    s3 += at(q.w);
                }
                float sum = (s0 + s1) + (s2 + s3);
                // segments of one row lie side by side: join them, add once
                const uint32_t r_prev = __shfl_up_sync(0xFFFFFFFFu, r, 1);
                const bool same = lane > 0 && r_prev == r && r != ~0u;
                bool last = true;
                if (__any_sync(0xFFFFFFFFu, same)) {
                    bool head = !same;
#pragma unroll
                    for (int k = 1; k < 32; k <<= 1) {
                        const float cu = __shfl_up_sync(0xFFFFFFFFu, sum, k);
                        const bool hu = __shfl_up_sync(0xFFFFFFFFu, head, k);
                        if (lane >= (uint32_t)k && !head) {
                            sum += cu;
                            head = hu;
                        }
                    }
                    last = !__shfl_down_sync(0xFFFFFFFFu, same, 1) || lane == 31;
                }
                if (last && r != ~0u) {
                    if (r >= kRlTop && a.n_top) atomicAdd(a.top_sum + (r - kRlTop), (double)sum);
                    else atomicAdd(a.y + r, sum);
                }
            }
        }
    }
    __syncthreads();   // every warp of the CTA has drawn its last unit
    if (tid == 0 && atomicAdd(a.tick + kRlMaxPanels, 1u) == gridDim.x - 1) {
        for (int k = 0; k <= (int)kRlMaxPanels; ++k) atomicExch(a.tick + k, 0u);   // and of every CTA
    }
}

// The longest rows' sums, and zero for the next sweep.  A row of 10^5 entries
// and more takes a hundred additions one after another, whose rounding in 32
// bits was most of the ranks' error (2-norm against 64 bits, five iterations of
// Kronecker 24: 1.6e-7, now 6.6e-8; 20: 7.9e-8 and 4.4e-8; propagation blocking
// 9.8e-8 and 5.2e-8).  A launch of its own, 2-4 us: a fence and the same loop in
// the last CTA of the sweep slowed the sweep itself (Kronecker 24: 1,024 ->
// 1,056 us).
__global__ void rl_top_kernel(double* __restrict__ sum, const uint32_t* __restrict__ vertex, uint32_t n,
                              float* __restrict__ y) {
    const uint32_t k = threadIdx.x;
    if (k >= n) return;
    y[vertex[k]] = (float)sum[k];
    sum[k] = 0.0;
}

// ------------------------------------------------------------------ build --
// Entries per destination and, with `out`, per source (the half grid: the same counts).
__global__ void rl_count_kernel(const gs_unit* __restrict__ units, uint64_t n_units, const uint32_t* __restrict__ rec,
                                int directed, uint32_t* __restrict__ in, uint32_t* __restrict__ out) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t u = warp; u < n_units; u += n_warps) {
        const gs_unit un = units[u];
        const uint32_t rb = (un.rc >> 16) << 16, cb = (un.rc & 0xFFFFu) << 16;
        for (uint32_t k = lane; k < un.n; k += 32) {
            const uint32_t r = __ldcs(rec + un.rec_beg + k);
            const uint32_t a = rb + (r & 0xFFFFu), b = cb + (r >> 16);
            atomicAdd(in + b, 1u);
            if (!directed) atomicAdd(in + a, 1u);
            else if (out) atomicAdd(out + a, 1u);
        }
    }
}

// Vertices by count: one bin per count below kSmallCounts, 64 per power of two
// above, whose counts are added up too (no bin: zero).
constexpr uint32_t kSmallCounts = 4096, kBigCounts = 20 * 64;
struct RlHistogram {
    unsigned long long big_sum[kBigCounts];
    uint32_t small[kSmallCounts], big[kBigCounts];
};

__global__ void __launch_bounds__(1024) rl_histogram_kernel(const uint32_t* __restrict__ count, uint64_t N, RlHistogram* h) {
    __shared__ uint32_t s[kSmallCounts];
    for (uint32_t i = threadIdx.x; i < kSmallCounts; i += blockDim.x) s[i] = 0;
    __syncthreads();
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < N; v += nth) {
        const uint32_t c = count[v];
        if (c == 0) continue;
        if (c < kSmallCounts) {
            atomicAdd(s + c, 1u);
        } else {
            const uint32_t e = 31 - __clz(c), bin = (e - 12) * 64 + (c >> (e - 6) & 63);
            atomicAdd(h->big + bin, 1u);
            atomicAdd(h->big_sum + bin, (unsigned long long)c);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kSmallCounts; i += blockDim.x)
        if (s[i]) atomicAdd(h->small + i, s[i]);
}

// Entries of the k vertices of the highest counts (exact up to the part of a
// bin above kSmallCounts that k cuts off).
uint64_t top_entries(const RlHistogram& h, uint64_t k) {
    uint64_t sum = 0;
    for (uint32_t b = kBigCounts; b-- > 0 && k;) {
        const uint64_t n = std::min<uint64_t>(k, h.big[b]);
        if (n) sum += n == h.big[b] ? h.big_sum[b] : h.big_sum[b] / h.big[b] * n;
        k -= n;
    }
    for (uint32_t c = kSmallCounts; c-- > 1 && k;) {
        const uint64_t n = std::min<uint64_t>(k, h.small[c]);
        sum += n * c;
        k -= n;
    }
    return sum;
}

// Entries of the vertices of at least `least` < kSmallCounts.
uint64_t long_entries(const RlHistogram& h, uint32_t least) {
    uint64_t sum = 0;
    for (uint32_t b = 0; b < kBigCounts; ++b) sum += h.big_sum[b];
    for (uint32_t c = least; c < kSmallCounts; ++c) sum += (uint64_t)h.small[c] * c;
    return sum;
}

__global__ void rl_iota_kernel(uint32_t* v, uint64_t n) {
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth) v[i] = (uint32_t)i;
}

__global__ void rl_rank_kernel(const uint32_t* __restrict__ order, uint64_t n, uint32_t* __restrict__ rank) {
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth) rank[order[i]] = (uint32_t)i;
}

// First index of a falling array whose value is below `below`.
__device__ __forceinline__ uint64_t falling_bound(const uint32_t* c, uint64_t n, uint32_t below) {
    uint64_t lo = 0, hi = n;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (c[mid] >= below) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__global__ void rl_bounds_kernel(const uint32_t* in_sorted, const uint32_t* out_sorted, uint64_t n,
                                 unsigned long long* res) {
    if (threadIdx.x == 0) res[0] = falling_bound(in_sorted, n, 1);
    if (threadIdx.x == 1) res[1] = falling_bound(out_sorted, n, 1);
    if (threadIdx.x == 2) res[2] = falling_bound(in_sorted, n, kRlHeavy);
}

// Entry keys: destination rank above `pos_bits` bits of source position.
__global__ void rl_keys_kernel(const gs_unit* __restrict__ units, uint64_t n_units, const uint32_t* __restrict__ rec,
                               int directed, const uint32_t* __restrict__ rank_in, const uint32_t* __restrict__ rank_out,
                               int pos_bits, uint64_t* __restrict__ keys) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t u = warp; u < n_units; u += n_warps) {
        const gs_unit un = units[u];
        const uint32_t rb = (un.rc >> 16) << 16, cb = (un.rc & 0xFFFFu) << 16;
        for (uint32_t k = lane; k < un.n; k += 32) {
            const uint64_t e = un.rec_beg + k;
            const uint32_t r = __ldcs(rec + e);
            const uint32_t a = rb + (r & 0xFFFFu), b = cb + (r >> 16);
            const uint64_t to_b = ((uint64_t)__ldg(rank_in + b) << pos_bits) | __ldg(rank_out + a);
            if (directed) {
                __stcs(keys + e, to_b);
            } else {
                const uint64_t to_a = ((uint64_t)__ldg(rank_in + a) << pos_bits) | __ldg(rank_out + b);
                __stcs(reinterpret_cast<ulonglong2*>(keys) + e, make_ulonglong2(to_b, to_a));
            }
        }
    }
}

// First key of [lo, hi) whose source position is at least `pos`.
__device__ __forceinline__ uint64_t pos_bound(const uint64_t* __restrict__ keys, uint64_t lo, uint64_t hi,
                                              uint64_t pos, uint64_t mask) {
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if ((keys[mid] & mask) < pos) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Entries of the heavy rows in panels 0 .. kRlMaxPanels - 1 (a warp per row).
__global__ void rl_panel_kernel(const uint64_t* __restrict__ keys, const unsigned long long* __restrict__ start,
                                uint64_t n_heavy, uint64_t mask, unsigned long long* count) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    unsigned long long local[kRlMaxPanels / 32] = {};
    for (uint64_t r = warp; r < n_heavy; r += n_warps) {
        const uint64_t lo = start[r], hi = start[r + 1];
#pragma unroll
        for (uint32_t k = 0; k < kRlMaxPanels / 32; ++k) {
            const uint64_t p = 32 * k + lane;
            const uint64_t b = pos_bound(keys, lo, hi, p * kRlPanel, mask);
            const uint64_t n = pos_bound(keys, b, hi, (p + 1) * kRlPanel, mask) - b;
            const uint32_t few = __ballot_sync(0xFFFFFFFFu, p > 0 && n < kRlPanelRow);
            if (!(few & ((2u << lane) - 1u))) local[k] += n;
            if (few) break;   // uniform
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < kRlMaxPanels / 32; ++k)
        if (local[k]) atomicAdd(count + 32 * k + lane, local[k]);
}

// The segments of a row: fn(group, first entry, length).
template <class F>
__device__ __forceinline__ void row_segments(const uint64_t* __restrict__ keys, uint64_t lo, uint64_t hi,
                                             uint64_t mask, uint32_t n_panels, uint32_t seg, F fn) {
    auto cut = [&](uint32_t group, uint64_t b, uint64_t e) {
        for (; b < e; b += seg) fn(group, b, (uint32_t)(e - b < seg ? e - b : seg));
    };
    if (hi - lo < kRlHeavy) {
        cut(1, lo, hi);
        return;
    }
    uint64_t b = lo;
    for (uint32_t p = 0; p < n_panels; ++p) {
        const uint64_t e = pos_bound(keys, b, hi, (uint64_t)(p + 1) * kRlPanel, mask);
        if (p && e - b < kRlPanelRow) break;
        cut(p ? p + 2 : 2, b, e);
        b = e;
    }
    cut(0, b, hi);
}

__global__ void rl_segment_count_kernel(const uint64_t* __restrict__ keys, const unsigned long long* __restrict__ start,
                                        uint64_t n_rows, uint64_t mask, uint32_t n_panels, uint32_t seg,
                                        uint32_t* __restrict__ n) {
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= n_rows; r += nth) {
        uint32_t c = 0;
        if (r < n_rows)
            row_segments(keys, start[r], start[r + 1], mask, n_panels, seg, [&](uint32_t, uint64_t, uint32_t) { ++c; });
        n[r] = c;
    }
}

// Sort key of a segment: its group, then falling length.
__global__ void rl_segment_emit_kernel(const uint64_t* __restrict__ keys, const unsigned long long* __restrict__ start,
                                       uint64_t n_rows, uint64_t mask, uint32_t n_panels, uint32_t seg,
                                       const uint32_t* __restrict__ at, const uint32_t* __restrict__ vertex,
                                       uint32_t n_top, uint32_t* __restrict__ key, uint32_t* __restrict__ beg,
                                       uint32_t* __restrict__ row) {
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += nth) {
        uint32_t o = at[r];
        const uint32_t v = r < n_top ? kRlTop + (uint32_t)r : vertex[r];
        row_segments(keys, start[r], start[r + 1], mask, n_panels, seg, [&](uint32_t g, uint64_t b, uint32_t len) {
            key[o] = g * (kRlSegMax + 1) + (kRlSegMax - len);
            beg[o] = (uint32_t)b;
            row[o] = v;
            ++o;
        });
    }
}

struct RlGroups {
    uint32_t beg[kGroups + 1];     // sorted segments of group g: [beg[g], beg[g + 1])
    uint32_t slice[kGroups + 1];   // slices of group g
};

__global__ void rl_group_kernel(const uint32_t* __restrict__ key, uint32_t n, uint32_t* __restrict__ beg) {
    const uint32_t g = threadIdx.x;
    if (g > kGroups) return;
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (key[mid] < g * (kRlSegMax + 1)) lo = mid + 1;
        else hi = mid;
    }
    beg[g] = lo;
}

__device__ __forceinline__ uint32_t group_of_slice(const RlGroups& G, uint32_t s) {
    uint32_t g = 0;
    while (s >= G.slice[g + 1]) ++g;
    return g;
}

// Steps (16-byte groups per lane) of every slice; its first segment is its longest.
__global__ void rl_slice_kernel(const RlGroups G, uint32_t n_slices, const uint32_t* __restrict__ key,
                                uint8_t* __restrict__ n4, uint32_t* __restrict__ off) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s <= n_slices; s += nth) {
        uint32_t n = 0;
        if (s < n_slices) {
            const uint32_t g = group_of_slice(G, s);
            const uint32_t k = key[G.beg[g] + (s - G.slice[g]) * 32];
            n = (kRlSegMax - (k - g * (kRlSegMax + 1)) + 3) >> 2;
            n4[s] = (uint8_t)n;
        }
        off[s] = n;
    }
}

// A warp per slice: its segments' entries, transposed and padded.
__global__ void rl_fill_kernel(const RlGroups G, uint32_t n_slices, const uint32_t* __restrict__ key,
                               const uint32_t* __restrict__ idx, const uint32_t* __restrict__ beg,
                               const uint32_t* __restrict__ seg_row, const uint64_t* __restrict__ keys, uint64_t mask,
                               const uint8_t* __restrict__ n4, const uint32_t* __restrict__ off,
                               uint4* __restrict__ ent, uint32_t* __restrict__ row) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < n_slices; s += n_warps) {
        const uint32_t g = group_of_slice(G, s);
        const uint32_t i = G.beg[g] + (s - G.slice[g]) * 32 + lane;
        uint32_t len = 0, r = ~0u;
        uint64_t b = 0;
        if (i < G.beg[g + 1]) {
            len = kRlSegMax - (key[i] - g * (kRlSegMax + 1));
            const uint32_t k = idx[i];
            b = beg[k];
            r = seg_row[k];
        }
        row[(uint64_t)s * 32 + lane] = r;
        const uint32_t panel0 = g >= 3 ? (g - 2) * kRlPanel : 0u;
        auto one = [&](uint32_t k) -> uint32_t {
            if (k >= len) return kRlPanel;   // padding
            const uint32_t pos = (uint32_t)(keys[b + k] & mask);
            if (g >= 3) return pos - panel0;
            return pos < kRlPanel ? pos : pos + 1;
        };
        uint4* out = ent + (uint64_t)off[s] * 32 + lane;
        for (uint32_t k = 0; k < n4[s]; ++k) out[32 * k] = make_uint4(one(4 * k), one(4 * k + 1), one(4 * k + 2), one(4 * k + 3));
    }
}

// Whether a pulled sweep beats what the graph would use instead, in
// picoseconds per entry over the chip; at[0..2]: entries whose source is among
// the first kRlPanel, all panels' and kRlL2Sources sources (panel 0, the further
// panels of long rows, L2; the rest DRAM), at[3]: entries of the long rows.  About four fifths of what the long rows have beyond panel 0
// falls into panels they have enough entries in.  0.9 and 5.0 fit the sweeps
// above (Kronecker 24: 2.0 estimated, 1.8 measured; 26: 3.0 and 2.7; uniform,
// 3 M vertices: 5.0 and 5.4); propagation blocking measured 3.5-4.9, the row
// slices 7.5 and more.  Up to kPbPullSources vertices its bins may be pulled:
// 18.4 us per iteration against the row lists' 19.6 at 50,000 vertices and 16
// entries each, uniform (3.1 estimated), 20.5 against 20.6 at 80,000, 20.6
// against 24.5 at 120,000 (3.5), 32.4 against 41.4 at 400,000.
bool rl_worth(const gs_graph* g, uint64_t n_ent, const unsigned long long at[4]) {
    const double n = (double)n_ent, hot = at[0] / n, all = at[1] / n, l2 = at[2] / n, heavy = at[3] / n;
    const double staged = hot + 0.8 * heavy * (all - hot), far = 1.0 - l2;
    const double pull = 0.9 * staged + 5.0 * std::max(0.0, l2 - staged) + 24.0 * far;
    if (!pb_layout_wanted(g)) return pull <= 7.5;
    return pull <= (g->N <= kPbPullSources ? 3.4 : 3.7);
}

// Vertices by falling count: order[i], and counts in that order.
gs_status sort_by_count(Temps& T, const uint32_t* count, uint64_t N, uint32_t** order, uint32_t** sorted,
                        uint32_t** rank) {
    gs_ctx* ctx = T.ctx;
    uint32_t* ids = nullptr;
    GS_TRY(T.get(&ids, N));
    GS_TRY(T.get(order, N));
    GS_TRY(T.get(sorted, N));
    rl_iota_kernel<<<grid_for(N, ctx), 256, 0, ctx->stream>>>(ids, N);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    GS_TRY(cub_run(T, "row lists: vertex sort", [&](void* t, size_t& b) {
        return cub::DeviceRadixSort::SortPairsDescending(t, b, count, *sorted, ids, *order, N, 0, 32, ctx->stream);
    }));
    GS_TRY(T.get(rank, N));
    rl_rank_kernel<<<grid_for(N, ctx), 256, 0, ctx->stream>>>(*order, N, *rank);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches += 2;
    return GS_OK;
}

// Exclusive scan of `n` counts and, at [n], their total.
gs_status scan_counts(Temps& T, const uint32_t* count, uint64_t n, unsigned long long total, unsigned long long** out) {
    gs_ctx* ctx = T.ctx;
    GS_TRY(T.get(out, n + 1));
    GS_TRY(cub_run(T, "row lists: count scan", [&](void* t, size_t& b) {
        return cub::DeviceScan::ExclusiveSum(t, b, count, *out, n, ctx->stream);
    }));
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(*out + n, &total, 8, cudaMemcpyHostToDevice, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return GS_OK;
}

// Reorders the units of the groups 0, 1 and 2 so that each group's are spread
// evenly over the whole list.
void interleave(std::vector<gs_rl_unit>& units, const RlGroups& G) {
    std::vector<std::pair<double, uint32_t>> key(units.size());
    uint32_t n[3] = {0, 0, 0}, k[3] = {0, 0, 0};
    auto group = [&](const gs_rl_unit& u) { return u.slice < G.slice[1] ? 0 : u.slice < G.slice[2] ? 1 : 2; };
    for (const gs_rl_unit& u : units) n[group(u)]++;
    for (uint32_t i = 0; i < units.size(); ++i) {
        const int g = group(units[i]);
        key[i] = {(k[g]++ + 0.5) / n[g], i};
    }
    std::sort(key.begin(), key.end());
    std::vector<gs_rl_unit> out(units.size());
    for (uint32_t i = 0; i < units.size(); ++i) out[i] = units[key[i].second];
    units.swap(out);
}

gs_status build(gs_graph* g, bool* worth) {
    gs_ctx* ctx = g->ctx;
    gs_rl_layout& L = g->rl;
    const uint64_t N = g->N, n_ent = g->directed ? g->E : 2 * g->E;
    const uint32_t many = gs_grid_size(ctx, 8);

    // Entries per destination and source (what the graph counted itself is not
    // counted again), and from their histograms whether the lists are worth
    // building at all: nothing is reserved or sorted for a graph that another
    // layout sweeps faster.  Making a PageRank state, uniform random graphs that
    // end up with pulled bins, against reserving and sorting first: 24 M entries
    // over 3 M vertices (directed) 7.1 -> 6.4 ms, 6.4 M over 400,009 5.2 -> 4.4,
    // 64 M over 4 M 10.6 -> 8.4 (accumulated bins without an attempt: 6.7, 4.9, 10.6).
    const bool have_out = g->degree_from_records;   // undirected: the same as in
    const uint64_t n_counted = (g->directed ? 1 : 0) + (have_out ? 0 : 1);
    struct Counts {
        gs_ctx* ctx;
        char* p = nullptr;
        size_t bytes;
        ~Counts() { gs_pool_put(ctx, p, bytes); }
    } C{ctx, nullptr, 2 * sizeof(RlHistogram) + n_counted * N * 4};
    GS_TRY(gs_pool_get(ctx, C.bytes, (void**)&C.p));
    RlHistogram* d_hist = (RlHistogram*)C.p;
    uint32_t* const counted = (uint32_t*)(d_hist + 2);
    const uint32_t* const own = (const uint32_t*)g->d_degree;
    const uint32_t* in = n_counted ? counted : own;
    const uint32_t* out = !g->directed ? in : have_out ? own : counted + N;
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(C.p, 0, C.bytes, ctx->stream));
    if (n_counted) {
        rl_count_kernel<<<many, 256, 0, ctx->stream>>>(g->d_units, g->U, g->d_rec, g->directed, counted,
                                                       have_out ? nullptr : counted + N);
        GS_CHECK_CUDA(ctx, cudaGetLastError());
        ctx->launches++;
    }
    const uint32_t by_vertex = std::min(grid_for(N, ctx), gs_grid_size(ctx, 2));
    rl_histogram_kernel<<<by_vertex, 1024, 0, ctx->stream>>>(in, N, d_hist);
    if (g->directed) rl_histogram_kernel<<<by_vertex, 1024, 0, ctx->stream>>>(out, N, d_hist + 1);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches += g->directed ? 2 : 1;
    std::vector<RlHistogram> hist(g->directed ? 2 : 1);
    GS_TRY(to_host(ctx, hist.data(), d_hist, hist.size()));
    const RlHistogram& by_use = hist.back();
    const unsigned long long where[4] = {top_entries(by_use, kRlPanel), top_entries(by_use, (uint64_t)kRlPanel * kRlMaxPanels),
                                         top_entries(by_use, kRlL2Sources), long_entries(hist[0], kRlHeavy)};
    *worth = rl_worth(g, n_ent, where);
    if (!*worth) return GS_OK;

    Temps T(ctx);
    // two key buffers; orders and ranks; cub's scratch
    GS_TRY(T.reserve(n_ent * 16 + n_ent / 4 + N * (g->directed ? 48 : 32) + N * 12 + (8ull << 20)));
    uint32_t *row_order, *row_cnt, *row_rank, *src_order, *src_cnt, *src_rank;
    GS_TRY(sort_by_count(T, in, N, &row_order, &row_cnt, &row_rank));
    if (g->directed) {
        GS_TRY(sort_by_count(T, out, N, &src_order, &src_cnt, &src_rank));
    } else {
        src_order = row_order;
        src_cnt = row_cnt;
        src_rank = row_rank;
    }
    unsigned long long* d_res = nullptr;
    GS_TRY(T.get(&d_res, 128));
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(d_res, 0, 128 * 8, ctx->stream));
    rl_bounds_kernel<<<1, 32, 0, ctx->stream>>>(row_cnt, src_cnt, N, d_res);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    unsigned long long h[128];
    GS_TRY(to_host(ctx, h, d_res, 3));
    const uint64_t n_rows = h[0], n_src = h[1], n_heavy = h[2];

    unsigned long long* start = nullptr;
    GS_TRY(scan_counts(T, row_cnt, n_rows, n_ent, &start));
    unsigned long long* pushes = start;   // pushes by source, scanned
    if (g->directed) GS_TRY(scan_counts(T, src_cnt, n_src, n_ent, &pushes));
    GS_TRY(to_host(ctx, h, pushes + std::min<uint64_t>(kRlPanel, n_src), 1));
    const uint64_t hot = h[0];

    // the entries, sorted by destination rank, then by source panel
    const int pos_bits = std::max(bits_for(n_src), kSortSkip);
    const uint64_t mask = (1ull << pos_bits) - 1;
    uint64_t *k0 = nullptr, *k1 = nullptr;
    GS_TRY(T.get(&k0, n_ent));
    GS_TRY(T.get(&k1, n_ent));
    rl_keys_kernel<<<many, 256, 0, ctx->stream>>>(g->d_units, g->U, g->d_rec, g->directed, row_rank, src_rank, pos_bits,
                                                  k0);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    cub::DoubleBuffer<uint64_t> db(k0, k1);
    GS_TRY(cub_run(T, "row lists: entry sort", [&](void* t, size_t& b) {
        return cub::DeviceRadixSort::SortKeys(t, b, db, n_ent, kSortSkip, pos_bits + bits_for(n_rows), ctx->stream);
    }));
    const uint64_t* keys = db.Current();
    T.reuse(db.Alternate(), n_ent * 8);

    // panels: the first, and the next ones while the long rows have enough
    // entries in them to pay for a CTA's staging
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(d_res, 0, kRlMaxPanels * 8, ctx->stream));
    if (n_heavy) {
        rl_panel_kernel<<<many, 256, 0, ctx->stream>>>(keys, start, n_heavy, mask, d_res);
        GS_CHECK_CUDA(ctx, cudaGetLastError());
        ctx->launches++;
    }
    GS_TRY(to_host(ctx, h, d_res, kRlMaxPanels));
    uint32_t n_panels = 1;
    uint64_t in_panels = 0;
    while (n_panels < kRlMaxPanels && (uint64_t)n_panels * kRlPanel < n_src && h[n_panels] >= kRlPanelMin)
        in_panels += h[n_panels++];

    // segments no longer than leaves every warp of the chip a few of them
    const uint64_t warps = (uint64_t)ctx->num_sms * kRlWarps;
    uint32_t seg = 32;
    while (seg < kRlSegMax && (uint64_t)seg * 2 * 32 * warps * 2 <= n_ent) seg *= 2;
    uint32_t* at = nullptr;
    GS_TRY(T.get(&at, n_rows + 1));
    rl_segment_count_kernel<<<grid_for(n_rows + 1, ctx), 256, 0, ctx->stream>>>(keys, start, n_rows, mask, n_panels, seg,
                                                                                at);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    GS_TRY(cub_run(T, "row lists: segment scan", [&](void* t, size_t& b) {
        return cub::DeviceScan::ExclusiveSum(t, b, at, at, n_rows + 1, ctx->stream);
    }));
    uint32_t n_seg = 0;
    GS_TRY(to_host(ctx, &n_seg, at + n_rows, 1));
    const uint32_t n_top = g->N <= kRlTop ? (uint32_t)std::min<uint64_t>(n_heavy, kRlTopRows) : 0;
    uint32_t *sk0, *sk1, *si0, *si1, *sbeg, *srow;
    GS_TRY(T.get(&sk0, n_seg));
    GS_TRY(T.get(&sk1, n_seg));
    GS_TRY(T.get(&si0, n_seg));
    GS_TRY(T.get(&si1, n_seg));
    GS_TRY(T.get(&sbeg, n_seg));
    GS_TRY(T.get(&srow, n_seg));
    rl_segment_emit_kernel<<<grid_for(n_rows, ctx), 256, 0, ctx->stream>>>(keys, start, n_rows, mask, n_panels, seg, at,
                                                                           row_order, n_top, sk0, sbeg, srow);
    rl_iota_kernel<<<grid_for(n_seg, ctx), 256, 0, ctx->stream>>>(si0, n_seg);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches += 2;
    GS_TRY(cub_run(T, "row lists: segment sort", [&](void* t, size_t& b) {
        return cub::DeviceRadixSort::SortPairs(t, b, sk0, sk1, si0, si1, n_seg, 0,
                                               bits_for((uint64_t)kGroups * (kRlSegMax + 1)), ctx->stream);
    }));
    RlGroups G;
    uint32_t* d_gb = nullptr;
    GS_TRY(T.get(&d_gb, kGroups + 1));
    rl_group_kernel<<<1, 32 * ((kGroups + 32) / 32), 0, ctx->stream>>>(sk1, n_seg, d_gb);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    GS_TRY(to_host(ctx, G.beg, d_gb, kGroups + 1));
    G.slice[0] = 0;
    for (uint32_t k = 0; k < kGroups; ++k) G.slice[k + 1] = G.slice[k] + (G.beg[k + 1] - G.beg[k] + 31) / 32;
    const uint32_t n_slices = G.slice[kGroups];
    uint32_t* off = nullptr;
    GS_TRY(T.get(&off, (uint64_t)n_slices + 1));
    const uint64_t row_bytes = ((uint64_t)n_slices * 128 + 255) & ~255ull;
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_row, row_bytes + std::max<uint32_t>(1, n_slices)));
    L.d_n4 = (uint8_t*)L.d_row + row_bytes;
    rl_slice_kernel<<<grid_for((uint64_t)n_slices + 1, ctx), 256, 0, ctx->stream>>>(G, n_slices, sk1, L.d_n4, off);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    GS_TRY(cub_run(T, "row lists: slice scan", [&](void* t, size_t& b) {
        return cub::DeviceScan::ExclusiveSum(t, b, off, off, (uint64_t)n_slices + 1, ctx->stream);
    }));
    uint32_t steps = 0;
    GS_TRY(to_host(ctx, &steps, off + n_slices, 1));
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_ent, std::max<uint64_t>(1, steps) * 512));
    rl_fill_kernel<<<many, 256, 0, ctx->stream>>>(G, n_slices, sk1, si1, sbeg, srow, keys, mask, L.d_n4, off,
                                                  reinterpret_cast<uint4*>(L.d_ent), L.d_row);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches++;

    // units: up to 32 slices and about 64 steps for a warp to draw at a time,
    // fewer when the graph has not that many for every warp
    std::vector<uint8_t> n4(n_slices);
    GS_TRY(to_host(ctx, n4.data(), L.d_n4, n_slices));
    const uint32_t target = (uint32_t)std::clamp<uint64_t>(steps / (warps * 4), seg / 4, 64);
    std::vector<gs_rl_unit> units;
    uint32_t at_step = 0;
    double cost[kRlMaxPanels];
    for (uint32_t p = 0; p < n_panels; ++p) {
        const uint32_t s0 = p ? G.slice[p + 2] : 0, s1 = p ? G.slice[p + 3] : G.slice[3];
        const uint32_t step0 = at_step;
        L.unit_beg[p] = (uint32_t)units.size();
        for (uint32_t s = s0; s < s1;) {
            gs_rl_unit u{s, 0, at_step, 0};
            while (s < s1 && u.n_slices < 32 && (u.n_slices == 0 || u.steps + n4[s] <= target)) {
                u.steps += n4[s++];
                u.n_slices++;
            }
            at_step += u.steps;
            units.push_back(u);
        }
        // long rows' sources beyond panel 0 wait on L2, those inside it keep
        // the shared-memory pipe busy: both kinds are in flight all the time
        // when the three groups' units take turns
        if (p == 0) interleave(units, G);
        // time per entry: 1 from L2, 0.5 from shared memory.  (The load path's
        // clocks are 1 and 0.13, but what the panels' CTAs run into is latency:
        // with 0.13 they finished last, 265 against 240 us per iteration at
        // Kronecker 22, 1,070 against 1,045 at 24; 0.8 and 1.5 are no better.)
        const double cold = p ? 0.0 : (double)(n_ent - hot - std::min<uint64_t>(in_panels, n_ent - hot));
        cost[p] = cold + 0.5 * ((double)(at_step - step0) * 128 - cold);
    }
    L.unit_beg[n_panels] = (uint32_t)units.size();
    L.n_panels = n_panels;
    L.grid = (uint32_t)std::clamp<uint64_t>((units.size() + 7) / 8, n_panels, std::max(ctx->num_sms, (int)n_panels));
    // every panel's own CTAs (the others join in when they have none left)
    double sum = 0;
    for (uint32_t p = 0; p < n_panels; ++p) sum += cost[p];
    uint32_t used = 0;
    for (uint32_t p = n_panels; p-- > 1;) {
        const uint32_t left = L.grid - used - p;   // a CTA at least for each panel below
        L.home_beg[p] = std::max<uint32_t>(1, std::min<uint32_t>(left, (uint32_t)(cost[p] / sum * L.grid + 0.5)));
        used += L.home_beg[p];
    }
    L.home_beg[0] = L.grid - used;
    for (uint32_t p = 0, b = 0; p <= n_panels; ++p) {
        const uint32_t n = p < n_panels ? L.home_beg[p] : 0;
        L.home_beg[p] = b;
        b += n;
    }
    L.n_src = (uint32_t)n_src;
    L.n_entries = (uint64_t)steps * 128;
    const uint64_t xn = (n_src + 3) & ~3ull;
    const uint64_t x_bytes = (xn * 4 + 255) & ~255ull, src_bytes = (n_src * 4 + 255) & ~255ull;
    const uint64_t unit_bytes = (units.size() * sizeof(gs_rl_unit) + 255) & ~255ull;
    const uint64_t tick_bytes = ((kRlMaxPanels + 1) * 4 + 255) & ~255ull, top_bytes = (uint64_t)n_top * 12;
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_x, x_bytes + src_bytes + unit_bytes + tick_bytes + top_bytes));
    L.d_src = (uint32_t*)((char*)L.d_x + x_bytes);
    L.d_units = (gs_rl_unit*)((char*)L.d_src + src_bytes);
    L.d_tick = (unsigned int*)((char*)L.d_units + unit_bytes);
    L.d_top_sum = (double*)((char*)L.d_tick + tick_bytes);
    L.d_top = (uint32_t*)(L.d_top_sum + n_top);
    L.n_top = n_top;
    if (!units.empty())
        GS_CHECK_CUDA(ctx, cudaMemcpyAsync(L.d_units, units.data(), units.size() * sizeof(gs_rl_unit),
                                           cudaMemcpyHostToDevice, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(L.d_src, src_order, n_src * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(L.d_x, 0, x_bytes, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(L.d_tick, 0, tick_bytes + (uint64_t)n_top * 8, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(L.d_top, row_order, (uint64_t)n_top * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    L.built = true;
    return GS_OK;
}

}  // namespace

void rl_layout_free(gs_graph* g) {
    gs_rl_layout& L = g->rl;
    for (void* p : {(void*)L.d_ent, (void*)L.d_row, (void*)L.d_x}) gs_dev_free(p);
    L = gs_rl_layout();
}

bool rl_layout_wanted(const gs_graph* g) {
    if (g->stream || g->E == 0) return false;
    const uint64_t n_ent = g->directed ? g->E : 2 * g->E;
    if (n_ent >= (1ull << 32) - (1ull << 20)) return false;   // entry and step numbers are 32-bit
    // under an HBM budget the layout must fit beside the records
    const uint64_t keep = n_ent * 9 / 2 + g->N * 16;
    if (g->ctx->budget && 4 * g->E + keep > g->ctx->budget) return false;
    // building needs the sort's two key buffers, the vertex orders and the segment tables too
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return false;
    const uint64_t need = keep + n_ent * 16 + g->N * 64 + (2ull << 30);
    // (idle pool blocks count as free: an allocation that fails releases them)
    return free_b + g->ctx->pool_bytes > need;
}

gs_status rl_layout_build(gs_graph* g) {
    rl_layout_free(g);
    bool worth = false;
    const gs_status st = build(g, &worth);
    if (st != GS_OK || !worth) rl_layout_free(g);
    if (st == GS_OK && !worth) g->rl.refused = true;
    return st;
}

gs_status rl_launch(gs_state* s) {
    gs_graph* g = s->g;
    gs_ctx* ctx = g->ctx;
    const gs_rl_layout& L = g->rl;
    if (!s->d_error) {
        GS_TRY(gs_state_alloc(s, (void**)&s->d_error, sizeof(uint64_t)));
        GS_CHECK_CUDA(ctx, cudaMemsetAsync(s->d_error, 0, sizeof(uint64_t), ctx->stream));
    }
    const int smem = (int)(kRlPanel + 4) * 4;
    GS_CHECK_CUDA(ctx, gs_smem_limit_once<rl_pull_kernel>(ctx->device, smem));
    RlArgs a{reinterpret_cast<const uint4*>(L.d_ent), L.d_row, L.d_n4, L.d_units, L.d_x, s->d_y, L.n_src, L.n_panels,
             {}, {}, L.d_top_sum, L.n_top, L.d_tick, (int*)s->d_error};
    for (uint32_t p = 0; p <= L.n_panels; ++p) {
        a.unit_beg[p] = L.unit_beg[p];
        a.home_beg[p] = L.home_beg[p];
    }
    gs_timer_begin(ctx);
    rl_permute_kernel<<<grid_for(L.n_src, ctx), 256, 0, ctx->stream>>>(s->d_x, L.d_src, L.n_src, L.d_x);
    rl_pull_kernel<<<L.grid, kRlThreads, smem, ctx->stream>>>(a);
    if (L.n_top) {
        rl_top_kernel<<<1, kRlTopRows, 0, ctx->stream>>>(L.d_top_sum, L.d_top, L.n_top, s->d_y);
        ctx->launches++;
    }
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches += 2;
    // algorithmic bytes per iteration: 4E + 12V (records, x, s, inv)
    gs_timer_end(ctx, GS_ALGO_PAGERANK, 4 * g->E + 12 * g->V);
    return GS_OK;
}
