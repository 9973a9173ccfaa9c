// PageRank sweep by propagation blocking (sm_100a): pagerank_onepart
// (pr.cpp:119-154) for a large resident graph.
//
// Per record (v0, v1) of tile (i, j) the reference does
//     rank[v1] += prior[v0];   rank[v0] += prior[v1]   (the second: half grid)
// i.e. every record pushes x of one end into s of the other, once per
// direction.  At Kronecker scale 26 both ends are random over 268 MB arrays,
// so a sweep that touches x and s per record pays two random L2/DRAM
// operations per record, and the L1 pipe that issues them is the limit.
//
// Here a sweep is two streaming passes over a layout built once per graph
// (Beamer, Asanovic, Patterson, "Reducing PageRank Communication via
// Propagation Blocking", IPDPS 2017, restated for the tile grid):
//
//   * entries: one per (record, direction), sorted by (source slice S =
//     src >> 14, destination bin D = dst >> 14, dst, src).  Two u16 streams
//     hold the source's offset in its slice and the destination's offset in
//     its bin; the (S, D) blocks of the stream are contiguous, each padded to
//     a multiple of 8 entries (padding points past every destination);
//   * gather (pass 1): a CTA stages x of one source slice (16,384 floats,
//     64 KB) in shared memory with one bulk copy and streams the slice's
//     entries: val[e] = x[src of e] -- a shared-memory gather, a coalesced
//     16-bit read and a coalesced 32-bit write per entry;
//   * accumulate (pass 2): a CTA owns one destination bin (16,384 floats,
//     64 KB of shared memory), walks the bin's blocks (one per source slice,
//     D-major table, each cut into chunks of at most 256 entries, a
//     half-warp per chunk) and adds val[e] into its shared-memory sums at
//     the destination offset (equal destinations, adjacent in a block, are
//     summed in registers and across lanes first: one atomic per run), then
//     writes the bin's sums to y.
//
//   * pull (pass 2 of graphs without hubs up to kPbPullSources vertices): bins of
//     512 to 2,048 destinations whose values fit into shared memory together;
//     there a lane sums each destination's, through a list of 16-bit positions
//     in place of the destination offsets, without atomics.  Hardly two entries
//     of a block share a destination in such graphs, so every entry cost the
//     accumulate pass a compare-and-swap loop on a shared float.  Us per
//     iteration, accumulated against pulled (both with the gather): uniform,
//     3,000,017 vertices, 24 M entries 129 -> 100, 400,009 vertices, 6.4 M
//     entries 53 -> 32, 4 M vertices, 64 M entries 254 -> 209.  The gather takes 38
//     and the pull 47 of the 100, each moving its bytes at 3.8 TB/s.
//
// Both passes stream; the random accesses stay in shared memory.  DRAM bytes
// per entry and sweep: 2 (source offset) + 4 + 4 (value written and read) +
// 2 (destination offset) = 12, plus x, y and the block table.  The sums are
// re-associated per bin (FP32), which only changes rounding.
#include "gs_internal.cuh"
#include "gs_temps.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <vector>

namespace {

constexpr uint32_t kSrcSlice = 1u << kPbSrcBits;   // 16,384
constexpr uint32_t kDstBin = 1u << kPbDstBits;     // 16,384
constexpr int kKeyLowBits = kPbSrcBits + kPbDstBits;
constexpr int kGatherThreads = 512;
constexpr int kGatherCtas = 3;       // resident gather CTAs per SM (64 KB of x each)
constexpr int kGatherGroups = 2;     // 8-entry groups per gather thread and step (two steps in flight)
constexpr int kAccThreads = 512;
constexpr int kAccCtas = 3;          // resident accumulate CTAs per SM (the bin's sums each)
constexpr int kAccGroups = 2;        // 8-entry groups in flight per accumulate lane
constexpr int kPullThreads = 512;
constexpr int kPullCtas = 3;         // resident pull CTAs per SM (a bin's values and sums each)
constexpr uint32_t kPullVals = 17088;   // values of a bin, padding included: 66.8 KB
constexpr uint32_t kPullRows = 2048;    // most destinations of a bin
constexpr uint32_t kPullMinRows = 512;  // fewest: a strip of 32 for each of the 16 warps
constexpr uint32_t kPullRowMax = 128;   // longest row (a lane sums it alone)
constexpr uint32_t kPullSteps = 4;      // steps of a strip in flight
constexpr size_t kPullSmem = (kPullVals + 4 + kPullRows) * 4;
static_assert(kPullVals % 8 == 0 && kPullVals < 0xFFFFu, "positions are 16-bit");
constexpr long long kWaitLimit = 1ll << 24;
// Blocks are padded to a multiple of 8 entries; a padding entry points at
// offset 0 of its slice (its value is read and never added) and at
// destination kPadDst, past every offset of a bin.
constexpr uint16_t kPadDst = 0xFFFFu;
static_assert(kPbDstBits < 16, "kPadDst must lie past every destination offset");

struct __align__(128) GatherSmem {
    float xs[kSrcSlice];
    unsigned long long bar;
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

// Pass 1.  Item: entries [e0, e0 + n) of source slice `slice`.
__global__ void __launch_bounds__(kGatherThreads, kGatherCtas)
    pb_gather_kernel(const gs_pb_item1* __restrict__ items, uint64_t n_items, const uint16_t* __restrict__ src,
                     const float* __restrict__ x, float* __restrict__ val, int* error, unsigned int* ticket) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    GatherSmem& m = *reinterpret_cast<GatherSmem*>(smem_raw);
    const uint32_t tid = threadIdx.x;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&m.bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    uint32_t parity = 0;
    __shared__ unsigned long long s_item;
    auto advance = [&](uint64_t i) -> uint64_t {
        if (!ticket) return i + gridDim.x;
        __syncthreads();   // every thread has read the previous draw
        if (tid == 0) s_item = atomicAdd(ticket, 1u);
        __syncthreads();
        return s_item;
    };
    for (uint64_t i = ticket ? advance(0) : blockIdx.x; i < n_items; i = advance(i)) {
        const gs_pb_item1 it = items[i];
        if (tid == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&m.bar)),
                         "r"(kSrcSlice * 4)
                         : "memory");
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    smem_u32(m.xs)),
                "l"(x + ((uint64_t)it.slice << kPbSrcBits)), "r"(kSrcSlice * 4), "r"(smem_u32(&m.bar))
                : "memory");
        }
        const bool got = wait_bar(&m.bar, parity);
        parity ^= 1;
        if (!__syncthreads_and(got)) {
            // the copy is late: flag it and give it one more bounded wait, so
            // that the CTA does not leave with its copy still in flight
            if (tid == 0) {
                atomicExch(error, 1);
                wait_bar(&m.bar, parity ^ 1);
            }
            break;   // uniform
        }
        const uint64_t e0 = it.e0, end = it.e0 + it.n;
        // head up to a multiple of 8 entries, 8-entry body (16-byte loads,
        // two 16-byte stores), tail
        const uint64_t a = ((e0 + 7) & ~7ull) < end ? ((e0 + 7) & ~7ull) : end;
        const uint64_t b = (end & ~7ull) > a ? (end & ~7ull) : a;
        for (uint64_t e = e0 + tid; e < a; e += kGatherThreads) val[e] = m.xs[src[e]];
        for (uint64_t e = b + tid; e < end; e += kGatherThreads) val[e] = m.xs[src[e]];
        const uint4* s8 = reinterpret_cast<const uint4*>(src);
        float4* v4 = reinterpret_cast<float4*>(val);
        const uint64_t c1 = b >> 3;
        auto emit = [&](const uint4 w, uint64_t ck) {
            v4[2 * ck] = make_float4(m.xs[w.x & 0xFFFFu], m.xs[w.x >> 16], m.xs[w.y & 0xFFFFu], m.xs[w.y >> 16]);
            v4[2 * ck + 1] = make_float4(m.xs[w.z & 0xFFFFu], m.xs[w.z >> 16], m.xs[w.w & 0xFFFFu], m.xs[w.w >> 16]);
        };
        // the next groups' offsets are loaded before this one's are used, so
        // the loads overlap the shared-memory gathers and the stores
        constexpr uint64_t kStride = (uint64_t)kGatherThreads * kGatherGroups;
        uint4 w[kGatherGroups];
        uint64_t c = (a >> 3) + tid;
#pragma unroll
        for (int k = 0; k < kGatherGroups; ++k) {
            const uint64_t ck = c + (uint64_t)k * kGatherThreads;
            if (ck < c1) w[k] = __ldcs(s8 + ck);
        }
        for (; c < c1; c += kStride) {
            uint4 nw[kGatherGroups];
#pragma unroll
            for (int k = 0; k < kGatherGroups; ++k) {
                const uint64_t ck = c + kStride + (uint64_t)k * kGatherThreads;
                nw[k] = ck < c1 ? __ldcs(s8 + ck) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int k = 0; k < kGatherGroups; ++k) {
                const uint64_t ck = c + (uint64_t)k * kGatherThreads;
                if (ck < c1) emit(w[k], ck);
                w[k] = nw[k];
            }
        }
        __syncthreads();   // xs is rewritten by the next item
    }
    if (ticket && tid == 0 && atomicAdd(ticket + 1, 1u) == gridDim.x - 1) {
        atomicExch(ticket, 0u);   // every CTA has drawn its last ticket
        atomicExch(ticket + 1, 0u);
    }
}

// Adds the 8 entries of every lane of a group of W lanes (lane l of the W:
// the l-th 8-entry group of a window of the bin's group list, its entries
// sorted by destination; `valid` false for a lane past the item) into the
// shared sums.  Equal destinations are adjacent inside a group, and a run may
// cross lanes (a high-degree vertex can fill many groups of a block; two
// groups of neighbouring blocks may also end and start on one destination,
// whose sum is the same either way): a lane sums its runs in registers and
// adds the ones inside it at once; its first and last runs join the
// neighbouring lanes' runs through a segmented prefix scan over the W lanes,
// and each run is added once, by the lane where it ends.  Without the
// cross-lane step all lanes of a run would hit one address in the same
// atomic instruction.  Padding entries carry kPadDst (past every offset) and
// are never added.
template <int W>
__device__ __forceinline__ void add_lane_groups(float* acc, uint32_t hl, unsigned mask, bool valid, const uint4 d,
                                                const float4 lo, const float4 hi) {
    const uint32_t o[8] = {d.x & 0xFFFFu, d.x >> 16, d.y & 0xFFFFu, d.y >> 16,
                           d.z & 0xFFFFu, d.z >> 16, d.w & 0xFFFFu, d.w >> 16};
    const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    // in-lane runs: the first (f, sf) and the last (t, run) stay open, the
    // ones between them are added here
    const uint32_t f = valid ? o[0] : 0x10000u + hl;   // past any offset: links nothing
    uint32_t t = f;
    float run = valid ? v[0] : 0.f, sf = 0.f;
    bool single = true;
#pragma unroll
    for (int j = 1; j < 8; ++j) {
        if (!valid) break;
        if (o[j] != t) {
            if (single) sf = run;
            else if (t < kDstBin) atomicAdd(acc + t, run);
            single = false;
            t = o[j];
            run = v[j];
        } else {
            run += v[j];
        }
    }
    // lane l's first run continues lane l-1's last run when their keys match
    const uint32_t t_prev = __shfl_up_sync(mask, t, 1, W);
    const bool link = hl > 0 && t_prev == f;
    // segmented prefix sums of the last runs: a segment starts at a lane
    // whose first run does not continue the previous lane's, or whose first
    // run is not its last (its last run starts a new chain)
    float c = run;
    bool head = !single || !link;
#pragma unroll
    for (int k = 1; k < W; k <<= 1) {
        const float cu = __shfl_up_sync(mask, c, k, W);
        const bool hu = __shfl_up_sync(mask, head, k, W);
        if (hl >= (uint32_t)k && !head) {
            c += cu;
            head = hu;
        }
    }
    const float carry_in = __shfl_up_sync(mask, c, 1, W);
    const bool link_next = __shfl_down_sync(mask, link, 1, W) && hl < W - 1;
    if (!valid) return;
    if (!single && f < kDstBin) atomicAdd(acc + f, sf + (link ? carry_in : 0.f));   // first run, closed here
    if (!link_next && t < kDstBin) atomicAdd(acc + t, c);                          // the last run's chain ends here
}

// Pass 2.  Item: groups [b0, b1) of the group list, all of bin `bin`;
// `whole` when the item holds every group of the bin (its sums are then
// stored, else added to y).  A warp takes windows of 32 consecutive groups
// (a lane per group: one 4-byte group index, then one 16-byte load of
// destination offsets and two of values), kAccGroups windows in flight.
__global__ void __launch_bounds__(kAccThreads, kAccCtas)
    pb_accumulate_kernel(const gs_pb_item2* __restrict__ items, uint64_t n_items, const uint32_t* __restrict__ groups,
                         const uint16_t* __restrict__ dst, const float* __restrict__ val, float* __restrict__ y,
                         unsigned int* ticket) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* acc = reinterpret_cast<float*>(smem_raw);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr uint32_t kWarps = kAccThreads / 32;
    constexpr uint32_t kStep = 32 * kAccGroups;
    __shared__ unsigned long long s_item;
    auto advance = [&](uint64_t i) -> uint64_t {
        if (!ticket) return i + gridDim.x;
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(ticket, 1u);
        __syncthreads();
        return s_item;
    };
    float4* acc4 = reinterpret_cast<float4*>(acc);
    const uint4* d8 = reinterpret_cast<const uint4*>(dst);
    const float4* v4 = reinterpret_cast<const float4*>(val);
    for (uint64_t i = ticket ? advance(0) : blockIdx.x; i < n_items; i = advance(i)) {
        const gs_pb_item2 it = items[i];
        for (uint32_t k = tid; k < kDstBin / 4; k += kAccThreads) acc4[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        for (uint64_t w0 = (uint64_t)it.b0 + warp * kStep; w0 < it.b1; w0 += kWarps * kStep) {   // uniform in the warp
            uint32_t gi[kAccGroups];
#pragma unroll
            for (int k = 0; k < kAccGroups; ++k) {
                const uint64_t gk = w0 + 32u * k + lane;
                gi[k] = gk < it.b1 ? __ldcs(groups + gk) : 0u;
            }
            uint4 d[kAccGroups];
            float4 lo[kAccGroups], hi[kAccGroups];
#pragma unroll
            for (int k = 0; k < kAccGroups; ++k) {
                d[k] = make_uint4(0, 0, 0, 0);
                lo[k] = hi[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (w0 + 32u * k + lane < it.b1) {
                    d[k] = __ldcs(d8 + gi[k]);
                    lo[k] = __ldcs(v4 + 2 * (uint64_t)gi[k]);
                    hi[k] = __ldcs(v4 + 2 * (uint64_t)gi[k] + 1);
                }
            }
#pragma unroll
            for (int k = 0; k < kAccGroups; ++k)
                add_lane_groups<32>(acc, lane, 0xFFFFFFFFu, w0 + 32u * k + lane < it.b1, d[k], lo[k], hi[k]);
        }
        __syncthreads();
        float4* y4 = reinterpret_cast<float4*>(y + ((uint64_t)it.bin << kPbDstBits));
        for (uint32_t k = tid; k < kDstBin / 4; k += kAccThreads) {
            const float4 s = acc4[k];
            if (it.whole) y4[k] = s;
            else if (s.x != 0.f || s.y != 0.f || s.z != 0.f || s.w != 0.f) atomicAdd(y4 + k, s);
        }
        __syncthreads();   // acc is cleared by the next item
    }
    if (ticket && tid == 0 && atomicAdd(ticket + 1, 1u) == gridDim.x - 1) {
        atomicExch(ticket, 0u);
        atomicExch(ticket + 1, 0u);
    }
}

// Pass 2, pulled bins.  Item: bin b.  Its values are copied into shared memory
// (a thread per 8-entry group, 16-byte asynchronous copies), then a lane sums
// one destination's: 32 destinations of about one count to a strip, the
// positions of their entries transposed, four to a lane's 8-byte load.  Three
// CTAs per SM cover one another's copies; the next bin's groups are loaded, and
// its positions brought into L2, while this one is summed (50 -> 47 us of a 100
// us iteration at 24 M entries; 2 or 6 steps in flight instead of 4: the same).
__global__ void __launch_bounds__(kPullThreads, kPullCtas)
    pb_pull_kernel(const uint32_t* __restrict__ bin_group, uint32_t n_bins, const uint32_t* __restrict__ groups,
                   const uint32_t* __restrict__ strip_beg, const uint16_t* __restrict__ perm,
                   const uint16_t* __restrict__ idx, const float* __restrict__ val, float* __restrict__ y,
                   uint32_t bin_rows, uint64_t N, unsigned int* ticket) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* vals = reinterpret_cast<float*>(smem_raw);   // kPullVals, then the padding's zero
    float* sums = vals + kPullVals + 4;                 // bin_rows
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr uint32_t kWarps = kPullThreads / 32;
    constexpr uint32_t kCopies = (kPullVals / 8 + kPullThreads - 1) / kPullThreads;
    __shared__ uint32_t s_item;
    const uint2* idx2 = reinterpret_cast<const uint2*>(idx);
    const uint32_t strips = bin_rows / 32;
    if (tid == 0) {
        vals[kPullVals] = 0.f;
        s_item = ticket ? atomicAdd(ticket, 1u) : blockIdx.x;
    }
    __syncthreads();
    uint32_t b = s_item, n = 0, gi[kCopies];
    // the groups of bin d, and its positions into L2
    auto fetch = [&](uint32_t d) {
        const uint32_t g0 = bin_group[d];
        n = bin_group[d + 1] - g0;   // <= kPullVals / 8 (pb_pull_build)
#pragma unroll
        for (uint32_t k = 0; k < kCopies; ++k) {
            const uint32_t at = tid + k * kPullThreads;
            gi[k] = at < n ? __ldcs(groups + g0 + at) : 0u;
        }
        const uint32_t q1 = strip_beg[(d + 1) * strips];
        for (uint32_t q = strip_beg[d * strips] + tid; q < q1; q += kPullThreads)   // a step is 256 bytes
            asm volatile("prefetch.global.L2 [%0];\n\tprefetch.global.L2 [%1];" ::"l"(idx2 + (uint64_t)q * 32),
                         "l"(idx2 + (uint64_t)q * 32 + 16));
    };
    __syncthreads();   // s_item has been read
    if (b < n_bins) fetch(b);
    while (b < n_bins) {
#pragma unroll
        for (uint32_t k = 0; k < kCopies; ++k) {
            const uint32_t at = tid + k * kPullThreads;
            if (at < n) {
                const uint32_t to = smem_u32(vals + 8 * at);
                const float* from = val + 8 * (uint64_t)gi[k];
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16), "l"(from + 4) : "memory");
            }
        }
        if (tid == 0) s_item = ticket ? atomicAdd(ticket, 1u) : b + gridDim.x;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const uint32_t next = s_item;   // written again after the barrier below
        if (next < n_bins) fetch(next);
        for (uint32_t k = warp; k < strips; k += kWarps) {
            const uint32_t st = b * strips + k, s1 = strip_beg[st + 1];
            const uint16_t row = perm[st * 32 + lane];
            float sum = 0.f;
            for (uint32_t q = strip_beg[st]; q < s1; q += kPullSteps) {   // uniform in the warp
                uint2 w[kPullSteps];
#pragma unroll
                for (uint32_t j = 0; j < kPullSteps; ++j)
                    if (q + j < s1) w[j] = __ldcs(idx2 + (uint64_t)(q + j) * 32 + lane);
#pragma unroll
                for (uint32_t j = 0; j < kPullSteps; ++j)
                    if (q + j < s1)
                        sum += (vals[w[j].x & 0xFFFFu] + vals[w[j].x >> 16]) + (vals[w[j].y & 0xFFFFu] + vals[w[j].y >> 16]);
            }
            sums[row] = sum;
        }
        __syncthreads();
        // (the next bin's first barrier stands between this read of sums and the next write)
        const uint64_t v0 = (uint64_t)b * bin_rows;
        const uint32_t rows = (uint32_t)(N - v0 < bin_rows ? N - v0 : bin_rows);   // a multiple of 32, as N is
        const float4* s4 = reinterpret_cast<const float4*>(sums);
        float4* y4 = reinterpret_cast<float4*>(y + v0);
        for (uint32_t k = tid; k < rows / 4; k += kPullThreads) y4[k] = s4[k];
        b = next;
    }
    if (ticket && tid == 0 && atomicAdd(ticket + 1, 1u) == gridDim.x - 1) {
        atomicExch(ticket, 0u);
        atomicExch(ticket + 1, 0u);
    }
}

// ------------------------------------------------------------------ build --
// One key per (record, direction): (S * nD + D) above kKeyLowBits, then the
// destination's and the source's offsets.
__device__ __forceinline__ uint64_t pb_key(uint32_t src, uint32_t dst, uint32_t nD, uint32_t bin_rows) {
    const uint32_t D = dst / bin_rows;
    const uint64_t blk = (uint64_t)(src >> kPbSrcBits) * nD + D;
    return (blk << kKeyLowBits) | ((uint64_t)(dst - D * bin_rows) << kPbSrcBits) | (src & (kSrcSlice - 1));
}

__global__ void pb_keys_kernel(const gs_unit* __restrict__ units, uint64_t n_units, const uint32_t* __restrict__ rec,
                               uint32_t nD, uint32_t bin_rows, int directed, uint64_t* __restrict__ keys) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t u = warp; u < n_units; u += n_warps) {
        const gs_unit un = units[u];
        const uint32_t rb = (un.rc >> 16) << 16, cb = (un.rc & 0xFFFFu) << 16;
        for (uint32_t k = lane; k < un.n; k += 32) {
            const uint64_t e = un.rec_beg + k;
            const uint32_t r = rec[e];
            const uint32_t a = rb + (r & 0xFFFFu), b = cb + (r >> 16);
            if (directed) {
                keys[e] = pb_key(a, b, nD, bin_rows);                  // push v0 -> v1 only (pr.cpp:141-146)
            } else {
                keys[2 * e] = pb_key(a, b, nD, bin_rows);              // rank[v1] += prior[v0]
                keys[2 * e + 1] = pb_key(b, a, nD, bin_rows);          // rank[v0] += prior[v1]
            }
        }
    }
}

// Block counts rounded up to 8 entries: pc[bid] (bid < n_blk), pc[n_blk] = 0.
__global__ void pb_padded_count_kernel(const uint64_t* __restrict__ start, uint64_t n_blk, uint64_t* __restrict__ pc) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t bid = tid; bid <= n_blk; bid += nth)
        pc[bid] = bid < n_blk ? (start[bid + 1] - start[bid] + 7) & ~7ull : 0;
}

// The sorted keys of block bid go to the padded streams at pstart[bid]
// (source and destination offsets), then the block's padding entries (a warp
// per block).
__global__ void pb_split_kernel(const uint64_t* __restrict__ keys, const uint64_t* __restrict__ start,
                                const uint64_t* __restrict__ pstart, uint64_t n_blk, uint16_t* __restrict__ src,
                                uint16_t* __restrict__ dst) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t bid = warp; bid < n_blk; bid += n_warps) {
        const uint64_t s0 = start[bid], n = start[bid + 1] - s0, p0 = pstart[bid], pn = pstart[bid + 1] - p0;
        for (uint64_t k = lane; k < pn; k += 32) {
            if (k < n) {
                const uint64_t key = keys[s0 + k];
                src[p0 + k] = (uint16_t)(key & (kSrcSlice - 1));
                dst[p0 + k] = (uint16_t)((key >> kPbSrcBits) & (kDstBin - 1));
            } else {
                src[p0 + k] = 0;
                dst[p0 + k] = kPadDst;
            }
        }
    }
}

// First entry of every block id in [0, n_blk] (n_blk: one past the last):
// a binary search over the sorted keys.
__global__ void pb_block_start_kernel(const uint64_t* __restrict__ keys, uint64_t n, uint64_t n_blk,
                                      uint64_t* __restrict__ start) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t bid = tid; bid <= n_blk; bid += nth) {
        uint64_t lo = 0, hi = n;
        while (lo < hi) {
            const uint64_t mid = (lo + hi) >> 1;
            if ((keys[mid] >> kKeyLowBits) < bid) lo = mid + 1;
            else hi = mid;
        }
        start[bid] = lo;
    }
}

// The D-major block table: blocks[D * nS + S] = block (S, D).
__global__ void pb_block_table_kernel(const uint64_t* __restrict__ start, uint32_t nS, uint32_t nD,
                                      gs_pb_block* __restrict__ blocks) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n_blk = (uint64_t)nS * nD;
    for (uint64_t p = tid; p < n_blk; p += nth) {
        const uint64_t D = p / nS, S = p % nS, bid = S * nD + D;
        blocks[p] = gs_pb_block{start[bid], (uint32_t)(start[bid + 1] - start[bid]), 0u};
    }
}

// The group list: block p of the D-major table (entries [e0, e0 + n), n a
// multiple of 8) lists its groups e0/8 .. (e0 + n)/8 - 1 from gpos[p] on.
// A warp per block.
__global__ void pb_group_list_kernel(const gs_pb_block* __restrict__ blocks, const uint64_t* __restrict__ gpos,
                                     uint64_t n_blk, uint32_t* __restrict__ groups) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t p = warp; p < n_blk; p += n_warps) {
        const gs_pb_block b = blocks[p];
        const uint64_t g0 = b.e0 >> 3, out = gpos[p];
        for (uint32_t k = lane; k < (b.n >> 3); k += 32) groups[out + k] = (uint32_t)(g0 + k);
    }
}

// In-entries of every vertex.
__global__ void pb_count_kernel(const gs_unit* __restrict__ units, uint64_t n_units, const uint32_t* __restrict__ rec,
                                int directed, uint32_t* __restrict__ count) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t u = warp; u < n_units; u += n_warps) {
        const gs_unit un = units[u];
        const uint32_t rb = (un.rc >> 16) << 16, cb = (un.rc & 0xFFFFu) << 16;
        for (uint32_t k = lane; k < un.n; k += 32) {
            const uint32_t r = rec[un.rec_beg + k];
            atomicAdd(count + cb + (r >> 16), 1u);
            if (!directed) atomicAdd(count + rb + (r & 0xFFFFu), 1u);
        }
    }
}

// Pulled bins: most[0] = the longest row, most[1] = the fullest bin's entries
// (a warp per bin).
__global__ void pb_bin_max_kernel(const uint32_t* __restrict__ count, uint64_t N, uint32_t bin_rows, uint32_t n_bins,
                                  uint32_t* __restrict__ most) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < n_bins; b += n_warps) {
        const uint64_t v0 = (uint64_t)b * bin_rows;
        unsigned long long sum = 0;
        uint32_t row = 0;
        for (uint64_t v = v0 + lane; v < v0 + bin_rows && v < N; v += 32) {
            sum += count[v];
            row = max(row, count[v]);
        }
        for (int o = 16; o; o >>= 1) {
            sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
            row = max(row, __shfl_xor_sync(0xFFFFFFFFu, row, o));
        }
        if (lane == 0) {
            atomicMax(most, row);
            atomicMax(most + 1, (uint32_t)min(sum, 0xFFFFFFFFull));
        }
    }
}

// Sort keys of the rows: by bin, then by falling count.
__global__ void pb_row_key_kernel(const uint32_t* __restrict__ count, uint64_t N, uint32_t n_rows, uint32_t bin_rows,
                                  uint32_t* __restrict__ key, uint32_t* __restrict__ row) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n_rows; v += nth) {
        key[v] = ((v / bin_rows) << 8) | (kPullRowMax - (v < N ? count[v] : 0u));
        row[v] = v;
    }
}

// Rows in order: rank and offset of each, steps of 4 entries of each strip.
__global__ void pb_row_rank_kernel(const uint32_t* __restrict__ key, const uint32_t* __restrict__ row, uint32_t n_rows,
                                   uint32_t bin_rows, uint16_t* __restrict__ rank, uint16_t* __restrict__ perm,
                                   uint32_t* __restrict__ steps) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n_rows; q += nth) {
        const uint32_t b = q / bin_rows, v = row[q];   // every bin has bin_rows rows
        rank[v] = (uint16_t)(q - b * bin_rows);
        perm[q] = (uint16_t)(v - b * bin_rows);
        if ((q & 31) == 0) steps[q / 32] = (kPullRowMax - (key[q] & 0xFFu) + 3) / 4;
        if (q == 0) steps[n_rows / 32] = 0;
    }
}

// Groups of the blocks, bin by bin: n[D * nS + S] = those of block (S, D).
__global__ void pb_group_count_kernel(const uint64_t* __restrict__ pstart, uint32_t nS, uint32_t nD,
                                      uint32_t* __restrict__ n) {
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x, n_blk = (uint64_t)nS * nD;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p <= n_blk; p += nth) {
        const uint64_t bid = p % nS * nD + p / nS;
        n[p] = p < n_blk ? (uint32_t)((pstart[bid + 1] - pstart[bid]) >> 3) : 0u;
    }
}

__global__ void pb_bin_group_kernel(const uint32_t* __restrict__ gpos, uint32_t nS, uint32_t nD,
                                    uint32_t* __restrict__ bin_group) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d <= nD; d += nth) bin_group[d] = gpos[(uint64_t)d * nS];
}

__global__ void pb_pad_kernel(uint32_t* __restrict__ idx2, uint64_t n) {
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += nth)
        idx2[k] = kPullVals | (kPullVals << 16);
}

// Pulled bins: block bid's sources to the padded stream, its groups to its
// bin's list, and every entry's position in the bin to its row (a warp per
// block; the order inside a row is that of the atomics).
__global__ void pb_pull_split_kernel(const uint64_t* __restrict__ keys, const uint64_t* __restrict__ start,
                                     const uint64_t* __restrict__ pstart, const uint32_t* __restrict__ gpos,
                                     uint32_t nS, uint32_t nD, uint32_t bin_rows, const uint16_t* __restrict__ rank,
                                     const uint32_t* __restrict__ strip_beg, uint32_t* __restrict__ cursor,
                                     uint16_t* __restrict__ src, uint32_t* __restrict__ groups,
                                     uint16_t* __restrict__ idx) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t bid = warp; bid < (uint64_t)nS * nD; bid += n_warps) {
        const uint64_t s0 = start[bid], n = start[bid + 1] - s0, p0 = pstart[bid], pn = pstart[bid + 1] - p0;
        const uint32_t D = (uint32_t)(bid % nD), S = (uint32_t)(bid / nD);
        const uint32_t g0 = gpos[(uint64_t)D * nS + S], at = (g0 - gpos[(uint64_t)D * nS]) * 8;
        for (uint64_t k = lane; k < pn; k += 32) {
            if ((k & 7) == 0) groups[g0 + (k >> 3)] = (uint32_t)((p0 + k) >> 3);
            if (k >= n) {
                src[p0 + k] = 0;
                continue;
            }
            const uint64_t key = keys[s0 + k];
            src[p0 + k] = (uint16_t)(key & (kSrcSlice - 1));
            const uint32_t v = D * bin_rows + ((uint32_t)(key >> kPbSrcBits) & (kDstBin - 1));
            const uint32_t r = rank[v], j = atomicAdd(cursor + v, 1u);
            const uint64_t step = strip_beg[D * (bin_rows / 32) + r / 32] + j / 4;
            idx[step * 128 + (r & 31) * 4 + (j & 3)] = (uint16_t)(at + k);
        }
    }
}

// Gather items of the slices, whose entries start at slice_start[0 .. nS].
// An item pays for staging its slice, so it holds 32,768 entries at least --
// unless that leaves the CTAs less than two items each (pulled bins, uniform,
// us per iteration: 400,009 vertices, 6.4 M entries 34.8 -> 32.8; 1,000,003 and
// 3,000,017 vertices of 8 entries, directed, 46.2 -> 43.9 and 102.9 -> 99.5).
std::vector<gs_pb_item1> gather_items(const gs_ctx* ctx, const std::vector<uint64_t>& slice_start) {
    const uint64_t ctas = (uint64_t)ctx->num_sms * kGatherCtas, n_pad = slice_start.back();
    const uint64_t per =
        std::clamp<uint64_t>(n_pad / (ctas * 4), std::clamp<uint64_t>(n_pad / (ctas * 2), 8192, 32768), 1ull << 20) &
        ~7ull;
    std::vector<gs_pb_item1> items;
    for (uint32_t s = 0; s + 1 < slice_start.size(); ++s)
        for (uint64_t e = slice_start[s]; e < slice_start[s + 1]; e += per)
            items.push_back(gs_pb_item1{e, (uint32_t)std::min<uint64_t>(per, slice_start[s + 1] - e), s});
    return items;
}

// Destinations per pulled bin, 0 where bins are accumulated.  A bin's values
// must fit into shared memory whatever the padding of its nS blocks (7 entries
// each at most), which is checked on the counted entries; blocks should hold 32
// entries on average and more (padding 11 %), a bin a strip for each of its
// warps, and no row keep a lane busy for long.
uint32_t pb_pull_rows(const gs_graph* g, uint64_t n_ent, uint64_t nS) {
    if (g->N > kPbPullSources || g->ctx->budget) return 0;
    const double mean = (double)n_ent / (double)std::max<uint64_t>(1, g->V);
    const double room = (double)kPullVals - 7.0 * (double)nS;
    uint64_t rows = kPullRows;
    while (rows >= kPullMinRows && rows * mean + 5.0 * std::sqrt(rows * mean) > room) rows -= 32;
    if (rows < kPullMinRows || rows * mean < 32.0 * (double)nS) return 0;
    const uint64_t n_bins = (g->N + rows - 1) / rows, n_blk = nS * n_bins;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return 0;
    const uint64_t need = n_ent * 32 + n_blk * 64 + g->N * 40 + (2ull << 30);
    return free_b + g->ctx->pool_bytes > need ? (uint32_t)rows : 0;
}

// The layout with pulled bins of `rows` destinations; *fits is false, and
// nothing is kept, when a row or a bin is too long for it.
gs_status pb_pull_build(gs_graph* g, uint32_t rows, bool* fits) {
    gs_ctx* ctx = g->ctx;
    gs_pb_layout& L = g->pb;
    const uint64_t n_ent = g->directed ? g->E : 2 * g->E;
    const uint32_t nS = (uint32_t)(g->N >> kPbSrcBits), nD = (uint32_t)((g->N + rows - 1) / rows), R = nD * rows;
    const uint64_t n_blk = (uint64_t)nS * nD;
    const uint32_t many = gs_grid_size(ctx, 8);
    Temps T(ctx);
    GS_TRY(T.reserve(n_ent * 17 + n_blk * 24 + (uint64_t)R * 28 + (4ull << 20)));
    uint32_t* most = nullptr;
    GS_TRY(T.get(&most, 2));
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(most, 0, 8, ctx->stream));
    const uint32_t* count = (const uint32_t*)g->d_degree;
    if (g->directed || !g->degree_from_records) {   // else the graph has counted them
        uint32_t* counted = nullptr;
        GS_TRY(T.get(&counted, g->N));
        GS_CHECK_CUDA(ctx, cudaMemsetAsync(counted, 0, g->N * 4, ctx->stream));
        pb_count_kernel<<<many, 256, 0, ctx->stream>>>(g->d_units, g->U, g->d_rec, g->directed, counted);
        GS_CHECK_CUDA(ctx, cudaGetLastError());
        ctx->launches++;
        count = counted;
    }
    pb_bin_max_kernel<<<many, 256, 0, ctx->stream>>>(count, g->N, rows, nD, most);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    uint32_t h_most[2];
    GS_TRY(to_host(ctx, h_most, most, 2));
    *fits = h_most[0] <= kPullRowMax && h_most[1] + 7ull * nS <= kPullVals;
    if (!*fits) return GS_OK;

    // rows by bin and falling count
    uint32_t *rk0, *rk1, *rv0, *rv1, *steps;
    uint16_t* rank;
    GS_TRY(T.get(&rk0, R));
    GS_TRY(T.get(&rk1, R));
    GS_TRY(T.get(&rv0, R));
    GS_TRY(T.get(&rv1, R));
    GS_TRY(T.get(&rank, R));
    GS_TRY(T.get(&steps, R / 32 + 1));
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_perm, (uint64_t)R * 2));
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_strip, ((uint64_t)R / 32 + 1) * 4));
    pb_row_key_kernel<<<grid_for(R, ctx), 256, 0, ctx->stream>>>(count, g->N, R, rows, rk0, rv0);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    GS_TRY(cub_run(T, "pulled bins: row sort", [&](void* t, size_t& b) {
        return cub::DeviceRadixSort::SortPairs(t, b, rk0, rk1, rv0, rv1, R, 0, 8 + bits_for(nD), ctx->stream);
    }));
    pb_row_rank_kernel<<<grid_for(R, ctx), 256, 0, ctx->stream>>>(rk1, rv1, R, rows, rank, L.d_perm, steps);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    GS_TRY(cub_run(T, "pulled bins: step scan", [&](void* t, size_t& b) {
        return cub::DeviceScan::ExclusiveSum(t, b, steps, L.d_strip, R / 32 + 1, ctx->stream);
    }));
    ctx->launches += 2;

    // entries by block, in any order inside one
    uint64_t *k0, *k1, *start, *pstart;
    uint32_t *gcount, *gpos;
    GS_TRY(T.get(&k0, n_ent));
    GS_TRY(T.get(&k1, n_ent));
    GS_TRY(T.get(&start, n_blk + 1));
    GS_TRY(T.get(&pstart, n_blk + 1));
    GS_TRY(T.get(&gcount, n_blk + 1));
    GS_TRY(T.get(&gpos, n_blk + 1));
    pb_keys_kernel<<<many, 256, 0, ctx->stream>>>(g->d_units, g->U, g->d_rec, nD, rows, g->directed, k0);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    cub::DoubleBuffer<uint64_t> db(k0, k1);
    GS_TRY(cub_run(T, "pulled bins: entry sort", [&](void* t, size_t& b) {
        return cub::DeviceRadixSort::SortKeys(t, b, db, n_ent, kKeyLowBits, kKeyLowBits + bits_for(n_blk), ctx->stream);
    }));
    const uint64_t* keys = db.Current();
    pb_block_start_kernel<<<grid_for(n_blk + 1, ctx), 256, 0, ctx->stream>>>(keys, n_ent, n_blk, start);
    pb_padded_count_kernel<<<grid_for(n_blk + 1, ctx), 256, 0, ctx->stream>>>(start, n_blk, pstart);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    GS_TRY(cub_run(T, "pulled bins: block scan", [&](void* t, size_t& b) {
        return cub::DeviceScan::ExclusiveSum(t, b, pstart, pstart, n_blk + 1, ctx->stream);
    }));
    pb_group_count_kernel<<<grid_for(n_blk + 1, ctx), 256, 0, ctx->stream>>>(pstart, nS, nD, gcount);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    GS_TRY(cub_run(T, "pulled bins: group scan", [&](void* t, size_t& b) {
        return cub::DeviceScan::ExclusiveSum(t, b, gcount, gpos, n_blk + 1, ctx->stream);
    }));
    ctx->launches += 4;
    std::vector<uint64_t> slice_start(nS + 1);
    GS_CHECK_CUDA(ctx, cudaMemcpy2DAsync(slice_start.data(), 8, pstart, (size_t)nD * 8, 8, nS + 1, cudaMemcpyDeviceToHost,
                                         ctx->stream));
    uint32_t n_steps = 0;
    GS_TRY(to_host(ctx, &n_steps, L.d_strip + R / 32, 1));
    const uint64_t n_pad = slice_start[nS];
    const std::vector<gs_pb_item1> items = gather_items(ctx, slice_start);
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_src, n_pad * 2));
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_val, n_pad * 4));
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_groups, n_pad / 2));
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_idx, std::max<uint64_t>(1, n_steps) * 256));
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_bin_group, ((uint64_t)nD + 1) * 4));
    GS_TRY(gs_dev_alloc(ctx, (void**)&L.d_items1, std::max<size_t>(1, items.size()) * sizeof(gs_pb_item1)));
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(rk0, 0, (uint64_t)R * 4, ctx->stream));   // now the rows' cursors
    pb_pad_kernel<<<many, 256, 0, ctx->stream>>>((uint32_t*)L.d_idx, (uint64_t)n_steps * 64);
    pb_pull_split_kernel<<<many, 256, 0, ctx->stream>>>(keys, start, pstart, gpos, nS, nD, rows, rank, L.d_strip, rk0,
                                                        L.d_src, L.d_groups, L.d_idx);
    pb_bin_group_kernel<<<grid_for(nD + 1, ctx), 256, 0, ctx->stream>>>(gpos, nS, nD, L.d_bin_group);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches += 3;
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(L.d_items1, items.data(), items.size() * sizeof(gs_pb_item1),
                                       cudaMemcpyHostToDevice, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    L.n_entries = n_pad;
    L.n_groups = n_pad / 8;
    L.n_items1 = items.size();
    L.n_items2 = nD;
    L.bin_rows = rows;
    L.built = true;
    return GS_OK;
}

// The second pass on stream q, with or without a ticket.
cudaError_t second_pass(const gs_graph* g, const float* val, float* y, unsigned int* ticket, cudaStream_t q) {
    const gs_ctx* ctx = g->ctx;
    const gs_pb_layout& L = g->pb;
    uint32_t grid = (uint32_t)L.n_items2;
    if (L.bin_rows) {
        const cudaError_t e = gs_smem_limit_once<pb_pull_kernel>(ctx->device, (int)kPullSmem);
        if (e != cudaSuccess) return e;
        if (ticket) grid = std::min(grid, gs_grid_size(ctx, kPullCtas));
        pb_pull_kernel<<<grid, kPullThreads, kPullSmem, q>>>(L.d_bin_group, (uint32_t)L.n_items2, L.d_groups, L.d_strip,
                                                             L.d_perm, L.d_idx, val, y, L.bin_rows, g->N, ticket);
    } else {
        const cudaError_t e = gs_smem_limit_once<pb_accumulate_kernel>(ctx->device, (int)(kDstBin * 4));
        if (e != cudaSuccess) return e;
        if (ticket) grid = std::min(grid, gs_grid_size(ctx, kAccCtas));
        pb_accumulate_kernel<<<grid, kAccThreads, kDstBin * 4, q>>>(L.d_items2, L.n_items2, L.d_groups, L.d_dst, val, y,
                                                                    ticket);
    }
    return cudaGetLastError();
}

}  // namespace

void pb_layout_free(gs_graph* g) {
    gs_pb_layout& L = g->pb;
    gs_dev_free(L.d_src);
    gs_dev_free(L.d_dst);
    gs_dev_free(L.d_val);
    gs_dev_free(L.d_groups);
    gs_dev_free(L.d_items1);
    gs_dev_free(L.d_items2);
    gs_dev_free(L.d_bin_group);
    gs_dev_free(L.d_strip);
    gs_dev_free(L.d_perm);
    gs_dev_free(L.d_idx);
    L = gs_pb_layout();
}

bool pb_layout_wanted(const gs_graph* g) {
    if (g->stream || g->E == 0) return false;
    const uint64_t n_ent = g->directed ? g->E : 2 * g->E;
    const uint64_t nS = g->N >> kPbSrcBits, nD = g->N >> kPbDstBits;
    // the block table is dense (every (S, D) pair): worth it when blocks hold
    // many entries on average; group indices (entry / 8) are 32-bit
    if (nS * nD * 64 > n_ent || nS * nD >= (1ull << 31) || n_ent + 8 * nS * nD >= (1ull << 34)) return false;
    // under an HBM budget the layout (8 B per entry) must fit beside the records
    if (g->ctx->budget && 4 * g->E + 8 * n_ent > g->ctx->budget) return false;
    // building needs the sort's two key buffers too
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return false;
    const uint64_t need = (n_ent + 8 * nS * nD) * 8 + n_ent / 2 + n_ent * 16 + (nS * nD + 1) * 40 + (2ull << 30);
    // (idle pool blocks count as free: an allocation that fails releases them)
    return free_b + g->ctx->pool_bytes > need;
}

gs_status pb_layout_build(gs_graph* g) {
    gs_ctx* ctx = g->ctx;
    gs_pb_layout& L = g->pb;
    pb_layout_free(g);
    const uint64_t n_ent = g->directed ? g->E : 2 * g->E;
    const uint32_t nS = (uint32_t)(g->N >> kPbSrcBits), nD = (uint32_t)(g->N >> kPbDstBits);
    const uint64_t n_blk = (uint64_t)nS * nD;
    if (const uint32_t rows = pb_pull_rows(g, n_ent, nS)) {
        bool fits = false;
        const gs_status st = pb_pull_build(g, rows, &fits);
        if (L.built) return GS_OK;
        pb_layout_free(g);
        if (st != GS_OK && st != GS_ERR_OOM) return st;
    }
    int end_bit = kKeyLowBits;
    while ((1ull << (end_bit - kKeyLowBits)) < n_blk) ++end_bit;

    uint64_t *d_k0 = nullptr, *d_k1 = nullptr, *d_start = nullptr, *d_pstart = nullptr;
    gs_pb_block* d_blocks = nullptr;   // the D-major block table (build only)
    uint64_t n_pad = 0;   // entries with every block padded to a multiple of 8
    void* d_tmp = nullptr;
    size_t tmp_bytes = 0;
    gs_status st = gs_dev_alloc(ctx, (void**)&d_k0, n_ent * 8);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&d_k1, n_ent * 8);
    if (st == GS_OK) {
        pb_keys_kernel<<<gs_grid_size(ctx, 8), 256, 0, ctx->stream>>>(g->d_units, g->U, g->d_rec, nD, kDstBin,
                                                                       g->directed, d_k0);
        ctx->launches++;
        cudaError_t e = cudaGetLastError();
        cub::DoubleBuffer<uint64_t> keys(d_k0, d_k1);
        if (e == cudaSuccess)
            e = cub::DeviceRadixSort::SortKeys(nullptr, tmp_bytes, keys, n_ent, 0, end_bit, ctx->stream);
        if (e == cudaSuccess) st = gs_dev_alloc(ctx, &d_tmp, tmp_bytes);
        if (e == cudaSuccess && st == GS_OK)
            e = cub::DeviceRadixSort::SortKeys(d_tmp, tmp_bytes, keys, n_ent, 0, end_bit, ctx->stream);
        ctx->launches++;
        if (e != cudaSuccess && st == GS_OK) st = gs_cuda_fail(ctx, e, "propagation-blocking key sort");
        const uint64_t* sorted = keys.Current();
        gs_dev_free(d_tmp);
        d_tmp = nullptr;
        if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&d_start, (n_blk + 1) * 8);
        if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&d_pstart, (n_blk + 1) * 8);
        if (st == GS_OK) {
            pb_block_start_kernel<<<grid_for(n_blk + 1, ctx), 256, 0, ctx->stream>>>(sorted, n_ent, n_blk, d_start);
            pb_padded_count_kernel<<<grid_for(n_blk + 1, ctx), 256, 0, ctx->stream>>>(d_start, n_blk, d_pstart);
            ctx->launches += 2;
            e = cudaGetLastError();
            size_t scan_bytes = 0;
            if (e == cudaSuccess)
                e = cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, d_pstart, d_pstart, n_blk + 1, ctx->stream);
            if (e == cudaSuccess) st = gs_dev_alloc(ctx, &d_tmp, scan_bytes);
            if (e == cudaSuccess && st == GS_OK)
                e = cub::DeviceScan::ExclusiveSum(d_tmp, scan_bytes, d_pstart, d_pstart, n_blk + 1, ctx->stream);
            ctx->launches++;
            if (e == cudaSuccess && st == GS_OK)
                e = cudaMemcpyAsync(&n_pad, d_pstart + n_blk, 8, cudaMemcpyDeviceToHost, ctx->stream);
            if (e == cudaSuccess && st == GS_OK) e = cudaStreamSynchronize(ctx->stream);
            gs_dev_free(d_tmp);
            d_tmp = nullptr;
            if (e != cudaSuccess && st == GS_OK) st = gs_cuda_fail(ctx, e, "propagation-blocking block starts");
        }
        if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&L.d_src, n_pad * 2);
        if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&L.d_dst, n_pad * 2);
        if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&d_blocks, std::max<uint64_t>(1, n_blk) * sizeof(gs_pb_block));
        if (st == GS_OK) {
            pb_split_kernel<<<gs_grid_size(ctx, 8), 256, 0, ctx->stream>>>(sorted, d_start, d_pstart, n_blk, L.d_src,
                                                                            L.d_dst);
            pb_block_table_kernel<<<grid_for(n_blk, ctx), 256, 0, ctx->stream>>>(d_pstart, nS, nD, d_blocks);
            ctx->launches += 2;
            e = cudaGetLastError();
            if (e != cudaSuccess) st = gs_cuda_fail(ctx, e, "propagation-blocking layout");
        }
    }
    gs_dev_free(d_k0);
    gs_dev_free(d_k1);
    std::vector<gs_pb_block> blocks(n_blk);
    std::vector<uint64_t> slice_start(nS + 1);
    if (st == GS_OK) {
        cudaError_t e = cudaMemcpyAsync(blocks.data(), d_blocks, n_blk * sizeof(gs_pb_block),
                                        cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        // entries of slice S start at block (S, 0), the first of the bin-major table
        for (uint32_t s = 0; s < nS; ++s) slice_start[s] = blocks[s].e0;
        slice_start[nS] = n_pad;
        if (e != cudaSuccess) st = gs_cuda_fail(ctx, e, "propagation-blocking tables");
    }
    gs_dev_free(d_start);
    gs_dev_free(d_pstart);
    if (st != GS_OK) {
        gs_dev_free(d_blocks);
        pb_layout_free(g);
        return st;
    }
    // The group list the accumulate pass walks: every bin's blocks in slice
    // order, as 8-entry groups, so that a bin is one flat sequence of groups
    // however its entries are spread over blocks (a lane per group).
    std::vector<uint64_t> gpos(n_blk + 1);
    gpos[0] = 0;
    for (uint64_t b = 0; b < n_blk; ++b) gpos[b + 1] = gpos[b] + (blocks[b].n >> 3);
    const uint64_t n_groups = gpos[n_blk];
    // Items: entry chunks of every slice (pass 1) and group ranges of every
    // bin (pass 2), sized so that each pass has a few items per resident CTA
    // (pass 2: ~16, so that the last wave of equal items leaves few SMs idle).
    // (item boundaries stay multiples of 8 entries: every block starts on one)
    // A bin's item holds 8,192 groups at least: every further item of a bin adds
    // its sums to y once more, in 32 bits.  2,048 groups, so that small graphs
    // have two items per CTA, took the served ranks of Kronecker 19 from 5.5e-8
    // to 9.4e-8 of the 64-bit ones (2-norm) and its request from 0.44 to 0.48 ms
    // (18: 0.40 and 0.42; 17: 0.26 and 0.18); 24 M entries over 1,500,007 vertices,
    // uniform, under a budget 106 and 119 us per iteration (400,009: 52 and 41).
    const uint64_t per2 =
        std::clamp<uint64_t>(n_groups / ((uint64_t)ctx->num_sms * kAccCtas * 16), 8192, 1ull << 19);
    const std::vector<gs_pb_item1> items1 = gather_items(ctx, slice_start);
    std::vector<gs_pb_item2> items2;
    for (uint32_t d = 0; d < nD; ++d) {
        const uint64_t g0 = gpos[(uint64_t)d * nS], g1 = gpos[(uint64_t)(d + 1) * nS];
        const uint64_t parts = (g1 - g0 + per2 - 1) / per2;
        for (uint64_t k = 0; k < parts; ++k)
            items2.push_back(gs_pb_item2{(uint32_t)(g0 + (g1 - g0) * k / parts),
                                         (uint32_t)(g0 + (g1 - g0) * (k + 1) / parts), d, parts == 1 ? 1u : 0u});
    }
    L.n_entries = n_pad;
    L.n_groups = n_groups;
    L.n_items1 = items1.size();
    L.n_items2 = items2.size();
    uint64_t* d_gpos = nullptr;
    st = gs_dev_alloc(ctx, (void**)&L.d_val, n_pad * 4);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&L.d_groups, std::max<uint64_t>(1, n_groups) * 4);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&d_gpos, (n_blk + 1) * 8);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&L.d_items1, std::max<size_t>(1, items1.size()) * sizeof(gs_pb_item1));
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&L.d_items2, std::max<size_t>(1, items2.size()) * sizeof(gs_pb_item2));
    cudaError_t e = cudaSuccess;
    if (st == GS_OK)
        e = cudaMemcpyAsync(d_gpos, gpos.data(), (n_blk + 1) * 8, cudaMemcpyHostToDevice, ctx->stream);
    if (st == GS_OK && e == cudaSuccess) {
        pb_group_list_kernel<<<gs_grid_size(ctx, 8), 256, 0, ctx->stream>>>(d_blocks, d_gpos, n_blk, L.d_groups);
        ctx->launches++;
        e = cudaGetLastError();
    }
    if (st == GS_OK && e == cudaSuccess && !items1.empty())
        e = cudaMemcpyAsync(L.d_items1, items1.data(), items1.size() * sizeof(gs_pb_item1), cudaMemcpyHostToDevice,
                            ctx->stream);
    if (st == GS_OK && e == cudaSuccess && !items2.empty())
        e = cudaMemcpyAsync(L.d_items2, items2.data(), items2.size() * sizeof(gs_pb_item2), cudaMemcpyHostToDevice,
                            ctx->stream);
    if (st == GS_OK && e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (st == GS_OK && e != cudaSuccess) st = gs_cuda_fail(ctx, e, "propagation-blocking items");
    gs_dev_free(d_gpos);
    gs_dev_free(d_blocks);
    if (st != GS_OK) {
        pb_layout_free(g);
        return st;
    }
    L.built = true;
    return GS_OK;
}

gs_status pb_sweep(gs_graph* g, const float* x, float* y, int* error) {
    gs_ctx* ctx = g->ctx;
    const gs_pb_layout& L = g->pb;
    if (L.n_items1 == 0) return GS_OK;
    GS_CHECK_CUDA(ctx, gs_smem_limit_once<pb_gather_kernel>(ctx->device, (int)sizeof(GatherSmem)));
    const uint32_t g1 = (uint32_t)std::min<uint64_t>(L.n_items1, gs_grid_size(ctx, kGatherCtas));
    pb_gather_kernel<<<g1, kGatherThreads, sizeof(GatherSmem), ctx->stream>>>(L.d_items1, L.n_items1, L.d_src, x,
                                                                             L.d_val, error, ctx->d_ticket + 4);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    GS_CHECK_CUDA(ctx, second_pass(g, L.d_val, y, ctx->d_ticket + 6, ctx->stream));
    ctx->launches += 2;
    return GS_OK;
}

gs_status pb_sweep_on(gs_graph* g, cudaStream_t stream, const float* x, float* y, int* error, float* val) {
    gs_ctx* ctx = g->ctx;
    const gs_pb_layout& L = g->pb;
    if (L.n_items1 == 0) return GS_OK;
    GS_CHECK_CUDA(ctx, gs_smem_limit_once<pb_gather_kernel>(ctx->device, (int)sizeof(GatherSmem)));
    // one CTA per item and no ticket: short CTAs, so that a higher-priority
    // stream's CTAs find free SMs between them
    pb_gather_kernel<<<(uint32_t)L.n_items1, kGatherThreads, sizeof(GatherSmem), stream>>>(
        L.d_items1, L.n_items1, L.d_src, x, val, error, nullptr);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    GS_CHECK_CUDA(ctx, second_pass(g, val, y, nullptr, stream));
    ctx->launches += 2;
    return GS_OK;
}

gs_status pb_launch(gs_state* s) {
    gs_graph* g = s->g;
    gs_ctx* ctx = g->ctx;
    if (!s->d_error) {
        GS_TRY(gs_state_alloc(s, (void**)&s->d_error, sizeof(uint64_t)));
        GS_CHECK_CUDA(ctx, cudaMemsetAsync(s->d_error, 0, sizeof(uint64_t), ctx->stream));
    }
    gs_timer_begin(ctx);
    GS_TRY(pb_sweep(g, s->d_x, s->d_y, (int*)s->d_error));
    // algorithmic bytes per iteration: 4E + 12V (records, x, s, inv)
    gs_timer_end(ctx, GS_ALGO_PAGERANK, 4 * g->E + 12 * g->V);
    return GS_OK;
}
