// Adjacency lists of a resident graph (sm_100a) and the queries that run on
// them: BFS, WCC and k-core (gs_run).
//
// A tile sweep reads every record of the tiles a level or round touches --
// from the third level of a BFS on, and in every k-core round, that is the
// whole grid -- whatever the few vertices concerned are.  With the records
// also listed by vertex, a BFS level costs its frontier's entries (top-down),
// or a few probes per vertex not reached yet (bottom-up: Beamer, Asanovic and
// Patterson, "Direction-Optimizing Breadth-First Search", SC 2012), a k-core
// round the entries of the vertices it removes, and WCC about two entries per
// vertex plus the entries of the vertices outside the largest tree (Sutton,
// Ben-Nun and Barak, "Optimizing Parallel Graph Connectivity Computation via
// Subgraph Sampling", IPDPS 2018).  Depths, labels and degrees are those of
// the sweeps (the same level sets, component minima and synchronous rounds).
//
// Device time per query, tile sweeps against lists: BFS at Kronecker 26 6.35
// -> 0.55 ms, WCC at 25 2.9 -> 0.68, k-core(8) at 25 3.4 -> 0.70 (edge factor
// 16).  What bounds them is random 4-byte accesses to L2 (about one per vertex
// looked at) and the latency of their chains, so every kernel keeps four
// independent ones per lane in flight and works on compacted lists of the
// vertices concerned instead of on words with a few bits set.
//
// The lists cost 8 bytes per record and 9 per vertex of HBM, and building
// them takes about 7 such queries' time (45 ms at Kronecker 26, 22 at 25).  So a
// graph gets them once its queries have swept it kAdjBuild times, eight BFS or
// k-core queries or eleven WCC (gs_adj_ready: a graph that is queried only a
// few times never pays for them, one that is queried often pays about as much
// as it had spent by then, in one query), and only while half of the free HBM
// stays free.  An allocation that fails drops them for good (gs_adj_release); a
// query that finds no room for its own scratch runs on the tiles.
#include "gs_internal.cuh"
#include "gs_ops.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cstring>
#include <vector>

namespace {

using namespace gsops;

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kCtas = 3;               // resident CTAs per SM of the cooperative launches
constexpr uint32_t kChunk = 1024;      // entries of a long row a warp takes at a time
constexpr uint32_t kProbe = 64;        // bottom-up: entries a lane looks at before its warp helps
constexpr uint32_t kLongRow = 4096;    // entries left after that which go to the whole grid

inline uint32_t blocks_for(uint64_t n, const gs_ctx* ctx) {
    const uint64_t b = (n + 255) / 256;
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(b, gs_grid_size(ctx, 16)));
}

// ------------------------------------------------------------------ build --
constexpr uint32_t kMixed = 16;        // windows whose lists are being filled at a time

// The lists are built in two passes over the records, one per end, each over
// the units in the order of that end's window, so that the CTAs in flight count
// into, take slots from and write a few windows' counters and lists, which L2
// holds.  kMixed windows take turns: fewer make every CTA wait for the same hub
// counters, more no longer fit.  The lists of Kronecker 26: file order (the
// second ends of a tile row touch every window) 157 ms, window order 89, with
// units drawn from a ticket and 1 / 4 / 8 / 16 windows taking turns 110 / 60 /
// 45 / 45 ms.
__global__ void adj_unit_key_kernel(const gs_unit* __restrict__ units, uint32_t n, int by_col, uint32_t* __restrict__ key,
                                    uint32_t* __restrict__ idx) {
    const uint32_t nth = gridDim.x * blockDim.x;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += nth) {
        key[u] = by_col ? units[u].rc & 0xFFFFu : units[u].rc >> 16;
        idx[u] = u;
    }
}

// fn(own ends, other ends, valid) for four records of every thread at a time,
// a unit per CTA and units drawn in the given order from a ticket, so that the
// records in flight are those of two or three windows (CTAs that took every
// gridDim.x-th unit drifted apart by tens of windows: 89 ms at Kronecker 26).
template <class F>
__device__ __forceinline__ void each_record(const gs_unit* __restrict__ units, const uint32_t* __restrict__ order,
                                            uint32_t n_units, uint32_t part, unsigned int* ticket,
                                            const uint32_t* __restrict__ rec, int by_col, F fn) {
    __shared__ uint32_t s_unit;
    // kMixed consecutive stretches of `part` units (about a window each) take turns
    const uint32_t turn = part * kMixed, n_all = (n_units + turn - 1) / turn * turn;
    while (true) {
        __syncthreads();   // every thread has read the previous draw
        if (threadIdx.x == 0) s_unit = atomicAdd(ticket, 1u);
        __syncthreads();
        const uint32_t t = s_unit;
        if (t >= n_all) return;
        const uint32_t in = t % turn, i = t - in + in % kMixed * part + in / kMixed;
        if (i >= n_units) continue;   // uniform
        const gs_unit un = units[order[i]];
        const uint32_t rb = (un.rc >> 16) << 16, cb = (un.rc & 0xFFFFu) << 16;
        for (uint32_t k = threadIdx.x; k < un.n; k += blockDim.x * 4) {
            uint32_t own[4], other[4];
            bool ok[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t x = k + j * blockDim.x;
                ok[j] = x < un.n;
                const uint32_t r = ok[j] ? __ldcs(rec + un.rec_beg + x) : 0u;
                const uint32_t a = rb + (r & 0xFFFFu), b = cb + (r >> 16);
                own[j] = by_col ? b : a;
                other[j] = by_col ? a : b;
            }
            fn(own, other, ok);
        }
    }
}

__global__ void adj_count_kernel(const gs_unit* __restrict__ units, const uint32_t* __restrict__ order, uint32_t n_units,
                                 uint32_t part, unsigned int* ticket, const uint32_t* __restrict__ rec, int by_col, uint32_t* count) {
    each_record(units, order, n_units, part, ticket, rec, by_col, [&](const uint32_t (&own)[4], const uint32_t (&)[4], const bool (&ok)[4]) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (ok[j]) atomicAdd(count + own[j], 1u);
    });
}

// Bit v of `none`: in[v] == 0; *some counts the others.
__global__ void adj_none_kernel(const uint32_t* __restrict__ in, uint64_t N, uint32_t* __restrict__ none,
                                unsigned long long* some) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t step = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    uint32_t local = 0;
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < N / 32; w += step) {
        const uint32_t bits = __ballot_sync(kFull, in[w * 32 + lane] == 0);
        if (lane == 0) none[w] = bits;
        local += lane == 0 ? 32 - __popc(bits) : 0;
    }
    warp_add_u64(some, local);
}

// The vertices of at least `least` out-entries: their bits, and their list (any
// order, at most `cap` of them).
__global__ void adj_hub_kernel(const uint32_t* __restrict__ out, uint64_t N, uint32_t least, uint32_t* __restrict__ hub,
                               uint32_t* __restrict__ hubs, uint32_t cap, unsigned int* n_hubs) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t step = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < N / 32; w += step) {
        const uint32_t bits = __ballot_sync(kFull, out[w * 32 + lane] >= least);
        if (lane == 0) hub[w] = bits;
        if (bits == 0) continue;   // uniform
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(n_hubs, __popc(bits));
        at = __shfl_sync(kFull, at, 0) + __popc(bits & ((1u << lane) - 1u));
        if ((bits >> lane & 1u) && at < cap) hubs[at] = (uint32_t)w * 32 + lane;
    }
}

// One end's entries.  With `hub`, hubs fill a list from its front, other
// vertices from its back: a bottom-up probe of a BFS meets the neighbours most
// likely to be in the frontier first.
__global__ void adj_fill_kernel(const gs_unit* __restrict__ units, const uint32_t* __restrict__ order, uint32_t n_units,
                                uint32_t part, unsigned int* ticket, const uint32_t* __restrict__ rec, int by_col,
                                const uint32_t* __restrict__ hub,
                                const uint32_t* __restrict__ off, uint32_t* __restrict__ adj, uint32_t* front,
                                uint32_t* back) {
    each_record(units, order, n_units, part, ticket, rec, by_col, [&](const uint32_t (&own)[4], const uint32_t (&other)[4], const bool (&ok)[4]) {
        bool fwd[4];
        uint32_t base[4], k[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) fwd[j] = !hub || !ok[j] || bit_of(hub, other[j]);
#pragma unroll
        for (int j = 0; j < 4; ++j) base[j] = ok[j] ? __ldg(off + own[j] + (fwd[j] ? 0 : 1)) : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) k[j] = ok[j] ? atomicAdd((fwd[j] ? front : back) + own[j], 1u) : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (ok[j]) adj[fwd[j] ? base[j] + k[j] : base[j] - 1 - k[j]] = other[j];
    });
}

// -------------------------------------------------------------------- BFS --
// A chunk of a long row, taken by any warp of the grid.
struct AdjItem {
    uint32_t v, beg, end;
};
// (lists change hands between SMs inside a launch: read through L2)
__device__ __forceinline__ AdjItem load_item(const AdjItem* p) {
    return AdjItem{__ldcg(&p->v), __ldcg(&p->beg), __ldcg(&p->end)};
}

struct BfsCtl {
    unsigned long long total[256];   // vertices found per level ([0]: the root)
    unsigned long long edges[256];   // their out-entries (after a bottom-up level: an estimate)
    unsigned int n_queue[4];         // frontier vertices listed, by level & 3
    unsigned int n_long[4];          // chunks of long rows, by level & 3
    unsigned int bar[2];
    int err;
    int levels;
    int overflow;
};

struct BfsArgs {
    const uint32_t *off_in, *adj_in, *first_in, *off_out, *adj_out;
    uint32_t* fr;            // two frontier bitmaps of N / 32 words
    uint32_t* vis;           // visited, or without in-entries
    uint8_t* depth;
    uint32_t* queue;         // [2][cap] frontier vertices, by level & 1
    AdjItem* items;          // [cap]
    uint32_t cap;
    uint32_t block;          // words a warp takes at a time (a power of two <= 32)
    uint64_t words;
    unsigned long long n_cand, n_ent;
    unsigned long long* read;   // [256] entries read per level
    BfsCtl* c;
};

// Visited bits from `none`, and the root (bfs.cpp:56-75).
__global__ void bfs_adj_seed_kernel(BfsArgs a, const uint32_t* __restrict__ none, uint32_t root) {
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x, tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t w = tid; w < a.words; w += nth) {
        uint32_t x = none[w];
        if (w == root >> 5) x |= 1u << (root & 31);
        a.vis[w] = x;
    }
    if (tid == 0) {
        a.fr[root >> 4] = 0;   // the tile sweep's seed (bfs_init)
        a.fr[root >> 5] = 1u << (root & 31);
        a.depth[root] = 1;
        a.queue[a.cap] = root;   // level 1
        a.c->total[0] = 1;
        a.c->edges[0] = a.off_out[root + 1] - a.off_out[root];
        a.c->n_queue[1] = 1;
    }
}

// One launch for all levels (Kronecker 16 takes 65 us in six levels of 4-20 us;
// two launches and a host round trip per level took 180 and more).  Kronecker
// 26, a root whose second level has 8.6 M entries: levels of 16, 177 (bulk
// top-down), 220 (bottom-up: 31.6 M first entries, 97 % of them hits), 54 and
// 47 us, 550 us in all.  Probing a candidate at a time per lane and word
// instead of four from a compacted list took 1,366 and 667 us for the two
// bottom-up levels; finding, marking and listing one by one took 380 us for the
// bulk level.  Every CTA is resident, levels are separated by a grid barrier
// (bounded, grid_barrier), and every CTA takes the same decisions from the
// counters behind it.
__global__ void __launch_bounds__(kThreads, kCtas) bfs_adj_kernel(const BfsArgs a) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t gw = blockIdx.x * kWarps + warp, nwarps = gridDim.x * kWarps;
    const uint32_t lt = (1u << lane) - 1u;
    __shared__ unsigned long long s_sum[3];
    __shared__ uint16_t s_list[kWarps][1024];   // a block's candidates, then those the first probe missed
    __shared__ uint32_t s_fresh[kWarps][32];
    BfsCtl* c = a.c;
    bool list = true;        // the queue holds the whole frontier
    unsigned long long seen = 0;
    for (int level = 1; level < 255; ++level) {
        uint32_t* cur = a.fr + (level & 1 ? 0 : a.words);
        uint32_t* nxt = a.fr + (level & 1 ? a.words : 0);
        uint32_t* now = a.queue + (level & 1 ? a.cap : 0);
        uint32_t* then = a.queue + (level & 1 ? 0 : a.cap);
        unsigned int* n_then = c->n_queue + ((level + 1) & 3);
        unsigned int* n_items = c->n_long + (level & 3);
        const unsigned long long m = __ldcg(c->edges + level - 1);
        seen += __ldcg(c->total + level - 1);
        uint32_t n_now = __ldcg(c->n_queue + (level & 3));
        if (threadIdx.x < 3) s_sum[threadIdx.x] = 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            c->n_queue[(level + 2) & 3] = 0;   // last used two levels ago
            c->n_long[(level + 2) & 3] = 0;
        }
        // Top-down reads the frontier's entries, two random words each and an
        // atomic per vertex found: 33-49 G entries/s at Kronecker 26.  Bottom-up
        // reads, for every vertex that is left, entries until one is in the
        // frontier -- about n_ent / m of them if the frontier's entries are
        // spread evenly, at most all, fewer as hubs come first -- at 150-170 G/s
        // (taken as equal rates, 3 of 17 roots went through 150 M entries top-down:
        // 4.2 ms for the level instead of under 1).
        const unsigned long long left = a.n_cand > seen ? a.n_cand - seen : 0;
        const unsigned long long all = a.n_ent / (a.n_cand ? a.n_cand : 1) + 1;
        const unsigned long long probes = m ? min(all, a.n_ent / m + 1) : all;
        bool down = m * 6 <= left * probes + a.words / 16;
        if (down && !list) {
            // the frontier came from a bottom-up level: list its vertices,
            // and clear the bitmap that this level writes
            unsigned int* n_here = c->n_queue + (level & 3);
            for (uint64_t w0 = (uint64_t)gw * 32; w0 < a.words; w0 += (uint64_t)nwarps * 32) {
                const uint64_t w = w0 + lane;
                uint32_t x = w < a.words ? __ldcg(cur + w) : 0u;
                if (w < a.words) __stcg(nxt + w, 0u);
                uint32_t at = __popc(x);
                const uint32_t mine = at;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFull, at, o);
                    if (lane >= (uint32_t)o) at += y;
                }
                const uint32_t sum = __shfl_sync(kFull, at, 31);
                if (sum == 0) continue;   // uniform
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(n_here, sum);
                at = __shfl_sync(kFull, base, 0) + at - mine;
                for (; x; x &= x - 1, ++at)
                    if (at < a.cap) now[at] = (uint32_t)w * 32 + __ffs(x) - 1;
            }
            if (!grid_barrier(c->bar, &c->err)) return;
            n_now = __ldcg(c->n_queue + (level & 3));
        }
        if (n_now > a.cap) down = false;   // too many to list
        // A small frontier's finds are marked, counted and listed one by one.  A
        // larger one's (the next level will hardly be top-down) are only OR-ed
        // into the next bitmap, which a pass over the words then reads: an
        // atomic without an answer per find instead of three with one.
        const bool bulk = down && m > a.n_ent / 1024 + 1024;
        // rows of over two chunks are spread over the grid
        const uint32_t chunk = down ? (uint32_t)min(4096ull, max(128ull, (m / nwarps + 127) & ~127ull)) : kChunk;
        __syncthreads();   // s_sum is zero
        unsigned long long found = 0, entries = 0, read = 0;
        // Top-down: up to four neighbours a lane (~0: none), the warp together.
        auto visit = [&](const uint32_t (&n)[4]) {
            bool hit[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) hit[j] = n[j] != ~0u && !(__ldcg(a.vis + (n[j] >> 5)) >> (n[j] & 31) & 1u);
            if (bulk) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (hit[j]) atomicOr(nxt + (n[j] >> 5), 1u << (n[j] & 31));
                return;
            }
            if (!__any_sync(kFull, hit[0] | hit[1] | hit[2] | hit[3])) return;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t bit = 1u << (n[j] & 31);
                if (hit[j]) hit[j] = !(atomicOr(a.vis + (n[j] >> 5), bit) & bit);
            }
            uint32_t bal[4], k = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                bal[j] = __ballot_sync(kFull, hit[j]);
                k += __popc(bal[j]);
            }
            uint32_t at = 0;
            if (lane == 0 && k) at = atomicAdd(n_then, k);
            at = __shfl_sync(kFull, at, 0);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (hit[j]) {
                    atomicOr(nxt + (n[j] >> 5), 1u << (n[j] & 31));
                    a.depth[n[j]] = (uint8_t)(level + 1);
                    const uint32_t q = at + __popc(bal[j] & lt);
                    if (q < a.cap) then[q] = n[j];
                    found += 1;
                    entries += __ldg(a.off_out + n[j] + 1) - __ldg(a.off_out + n[j]);
                }
                at += __popc(bal[j]);
            }
        };
        auto visit_row = [&](uint32_t b, uint32_t e) {   // the warp together
            for (uint32_t k = b; k < e; k += 128) {
                uint32_t n[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t x = k + 32 * j + lane;
                    n[j] = x < e ? __ldg(a.adj_out + x) : ~0u;
                }
                visit(n);
            }
        };
        // Bottom-up: is any of a row's entries in the frontier?  The warp together.
        auto probe_row = [&](uint32_t b, uint32_t e, uint32_t& looked) -> bool {
            uint32_t got = 0, p = b;
            for (; p < e && !got; p += 128) {
                uint32_t x = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t q = p + 32 * j + lane;
                    if (q < e) {
                        const uint32_t n = __ldg(a.adj_in + q);
                        x |= __ldcg(cur + (n >> 5)) >> (n & 31);
                    }
                }
                got = __any_sync(kFull, x & 1u);
            }
            looked = min(p, e) - b;
            return got != 0;
        };
        // Lists a long row's chunks for the grid; false when there is no room.
        auto defer = [&](uint32_t v, uint32_t b, uint32_t e) -> bool {
            const uint32_t n = (e - b + chunk - 1) / chunk;
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(n_items, n);
            at = __shfl_sync(kFull, at, 0);
            for (uint32_t j = lane; j < n; j += 32)
                if (at + j < a.cap) a.items[at + j] = AdjItem{v, b + j * chunk, min(b + (j + 1) * chunk, e)};
            return at + n <= a.cap;
        };
        if (down) {
            // a vertex a warp, or 32 when there are enough for every warp
            const uint32_t some = n_now <= nwarps * 2 ? 1 : 32;
            for (uint32_t i = gw * some; i < n_now; i += nwarps * some) {
                const bool mine = lane < some && i + lane < n_now;
                const uint32_t v = mine ? __ldcg(now + i + lane) : 0u;
                uint32_t b = mine ? __ldg(a.off_out + v) : 0u;
                const uint32_t e = mine ? __ldg(a.off_out + v + 1) : 0u;
                if (mine) __stcg(cur + (v >> 5), 0u);   // the bitmap the next level writes
                read += e - b;
                uint32_t wide = __ballot_sync(kFull, some == 1 ? lane == 0 : e - b > 16);
                const uint32_t own = wide >> lane & 1u ? b : e;   // short rows: a lane each
                for (uint32_t k = b; __any_sync(kFull, own != b && k < e); k += 4) {
                    uint32_t n[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) n[j] = own != b && k + j < e ? __ldg(a.adj_out + k + j) : ~0u;
                    visit(n);
                }
                while (wide) {
                    const uint32_t l = __ffs(wide) - 1;
                    wide &= wide - 1;
                    const uint32_t rv = __shfl_sync(kFull, v, l), rb = __shfl_sync(kFull, b, l),
                                   re = __shfl_sync(kFull, e, l);
                    if (re - rb > 2 * chunk && defer(rv, rb, re)) continue;
                    visit_row(rb, re);
                }
            }
            list = !bulk;
        } else {
            for (uint64_t w0 = (uint64_t)gw * a.block; w0 < a.words; w0 += (uint64_t)nwarps * a.block) {
                const bool mine = lane < a.block && w0 + lane < a.words;
                const uint32_t vw = mine ? __ldcg(a.vis + w0 + lane) : ~0u;
                const uint32_t base = (uint32_t)w0 * 32;
                const uint32_t n_cand = list_bits(s_list[warp], ~vw, lane);
                if (n_cand == 0) {   // uniform
                    if (mine) __stcg(nxt + w0 + lane, 0u);
                    continue;
                }
                s_fresh[warp][lane] = 0;
                __syncwarp();
                auto hit_one = [&](uint32_t o) {
                    atomicOr(&s_fresh[warp][o >> 5], 1u << (o & 31));
                    a.depth[base + o] = (uint8_t)(level + 1);
                    found += 1;
                };
                // every candidate's first entry, four a lane in flight: it
                // leads to a hub and hits most of the time
                uint32_t n_miss = 0;
                for (uint32_t t = 0; t < n_cand; t += 128) {
                    uint32_t o[4], n[4];
                    bool miss[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t k = t + 32 * j + lane;
                        o[j] = k < n_cand ? s_list[warp][k] : ~0u;
                        n[j] = o[j] != ~0u ? __ldg(a.first_in + base + o[j]) : 0u;
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) n[j] = o[j] != ~0u ? __ldcg(cur + (n[j] >> 5)) >> (n[j] & 31) & 1u : 0u;
                    __syncwarp();   // the list up to t + 128 has been read
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        miss[j] = o[j] != ~0u && !n[j];
                        if (n[j]) hit_one(o[j]);
                        const uint32_t bal = __ballot_sync(kFull, miss[j]);
                        if (miss[j]) s_list[warp][n_miss + __popc(bal & lt)] = (uint16_t)o[j];
                        n_miss += __popc(bal);
                    }
                    __syncwarp();
                }
                if (lane == 0) read += n_cand;
                // the others' further entries
                for (uint32_t t = 0; t < n_miss; t += 32) {
                    const bool has = t + lane < n_miss;
                    const uint32_t o = has ? s_list[warp][t + lane] : 0u, v = base + o;
                    uint32_t i = has ? __ldg(a.off_in + v) + 1 : 0u;
                    const uint32_t e = has ? __ldg(a.off_in + v + 1) : 0u, i0 = i;
                    const uint32_t stop = i < e && e - i > kProbe ? i + kProbe : e;
                    bool hit = false;
                    while (!hit && i < stop) {
                        uint32_t n[4], x[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) n[j] = i + j < stop ? __ldg(a.adj_in + i + j) : 0u;
#pragma unroll
                        for (int j = 0; j < 4; ++j) x[j] = i + j < stop ? __ldcg(cur + (n[j] >> 5)) >> (n[j] & 31) : 0u;
                        hit = (x[0] | x[1] | x[2] | x[3]) & 1u;
                        i = min(i + 4, stop);
                    }
                    read += i - i0;
                    // long rows: the warp together, or, very long ones, the grid
                    uint32_t more = __ballot_sync(kFull, !hit && i < e);
                    while (more) {
                        const uint32_t l = __ffs(more) - 1;
                        more &= more - 1;
                        const uint32_t rb = __shfl_sync(kFull, i, l), re = __shfl_sync(kFull, e, l);
                        if (re - rb > kLongRow && defer(__shfl_sync(kFull, v, l), rb, re)) continue;
                        uint32_t looked;
                        const bool got = probe_row(rb, re, looked);
                        if (lane == l) hit = got;
                        if (lane == 0) read += looked;
                    }
                    if (hit) hit_one(o);
                }
                __syncwarp();
                const uint32_t fresh = s_fresh[warp][lane];
                if (mine) {
                    __stcg(nxt + w0 + lane, fresh);
                    if (fresh) __stcg(a.vis + w0 + lane, vw | fresh);
                }
                __syncwarp();   // s_list and s_fresh are rewritten
            }
            list = false;
        }
        auto add_up = [&]() {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                found += __shfl_xor_sync(kFull, found, o);
                entries += __shfl_xor_sync(kFull, entries, o);
                read += __shfl_xor_sync(kFull, read, o);
            }
            // bottom-up levels do not look the found vertices' rows up
            if (!down) entries = found * all;
            if (lane == 0) {
                if (found) atomicAdd(s_sum, found);
                if (entries) atomicAdd(s_sum + 1, entries);
                if (read) atomicAdd(s_sum + 2, read);
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                if (s_sum[0]) atomicAdd(c->total + level, s_sum[0]);
                if (s_sum[1]) atomicAdd(c->edges + level, s_sum[1]);
                if (s_sum[2]) atomicAdd(a.read + level - 1, s_sum[2]);
            }
            found = entries = read = 0;
        };
        add_up();
        if (!grid_barrier(c->bar, &c->err)) return;
        const uint32_t n_long = min(__ldcg(n_items), a.cap);
        if (n_long) {
            if (threadIdx.x < 3) s_sum[threadIdx.x] = 0;
            __syncthreads();
            for (uint32_t i = gw; i < n_long; i += nwarps) {
                const AdjItem it = load_item(a.items + i);
                if (down) {
                    visit_row(it.beg, it.end);
                    continue;
                }
                const uint32_t bit = 1u << (it.v & 31);
                if (__ldcg(a.vis + (it.v >> 5)) & bit) continue;   // uniform: another chunk found it
                uint32_t looked;
                const bool got = probe_row(it.beg, it.end, looked);
                if (lane == 0) {
                    read += looked;
                    if (got && !(atomicOr(a.vis + (it.v >> 5), bit) & bit)) {
                        atomicOr(nxt + (it.v >> 5), bit);
                        a.depth[it.v] = (uint8_t)(level + 1);
                        found += 1;
                    }
                }
                __syncwarp();
            }
            add_up();
            if (!grid_barrier(c->bar, &c->err)) return;
        }
        if (bulk) {
            if (threadIdx.x < 3) s_sum[threadIdx.x] = 0;
            __syncthreads();
            for (uint64_t w0 = (uint64_t)gw * a.block; w0 < a.words; w0 += (uint64_t)nwarps * a.block) {
                const bool mine = lane < a.block && w0 + lane < a.words;
                const uint32_t x = mine ? __ldcg(nxt + w0 + lane) : 0u;
                if (x) __stcg(a.vis + w0 + lane, __ldcg(a.vis + w0 + lane) | x);
                const uint32_t n = list_bits(s_list[warp], x, lane);
                for (uint32_t t = lane; t < n; t += 32) {
                    const uint32_t v = (uint32_t)w0 * 32 + s_list[warp][t];
                    a.depth[v] = (uint8_t)(level + 1);
                    entries += __ldg(a.off_out + v + 1) - __ldg(a.off_out + v);
                }
                if (lane == 0) found += n;
                __syncwarp();   // s_list is rewritten
            }
            add_up();
            if (!grid_barrier(c->bar, &c->err)) return;
        }
        if (__ldcg(c->total + level) == 0) {
            if (blockIdx.x == 0 && threadIdx.x == 0) c->levels = level;
            return;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        c->levels = 254;
        c->overflow = 1;   // vertices at depth 255
    }
}

// Window flags per level from the depths: hist[l][w] = 1 when window w holds a
// vertex of depth l + 1 (a block per window).
__global__ void depth_windows_kernel(const uint8_t* __restrict__ depth, uint32_t nw, int levels,
                                     uint8_t* __restrict__ hist) {
    __shared__ uint8_t s[256];
    for (uint32_t w = blockIdx.x; w < nw; w += gridDim.x) {
        for (int l = threadIdx.x; l < 256; l += blockDim.x) s[l] = 0;
        __syncthreads();
        const uint4* d = reinterpret_cast<const uint4*>(depth + ((uint64_t)w << kTileBits));
        for (uint32_t i = threadIdx.x; i < (1u << kTileBits) / 16; i += blockDim.x) {
            const uint4 x = d[i];
            const uint32_t q[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int b = 0; b < 4; ++b) s[q[j] >> (8 * b) & 255u] = 1;
        }
        __syncthreads();
        for (int l = threadIdx.x; l < levels; l += blockDim.x) hist[(uint64_t)l * nw + w] = s[l + 1];
        __syncthreads();
    }
}

// ----------------------------------------------------------------- k-core --
struct KcoreCtl {
    unsigned long long removed[4];   // by round & 3
    unsigned int n_items[4];
    unsigned int bar[2];
    int err;
    int rounds;                      // rounds that removed a vertex
};

struct KcoreArgs {
    const uint32_t *off, *adj;
    int32_t* deg;
    uint32_t* removed;       // N / 32 words, zero
    uint32_t* cand;          // N / 32 words, zero: vertices whose degree fell into (0, k)
    AdjItem* items;
    uint32_t cap, block;
    uint64_t words;
    int k;
    KcoreCtl* c;
};

// iteration_finalize and the decrement sweeps of kcore.cpp:63-217, round by
// round: every vertex with 0 < (int16)degree < k is removed (degree 0), then
// every entry of a removed vertex takes one from its neighbour's degree.  From
// the second round on only the vertices whose degree was lowered into (0, k)
// can be removed: the last decrement of a round leaves the degree that the
// next round looks at, so marking on every decrement misses none.
// (a large round decrements without waiting for the old degree and has the
// next round look at every vertex instead: 25 us at 33 M vertices).
__global__ void __launch_bounds__(kThreads, kCtas) kcore_adj_kernel(const KcoreArgs a) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t gw = blockIdx.x * kWarps + warp, nwarps = gridDim.x * kWarps;
    __shared__ unsigned long long s_sum;
    __shared__ uint16_t s_list[kWarps][1024];
    __shared__ uint32_t s_gone[kWarps][32];
    KcoreCtl* c = a.c;
    bool all = true;    // this round looks at every vertex
    bool bulk = false;  // this round removes many
    auto lower4 = [&](const uint32_t (&n)[4]) {   // ~0: none
        if (bulk) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n[j] != ~0u) atomicSub(a.deg + n[j], 1);
            return;
        }
        int was[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) was[j] = n[j] != ~0u ? atomicSub(a.deg + n[j], 1) : 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int16_t m = (int16_t)(was[j] - 1);
            if (n[j] != ~0u && m > 0 && m < a.k) atomicOr(a.cand + (n[j] >> 5), 1u << (n[j] & 31));
        }
    };
    auto lower_row = [&](uint32_t b, uint32_t e) {   // the warp together
        for (uint32_t p = b + lane; p < e; p += 128) {
            uint32_t n[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) n[j] = p + 32 * j < e ? __ldg(a.adj + p + 32 * j) : ~0u;
            lower4(n);
        }
    };
    for (int round = 0;; ++round) {
        if (threadIdx.x == 0) s_sum = 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            c->removed[(round + 2) & 3] = 0;
            c->n_items[(round + 2) & 3] = 0;
        }
        __syncthreads();
        unsigned long long gone_here = 0;
        for (uint64_t w0 = (uint64_t)gw * a.block; w0 < a.words; w0 += (uint64_t)nwarps * a.block) {
            const bool mine = lane < a.block && w0 + lane < a.words;
            uint32_t rem = 0;
            if (all) {
                const uint32_t nb = a.words - w0 < a.block ? (uint32_t)(a.words - w0) : a.block;
                for (uint32_t k0 = 0; k0 < nb; k0 += 4) {
                    int32_t d[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        d[j] = k0 + j < nb ? __ldcg(a.deg + (w0 + k0 + j) * 32 + lane) : 0;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int16_t m = (int16_t)d[j];   // kcore.cpp:189
                        const bool gone = m < a.k && m > 0;
                        if (gone) __stcg(a.deg + (w0 + k0 + j) * 32 + lane, 0);
                        const uint32_t bits = __ballot_sync(kFull, gone);
                        if (lane == k0 + j) rem = bits;
                    }
                }
            } else {
                const uint32_t cw = mine ? __ldcg(a.cand + w0 + lane) : 0u;
                if (cw) __stcg(a.cand + w0 + lane, 0u);
                const uint32_t n = list_bits(s_list[warp], cw, lane);
                if (n == 0) continue;   // uniform
                s_gone[warp][lane] = 0;
                __syncwarp();
                for (uint32_t t = lane; t < n; t += 32) {
                    const uint32_t o = s_list[warp][t];
                    const int16_t m = (int16_t)__ldcg(a.deg + w0 * 32 + o);
                    if (m < a.k && m > 0) {
                        __stcg(a.deg + w0 * 32 + o, 0);
                        atomicOr(&s_gone[warp][o >> 5], 1u << (o & 31));
                    }
                }
                __syncwarp();
                rem = s_gone[warp][lane];
                __syncwarp();   // s_list and s_gone are rewritten
            }
            if (rem) __stcg(a.removed + w0 + lane, rem);
            gone_here += __popc(rem);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) gone_here += __shfl_xor_sync(kFull, gone_here, o);
        if (lane == 0 && gone_here) atomicAdd(&s_sum, gone_here);
        __syncthreads();
        if (threadIdx.x == 0 && s_sum) atomicAdd(c->removed + (round & 3), s_sum);
        if (!grid_barrier(c->bar, &c->err)) return;
        const unsigned long long removed = __ldcg(c->removed + (round & 3));
        if (removed == 0) {
            if (blockIdx.x == 0 && threadIdx.x == 0) c->rounds = round;
            return;
        }
        bulk = removed * 64 > a.words * 32;
        all = bulk;   // next round
        for (uint64_t w0 = (uint64_t)gw * a.block; w0 < a.words; w0 += (uint64_t)nwarps * a.block) {
            const bool mine = lane < a.block && w0 + lane < a.words;
            const uint32_t rw = mine ? __ldcg(a.removed + w0 + lane) : 0u;   // written by this thread
            if (rw) __stcg(a.removed + w0 + lane, 0u);
            const uint32_t n_rows = list_bits(s_list[warp], rw, lane);
            for (uint32_t t = 0; t < n_rows; t += 32) {
                const bool gone = t + lane < n_rows;
                const uint32_t v = (uint32_t)w0 * 32 + (gone ? s_list[warp][t + lane] : 0u);
                uint32_t i = gone ? __ldg(a.off + v) : 0u;
                const uint32_t e = gone ? __ldg(a.off + v + 1) : 0u;
                const bool is_long = e - i > kProbe;
                if (!is_long)
                    for (; i < e; i += 4) {
                        uint32_t n[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) n[j] = i + j < e ? __ldg(a.adj + i + j) : ~0u;
                        lower4(n);
                    }
                uint32_t more = __ballot_sync(kFull, is_long);
                while (more) {
                    const uint32_t l = __ffs(more) - 1;
                    more &= more - 1;
                    const uint32_t b = __shfl_sync(kFull, i, l), re = __shfl_sync(kFull, e, l);
                    if (re - b > kLongRow) {   // the grid takes it, chunk by chunk
                        const uint32_t n = (re - b + kChunk - 1) / kChunk;
                        uint32_t at = 0;
                        if (lane == 0) at = atomicAdd(c->n_items + (round & 3), n);
                        at = __shfl_sync(kFull, at, 0);
                        // chunks past the list's end are taken here
                        for (uint32_t j = 0; j < n; ++j) {
                            const uint32_t cb = b + j * kChunk, ce = min(cb + kChunk, re);
                            if (at + j >= a.cap) lower_row(cb, ce);
                            else if (lane == 0) a.items[at + j] = AdjItem{0u, cb, ce};
                        }
                    } else {
                        lower_row(b, re);
                    }
                }
            }
            __syncwarp();   // s_list is rewritten
        }
        if (!grid_barrier(c->bar, &c->err)) return;
        const uint32_t n_items = min(__ldcg(c->n_items + (round & 3)), a.cap);
        if (n_items) {
            for (uint32_t i = gw; i < n_items; i += nwarps) {
                const AdjItem it = load_item(a.items + i);
                lower_row(it.beg, it.end);
            }
            if (!grid_barrier(c->bar, &c->err)) return;
        }
    }
}

// -------------------------------------------------------------------- WCC --
// Root of v's tree, read through L1: a stale parent is still an ancestor, so
// the result is an ancestor that was a root when its line was read.  The
// compare-and-swap of hook() is what decides; after a failed one the roots
// are found again through L2.  (Every vertex of the largest tree points at one
// root, whose own entry all warps would otherwise read from one L2 slice.)
__device__ __forceinline__ uint32_t find_root_l1(uint32_t* parent, uint32_t v) {
    const uint32_t first = parent[v];
    uint32_t r = first, p = first;
    if (first == v) return v;
    while ((p = parent[r]) != r) r = p;
    if (r != first) __stcg(parent + v, r);   // v is no root and never becomes one again
    return r;
}

__device__ __forceinline__ bool hook_l1(uint32_t* parent, uint32_t a, uint32_t b) {
    const uint32_t ra = find_root_l1(parent, a), rb = find_root_l1(parent, b);
    if (ra == rb) return true;
    const uint32_t hi = ra > rb ? ra : rb, lo = ra > rb ? rb : ra;
    if (atomicCAS(parent + hi, hi, lo) == hi) return true;   // parents are smaller than children: no cycle
    return hook(parent, hi, lo);
}

// The hubs hooked to their first neighbours (hubs themselves, as the lists go),
// a neighbour a launch, each followed by pointing every hub at its root: after
// the first round most hubs share a root and the others' hooks find it in two
// reads.  (All links in one launch contend for the few roots left: 370-405 us at
// Kronecker 25 instead of 245.)
constexpr uint32_t kHubLinks = 3;
__global__ void wcc_adj_hub_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj,
                                   const uint32_t* __restrict__ hubs, uint32_t n, uint32_t link, uint32_t* parent,
                                   unsigned long long* unresolved) {
    const uint32_t nth = gridDim.x * blockDim.x;
    uint32_t bad = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth) {
        const uint32_t v = __ldg(hubs + i), at = __ldg(off + v) + link;
        if (at < __ldg(off + v + 1)) bad += !hook_l1(parent, v, __ldg(adj + at));
    }
    warp_add_u64(unresolved, bad);
}

__global__ void wcc_adj_hub_root_kernel(const uint32_t* __restrict__ hubs, uint32_t n, uint32_t* parent) {
    const uint32_t nth = gridDim.x * blockDim.x;
    uint32_t known = ~0u, first;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nth) {
        const uint32_t v = hubs[i], r = find_root_known(parent, v, known, &first);
        if (r != first) parent[v] = r;
    }
}

// Every other vertex hooked to its first neighbour, four a thread in flight:
// nearly all of the largest tree.  A vertex of a record is touched
// (wcc.cpp:203-217).
__global__ void wcc_adj_first_kernel(const uint32_t* __restrict__ none, const uint32_t* __restrict__ first,
                                     const uint32_t* __restrict__ hub, const uint32_t* __restrict__ off_out,
                                     const uint32_t* __restrict__ adj_out, int directed, uint32_t* parent,
                                     uint8_t* __restrict__ touched, uint64_t N, unsigned long long* unresolved) {
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x, tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    // the pairs whose hook takes a search, run 32 at a time, one per lane (a
    // few lanes of nearly every warp: searched where they were found, their
    // chains of dependent reads took 280 of the 480 us at Kronecker 25)
    __shared__ uint2 s_q[8][64];
    uint2* q = s_q[threadIdx.x >> 5];
    uint32_t bad = 0, qn = 0;   // qn: uniform in the warp, below 32 between pushes
    auto push = [&](bool need, uint32_t v, uint32_t n) {
        const uint32_t bal = __ballot_sync(kFull, need);
        if (need) q[qn + __popc(bal & lt)] = make_uint2(v, n);
        qn += __popc(bal);
        __syncwarp();
        if (qn >= 32) {
            const uint2 mine = q[lane], rest = lane + 32 < qn ? q[lane + 32] : make_uint2(0, 0);
            __syncwarp();
            if (lane + 32 < qn) q[lane] = rest;
            qn -= 32;
            bad += !hook_l1(parent, mine.x, mine.y);
            __syncwarp();
        }
    };
    // (N is a multiple of 65,536: the warp stays together)
    for (uint64_t v0 = tid; v0 < N; v0 += 4 * nth) {
        uint32_t n[4], pn[4], rn[4];
        bool link[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint64_t v = v0 + j * nth;
            link[j] = v < N && !(__ldg(none + (v >> 5)) >> (v & 31) & 1u);
            n[j] = link[j] ? __ldg(first + v) : 0u;
            if (directed && v < N && !link[j]) {   // only out-entries?
                const uint32_t b = __ldg(off_out + v);
                link[j] = b < __ldg(off_out + v + 1);
                if (link[j]) n[j] = __ldg(adj_out + b);
            }
            if (link[j]) touched[v] = 1;
            link[j] = link[j] && !(__ldg(hub + (v >> 5)) >> (v & 31) & 1u);
        }
        // a neighbour's root is its parent more often than not
#pragma unroll
        for (int j = 0; j < 4; ++j) pn[j] = link[j] ? parent[n[j]] : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) rn[j] = link[j] ? parent[pn[j]] : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t v = (uint32_t)(v0 + j * nth);
            // v is mostly still alone: linked under the neighbour's root at once
            const bool at_once = link[j] && rn[j] == pn[j] && pn[j] < v && atomicCAS(parent + v, v, pn[j]) == v;
            link[j] = link[j] && !at_once;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) push(link[j], (uint32_t)(v0 + j * nth), n[j]);
    }
    if (lane < qn) bad += !hook_l1(parent, q[lane].x, q[lane].y);
    warp_add_u64(unresolved, bad);
}

// The entries of the vertices outside the largest tree (bit clear in `giant`):
// the records with both ends in it join nothing new.  A vertex that has joined
// it meanwhile is done too -- a neighbour still outside has the record in its
// own list.  A warp takes 32 words and compacts their vertices; short rows a
// lane each, long ones the warp together.
__global__ void wcc_adj_rest_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj,
                                    const uint32_t* __restrict__ none, uint32_t* parent,
                                    const uint32_t* __restrict__ giant, const uint32_t* __restrict__ root,
                                    uint64_t words, unsigned long long* unresolved) {
    __shared__ uint16_t s_list[8][1024];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t step = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint32_t c = *root;   // ~0: no tree was found
    uint32_t bad = 0;
    auto joined = [&](uint32_t v) { return c != ~0u && find_root_l1(parent, v) == find_root_l1(parent, c); };
    for (uint64_t w0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; w0 < words; w0 += step * 32) {
        const uint64_t w = w0 + lane;
        const uint32_t n = list_bits(s_list[warp], w < words ? ~(__ldg(giant + w) | (none ? __ldg(none + w) : 0u)) : 0u,
                                     lane);
        for (uint32_t t = 0; t < n; t += 32) {
            const bool has = t + lane < n;
            const uint32_t v = (uint32_t)w0 * 32 + (has ? s_list[warp][t + lane] : 0u);
            const uint32_t b = has ? __ldg(off + v) : 0u, e = has ? __ldg(off + v + 1) : 0u;
            const bool is_long = e - b > kProbe;
            if (!is_long)
                for (uint32_t i = b; i < e; ++i) {
                    bad += !hook_l1(parent, v, __ldg(adj + i));
                    if ((i - b) % 4 == 0 && joined(v)) break;
                }
            uint32_t more = __ballot_sync(kFull, is_long);
            while (more) {
                const uint32_t l = __ffs(more) - 1;
                more &= more - 1;
                const uint32_t lb = __shfl_sync(kFull, b, l), le = __shfl_sync(kFull, e, l), lv = __shfl_sync(kFull, v, l);
                for (uint32_t i = lb; i < le; i += 32) {   // uniform
                    if (i + lane < le) bad += !hook_l1(parent, lv, __ldg(adj + i + lane));
                    if (__any_sync(kFull, lane == 0 && joined(lv))) break;
                }
            }
        }
        __syncwarp();   // s_list is rewritten
    }
    warp_add_u64(unresolved, bad);
}

// CTAs of a cooperative launch over `words` 32-vertex words.
template <class K>
gs_status coop_grid(gs_ctx* ctx, K kernel, int* per_sm, uint64_t words, uint32_t* grid, uint32_t* block) {
    if (*per_sm == 0) {
        GS_CHECK_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kernel, kThreads, 0));
        *per_sm = std::max(1, std::min(*per_sm, kCtas));
    }
    const uint64_t most = (uint64_t)ctx->num_sms * *per_sm;
    *grid = (uint32_t)std::clamp<uint64_t>((words + kWarps - 1) / kWarps, 1, most);
    // words a warp takes at a time: 32 (one line) while that leaves every warp two turns
    *block = 32;
    while (*block > 1 && words < (uint64_t)*block * *grid * kWarps * 2) *block /= 2;
    return GS_OK;
}

// The first in-entry of every vertex that has one.
__global__ void adj_first_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj, uint64_t N,
                                 uint32_t* __restrict__ first) {
    const uint64_t nth = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < N; v += nth)
        first[v] = off[v] < off[v + 1] ? adj[off[v]] : 0u;
}

// Entries of all lists together.
uint64_t n_lists(const gs_graph* g) { return 2 * g->E; }

uint32_t items_cap(const gs_graph* g) {
    return (uint32_t)(std::min<uint64_t>(g->N / 16, 1u << 20) + n_lists(g) / kChunk + 4096);
}

gs_status adj_build(gs_graph* g) {
    gs_ctx* ctx = g->ctx;
    gs_adj& A = g->adj;
    const uint64_t N = g->N, E = g->E, words = N / 32;
    const uint32_t U = (uint32_t)g->U;
    const bool dir = g->directed != 0;
    const uint32_t many = gs_grid_size(ctx, 8);
    cudaStream_t q = ctx->stream;
    size_t scan_bytes = 0, sort_bytes = 0;
    GS_CHECK_CUDA(ctx, cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                                     N + 1, q));
    GS_CHECK_CUDA(ctx, cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                                       (const uint32_t*)nullptr, (uint32_t*)nullptr, U, 0, 16, q));
    const size_t cub_bytes = (std::max(scan_bytes, sort_bytes) + 255) & ~(size_t)255;
    // scratch: a scalar and the tickets, cub's, the unit orders, the cursors
    const uint64_t u4 = ((uint64_t)U + 63) & ~63ull;
    const size_t tmp_bytes = 256 + cub_bytes + u4 * 4 * 5 + N * 4 * (dir ? 3 : 2);
    char* tmp = nullptr;
    gs_status st = gs_dev_alloc(ctx, (void**)&tmp, tmp_bytes);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&A.off_in, (N + 1) * 4);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&A.adj_in, std::max<uint64_t>(1, dir ? E : 2 * E) * 4);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&A.none, words * 4);
    const uint32_t hub_cap = (uint32_t)(N / 32);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&A.hub, words * 4);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&A.hubs, (uint64_t)hub_cap * 4);
    if (st == GS_OK) st = gs_dev_alloc(ctx, (void**)&A.first_in, N * 4);
    if (st == GS_OK && dir) st = gs_dev_alloc(ctx, (void**)&A.off_out, (N + 1) * 4);
    if (st == GS_OK && dir) st = gs_dev_alloc(ctx, (void**)&A.adj_out, std::max<uint64_t>(1, E) * 4);
    cudaError_t e = cudaSuccess;
    if (st == GS_OK) {
        if (!dir) {
            A.off_out = A.off_in;
            A.adj_out = A.adj_in;
        }
        unsigned long long* d_some = (unsigned long long*)tmp;
        char* cub_tmp = tmp + 256;
        uint32_t* key0 = (uint32_t*)(cub_tmp + cub_bytes);
        uint32_t *key1 = key0 + u4, *idx = key1 + u4, *order[2] = {idx + u4, idx + 2 * u4};   // by row, by column
        uint32_t* front = idx + 3 * u4;
        uint32_t *back = front + N, *cursor = back + N;
        A.n_in = dir ? E : 2 * E;
        const uint32_t part = U / g->nw + 1;
        unsigned int* ticket = (unsigned int*)tmp + 8;   // one per pass over the units
        auto run = [&](cudaError_t x) {
            if (e == cudaSuccess) e = x;
            return e == cudaSuccess;
        };
        for (int by_col = 0; by_col < 2 && e == cudaSuccess; ++by_col) {
            adj_unit_key_kernel<<<blocks_for(U, ctx), 256, 0, q>>>(g->d_units, U, by_col, key0, idx);
            run(cub::DeviceRadixSort::SortPairs(cub_tmp, sort_bytes, key0, key1, idx, order[by_col], U, 0, 16, q));
        }
        // the counts go into the offset arrays and are scanned in place
        run(cudaMemsetAsync(front, 0, N * 4 * (dir ? 3 : 2), q));
        run(cudaMemsetAsync(tmp, 0, 256, q));
        run(cudaMemsetAsync(A.off_in + N, 0, 4, q));
        if (!dir && g->degree_from_records) {
            run(cudaMemcpyAsync(A.off_in, g->d_degree, N * 4, cudaMemcpyDeviceToDevice, q));
        } else {
            run(cudaMemsetAsync(A.off_in, 0, N * 4, q));
            if (dir) run(cudaMemsetAsync(A.off_out, 0, (N + 1) * 4, q));
            if (e == cudaSuccess) {
                adj_count_kernel<<<many, 256, 0, q>>>(g->d_units, order[0], U, part, ticket + 0, g->d_rec, 0, A.off_out);
                adj_count_kernel<<<many, 256, 0, q>>>(g->d_units, order[1], U, part, ticket + 1, g->d_rec, 1, A.off_in);
            }
        }
        if (e == cudaSuccess) adj_none_kernel<<<blocks_for(N, ctx), 256, 0, q>>>(A.off_in, N, A.none, d_some);
        run(cudaMemcpyAsync(ctx->h_scalars, d_some, 8, cudaMemcpyDeviceToHost, q));
        if (run(cudaStreamSynchronize(q))) {
            A.n_cand = ctx->h_scalars[0];
            // 32 times the mean: the bottom-up level that counts has a frontier of
            // the largest hubs only (17 roots at Kronecker 26, mean: 4 times the
            // mean 0.95 ms, 8 0.93, 16 0.90, 32 and 64 0.84)
            const uint32_t least = (uint32_t)std::min<uint64_t>(
                32 * ((A.n_in + A.n_cand - 1) / std::max<uint64_t>(1, A.n_cand)), 0xFFFFFFFFu);
            // (so at most one vertex in 32 is a hub)
            adj_hub_kernel<<<blocks_for(N, ctx), 256, 0, q>>>(A.off_out, N, least, A.hub, A.hubs, hub_cap,
                                                              (unsigned int*)tmp + 2);
            run(cudaMemcpyAsync(ctx->h_scalars, tmp, 16, cudaMemcpyDeviceToHost, q));
        }
        run(cub::DeviceScan::ExclusiveSum(cub_tmp, scan_bytes, (const uint32_t*)A.off_in, A.off_in, N + 1, q));
        if (dir) run(cub::DeviceScan::ExclusiveSum(cub_tmp, scan_bytes, (const uint32_t*)A.off_out, A.off_out, N + 1, q));
        if (e == cudaSuccess) {
            adj_fill_kernel<<<many, 256, 0, q>>>(g->d_units, order[0], U, part, ticket + 2, g->d_rec, 0, dir ? nullptr : A.hub, A.off_out,
                                                 A.adj_out, dir ? cursor : front, back);
            adj_fill_kernel<<<many, 256, 0, q>>>(g->d_units, order[1], U, part, ticket + 3, g->d_rec, 1, A.hub, A.off_in, A.adj_in, front,
                                                 back);
            adj_first_kernel<<<blocks_for(N, ctx), 256, 0, q>>>(A.off_in, A.adj_in, N, A.first_in);
        }
        run(cudaGetLastError());
        run(cudaStreamSynchronize(q));
        A.n_hub = std::min<uint64_t>(((const uint32_t*)ctx->h_scalars)[2], hub_cap);
        ctx->launches += 14;
        if (e != cudaSuccess) st = gs_cuda_fail(ctx, e, "adjacency lists");
    }
    gs_dev_free(tmp);   // (waits for the build)
    if (st != GS_OK) {
        gs_adj_free(g);
        return st;
    }
    A.built = true;
    return GS_OK;
}

}  // namespace

void gs_adj_free(gs_graph* g) {
    gs_adj& A = g->adj;
    // not pool blocks: their gigabytes would keep the records of the next
    // uploads out of the pool
    if (A.off_out != A.off_in) gs_dev_free(A.off_out);
    if (A.adj_out != A.adj_in) gs_dev_free(A.adj_out);
    for (void* p : {(void*)A.off_in, (void*)A.adj_in, (void*)A.first_in, (void*)A.none, (void*)A.hub, (void*)A.hubs})
        gs_dev_free(p);
    const uint32_t credit = A.credit;
    A = gs_adj();
    A.credit = credit;
}

void gs_adj_credit(gs_graph* g, uint32_t sweeps) {
    if (!g->adj.built && g->adj.credit < kAdjBuild) g->adj.credit += sweeps;
}

bool gs_adj_ready(gs_graph* g, uint32_t sweeps) {
    gs_adj& A = g->adj;
    if (A.built) return true;
    if (g->stream || g->E == 0 || A.refused) return false;
    gs_ctx* ctx = g->ctx;
    if (A.credit < kAdjBuild) {
        gs_adj_credit(g, sweeps);
        return false;
    }
    A.refused = true;   // unless all goes well
    if (n_lists(g) >= (1ull << 32) - (1ull << 20)) return false;   // 32-bit offsets
    const uint64_t keep = n_lists(g) * 4 + g->N * (g->directed ? 13 : 9);
    if (ctx->budget && 4 * g->E + keep > ctx->budget) return false;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return false;
    if ((keep + g->N * 16 + g->U * 32) * 2 > free_b || g->U >= (1ull << 32)) return false;
    if (adj_build(g) != GS_OK) {
        A.refused = true;   // out of memory after all: the sweeps still run
        return false;
    }
    A.refused = false;
    ctx->adj_graphs.push_back(g);
    return true;
}

void gs_adj_release(gs_ctx* ctx) {
    if (ctx->adj_graphs.empty()) return;
    cudaStreamSynchronize(ctx->stream);
    for (gs_graph* g : ctx->adj_graphs) {
        gs_adj_free(g);
        g->adj.refused = true;
    }
    ctx->adj_graphs.clear();
}

// s->d_adj, which stays null when there is no memory for it (an allocation that
// fails drops the lists before it gives up).
static gs_status query_scratch(gs_state* s, size_t bytes) {
    if (s->d_adj) return GS_OK;
    const gs_status st = gs_state_alloc(s, &s->d_adj, bytes);
    return st == GS_ERR_OOM ? GS_OK : st;
}

gs_status bfs_adj_run(gs_state* s, int64_t* steps) {
    gs_graph* g = s->g;
    gs_ctx* ctx = g->ctx;
    if (s->on_lists) return s->lists_status;   // failed before: a reset starts anew
    const uint64_t words = g->N / 32;
    const uint32_t cap = items_cap(g);
    // both frontier queues, the long rows' chunks
    GS_TRY(query_scratch(s, (size_t)cap * (8 + sizeof(AdjItem))));
    const gs_adj& A = g->adj;
    if (!A.built || !s->d_adj) return GS_OK;   // no room: the sweeps need none
    s->on_lists = true;
    s->lists_status = GS_ERR_CUDA;             // unless all goes well
    static_assert(sizeof(BfsCtl) <= kBfsCtlBytes, "control block");
    BfsCtl* c = (BfsCtl*)s->d_bfs_ctl;   // zero since bfs_init
    uint32_t grid = 1, block = 32;
    GS_TRY(coop_grid(ctx, bfs_adj_kernel, &ctx->adj_ctas[0], words, &grid, &block));
    BfsArgs a{A.off_in, A.adj_in, A.first_in, A.off_out, A.adj_out, s->d_front, s->d_visited, s->d_depth,
              (uint32_t*)s->d_adj, (AdjItem*)((uint32_t*)s->d_adj + (size_t)cap * 2), cap, block, words, A.n_cand, A.n_in,
              s->d_read, c};
    bfs_adj_seed_kernel<<<blocks_for(words, ctx), 256, 0, ctx->stream>>>(a, A.none, (uint32_t)s->arg);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    void* args[] = {&a};
    gs_timer_begin(ctx);
    GS_CHECK_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)bfs_adj_kernel, dim3(grid), dim3(kThreads), args, 0,
                                                   ctx->stream));
    ctx->launches += 2;
    gs_timer_end(ctx, GS_ALGO_BFS, 0);
    BfsCtl h;
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(&h, c, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (h.err) {
        s->lists_status = GS_ERR_TIMEOUT;
        return gs_fail(ctx, GS_ERR_TIMEOUT, "BFS: a grid barrier wait gave up");
    }
    s->lists_status = h.overflow ? GS_ERR_RANGE : GS_OK;
    s->level_counts.assign(h.total + 1, h.total + h.levels + 1);
    s->level_skip.assign(h.levels, 1);   // entries read are counted
    s->level = (uint8_t)h.levels;
    s->step = h.levels;
    s->swept = false;
    s->last_count = 0;
    *steps = h.levels;
    if (h.overflow) return gs_fail(ctx, GS_ERR_RANGE, "BFS exceeds 254 levels (u8 depth_t)");
    s->done = true;
    return GS_OK;
}

gs_status kcore_adj_run(gs_state* s, int64_t* steps) {
    gs_graph* g = s->g;
    gs_ctx* ctx = g->ctx;
    const uint64_t words = g->N / 32;
    const uint32_t cap = (uint32_t)(n_lists(g) / kChunk + 4096);
    const size_t item_bytes = ((size_t)cap * sizeof(AdjItem) + 255) & ~(size_t)255;
    // the row chunks, the control block and the candidates
    GS_TRY(query_scratch(s, item_bytes + 256 + words * 4));
    const gs_adj& A = g->adj;
    if (!A.built || !s->d_adj) return GS_OK;   // no room: the sweeps need none
    static_assert(sizeof(KcoreCtl) <= 256, "control block");
    KcoreCtl* c = (KcoreCtl*)((char*)s->d_adj + item_bytes);
    GS_CHECK_CUDA(ctx, cudaMemsetAsync(c, 0, 256 + words * 4, ctx->stream));
    uint32_t grid = 1, block = 32;
    GS_TRY(coop_grid(ctx, kcore_adj_kernel, &ctx->adj_ctas[1], words, &grid, &block));
    KcoreArgs a{A.off_in, A.adj_in, s->d_deg, s->d_kactive, (uint32_t*)((char*)c + 256), (AdjItem*)s->d_adj, cap, block,
                words, (int)s->arg, c};
    void* args[] = {&a};
    gs_timer_begin(ctx);
    GS_CHECK_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)kcore_adj_kernel, dim3(grid), dim3(kThreads), args, 0,
                                                   ctx->stream));
    ctx->launches += 1;
    gs_timer_end(ctx, GS_ALGO_KCORE, 0);   // (the entries read depend on the rounds: no bytes claimed)
    KcoreCtl h;
    GS_CHECK_CUDA(ctx, cudaMemcpyAsync(&h, c, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
    GS_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (h.err) return gs_fail(ctx, GS_ERR_TIMEOUT, "k-core: a grid barrier wait gave up");
    s->step = h.rounds;
    s->last_count = 0;
    s->done = true;
    *steps = h.rounds;
    return GS_OK;
}

gs_status wcc_adj_hook(gs_state* s, void (*vote)(gs_state*), unsigned long long* unresolved) {
    gs_graph* g = s->g;
    gs_ctx* ctx = g->ctx;
    const gs_adj& A = g->adj;
    const uint64_t N = g->N, words = N / 32;
    const uint32_t grid = gs_grid_size(ctx, 8), by_block = (uint32_t)std::min<uint64_t>((words + 255) / 256, grid);
    const uint32_t by_hub = (uint32_t)std::min<uint64_t>((A.n_hub + 255) / 256, grid);
    for (uint32_t link = 0; link < kHubLinks && A.n_hub; ++link) {
        wcc_adj_hub_kernel<<<by_hub, 256, 0, ctx->stream>>>(A.off_in, A.adj_in, A.hubs, (uint32_t)A.n_hub, link,
                                                            s->d_parent, unresolved);
        wcc_adj_hub_root_kernel<<<by_hub, 256, 0, ctx->stream>>>(A.hubs, (uint32_t)A.n_hub, s->d_parent);
        ctx->launches += 2;
    }
    wcc_adj_first_kernel<<<(uint32_t)std::min<uint64_t>((N + 1023) / 1024, grid), 256, 0, ctx->stream>>>(
        A.none, A.first_in, A.hub, A.off_out, A.adj_out, g->directed, s->d_parent, s->d_touched, N, unresolved);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    vote(s);
    const uint32_t* root = s->d_giant + words;
    wcc_adj_rest_kernel<<<by_block, 256, 0, ctx->stream>>>(A.off_in, A.adj_in, A.none, s->d_parent, s->d_giant, root,
                                                           words, unresolved);
    if (g->directed)
        wcc_adj_rest_kernel<<<by_block, 256, 0, ctx->stream>>>(A.off_out, A.adj_out, nullptr, s->d_parent, s->d_giant,
                                                               root, words, unresolved);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches += g->directed ? 3 : 2;
    return GS_OK;
}

gs_status gs_level_windows(gs_state* s, int levels) {
    gs_graph* g = s->g;
    gs_ctx* ctx = g->ctx;
    if (!s->d_act_hist) GS_TRY(gs_state_alloc(s, (void**)&s->d_act_hist, (size_t)g->nw * 256));
    depth_windows_kernel<<<std::min<uint32_t>(g->nw, gs_grid_size(ctx, 4)), 256, 0, ctx->stream>>>(s->d_depth, g->nw,
                                                                                                 levels, s->d_act_hist);
    GS_CHECK_CUDA(ctx, cudaGetLastError());
    ctx->launches++;
    return GS_OK;
}
