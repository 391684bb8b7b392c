// walk_whole.cu -- persistent step kernel for a graph resident in HBM.
//
// Replaces randomWalkKernel / randomWalkInsidePool[AllBatch]
// (src/WalkManager.h:229-274) for the case where every partition is cached on
// the device: walkers never need re-bucketing, so each one is stepped from
// creation to termination without leaving the SM.
//
// Design (GB300-first):
//  * Persistent grid: SMs x resident CTAs; each lane owns one walker at a time.
//  * Lazy walker creation: walker i is created from its index alone (start
//    vertex and, for PPR, its geometric length are pure functions of
//    (seed, run, i)), so no walker array is ever materialised.  The first
//    walkers are dealt out; a warp takes further ones from an atomic counter
//    (one atomic per refill; PPR: per pool of walkers with their lengths
//    drawn), keeping its lanes busy despite the spread of PPR's lengths.
//  * Graph reads: rowptr[cur], rowptr[cur+1] (16 B) and col[e] (4 B) through
//    the read-only path; counters are u64 reductions resolved in L2.  Column
//    loads are evict-first, row offsets and counters evict-last (mem.cuh).
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.h"
#include "lt_core.cuh"
#include "mem.cuh"
#include "ppr_pool.cuh"
#include "walk_whole.h"

namespace lt {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
// idle lanes a warp waits for before it asks for more walkers (PPR: for
// another pool, whose lengths it then draws)
constexpr int kRefillMin = 16;
// PPR: idle lanes before a warp takes walkers out of its pool (2|V| walks on
// RMAT 2^20 / 2^24, whole call: 1 224 us, 4 223, 8 219, 12 222)
constexpr int kTakeMin = 8;

struct Hints {
    uint64_t keep, stream;
};

// first edge and degree of v
template <int L>
struct Row {
    using Edge = typename std::conditional<L == kLayoutWide, uint64_t, uint32_t>::type;
    Edge first, deg;
};

template <int L>
__device__ __forceinline__ Row<L> row_range(const WholeArgs &a, uint32_t v, const Hints &h)
{
    Row<L> r;
    if constexpr (L == kLayoutPacked) {
        // the even words never change during a launch (only the counters
        // beside them do), so the read-only path serves them
        r.first = ld_nc_u32(a.rows + 2ull * v, h.keep);
        r.deg = ld_nc_u32(a.rows + 2ull * v + 2, h.keep) - r.first;
    } else if constexpr (L == kLayoutCompact) {
        r.first = ld_nc_u32(a.rowptr32 + v, h.keep);
        r.deg = ld_nc_u32(a.rowptr32 + v + 1, h.keep) - r.first;
    } else {
        r.first = ld_nc_u64(a.rowptr + v, h.keep);
        r.deg = ld_nc_u64(a.rowptr + v + 1, h.keep) - r.first;
    }
    return r;
}

// the neighbour that draw r picks from a row that is not empty
template <int L>
__device__ __forceinline__ uint32_t pick(const WholeArgs &a, const Row<L> &row, const Rand4 &r, const Hints &h)
{
    return ld_nc_stream64_u32(a.col + row.first + mod_u64(r64_of(r), row.deg), h.stream);
}

template <int L>
__device__ __forceinline__ void count_n(const WholeArgs &a, uint32_t v, uint32_t n, const Hints &h)
{
    if (L == kLayoutPacked)
        red_add_u32(a.rows + 2ull * v + 1, n, h.keep);
    else if (L == kLayoutCompact)
        red_add_u32(a.counts32 + v, n, h.keep);
    else
        red_add_u64((unsigned long long *)(a.counts + v), n, h.keep);
}
template <int L>
__device__ __forceinline__ void count1(const WholeArgs &a, uint32_t v, const Hints &h)
{
    count_n<L>(a, v, 1, h);
}

// Hub counters of PageRank.  Counter updates crowd the few lines that hold the
// hubs' counters (RMAT 2^23 / 2^27: 1 % of 92 M updates go to one line), and
// the L2 slice of such a line, at 105 % of its tag rate against 64 % on
// average, set the kernel's time.  A CTA therefore counts up to 4096 vertices
// of at least E / 2^15 out-edges in shared memory and adds them up once at its
// end; a vertex takes its slot at its first visit whose row is read (the first
// to come keeps it: a hub is likely to be that).  The CTAs are as large as they
// can be: each adds up its own table, which for a short launch on a small graph
// is as much traffic as the updates it spares.  No tables -> 512 slots (from
// E / 2^13) and 256 threads -> this: 10 steps from 3 million vertices drawn on
// RMAT 2^16 / 7e5 - -> 515 -> 274 us, on 2^18 / 2^22 - -> 369 -> 289, on 2^20 /
// 2^24 - -> 376 -> 306; RMAT 2^23 / 2^27 1759 -> 1557 -> 1561, u64 on RMAT 2^21 /
// 4e7 228 -> 201 -> 190.  512 slots and 1024 threads on 2^16 495, 1024 slots 348,
// 2048 293; serving the hubs' rows from shared memory as well gave nothing.
constexpr int kHotBits = 12;
constexpr uint32_t kHotSlots = 1u << kHotBits;
constexpr uint32_t kHotMinDegree = 64;
constexpr uint32_t kNoVertex = 0xFFFFFFFFu;

template <int L>
__device__ __forceinline__ uint32_t hot_degree(const WholeArgs &a)
{
    const uint64_t E = L == kLayoutPacked ? a.rows[2ull * a.V] : L == kLayoutCompact ? a.rowptr32[a.V] : a.rowptr[a.V];
    return (uint32_t)min(0xFFFFFFFFull, max((unsigned long long)kHotMinDegree, (unsigned long long)E >> 15));
}

template <int START>
__device__ __forceinline__ uint32_t first_vertex(const WholeArgs &a, uint64_t idx)
{
    if (START == kStartSource) return a.source;
    if (START == kStartPerVertex) return mod_by(a.by_v, idx);
    return mod_by(a.by_v, r64_of(walk_draw(a.keys, 0, kTagInit, a.run, idx)));
}

// Makes the draw here: the compiler would move it behind the branch on the
// row's degree, where it would wait for the row's loads first.
template <int APP>
__device__ __forceinline__ void settle(Rand4 &r)
{
    asm volatile("" : "+r"(r.x0), "+r"(r.x1));
    if (APP == kPageRank) asm volatile("" : "+r"(r.x2), "+r"(r.x3));
}

// n more walkers for the calling warp: the first one's index past the dealt ones
__device__ __forceinline__ uint64_t take(uint64_t *next, uint32_t n)
{
    unsigned long long got = 0;
    if ((threadIdx.x & 31) == 0) got = atomicAdd((unsigned long long *)next, (unsigned long long)n);
    return __shfl_sync(kFull, got, 0);
}

// Paths of generic walks.  A lane gathers up to kPathWords vertices of its path
// in shared memory; the warp writes the segments of its lanes that are full or
// ended, 16 threads to a segment, so that a store instruction covers two
// segments instead of 32 scattered words (one L2 request each).  4.7 M walks of
// 10 hops on RMAT 2^22 / 2^26 637 -> 602 us, 1 M of 40 hops on 2^18 / 2^22 518
// -> 448 us.  Walks of fewer than kPathGatherMin hops are too short for it
// (5 hops: 64 -> 75 us, 9: 103 either way) and in a launch that does not fill
// the chip its instructions cost more than the requests (20 000 walks of 10
// hops: 30 -> 33 us; 400 000 of 20: 97 -> 101): two walkers per lane of the chip
// at least.
constexpr uint32_t kPathWords = 16, kPathStride = kPathWords + 1;  // an odd stride: no bank conflicts
constexpr uint32_t kPathGatherMin = 10;
constexpr size_t kPathSmem = 4ull * kWholeBlock * kPathStride;

struct PathSegment {
    uint32_t *buf;  // of this lane
    uint32_t *out;  // where buf[0] goes
    uint32_t n;     // vertices gathered
};

// Writes the segments of the lanes with `due`; the whole warp, converged.
__device__ __forceinline__ void path_flush(PathSegment &p, bool due)
{
    unsigned m = __ballot_sync(kFull, due && p.n != 0u);
    __syncwarp();
    const uint32_t lane = threadIdx.x & 31u, w = lane & (kPathWords - 1u);
    const uint32_t *warp_buf = p.buf - lane * kPathStride;
    while (m) {
        uint32_t src = (uint32_t)__ffs((int)m) - 1u;
        m &= m - 1u;
        const bool second = m != 0u;
        if (lane >= 16u && second) src = (uint32_t)__ffs((int)m) - 1u;
        if (second) m &= m - 1u;
        const uint32_t n = __shfl_sync(kFull, p.n, src);
        uint32_t *out = (uint32_t *)__shfl_sync(kFull, (unsigned long long)p.out, src);
        if (w < n && (lane < 16u || second)) out[w] = warp_buf[src * kPathStride + w];
    }
    __syncwarp();
    if (due) {
        p.out += p.n;
        p.n = 0;
    }
}

// Threads of a CTA (2048 per SM either way): PageRank's share the hub counters.
template <int APP>
constexpr int block_of = APP == kPageRank ? 1024 : kWholeBlock;

// GATHER: paths go through shared memory (kWalk only).
template <int APP, int START, int C, bool GATHER>
__global__ void __launch_bounds__(block_of<APP>, 2048 / block_of<APP>) walk_whole_kernel(const __grid_constant__ WholeArgs a)
{
    const int lane = threadIdx.x & 31;
    const Hints h{l2_policy_evict_last(), l2_policy_evict_first()};

    uint32_t cur = 0, step = 0;
    uint64_t idx = 0;
    bool active = false;
    // walkers no longer to be had: the counter has passed W
    bool exhausted = false;
    // the first walkers are dealt out without the counter, 32 (PPR: a pool) to
    // each warp, the warps of the same number in their CTAs before the next
    // ones, so that few walkers spread over all SMs
    const uint64_t dealt = (uint64_t)gridDim.x * (APP == kPPR ? kWholeBlock / 32 * a.pool : block_of<APP>);
    bool first_deal = true;
    // PPR: the warp's pool of walkers with their lengths drawn
    __shared__ PprPool pools[APP == kPPR ? kWholeBlock / 32 : 1];
    PprPool &pool = pools[APP == kPPR ? threadIdx.x >> 5 : 0];
    uint32_t pool_at = 0, pool_n = 0;
    uint64_t pool_base = 0;
    extern __shared__ uint32_t path_buf[];  // GATHER: kPathSmem bytes
    PathSegment path{path_buf + threadIdx.x * kPathStride, nullptr, 0};
    constexpr bool kHot = APP == kPageRank;
    __shared__ uint32_t hot_v[kHot ? kHotSlots : 1], hot_n[kHot ? kHotSlots : 1];
    uint32_t hot_min = 0;
    if (kHot) {
        for (uint32_t i = threadIdx.x; i < kHotSlots; i += block_of<APP>) {
            hot_v[i] = a.hot ? kNoVertex : kNoVertex - 1u;  // free, or taken
            hot_n[i] = 0;
        }
        hot_min = hot_degree<C>(a);
        __syncthreads();
    }
    uint32_t n_mov = 0, n_end = 0;  // hops taken; walks that ended at a vertex without out-edges
    Rand4 r{};                      // PageRank: the draw of the walker's next step

    // one hop or update of the lane's walker
    auto hop = [&]() {
        // The draws do not depend on the graph: they are made between the
        // row's loads and their first use.
        if (APP == kPPR) {
            // app/ppr.cu:22-42; step >= 2 here, and a walk whose step comes
            // down to 1 is counted right away
            const Row<C> row = row_range<C>(a, cur, h);
            r = walk_draw(a.keys, step, kTagStep, a.run, idx);
            settle<APP>(r);
            if (row.deg > 0) {
                cur = pick<C>(a, row, r, h);
                n_mov++;
                step--;
            } else {
                step = 1;
            }
            active = step != 1;
            if (!active) count1<C>(a, cur, h);
        } else if (APP == kPageRank) {
            // app/pagerank.cu:26-44; a vertex without out-edges teleports.
            const uint32_t slot = (cur * 0x9E3779B1u) >> (32 - kHotBits);
            const uint32_t held = *(volatile uint32_t *)&hot_v[slot];
            if (held == cur)
                atomicAdd(&hot_n[slot], 1u);
            else
                count1<C>(a, cur, h);
            step--;
            if (step == 0) {
                active = false;
            } else {
                const Rand4 now = r;
                Row<C> row{};
                if (below(now, a.lim)) row = row_range<C>(a, cur, h);
                r = walk_draw(a.keys, step, kTagStep, a.run, idx);
                settle<APP>(r);
                if (held == kNoVertex && row.deg >= hot_min) atomicCAS(&hot_v[slot], kNoVertex, cur);
                if (row.deg > 0) {
                    cur = pick<C>(a, row, now, h);
                    n_mov++;
                } else {
                    cur = mod_by(a.by_v, r64_of(now));
                }
            }
        } else {
            // app/genericwalk.cu:22-32
            const Row<C> row = row_range<C>(a, cur, h);
            r = walk_draw(a.keys, step, kTagStep, a.run, idx);
            settle<APP>(r);
            uint32_t *out = !GATHER && a.paths ? a.paths + idx * (uint64_t)(a.length + 1) + (a.length - step) : nullptr;
            if (row.deg > 0) {
                cur = pick<C>(a, row, r, h);
                n_mov++;
                if (GATHER)
                    path.buf[path.n++] = cur;
                else if (out)
                    out[1] = cur;
                step--;
            } else {
                // the rest of the path (gathered as far as it fits)
                if (GATHER) {
                    const uint32_t fits = min(step, kPathWords - path.n);
                    for (uint32_t k = 0; k < fits; k++) path.buf[path.n + k] = kInvalidNode;
                    path.n += fits;
                    for (uint32_t k = fits; k < step; k++) path.out[path.n + (k - fits)] = kInvalidNode;
                } else if (out) {
                    for (uint32_t k = 1; k <= step; k++) out[k] = kInvalidNode;
                }
                n_end++;
                step = 0;
            }
            active = step != 0;
        }
        if (!active && a.endpoints) a.endpoints[idx] = cur;
    };

    while (true) {
        const unsigned busy = __ballot_sync(kFull, active);
        const int idle = 32 - __popc(busy);
        // ended walks keep their segments until a lane's is full or their lanes
        // are refilled (or nothing is left to do)
        if (GATHER && (__any_sync(kFull, path.n == kPathWords) || (exhausted ? idle == 32 : idle >= kRefillMin)))
            path_flush(path, path.n == kPathWords || !active);
        const uint32_t rank = __popc(~busy & ((1u << lane) - 1u));  // of an idle lane among them
        if (APP == kPPR) {
            if (pool_at == pool_n && idle >= kRefillMin && !exhausted) {
                pool_base = first_deal ? a.pool * ((uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x)
                                       : dealt + take(a.next, a.pool);
                first_deal = false;
                exhausted = pool_base + a.pool >= a.W;
                pool_at = 0;
                pool_n = pool_base >= a.W ? 0u : (uint32_t)min((uint64_t)a.pool, a.W - pool_base);
                ppr_pool_fill(pool, pool_n, a.long_len, a.lim, [&](uint32_t t, uint32_t at) {
                    return walk_draw(a.keys, t, kTagInit, a.run, pool_base + at);
                });
            }
            if (pool_at < pool_n && idle >= kTakeMin) {
                if (!active && pool_at + rank < pool_n) {
                    idx = pool_base + pool.at[pool_at + rank];
                    step = pool.len[pool_at + rank];
                    cur = first_vertex<START>(a, idx);
                    active = true;
                }
                pool_at = min(pool_n, pool_at + (uint32_t)idle);
            } else if (idle == 32 && exhausted) {
                break;
            }
        } else if (idle >= kRefillMin && !exhausted) {
            const uint64_t base = first_deal ? 32ull * ((uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x)
                                             : dealt + take(a.next, (uint32_t)idle);
            exhausted = first_deal ? dealt >= a.W : base + idle >= a.W;
            first_deal = false;
            if (!active && base + rank < a.W) {
                idx = (kHot ? a.first : 0u) + base + rank;
                cur = first_vertex<START>(a, idx);
                step = a.length;
                active = true;
                if (GATHER) {
                    path.out = a.paths + idx * (uint64_t)(a.length + 1);
                    path.buf[0] = cur;
                    path.n = 1;
                } else if (APP == kWalk && a.paths) {
                    a.paths[idx * (uint64_t)(a.length + 1)] = cur;
                }
                if (APP == kPageRank) r = walk_draw(a.keys, step, kTagStep, a.run, idx);
            }
        } else if (idle == 32) {
            break;
        }
        // No walkers to come: the lanes finish theirs without asking.  In a launch
        // that does not fill the chip a warp's instructions wait for one another,
        // and the votes and branches of a refill were a quarter of a hop's time
        // (device arrays, RMAT 2^16 / 2^20, p = 0.15: 5 000 PPR walks 41 -> 32 us,
        // 20 000 65 -> 49, 300 000 72 -> 61; 300 000 walks of 20 hops 44 -> 39;
        // 20 000 PageRank walks of 10 33 -> 30; large launches the same).
        if (!GATHER && exhausted && (APP != kPPR || pool_at == pool_n)) {
            while (active) hop();
            break;
        }
        if (active) hop();
    }

    // Statistics: one atomic per CTA and counter (one per warp would queue
    // some 30 000 atomics on one line at the end of every launch).  A PPR
    // walk makes one update per hop and one that ends it, a PageRank walk
    // a.length updates of which all but the last hop or teleport, a generic
    // walk one per hop and one where it ends early.
    if (kHot) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kHotSlots; i += block_of<APP>)
            if (hot_n[i]) count_n<C>(a, hot_v[i], hot_n[i], h);
    }
    if (!a.stats) return;
    __shared__ unsigned long long s_mov, s_end;
    if (threadIdx.x == 0) s_mov = s_end = 0;
    __syncthreads();
    uint64_t w_mov = n_mov, w_end = n_end;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        w_mov += __shfl_down_sync(kFull, w_mov, o);
        if (APP == kWalk) w_end += __shfl_down_sync(kFull, w_end, o);
    }
    if (lane == 0 && w_mov + w_end) {
        atomicAdd(&s_mov, (unsigned long long)w_mov);
        if (APP == kWalk) atomicAdd(&s_end, (unsigned long long)w_end);
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    unsigned long long upd = APP == kWalk ? s_mov + s_end : APP == kPPR ? s_mov : 0, tel = 0;
    if (APP == kPageRank) tel = 0ull - s_mov;
    if (blockIdx.x == 0) {
        if (APP == kPPR) upd += a.W;
        if (APP == kPageRank) {
            upd += a.W * a.length;
            tel += a.W * (a.length - 1);
        }
    }
    if (upd) atomicAdd((unsigned long long *)&a.stats[0], upd);
    if (s_mov) atomicAdd((unsigned long long *)&a.stats[1], s_mov);
    if (tel) atomicAdd((unsigned long long *)&a.stats[2], tel);
}

// CTAs of a launch with W walkers, at most: no more than have walkers, but one
// per SM.  PPR walks differ in length, so that a lane's second and third walker
// fill the time its warp would wait for its longest one: six walkers per lane
// (whole CTAs per SM, two at least, for the latencies of a graph in DRAM).  One
// walker per lane -> this, device arrays, p = 0.15: 150 000 walks on RMAT 2^16 /
// 7e5 59 -> 53 us, 300 000 86 -> 65, on 2^20 / 2^24 96 -> 84, on 2^22 / 2^26
// 106 -> 106; 600 000 105 -> 88, 114 -> 96, 128 -> 121; 1.2 million 126 -> 128,
// 140 -> 133, 171 -> 170.  Three walkers per lane 600 000 95, 103, 125; eight 88,
// 112, 128; one CTA per SM 150 000 on 2^22 / 2^26 101, two 95.
template <int APP>
uint64_t most_ctas(uint64_t W, int sms)
{
    const uint64_t full = std::max<uint64_t>(sms, (W + block_of<APP> - 1) / block_of<APP>);
    if (APP != kPPR) return full;
    const uint64_t six = sms * ((W - 1) / (6ull * sms * kWholeBlock) + 1);
    return std::min(full, std::max<uint64_t>(2ull * sms, six));
}

// A hub counter of a CTA has 32 bits, and nothing bounds the share of a launch's
// walkers that one CTA takes while others wait for SMs that another stream's
// kernels hold.  So PageRank calls of 2^32 updates and more become launches of
// fewer, one after the other, where each still fills the chip several times
// over (a launch's start and end are then 1e-4 of its time), and one launch
// without tables where the walks are too long for that.  4.8e9 updates in two
// launches, and in one without tables: RMAT 2^21 / 4e7 49.8 ms, 61.5; 2^23 / 2^27 93.0,
// 113.5; 2^16 / 2^20 34.0, 153.6.
constexpr uint64_t kHotUpdates = (1ull << 32) - 1;

uint64_t hot_walkers(uint32_t length) { return length ? kHotUpdates / length : 0; }

bool pagerank_hot(uint64_t W, uint32_t length, int sms)
{
    return W <= hot_walkers(length) || hot_walkers(length) >= 4 * 2048ull * sms;
}

template <int APP, int START, int C>
cudaError_t launch_t(const WholeArgs &a, int grid, cudaStream_t st)
{
    WholeArgs b = a;
    if constexpr (APP == kPageRank) {
        b.hot = pagerank_hot(a.W, a.length, a.sms);
        const uint64_t n = whole_launches(APP, a.W, a.length, a.sms);
        if (n > 1) {
            b.W = (a.W + n - 1) / n;
            for (b.first = 0; b.first < a.W; b.first += b.W) {
                b.W = std::min(b.W, a.W - b.first);
                if (b.first) {
                    const cudaError_t cleared = cudaMemsetAsync(b.next, 0, sizeof *b.next, st);
                    if (cleared != cudaSuccess) return cleared;
                }
                const int ctas = (int)std::min<uint64_t>((uint64_t)grid, most_ctas<APP>(b.W, a.sms));
                walk_whole_kernel<APP, START, C, false><<<ctas, block_of<APP>, 0, st>>>(b);
                const cudaError_t launched = cudaGetLastError();
                if (launched != cudaSuccess) return launched;
            }
            return cudaSuccess;
        }
    }
    grid = (int)std::min<uint64_t>((uint64_t)grid, most_ctas<APP>(a.W, a.sms));
    b.pool = pool_walkers(a.W, (uint64_t)grid * (kWholeBlock / 32));
    if constexpr (APP == kWalk) {
        if (a.paths && a.length >= kPathGatherMin && a.W > 2ull * a.sms * kWholeBlock * 8) {
            walk_whole_kernel<APP, START, C, true><<<grid, kWholeBlock, kPathSmem, st>>>(b);
            return cudaGetLastError();
        }
    }
    walk_whole_kernel<APP, START, C, false><<<grid, block_of<APP>, 0, st>>>(b);
    return cudaGetLastError();
}

template <int APP, int C>
cudaError_t launch_app(const WholeArgs &a, int start, int grid, cudaStream_t st)
{
    switch (start) {
    case kStartSource: return launch_t<APP, kStartSource, C>(a, grid, st);
    case kStartUniform: return launch_t<APP, kStartUniform, C>(a, grid, st);
    default: return launch_t<APP, kStartPerVertex, C>(a, grid, st);
    }
}

template <int APP, int START, int C>
int occupancy_t()
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, walk_whole_kernel<APP, START, C, false>, block_of<APP>, 0);
    return n;
}

template <int C>
int occupancy_c(int app, int start)
{
    switch (app * 3 + start) {
    case 0: return occupancy_t<kPPR, kStartSource, C>();
    case 1: return occupancy_t<kPPR, kStartUniform, C>();
    case 2: return occupancy_t<kPPR, kStartPerVertex, C>();
    case 3: return occupancy_t<kPageRank, kStartSource, C>();
    case 4: return occupancy_t<kPageRank, kStartUniform, C>();
    case 5: return occupancy_t<kPageRank, kStartPerVertex, C>();
    case 6: return occupancy_t<kWalk, kStartSource, C>();
    case 7: return occupancy_t<kWalk, kStartUniform, C>();
    default: return occupancy_t<kWalk, kStartPerVertex, C>();
    }
}

}  // namespace

uint64_t whole_launches(int app, uint64_t W, uint32_t length, int sms)
{
    if (app != kPageRank || !pagerank_hot(W, length, sms)) return 1;
    return (W + hot_walkers(length) - 1) / hot_walkers(length);
}

// SMs of the device and resident CTAs per SM of a kernel instance: properties
// of the device and the code, asked for once (the occupancy query costs a
// small call some 5 us).
namespace {
constexpr int kMaxDevices = 64;
std::atomic<int> g_sms[kMaxDevices], g_occ[kMaxDevices][3][9];
}  // namespace

int whole_sms(int device)
{
    int n = device < kMaxDevices ? g_sms[device].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
        if (device < kMaxDevices) g_sms[device].store(n, std::memory_order_relaxed);
    }
    return n;
}

int whole_grid(int app, int start, int device, int ctas_per_sm, int layout)
{
    int occ = device < kMaxDevices ? g_occ[device][layout][app * 3 + start].load(std::memory_order_relaxed) : 0;
    if (occ == 0) {
        occ = layout == kLayoutPacked    ? occupancy_c<kLayoutPacked>(app, start)
              : layout == kLayoutCompact ? occupancy_c<kLayoutCompact>(app, start)
                                         : occupancy_c<kLayoutWide>(app, start);
        if (occ < 1) occ = 1;
        if (device < kMaxDevices) g_occ[device][layout][app * 3 + start].store(occ, std::memory_order_relaxed);
    }
    if (ctas_per_sm > 0 && ctas_per_sm < occ) occ = ctas_per_sm;
    return whole_sms(device) * occ;
}

template <int C>
cudaError_t launch_layout(const WholeArgs &a, int app, int start, int grid, cudaStream_t st)
{
    switch (app) {
    case kPPR: return launch_app<kPPR, C>(a, start, grid, st);
    case kPageRank: return launch_app<kPageRank, C>(a, start, grid, st);
    default: return launch_app<kWalk, C>(a, start, grid, st);
    }
}

cudaError_t launch_walk_whole(const WholeArgs &a, int app, int start, int grid, cudaStream_t st, int layout)
{
    if (layout == kLayoutPacked) return launch_layout<kLayoutPacked>(a, app, start, grid, st);
    if (layout == kLayoutCompact) return launch_layout<kLayoutCompact>(a, app, start, grid, st);
    return launch_layout<kLayoutWide>(a, app, start, grid, st);
}

namespace {

__global__ void mod_check_kernel(uint64_t n, const uint64_t *x, const uint64_t *d, uint64_t *out)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        out[i] = d[i] ? mod_u64(x[i], d[i]) : ~0ull;
}

}  // namespace

}  // namespace lt

// The device build of the walk kernels' remainder, for checking it against
// native division (a zero divisor gives all ones).
extern "C" lt_status lt_mod_check_device(uint64_t n, const uint64_t *d_x, const uint64_t *d_d, uint64_t *d_out,
                                         void *stream)
{
    if (n == 0) return LT_OK;
    if (!d_x || !d_d || !d_out) return lt::fail(LT_ERR_INVALID, "null argument");
    const uint64_t blocks = std::min<uint64_t>((n + 255) / 256, 152ull * 8);
    lt::mod_check_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(n, d_x, d_d, d_out);
    LT_CUDA_TRY(cudaGetLastError());
    return LT_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of lt_walk_device.
//
// Some callers cannot allocate device memory: plugins handed fixed input and
// output buffers by a host framework that owns every allocation, and
// processes whose device memory another allocator has reserved in full.
// lt_walk_device asks them for a scratch buffer; this entry point needs none.  Its scratch (the
// next-walker counter of the step kernel) lives in the file-scope array below,
// which every GPU that loads this library holds until the process exits.
//
// The array is kNoAllocScratchBytes (256 B); the step kernel's scratch does not
// grow with the graph or the walker count (one 8-byte counter inside a
// walk_scratch_bytes()-byte block), and a call whose scratch need exceeds the
// array is rejected with LT_ERR_CAPACITY.
//
// All calls share the one array: it keeps the previous call's contents, so the
// counter is cleared on the caller's stream before each launch, and two calls
// whose kernels overlap on the GPU (different streams, no ordering between
// them) race on the counter and produce wrong results.  Order such calls on one
// stream.
//
// The device address of the array is looked up once per device, on the first
// call made with that device current (cudaGetSymbolAddress), and kept for the
// life of the process; make that first call before any stream capture begins.
// The kept address assumes the device's primary context is never reset: after
// a cudaDeviceReset the module is loaded again and the address may be stale.
// ---------------------------------------------------------------------------

#include <mutex>

#include "common.h"
#include "engine.h"

namespace lt {
namespace {

constexpr size_t kNoAllocScratchBytes = 256;
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

std::mutex g_noalloc_mu;
void *g_noalloc_ptr[kNoAllocMaxDevices] = {};

lt_status noalloc_scratch(void **out)
{
    int device = 0;
    LT_CUDA_TRY(cudaGetDevice(&device));
    if (device < 0 || device >= kNoAllocMaxDevices)
        return fail(LT_ERR_UNSUPPORTED, "device ordinal %d is beyond the %d devices the static scratch tracks", device,
                    kNoAllocMaxDevices);
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[device]) {
        void *p = nullptr;
        const cudaError_t err = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (err != cudaSuccess || !p)
            return fail(LT_ERR_CUDA, "cudaGetSymbolAddress of the static walk scratch failed on device %d: %s",
                        device, cudaGetErrorString(err));
        g_noalloc_ptr[device] = p;
    }
    *out = g_noalloc_ptr[device];
    return LT_OK;
}

}  // namespace
}  // namespace lt

extern "C" lt_status lt_walk_device_noalloc(int app, int start_mode, const uint64_t *d_rowptr, const uint32_t *d_col,
                                            uint32_t num_nodes, uint32_t source, uint64_t num_walkers,
                                            uint32_t length, float prob, uint32_t run, uint64_t seed,
                                            uint64_t *d_counts, uint32_t *d_endpoints, uint32_t *d_paths,
                                            uint64_t *d_stats, void *stream)
{
    const size_t need = lt::walk_scratch_bytes();
    if (need > lt::kNoAllocScratchBytes)
        return lt::fail(LT_ERR_CAPACITY, "the step kernel needs %zu scratch bytes; the static array holds %zu", need,
                        lt::kNoAllocScratchBytes);
    void *scratch = nullptr;
    LT_TRY(lt::noalloc_scratch(&scratch));
    return lt::walk_device(app, start_mode, d_rowptr, d_col, num_nodes, source, num_walkers, length, prob, run, seed,
                           d_counts, d_endpoints, d_paths, scratch, d_stats, (cudaStream_t)stream, 0);
}
