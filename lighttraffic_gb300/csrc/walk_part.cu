// walk_part.cu -- step kernel for partially cached graphs and the bucketing
// (scatter) kernel.
//
// Replaces randomWalkInsidePool[AllBatch] / randomWalkOutsidePool and the
// insertToQueue kernels (src/WalkManager.h:60-282) together with the 1-thread
// page kernels of src/buffer/Pool.h:484-528.
//
// Step kernel (persistent, one walker per lane; a warp takes blocks of input
// ordinals from one counter):
//   input  = the chunks queued for the partitions drained, plus walkers created
//            lazily from their ordinal (PPR source walkers, per-vertex starts);
//   a walker keeps stepping while the partition holding its vertex is readable
//   -- cached in a device slot, or mapped from pinned host memory for a
//   zero-copy pass -- which generalises the reference's "walk while inside the
//   partition" (src/WalkManager.h:239-240) to every cached partition;
//   updates that read no graph data (the final PPR / PageRank count, PageRank
//   teleports) run wherever the walker is;
//   a walker whose next update needs an unreadable partition is written to a
//   staging area (gathered in the warp's shared memory, one reservation for 32)
//   and counted in a per-destination histogram (shared memory, flushed once per
//   CTA).
// Bucketing: appends staged walkers to their destination queues; a CTA sorts
// its tile by destination in shared memory and reserves one range per
// destination with one global atomic (the two-level scheme of
// src/WalkManager.h:122-190), into chunks that the plan kernel or the host has
// taken from the free ones.
#include <algorithm>

#include "lt_core.cuh"
#include "mem.cuh"
#include "ppr_pool.cuh"
#include "scan.cuh"
#include "walk_part.h"

namespace lt {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
// idle lanes a warp waits for before it takes more walkers, and before it
// draws another pool of PPR lengths
constexpr int kTakeMin = 8;
constexpr int kRefillMin = 16;

// Row offsets stay in L2 (evict-last), column entries stream (evict-first).
__device__ __forceinline__ uint64_t ld_u64(unsigned long long addr, uint64_t keep)
{
    return ld_nc_u64(reinterpret_cast<const void *>(addr), keep);
}
__device__ __forceinline__ uint32_t ld_u32(unsigned long long addr, uint64_t stream)
{
    return ld_nc_stream_u32(reinterpret_cast<const void *>(addr), stream);
}

// Address of the first column entry of marked vertex v in the tier.
__device__ __forceinline__ unsigned long long hot_first(const StepArgs &a, uint32_t v, uint64_t keep)
{
    const uint2 w = ld_nc_u2(a.hot_words + (v >> 5), keep);
    const uint32_t rank = w.y + __popc(w.x & ((1u << (v & 31)) - 1u));
    return (unsigned long long)(a.hot_pool + ld_nc_u32(a.hot_off + rank, keep));
}

// What a warp keeps in shared memory: its pool of drawn PPR lengths, the
// walkers that have left (written out 32 at a time: one reservation and
// 128-byte stores instead of an atomic on one address in nearly every
// iteration), and, serving, the walks that have ended.
constexpr uint32_t kPartPool = 128;
template <bool POOL, bool SERVE>
struct PartWarp {
    struct {
        uint32_t at[POOL ? kPartPool : 1], len[POOL ? kPartPool : 1];
    } pool;
    uint32_t cur[64], step[64], idx[64], dest[64], q[SERVE ? 64 : 1];
    uint2 ends[SERVE ? 64 : 1];  // (query slot, vertex)
    // its block of input ordinals, the ordinal its pool begins at (of a queued
    // walker, or of one to be created) and the work chunk holding that
    uint64_t at, end, base;
    uint32_t work, exits;
};

// Shared-memory copy of the partition table of one launch (P <= kSmemPartMax).
struct SmemTable {
    const uint32_t *off;            // P + 1
    uint32_t *hist, *visit;         // P
    const uint32_t *zc;             // zero-copy mask
    const unsigned long long *col;  // P: column address, bit 0: zero-copy, 0: unreadable (RP32, P <= kColTableMax)
    const uint16_t *map;            // kPartMapN + 1
};

// The partition of v: between the partitions of the first vertices of v's
// block of 2^map_shift vertices and of the next one.
__device__ __forceinline__ uint32_t find_part(const StepArgs &a, const SmemTable &t, bool in_smem, uint32_t v)
{
    uint32_t lo = 0, hi = a.t.P - 1;
    if (in_smem) {
        const uint32_t b = v >> a.map_shift;
        lo = t.map[b];
        hi = t.map[b + 1];
    }
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo + 1) / 2;
        if (v < t.off[mid])
            hi = mid - 1;
        else
            lo = mid;
    }
    return lo;
}

// Walker index of lazily created ordinal t.
__device__ __forceinline__ uint32_t lazy_id(const StepArgs &a, uint64_t t)
{
    if (a.lazy_mode != kStartPerVertex) return (uint32_t)t;
    const uint32_t rem = mod_by(a.by_lazy, t);
    return (uint32_t)(div_exact(a.by_lazy, t - rem) * a.V + a.lazy_nb + rem);
}

__device__ __forceinline__ void count1(const StepArgs &a, uint32_t v, uint64_t keep)
{
    red_add1_u64((unsigned long long *)&a.counts[v], keep);
}

// A finished walk's endpoints of 32 lanes (or fewer) go to their queries'
// tables (linear probing, u32 counts); then each query has that many more
// walkers done.
__device__ __forceinline__ void serve_count(const StepArgs &a, bool have, uint2 e)
{
    const unsigned all = __ballot_sync(kFull, have);
    if (have) {
        const uint64_t base = a.q_toff[e.x];
        const uint64_t mask = (1ull << a.q_tlog[e.x]) - 1;
        uint64_t slot = ((uint64_t)(e.y * 0x9E3779B1u)) & mask;
        bool added = false;
        for (uint64_t probe = 0; probe <= mask && !added; probe++) {
            uint32_t *k = &a.q_keys[base + slot];
            uint32_t old = *(volatile uint32_t *)k;
            if (old == 0xFFFFFFFFu) old = atomicCAS(k, 0xFFFFFFFFu, e.y);
            if (old == 0xFFFFFFFFu || old == e.y) {
                atomicAdd(&a.q_cnt[base + slot], 1u);
                added = true;
            }
            slot = (slot + 1) & mask;
        }
        if (!added) atomicAdd(a.q_error, 1ull);
        __threadfence();
        const unsigned same = __match_any_sync(all, e.x);
        if ((threadIdx.x & 31) == (unsigned)__ffs((int)same) - 1u)
            atomicAdd(&a.q_done[e.x], (unsigned long long)__popc(same));
    }
    __syncwarp();
}

// Resident CTAs per SM the register budget is sized for: 64 registers a thread,
// no spills.  With 5 (PPR) and 6 (the others) 20 to 88 bytes spilled: cached
// partitions alone 25 -> 14 ms per run (PPR of 100 M walks on RMAT 2^26 / 2^30),
// PageRank of 7e5 walkers on RMAT 2^20 / 2^24, 21 of 70 partitions cached, 1.42 ->
// 1.36 ms, walks of 20 hops on RMAT 2^22 / 2^26 by the plain scheduler 30.8 ->
// 29.7; kernels that wait for host reads are the same.
constexpr int kPartMinBlocks = 4;

// HOT: the hot-vertex tier is on (a.hot_on); SERVE: query mode (a.q_seed);
// RP32: row offsets are u32 offsets from the partition's first edge, all
// partitions' back to back at a.zc_rp_base.  Separate instances keep the
// registers of the others.
template <int APP, bool HOT, bool SERVE, bool RP32>
__global__ void __launch_bounds__(kPartBlock, kPartMinBlocks) walk_part_kernel(const __grid_constant__ StepArgs a)
{
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ PartWarp<APP == kPPR && !SERVE, SERVE> s_warp[kPartBlock / 32];
    if (blockIdx.x == 0 && threadIdx.x == 0) a.clk[0] = globaltimer_ns();
    const uint32_t P = a.t.P;
    const bool in_smem = P <= kSmemPartMax;
    const bool col_table = RP32 && P <= kColTableMax;
    SmemTable t{a.t.node_off, a.hist, a.visits, nullptr, nullptr, nullptr};
    if (in_smem) {
        uint32_t *s_off = smem + (col_table ? 2 * P : 0), *s_hist = s_off + P + 1, *s_visit = s_hist + P;
        uint32_t *s_zc = s_visit + P;
        uint16_t *s_map = reinterpret_cast<uint16_t *>(s_zc + (P + 31) / 32);
        unsigned long long *s_col = reinterpret_cast<unsigned long long *>(smem);
        for (uint32_t i = threadIdx.x; i <= P; i += kPartBlock) s_off[i] = a.t.node_off[i];
        for (uint32_t i = threadIdx.x; i < P; i += kPartBlock) {
            s_hist[i] = 0;
            s_visit[i] = 0;
            if (col_table) {
                unsigned long long c = *(volatile const unsigned long long *)&a.t.rp_addr[i] ? a.t.col_addr[i] : 0ull;
                if (i == a.zc_part)
                    c = a.zc_col | 1ull;
                else if (c == 0ull && ((a.zc_mask[i >> 5] >> (i & 31)) & 1u))
                    c = (a.zc_col_base + 4ull * a.t.edge_off[i]) | 1ull;
                s_col[i] = c;
            }
        }
        for (uint32_t i = threadIdx.x; i < (P + 31) / 32; i += kPartBlock) s_zc[i] = a.zc_mask[i];
        for (uint32_t i = threadIdx.x; i <= kPartMapN / 2; i += kPartBlock)
            reinterpret_cast<uint32_t *>(s_map)[i] = reinterpret_cast<const uint32_t *>(a.t.map)[i];
        t = SmemTable{s_off, s_hist, s_visit, s_zc, s_col, s_map};
    }
    __syncthreads();

    const int lane = threadIdx.x & 31;
    const unsigned below_me = (1u << lane) - 1u;
    const uint64_t total = a.n_chunk_walkers + a.lazy_count;
    const uint64_t keep = l2_policy_evict_last(), stream = l2_policy_evict_first();
    PartWarp<APP == kPPR && !SERVE, SERVE> &sw = s_warp[threadIdx.x >> 5];

    // the warp's block of input ordinals (the first one without the counter),
    // of which [pool_at, pool_n) are at hand: queued walkers, or walkers to be
    // created (PPR: with their lengths drawn)
    const uint64_t dealt = (uint64_t)a.block * ((threadIdx.x >> 5) * gridDim.x + blockIdx.x);
    bool exhausted = dealt >= total, pool_lazy = false;
    uint32_t pool_at = 0, pool_n = 0;
    if (lane == 0) {
        sw.at = dealt;
        sw.end = min(dealt + a.block, total);
        sw.work = sw.exits = 0;
    }
    __syncwarp();

    uint32_t cur = 0, step = 0, idx = 0, qs = 0;
    uint64_t seed = 0;  // SERVE: of the lane's query
    bool active = false, emit = false, ended = false;
    uint32_t dest = 0;
    Rand4 r{};  // PageRank: the draw of the walker's next step
    // readable range of the lane's partition.  The empty range (1, 0) makes
    // the next look-up count as an entry into its partition, (2, 1) does not.
    uint32_t cp_nb = 1, cp_ne = 0;
    unsigned long long cp_rp = 0, cp_col = 0;  // cp_rp: !RP32, or HOT's one-vertex ranges
    uint64_t cp_eb = 0;                        // !RP32: the partition's first edge
    bool cp_zc = false;
    // statistics of this launch (a thread makes far fewer than 2^32 updates)
    // n_end: teleports (PageRank), walks that ended early (generic)
    uint32_t n_mov = 0, n_zc = 0, n_fin = 0, n_end = 0;
    uint32_t n_out = 0, n_ends = 0;  // walkers / ended walks gathered by the warp

    auto draw = [&](uint32_t s) {
        return SERVE ? walk_draw(seed, s, kTagStep, a.run, idx) : walk_draw(a.keys, s, kTagStep, a.run, idx);
    };
    auto write_out = [&](uint32_t first, uint32_t n) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(a.out_n, (unsigned long long)n);
        base = __shfl_sync(kFull, base, 0);
        if ((uint32_t)lane < n) {
            const uint64_t pos = base + lane;
            a.out_cur[pos] = sw.cur[first + lane];
            a.out_step[pos] = sw.step[first + lane];
            a.out_idx[pos] = sw.idx[first + lane];
            a.out_dest[pos] = sw.dest[first + lane];
            a.out_q[pos] = SERVE ? sw.q[first + lane] : 0u;
        }
        if (lane == 0) sw.exits += n;
        __syncwarp();
    };

    while (true) {
        const unsigned left = __ballot_sync(kFull, emit);
        if (left) {
            if (emit) {
                const uint32_t k = n_out + __popc(left & below_me);
                sw.cur[k] = cur;
                sw.step[k] = step;
                sw.idx[k] = idx;
                sw.dest[k] = dest;
                if (SERVE) sw.q[k] = qs;
                atomicAdd(&t.hist[dest], 1u);
                emit = false;
            }
            n_out += __popc(left);
            __syncwarp();
            if (n_out >= 32u) {
                n_out -= 32u;
                write_out(n_out, 32u);
            }
        }
        if (SERVE) {
            const unsigned over = __ballot_sync(kFull, ended);
            if (over) {
                if (ended) sw.ends[n_ends + __popc(over & below_me)] = make_uint2(qs, cur);
                ended = false;
                n_ends += __popc(over);
                __syncwarp();
                if (n_ends >= 32u) {
                    n_ends -= 32u;
                    serve_count(a, true, sw.ends[n_ends + lane]);
                }
            }
        }
        const unsigned busy = __ballot_sync(kFull, active);
        const int idle = 32 - __popc(busy);
        if (pool_at == pool_n && idle >= kRefillMin && !exhausted) {
            uint64_t at = sw.at;
            const uint64_t end = sw.end;
            pool_at = 0;
            pool_lazy = at >= a.n_chunk_walkers;
            const uint64_t base = pool_lazy ? at - a.n_chunk_walkers + a.lazy_begin : at;
            uint32_t work = sw.work;
            if (pool_lazy) {
                pool_n = (uint32_t)(end - at);
                if (APP == kPPR && !SERVE)
                    ppr_pool_fill(sw.pool, pool_n, a.long_len, a.lim, [&](uint32_t d, uint32_t w) {
                        return walk_draw(a.keys, d, kTagInit, a.run, lazy_id(a, base + w));
                    });
            } else {
                pool_n = (uint32_t)(min(end, (uint64_t)a.n_chunk_walkers) - at);
                if (a.work_off) work = (uint32_t)warp_find_last(a.work_off, work, a.n_work, at);
            }
            at += pool_n;
            if (at == end) {
                unsigned long long got = 0;
                if (lane == 0) got = atomicAdd(a.next, (unsigned long long)a.block);
                at = (uint64_t)a.block * gridDim.x * (kPartBlock / 32) + __shfl_sync(kFull, got, 0);
            }
            exhausted = at >= total;
            __syncwarp();
            if (lane == 0) {
                sw.at = at;
                sw.end = at < end ? end : min(at + a.block, total);
                sw.base = base;
                sw.work = work;
            }
            __syncwarp();
        }
        if (pool_at < pool_n && idle >= kTakeMin) {
            const uint32_t mine = pool_at + __popc(~busy & below_me);
            if (!active && mine < pool_n) {
                active = true;
                const uint64_t pool_base = sw.base;
                if (!pool_lazy) {
                    const uint64_t my = pool_base + mine;
                    uint32_t wi, j;
                    if (!a.work_off) {
                        wi = (uint32_t)(my / kChunk);
                        j = (uint32_t)(my % kChunk);
                    } else {
                        wi = sw.work;
                        while (wi + 1 < a.n_work && a.work_off[wi + 1] <= my) wi++;
                        j = (uint32_t)(my - a.work_off[wi]);
                    }
                    const uint32_t *c =
                        reinterpret_cast<const uint32_t *>(a.arena + (uint64_t)a.work_chunks[wi] * kChunkBytes);
                    cur = c[j];
                    step = c[kChunk + j];
                    idx = c[2 * kChunk + j];
                    // A walker taken from a queue chunk was counted as
                    // entering its partition when it was staged there
                    // (counting it again would rank uncached partitions by
                    // the walkers that queued at them, i.e. by the cache
                    // state).
                    cp_nb = 2;
                    cp_ne = 1;
                    if (SERVE) {
                        qs = c[3 * kChunk + j];
                        seed = a.q_seed[qs];
                    }
                } else {
                    const uint32_t w = APP == kPPR && !SERVE ? sw.pool.at[mine] : mine;
                    idx = lazy_id(a, pool_base + w);
                    if (a.lazy_mode == kStartPerVertex)
                        cur = a.lazy_nb + mod_by(a.by_lazy, pool_base + w);
                    else if (a.lazy_mode == kStartSource)
                        cur = a.source;
                    else
                        cur = mod_by(a.by_v, r64_of(walk_draw(a.keys, 0, kTagInit, a.run, idx)));
                    step = APP == kPPR && !SERVE ? sw.pool.len[mine] : a.length;
                    if (APP == kWalk && a.paths) a.paths[(uint64_t)idx * (a.length + 1)] = cur;
                    // the lane's range holds from its previous walker
                }
                if (APP == kPageRank) r = draw(step);
            }
            pool_at = min(pool_n, pool_at + (uint32_t)idle);
        } else if (idle == 32 && exhausted && pool_at == pool_n) {
            break;
        }
        if (!active) continue;

        // Does the next update read the graph, and is the walker's partition readable?
        const bool need_graph = APP != kPageRank || (step >= 2 && below(r, a.lim));
        if (need_graph && (cur < cp_nb || cur >= cp_ne)) {
            const uint32_t p = find_part(a, t, in_smem, cur);
            if (!(cp_nb == 2 && cp_ne == 1)) atomicAdd(&t.visit[p], 1u);
            unsigned long long rp = 1ull, col = 0;
            if (col_table) {
                col = t.col[p];
                cp_zc = (col & 1ull) != 0;
                rp = col;
                col &= ~1ull;
            } else if (p == a.zc_part) {
                rp = a.zc_rp;
                col = a.zc_col;
                cp_zc = true;
            } else {
                rp = *(volatile const unsigned long long *)&a.t.rp_addr[p];
                cp_zc = false;
                if (rp != 0ull) {
                    col = *(volatile const unsigned long long *)&a.t.col_addr[p];
                } else if (in_smem && ((t.zc[p >> 5] >> (p & 31)) & 1u)) {
                    rp = a.zc_rp_base + (RP32 ? 4ull : 8ull) * t.off[p];
                    col = a.zc_col_base + 4ull * a.t.edge_off[p];
                    cp_zc = true;
                }
            }
            bool hot = false;
            if (HOT && rp == 0ull) {
                // unreadable partition: a marked vertex is read from the
                // tier, as a one-vertex readable range of the lane
                const uint32_t lo_m = ld_nc_u32(reinterpret_cast<const void *>(a.zc_rp_base + 4ull * cur), keep);
                if (lo_m & kHotMark) {
                    cp_nb = cur;
                    cp_ne = cur + 1;
                    cp_col = hot_first(a, cur, keep) - 4ull * (lo_m & ~kHotMark);
                    cp_zc = false;
                    hot = true;
                }
            }
            if (hot) {
            } else if (rp == 0ull) {
                emit = true;
                active = false;
                dest = p;
                cp_nb = 1;
                cp_ne = 0;
                continue;
            } else {
                cp_nb = t.off[p];
                cp_ne = t.off[p + 1];
                cp_col = col;
                if (!RP32) {
                    cp_rp = rp;
                    cp_eb = a.t.edge_off[p];
                }
            }
        }

        // The row: first column entry and degree.  With RP32 the partition's
        // edge count ends its last vertex's row.
        unsigned long long fa = 0;
        uint64_t deg = 0;
        bool zc_read = cp_zc;
        if (need_graph) {
            if (RP32) {
                const uint32_t lo_m = ld_nc_u32(reinterpret_cast<const void *>(a.zc_rp_base + 4ull * cur), keep);
                uint32_t hi;
                if (cur + 1 < cp_ne) {
                    hi = ld_nc_u32(reinterpret_cast<const void *>(a.zc_rp_base + 4ull * (cur + 1)), keep);
                } else {
                    const uint32_t p = find_part(a, t, in_smem, cur);
                    hi = HOT && cur + 1 < t.off[p + 1]
                             ? ld_nc_u32(reinterpret_cast<const void *>(a.zc_rp_base + 4ull * (cur + 1)), keep)
                             : (uint32_t)(a.t.edge_off[p + 1] - a.t.edge_off[p]);
                }
                if (APP == kPageRank) count1(a, cur, keep);
                if (APP != kPageRank) {
                    r = draw(step);
                    asm volatile("" : "+r"(r.x0), "+r"(r.x1));  // here, under the loads
                }
                const uint32_t lo = lo_m & ~kHotMark;
                fa = cp_col + 4ull * lo;
                deg = (hi & ~kHotMark) - lo;
                if (HOT && (lo_m & kHotMark) && cp_zc) {
                    // a marked vertex of a zero-copy partition: from the tier
                    fa = hot_first(a, cur, keep);
                    zc_read = false;
                }
            } else {
                const uint32_t rel = cur - cp_nb;
                const uint64_t first = ld_u64(cp_rp + 8ull * rel, keep);
                const uint64_t next = ld_u64(cp_rp + 8ull * (rel + 1), keep);
                if (APP == kPageRank) count1(a, cur, keep);
                if (APP != kPageRank) {
                    r = draw(step);
                    asm volatile("" : "+r"(r.x0), "+r"(r.x1));
                }
                deg = next - first;
                fa = cp_col + 4ull * (first - cp_eb);
            }
        } else if (APP == kPageRank) {
            count1(a, cur, keep);
        }

        bool done = false;
        if (APP == kPPR) {
            // app/ppr.cu:22-42; step >= 2 here, and a walk whose step comes
            // down to 1 is counted right away
            if (deg > 0) {
                cur = ld_u32(fa + 4ull * mod_u64(r64_of(r), deg), stream);
                n_mov++;
                n_zc += zc_read;
                step--;
            } else {
                step = 1;
            }
            done = step == 1;
            if (done) {
                if (SERVE)
                    ended = true;
                else
                    red_add1_u64((unsigned long long *)&a.counts[cur], keep);
            }
        } else if (APP == kPageRank) {
            // app/pagerank.cu:26-44; a vertex without out-edges teleports.
            step--;
            done = step == 0;
            if (!done) {
                const uint64_t r64 = r64_of(r);
                if (deg > 0) {
                    cur = ld_u32(fa + 4ull * mod_u64(r64, deg), stream);
                    n_mov++;
                    n_zc += zc_read;
                } else {
                    cur = mod_by(a.by_v, r64);
                    n_end++;
                }
                r = draw(step);
                asm volatile("" : "+r"(r.x0), "+r"(r.x1), "+r"(r.x2), "+r"(r.x3));
            }
        } else {
            // app/genericwalk.cu:22-32
            uint32_t *path = a.paths ? a.paths + (uint64_t)idx * (a.length + 1) + (a.length - step) : nullptr;
            if (deg > 0) {
                cur = ld_u32(fa + 4ull * mod_u64(r64_of(r), deg), stream);
                n_mov++;
                n_zc += zc_read;
                if (path) path[1] = cur;
                step--;
            } else {
                if (path)
                    for (uint32_t k = 1; k <= step; k++) path[k] = kInvalidNode;
                n_end++;
                step = 0;
            }
            done = step == 0;
        }
        if (done) {
            active = false;
            n_fin++;
            if (a.endpoints) a.endpoints[idx] = cur;
        }
    }
    if (n_out) write_out(0, n_out);
    if (SERVE && n_ends) serve_count(a, (uint32_t)lane < n_ends, sw.ends[lane]);

    // Statistics: one atomic per CTA and counter.  A PPR walk makes one update
    // per hop and one that ends it, a PageRank walk one per hop, teleport and
    // end, a generic walk one per hop and one where it ends early.
    __shared__ unsigned long long s_stats[5];
    if (threadIdx.x < 5) s_stats[threadIdx.x] = 0;
    __syncthreads();
    uint64_t w_mov = n_mov, w_zc = n_zc, w_fin = n_fin, w_upd = n_end;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        w_mov += __shfl_down_sync(kFull, w_mov, o);
        w_zc += __shfl_down_sync(kFull, w_zc, o);
        w_fin += __shfl_down_sync(kFull, w_fin, o);
        w_upd += __shfl_down_sync(kFull, w_upd, o);
    }
    if (lane == 0) {
        if (w_upd) atomicAdd(&s_stats[0], (unsigned long long)w_upd);
        if (w_mov) atomicAdd(&s_stats[1], (unsigned long long)w_mov);
        if (w_zc) atomicAdd(&s_stats[2], (unsigned long long)w_zc);
        if (sw.exits) atomicAdd(&s_stats[3], (unsigned long long)sw.exits);
        if (w_fin) atomicAdd(&s_stats[4], (unsigned long long)w_fin);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long end_n = s_stats[0], mov = s_stats[1], fin = s_stats[4];
        const unsigned long long tel = APP == kPageRank ? end_n : 0ull;
        const unsigned long long upd = mov + (APP == kPageRank ? tel + fin : APP == kPPR ? fin : end_n);
        if (upd) atomicAdd(&a.stats[0], upd);
        if (mov) atomicAdd(&a.stats[1], mov);
        if (tel) atomicAdd(&a.stats[2], tel);
        if (s_stats[2]) atomicAdd(&a.stats[3], s_stats[2]);
        if (s_stats[3]) atomicAdd(&a.stats[4], s_stats[3]);
        if (fin) atomicAdd(&a.stats[5], fin);
        atomicMax(&a.clk[1], (unsigned long long)globaltimer_ns());
    }
    if (in_smem)
        for (uint32_t i = threadIdx.x; i < P; i += kPartBlock) {
            if (t.hist[i]) atomicAdd(&a.hist[i], t.hist[i]);
            if (t.visit[i]) atomicAdd(&a.visits[i], t.visit[i]);
        }
}

// Bucketing above kSmemPartMax partitions, whose counts do not fit shared
// memory: one global atomic per walker, kScatterItems of a thread in flight.
constexpr int kScatterItems = 4;

__global__ void __launch_bounds__(kPartBlock) scatter_kernel(ScatterArgs a)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) a.clk[0] = globaltimer_ns();
    const uint64_t tile = (uint64_t)kPartBlock * kScatterItems;
    for (uint64_t t0 = (uint64_t)blockIdx.x * tile; t0 < a.n; t0 += (uint64_t)gridDim.x * tile) {
        uint32_t pos[kScatterItems], dest[kScatterItems];
#pragma unroll
        for (int k = 0; k < kScatterItems; k++) {
            const uint64_t i = t0 + (uint64_t)k * kPartBlock + threadIdx.x;
            dest[k] = 0xFFFFFFFFu;
            if (i < a.n) {
                dest[k] = a.in_dest[i];
                pos[k] = atomicAdd(&a.cursor[dest[k]], 1u);
            }
        }
#pragma unroll
        for (int k = 0; k < kScatterItems; k++) {
            const uint64_t i = t0 + (uint64_t)k * kPartBlock + threadIdx.x;
            if (i < a.n) {
                const uint32_t chunk = a.plan_chunks[a.win_off[dest[k]] + pos[k] / kChunk];
                uint32_t *c = reinterpret_cast<uint32_t *>(a.arena + (uint64_t)chunk * kChunkBytes);
                const uint32_t j = pos[k] % kChunk;
                c[j] = a.in_cur[i];
                c[kChunk + j] = a.in_step[i];
                c[2 * kChunk + j] = a.in_idx[i];
                c[3 * kChunk + j] = a.in_q[i];
            }
        }
    }
    if (threadIdx.x == 0) atomicMax(&a.clk[1], (unsigned long long)globaltimer_ns());
}

// Bucketing by a block-local counting sort (P <= kSmemPartMax).  A tile of
// T = BLOCK x items staged walkers is ranked per destination in shared
// memory (shared atomics), the per-destination counts are scanned across the
// block and reserved in the destination windows with one global atomic per
// (tile, destination) -- the two-level scheme of insertToQueueKernel
// (src/WalkManager.h:122-190) -- and the tile is written back through its
// sort permutation as per-destination runs: consecutive threads write
// consecutive queue slots.
//
// The CTAs are persistent.  The bulk-copy unit (cp.async.bulk, one copy per
// field, completion counted on an mbarrier) brings a tile from the staging area
// into shared memory, so the kernel issues no global loads of walker fields.  A
// tile's chunk ids are looked up once per destination, not per walker.  The
// staged field arrays start 16-byte aligned and hold n rounded up to 4 words
// (the copies round up to 16 bytes).  If a copy does not complete within a
// second, the CTA records it in *err and reads the remaining tiles from global
// memory directly, so no walker is lost.
// What bounds it is the runs, one per tile and destination, each its own add,
// lookups and partly written sectors: with 1 090 partitions and 5.8 M walkers a
// pass took 162 us in tiles of 2048, 105 of 4096 and 81 of 8192, whether one or
// two CTAs shared an SM and whether a second buffer held the next tile (4096
// walkers: 104, 113, 105 us).  So a tile is as large as shared memory holds: 1024
// threads x 8 walkers, fewer where that would leave SMs without a tile.  PPR on
// RMAT 2^30 / 2^33, 1 112 partitions: bucketing 80 -> 54 ms of an 834 -> 803 ms
// run.  512 threads x 4 walkers, two CTAs per SM, are the autotuner's other
// choice.  256-thread CTAs of a 4096-walker tile left 8 warps per SM to hide the
// latencies (46 against 38 us).
constexpr int kBucketFields = 5;                    // cur, step, idx, query, dest
constexpr uint64_t kBulkWaitNs = 1000000000ull;     // bounded wait on one tile's copies

// a tile of kBucketFields u32 fields | mbarrier | 4 u32 per destination | u16 permutation
size_t bucket_smem(uint32_t P, uint64_t T) { return 4 * kBucketFields * T + 16 + 16ull * P + 2 * T; }

template <int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) bucket_sort_kernel(ScatterArgs a, uint32_t most)
{
    static_assert(BLOCK * ITEMS <= (int)kChunk);
    constexpr uint32_t kPerMax = kSmemPartMax / BLOCK;
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ uint32_t warp_tot[BLOCK / 32];
    __shared__ uint32_t tile_total;
    const uint32_t P = a.P;
    const uint64_t n = a.n_dev ? *a.n_dev : a.n;
    // items per thread: as few as one tile per CTA needs
    uint32_t items = 1;
    while (items < most && n > (uint64_t)gridDim.x * BLOCK * items) items *= 2;
    const uint32_t T = BLOCK * items;
    uint64_t *mbar = reinterpret_cast<uint64_t *>(smem + kBucketFields * T);
    uint32_t *s_off = reinterpret_cast<uint32_t *>(mbar + 2);  // P: tile count, then offset in the sorted tile
    uint32_t *s_base = s_off + P;                              // P: first reserved slot of the window
    uint32_t *s_ch0 = s_base + P;                              // P: chunk holding s_base
    uint32_t *s_ch1 = s_ch0 + P;                               // P: the next chunk, where the run crosses into it
    uint16_t *s_inv = reinterpret_cast<uint16_t *>(s_ch1 + P); // T: tile position at sorted position j
    if (blockIdx.x == 0 && threadIdx.x == 0 && !a.n_dev) a.clk[0] = globaltimer_ns();
    const uint32_t *src[kBucketFields] = {a.in_cur, a.in_step, a.in_idx, a.in_q, a.in_dest};
    if (a.err && (*(volatile unsigned int *)a.err & 2u)) return;
    const uint64_t tiles = (n + T - 1) / T;
    bool bulk = true;
#pragma unroll
    for (int f = 0; f < kBucketFields; f++) bulk = bulk && ((uintptr_t)src[f] & 15) == 0;
    if (threadIdx.x == 0) {
        mbar_init(mbar, 1);
        mbar_init_fence();
    }
    __syncthreads();
    // thread 0: copies of tile `tile`
    auto issue = [&](uint64_t tile) {
        const uint64_t t0 = tile * T;
        const uint32_t m = (uint32_t)(n - t0 < T ? n - t0 : T);
        const uint32_t bytes = (4 * m + 15) & ~15u;
        mbar_arrive_expect_tx(mbar, kBucketFields * bytes);
#pragma unroll
        for (int f = 0; f < kBucketFields; f++) bulk_load_smem(smem + f * T, src[f] + t0, bytes, mbar);
    };
    uint32_t issued = 0, waited = 0;  // copies issued / completions waited for
    uint64_t tile = blockIdx.x;
    if (bulk && tile < tiles) {
        if (threadIdx.x == 0) issue(tile);
        issued++;
    }
    const uint32_t per = (P + BLOCK - 1) / BLOCK;  // destinations a thread reserves and scans
    for (; tile < tiles; tile += gridDim.x) {
        const uint64_t t0 = tile * T;
        const uint32_t m = (uint32_t)(n - t0 < T ? n - t0 : T);
        for (uint32_t i = threadIdx.x; i < P; i += BLOCK) s_off[i] = 0;
        if (bulk) {
            const bool ok = mbar_wait_bounded(mbar, waited & 1, kBulkWaitNs);
            waited += ok;
            if (__syncthreads_or(!ok)) {
                if (threadIdx.x == 0 && a.err) atomicOr(a.err, 1u);
                bulk = false;
            }
        } else {
            __syncthreads();
        }
        const uint32_t *f_cur, *f_step, *f_idx, *f_q, *f_dest;
        if (bulk) {
            const uint32_t *buf = smem;
            f_cur = buf, f_step = buf + T, f_idx = buf + 2 * T, f_q = buf + 3 * T, f_dest = buf + 4 * T;
        } else {
            f_cur = a.in_cur + t0, f_step = a.in_step + t0, f_idx = a.in_idx + t0, f_q = a.in_q + t0,
            f_dest = a.in_dest + t0;
        }
        uint32_t dest[ITEMS], rank[ITEMS];
#pragma unroll
        for (uint32_t k = 0; k < ITEMS; k++) {
            const uint32_t i = k * BLOCK + threadIdx.x;
            dest[k] = k < items && i < m ? f_dest[i] : 0xFFFFFFFFu;
            rank[k] = dest[k] != 0xFFFFFFFFu ? atomicAdd(&s_off[dest[k]], 1u) : 0u;
        }
        __syncthreads();
        // reserve each destination's run: window starts and atomics first,
        // then the chunk lookups that depend on both
        uint32_t cnt[kPerMax], base[kPerMax], win[kPerMax];
        uint32_t mine = 0;
#pragma unroll
        for (uint32_t j = 0; j < kPerMax; j++) {
            const uint32_t d = threadIdx.x * per + j;
            cnt[j] = j < per && d < P ? s_off[d] : 0;
            win[j] = cnt[j] ? a.win_off[d] : 0;
        }
#pragma unroll
        for (uint32_t j = 0; j < kPerMax; j++) {
            const uint32_t d = threadIdx.x * per + j;
            base[j] = cnt[j] ? atomicAdd(&a.cursor[d], cnt[j]) : 0;
            mine += cnt[j];
        }
#pragma unroll
        for (uint32_t j = 0; j < kPerMax; j++) {
            if (!cnt[j]) continue;
            const uint32_t d = threadIdx.x * per + j;
            const uint32_t w = win[j] + base[j] / kChunk;
            s_base[d] = base[j];
            s_ch0[d] = a.plan_chunks[w];
            // a run (at most T <= kChunk walkers) spans one chunk or two
            s_ch1[d] = (base[j] + cnt[j] - 1) / kChunk != base[j] / kChunk ? a.plan_chunks[w + 1] : 0u;
        }
        uint32_t off = scan_detail::block_exclusive<uint32_t, BLOCK>(mine, warp_tot, &tile_total);
#pragma unroll
        for (uint32_t j = 0; j < kPerMax; j++) {
            const uint32_t d = threadIdx.x * per + j;
            if (j < per && d < P) {
                s_off[d] = off;
                off += cnt[j];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; k++)
            if (dest[k] != 0xFFFFFFFFu) s_inv[s_off[dest[k]] + rank[k]] = (uint16_t)(k * BLOCK + threadIdx.x);
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < m; j += BLOCK) {
            const uint32_t i = s_inv[j];
            const uint32_t d = f_dest[i];
            const uint32_t b0 = s_base[d];
            const uint32_t g = b0 + (j - s_off[d]);
            const uint32_t chunk = g / kChunk == b0 / kChunk ? s_ch0[d] : s_ch1[d];
            uint32_t *c = reinterpret_cast<uint32_t *>(a.arena + (uint64_t)chunk * kChunkBytes);
            const uint32_t jj = g % kChunk;
            c[jj] = f_cur[i];
            c[kChunk + jj] = f_step[i];
            c[2 * kChunk + jj] = f_idx[i];
            c[3 * kChunk + jj] = f_q[i];
        }
        __syncthreads();
        // the tile's fields have been read: the next one's come in
        if (bulk && tile + gridDim.x < tiles) {
            if (threadIdx.x == 0) issue(tile + gridDim.x);
            issued++;
        }
    }
    // copies still in flight exist only after a wait gave up: wait for them
    // (bounded) before this CTA's shared memory is released
    while (waited < issued && mbar_wait_bounded(mbar, waited & 1, kBulkWaitNs)) waited++;
    if (threadIdx.x == 0) atomicMax(&a.clk[1], (unsigned long long)globaltimer_ns());
}

// One CTA plans every destination: per destination the chunks its arrivals
// need (new ones and, with an open tail chunk, that one), two block scans for
// the stack and window positions, then the windows in destination order.
constexpr int kPlanBlock = 1024;

__global__ void __launch_bounds__(kPlanBlock) plan_kernel(PlanArgs a)
{
    constexpr uint32_t kPerMax = kSmemPartMax / kPlanBlock;
    __shared__ uint32_t warp_tot[kPlanBlock / 32];
    __shared__ uint32_t tot_new, tot_slots;
    if (threadIdx.x == 0) a.clk[0] = globaltimer_ns();
    const uint32_t P = a.P;
    const uint32_t per = (P + kPlanBlock - 1) / kPlanBlock;
    for (uint32_t i = threadIdx.x; i < a.ctl_words; i += kPlanBlock) a.ctl_host[i] = a.ctl[i];
    for (uint32_t i = threadIdx.x; i < a.n_done; i += kPlanBlock) a.done_host[i] = a.done[i];
    uint32_t h[kPerMax], fill[kPerMax], tail[kPerMax], nnew[kPerMax];
    uint32_t my_new = 0, my_slots = 0;
#pragma unroll
    for (uint32_t j = 0; j < kPerMax; j++) {
        const uint32_t d = threadIdx.x * per + j;
        h[j] = j < per && d < P ? a.hist[d] : 0;
        fill[j] = 0;
        tail[j] = kNoChunk;
        nnew[j] = 0;
        if (h[j]) {
            const uint32_t tc = a.tail_chunk[d], tf = a.tail_fill[d];
            const bool open = tc != kNoChunk && tf < kChunk;
            fill[j] = open ? tf : 0;
            tail[j] = open ? tc : kNoChunk;
            const uint32_t chunks = (uint32_t)(((uint64_t)fill[j] + h[j] + kChunk - 1) / kChunk);
            nnew[j] = chunks - (open ? 1u : 0u);
            my_new += nnew[j];
            my_slots += chunks;
        }
    }
    uint32_t pos_new = scan_detail::block_exclusive<uint32_t, kPlanBlock>(my_new, warp_tot, &tot_new);
    uint32_t pos_slot = scan_detail::block_exclusive<uint32_t, kPlanBlock>(my_slots, warp_tot, &tot_slots);
    if (tot_new > a.n_stack || tot_slots > a.plan_cap) {
        if (threadIdx.x == 0 && a.err) atomicOr(a.err, 2u);
        return;
    }
#pragma unroll
    for (uint32_t j = 0; j < kPerMax; j++) {
        const uint32_t d = threadIdx.x * per + j;
        if (j >= per || d >= P) continue;
        a.cursor[d] = fill[j];
        a.win_off[d] = h[j] ? pos_slot : 0;
        if (!h[j]) continue;
        if (tail[j] != kNoChunk) a.plan_chunks[pos_slot++] = tail[j];
        for (uint32_t c = 0; c < nnew[j]; c++) a.plan_chunks[pos_slot++] = a.stack[pos_new++];
    }
}

template <int APP, bool HOT, bool SERVE, bool RP32>
cudaError_t launch_part(const StepArgs &a, int grid, size_t smem, cudaStream_t st)
{
    walk_part_kernel<APP, HOT, SERVE, RP32><<<grid, kPartBlock, smem, st>>>(a);
    return cudaGetLastError();
}

// The limit on a kernel's dynamic shared memory belongs to the kernel, not to
// the engine whose partition count asks for it, and part_smem is not monotonic
// (35 016 bytes at 1 536 partitions, 22 744 at 1 537): it is set to the most any
// engine takes, so that engines of different partition counts run side by side.
template <int APP, bool HOT, bool SERVE, bool RP32>
int occ_part(size_t smem)
{
    static const int most = (int)std::max(part_smem(kColTableMax), part_smem(kSmemPartMax));
    cudaFuncSetAttribute(walk_part_kernel<APP, HOT, SERVE, RP32>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, walk_part_kernel<APP, HOT, SERVE, RP32>, kPartBlock, smem);
    return n;
}

// The instances' common occupancy (and their shared-memory limits set).
template <int APP>
int occ_app(size_t smem)
{
    int n = std::min(occ_part<APP, false, false, true>(smem), occ_part<APP, false, false, false>(smem));
    n = std::min(n, occ_part<APP, true, false, true>(smem));
    if (APP == kPPR) {
        n = std::min(n, occ_part<kPPR, false, true, true>(smem));
        n = std::min(n, occ_part<kPPR, false, true, false>(smem));
        n = std::min(n, occ_part<kPPR, true, true, true>(smem));
    }
    return n;
}

template <int APP>
cudaError_t launch_app(const StepArgs &a, int grid, size_t smem, cudaStream_t st)
{
    if (a.rp32) return a.hot_on ? launch_part<APP, true, false, true>(a, grid, smem, st)
                                : launch_part<APP, false, false, true>(a, grid, smem, st);
    return launch_part<APP, false, false, false>(a, grid, smem, st);
}

}  // namespace

size_t part_smem(uint32_t P)
{
    if (P > kSmemPartMax) return 0;
    return (P <= kColTableMax ? 8ull * P : 0) + 4 * (3ull * P + 1 + (P + 31) / 32) + 2 * (kPartMapN + 2);
}

int part_grid(int app, int /*start*/, int device, size_t smem, int ctas_per_sm)
{
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    int occ = app == kPPR ? occ_app<kPPR>(smem) : app == kPageRank ? occ_app<kPageRank>(smem) : occ_app<kWalk>(smem);
    if (ctas_per_sm > 0 && ctas_per_sm < occ) occ = ctas_per_sm;
    if (occ < 1) occ = 1;
    return sms * occ;
}

uint32_t part_map_shift(uint32_t V)
{
    uint32_t shift = 0;
    while (((uint64_t)V - 1) >> shift >= kPartMapN) shift++;
    return shift;
}

cudaError_t launch_walk_part(const StepArgs &args, int app, int grid, cudaStream_t st)
{
    const size_t smem = part_smem(args.t.P);
    StepArgs a = args;
    const uint64_t total = a.n_chunk_walkers + a.lazy_count;
    // no more CTAs than have walkers, but half the grid's
    const uint64_t need = std::max<uint64_t>((uint64_t)grid / 2, (total + kPartBlock - 1) / kPartBlock);
    if ((uint64_t)grid > need) grid = (int)std::max<uint64_t>(1, need);
    const uint64_t warps = (uint64_t)grid * (kPartBlock / 32);
    const uint64_t rounds = std::max<uint64_t>(1, (total + warps * kPartPool - 1) / (warps * kPartPool));
    a.block = (uint32_t)std::max<uint64_t>(16, (total + warps * rounds - 1) / (warps * rounds));
    a.map_shift = part_map_shift(a.V);
    if (app == kPPR && a.q_seed) {
        if (!a.rp32) return launch_part<kPPR, false, true, false>(a, grid, smem, st);
        return a.hot_on ? launch_part<kPPR, true, true, true>(a, grid, smem, st)
                        : launch_part<kPPR, false, true, true>(a, grid, smem, st);
    }
    switch (app) {
    case kPPR: return launch_app<kPPR>(a, grid, smem, st);
    case kPageRank: return launch_app<kPageRank>(a, grid, smem, st);
    default: return launch_app<kWalk>(a, grid, smem, st);
    }
}

cudaError_t launch_plan(const PlanArgs &a, cudaStream_t st)
{
    if (a.P > kSmemPartMax) return cudaErrorInvalidValue;
    plan_kernel<<<1, kPlanBlock, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_scatter(const ScatterArgs &a, int device, cudaStream_t st)
{
    if (a.n == 0) return cudaSuccess;
    // per device: SMs and the shared memory of a CTA (one launch per wave
    // iteration: no attribute queries on that path)
    static thread_local int cached_device = -1;
    static thread_local int sms = 0, smem_most = 0;
    if (cached_device != device) {
        cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&smem_most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
        smem_most -= 1024;  // room for the kernels' static shared memory
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(bucket_sort_kernel<1024, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_most);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(bucket_sort_kernel<512, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_most);
        if (e != cudaSuccess) return e;
        cached_device = device;
    }
    if (a.P <= kSmemPartMax) {
        if (a.items == 8) {
            const uint64_t blocks = std::min<uint64_t>((a.n + 511) / 512, 2ull * sms);
            bucket_sort_kernel<512, 4><<<(unsigned)blocks, 512, bucket_smem(a.P, 2048), st>>>(a, 4);
        } else {
            // where 8192 walkers do not fit beside the tables (P above 3 199) 4096 do
            const uint32_t most = bucket_smem(a.P, 8192) <= (size_t)smem_most ? 8 : 4;
            const uint64_t blocks = std::min<uint64_t>((a.n + 1023) / 1024, (uint64_t)sms);
            bucket_sort_kernel<1024, 8><<<(unsigned)blocks, 1024, bucket_smem(a.P, 1024ull * most), st>>>(a, most);
        }
        return cudaGetLastError();
    }
    const uint64_t tile = (uint64_t)kPartBlock * kScatterItems;
    const uint64_t blocks = std::min<uint64_t>((a.n + tile - 1) / tile, (uint64_t)sms * 8);
    scatter_kernel<<<(unsigned)blocks, kPartBlock, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace lt
