// ppr_pool.cuh -- PPR walk lengths drawn by a warp for a block of walkers ahead
// of the walks.
//
// A PPR walk's length takes 1 / (2 p) draws on average (3.6 at p = 0.15) and
// many more for the longest of a warp's walkers, so drawing the lengths of the
// walkers of one refill leaves most lanes waiting for the longest: 41 warp
// instructions per walk against some 15 here (2|V| walks on RMAT 2^20 / 2^24:
// step kernel 169 -> 137 us; pools of 128 walkers 148 us).  A warp draws for up to
// kPoolWalkers walkers at a time instead, a lane taking the block's next
// walker as soon as its own length is known; only the last ones leave lanes
// without a walker, which then help (2, 4, ... lanes per walker take its next
// draws in parallel).  Walks longer than `long_len` come first in the pool:
// a long walk begun last would run on alone at the end of the launch.
#pragma once

#include "lt_core.cuh"

namespace lt {

constexpr uint32_t kPoolWalkers = 256, kPoolMin = 16;

// One warp's pool, in shared memory: walker base + at[i] has length len[i].
struct PprPool {
    uint32_t at[kPoolWalkers];
    uint32_t len[kPoolWalkers];
};

// Fills the pool with walkers base .. base + n - 1 (n at most its
// arrays' size); the whole warp, converged.  Draw is a callable (t, at) -> Rand4: draw t of the
// init draws of walker base + at.
template <typename Pool, typename Draw>
__device__ __forceinline__ void ppr_pool_fill(Pool &pool, uint32_t n, uint32_t long_len, const Limit53 &lim,
                                              const Draw &draw)
{
    const unsigned full = 0xFFFFFFFFu, lane = threadIdx.x & 31u, below_me = (1u << lane) - 1u;
    uint32_t next = 0, front = 0, back = n;  // same in every lane
    uint32_t at = 0, t = 0;
    bool open = false;
    __syncwarp();  // the pool's last entries have been read
    while (true) {
        unsigned m = __ballot_sync(full, open);
        if (next < n && m != full) {
            const uint32_t mine = next + (uint32_t)__popc(~m & below_me);
            next += 32u - (uint32_t)__popc(m);
            if (!open && mine < n) {
                at = mine;
                t = 0;
                open = true;
            }
            m = __ballot_sync(full, open);
        }
        if (m == 0u) break;
        uint32_t len = 0;  // > 0: drawn in this round
        if (__popc(m) > 16) {
            if (open) {
                const Rand4 r = draw(t, at), q = draw(t + 1u, at);
                const bool a = below_hi(r, lim), b = below(r, lim), c = below_hi(q, lim), d = below(q, lim);
                if (a || b || c || d) len = 2u + 2u * t + (a ? 0u : b ? 1u : c ? 2u : 3u);
                t += 2u;
            }
        } else {
            // g = 2^lg lanes per open walker; lane's group draws for the
            // (lane >> lg)-th open one (the last one in the lanes left over)
            const uint32_t k = (uint32_t)__popc(m);
            const uint32_t lg = 31u - (uint32_t)__clz((int)(32u / k)), g = 1u << lg;
            const uint32_t want = (lane >> lg) < k ? lane >> lg : k - 1u;
            uint32_t src = 0;
#pragma unroll
            for (uint32_t b = 16; b > 0; b >>= 1)
                if ((uint32_t)__popc(m & ((1u << (src + b)) - 1u)) <= want) src += b;
            const uint32_t wt = __shfl_sync(full, t, src) + (lane & (g - 1u)), wa = __shfl_sync(full, at, src);
            const Rand4 r = draw(wt, wa);
            const bool a = below_hi(r, lim);
            const unsigned ends = __ballot_sync(full, a || below(r, lim)), at_a = __ballot_sync(full, a);
            if (open) {
                const uint32_t first = (uint32_t)__popc(m & below_me) << lg;
                const unsigned mine = (ends >> first) & (g == 32u ? full : (1u << g) - 1u);
                if (mine) {
                    const uint32_t f = (uint32_t)__ffs((int)mine) - 1u;
                    len = 2u + 2u * (t + f) + ((at_a >> (first + f)) & 1u ? 0u : 1u);
                }
                t += g;
            }
        }
        const unsigned is_long = __ballot_sync(full, len > long_len);
        const unsigned is_short = __ballot_sync(full, len != 0u) & ~is_long;
        if (len) {
            const uint32_t pos = len > long_len ? front + (uint32_t)__popc(is_long & below_me)
                                                : back - 1u - (uint32_t)__popc(is_short & below_me);
            pool.at[pos] = at;
            pool.len[pos] = len;
            open = false;
        }
        front += (uint32_t)__popc(is_long);
        back -= (uint32_t)__popc(is_short);
    }
    __syncwarp();
}

// Walkers per pool when W walkers are shared by `warps` warps: an equal share
// of W, cut into as few pools as hold it.
LT_HD uint32_t pool_walkers(uint64_t W, uint64_t warps)
{
    const uint64_t rounds = (W + warps * kPoolWalkers - 1) / (warps * kPoolWalkers);
    const uint64_t n = rounds ? (W + warps * rounds - 1) / (warps * rounds) : 0;
    return n < kPoolMin ? kPoolMin : (uint32_t)n;
}

}  // namespace lt
