// lt_core.cuh -- types, the per-walker random stream and the three apps' step
// semantics, shared by every kernel of the engine.
//
// Random stream (replaces cuRAND XORWOW with per-thread state, src/Rand.h:1-37):
//   Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC 2011)
//   key     = (seed lo32, seed hi32)
//   counter = (c0, tag | run << 8, walker index lo32, walker index hi32)
//     init draws: tag 1, c0 = draw number; step draws: tag 2, c0 = walker.step
//     before the update.  Every (walker, step) pair therefore owns one draw,
//     whatever thread, launch or schedule runs it.
//   r64 = x0 << 32 | x1 picks a neighbour or vertex as r64 % n (the integer
//   form of uniform_discrete_distribution, src/Rand.h:17-19);
//   m53 = (x2 << 32 | x3) >> 11 is the uniform double U = (m53 + 1) 2^-53 in
//   (0, 1]; the test U > p is done exactly in integers as m53 >= floor(p 2^53).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#ifdef __CUDACC__
#define LT_HD __host__ __device__ __forceinline__
#else
#define LT_HD inline
#endif

namespace lt {

using nodeId = uint32_t;       // src/Type.h:5
using edgeId = uint64_t;       // src/Type.h:6
using walkId = uint64_t;       // src/Type.h:7
using partitionId = uint32_t;  // u16 in the reference (src/Type.h:8); the .part file keeps u16

constexpr nodeId kInvalidNode = 0xFFFFFFFFu;  // src/Type.h:18
constexpr uint32_t kTagInit = 1u;
constexpr uint32_t kTagStep = 2u;
constexpr uint32_t kTagRmatSrc = 0x10u;
constexpr uint32_t kTagRmatDst = 0x11u;

enum App : int { kPPR = 0, kPageRank = 1, kWalk = 2 };
enum Start : int { kStartSource = 0, kStartUniform = 1, kStartPerVertex = 2 };

struct Rand4 {
    uint32_t x0, x1, x2, x3;
};

LT_HD uint32_t mulhi32(uint32_t a, uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// Philox4x32 with 10 rounds.
LT_HD Rand4 philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0, uint32_t k1)
{
    constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
    constexpr uint32_t W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint32_t hi0 = mulhi32(M0, c0), lo0 = M0 * c0;
        const uint32_t hi1 = mulhi32(M1, c2), lo1 = M1 * c2;
        const uint32_t n0 = hi1 ^ c1 ^ k0;
        const uint32_t n2 = hi0 ^ c3 ^ k1;
        c0 = n0;
        c1 = lo1;
        c2 = n2;
        c3 = lo0;
        k0 += W0;
        k1 += W1;
    }
    return Rand4{c0, c1, c2, c3};
}

// The ten round keys of one seed.  A kernel whose walkers share a seed takes
// them as an argument: its draws then read them as constant operands instead
// of adding the Weyl increments in every round.
struct RoundKeys {
    uint32_t k0[10], k1[10];
};

inline RoundKeys round_keys(uint64_t seed)
{
    RoundKeys k;
    for (int r = 0; r < 10; r++) {
        k.k0[r] = (uint32_t)seed + (uint32_t)r * 0x9E3779B9u;
        k.k1[r] = (uint32_t)(seed >> 32) + (uint32_t)r * 0xBB67AE85u;
    }
    return k;
}

LT_HD Rand4 philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, const RoundKeys &k)
{
    constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint64_t p0 = (uint64_t)M0 * c0, p1 = (uint64_t)M1 * c2;
        c0 = (uint32_t)(p1 >> 32) ^ c1 ^ k.k0[r];
        c1 = (uint32_t)p1;
        c2 = (uint32_t)(p0 >> 32) ^ c3 ^ k.k1[r];
        c3 = (uint32_t)p0;
    }
    return Rand4{c0, c1, c2, c3};
}

LT_HD Rand4 walk_draw(const RoundKeys &k, uint32_t c0, uint32_t tag, uint32_t run, uint64_t idx)
{
    return philox4x32_10(c0, tag | (run << 8), (uint32_t)idx, (uint32_t)(idx >> 32), k);
}

LT_HD Rand4 walk_draw(uint64_t seed, uint32_t c0, uint32_t tag, uint32_t run, uint64_t idx)
{
    return philox4x32_10(c0, tag | (run << 8), (uint32_t)idx, (uint32_t)(idx >> 32), (uint32_t)seed,
                         (uint32_t)(seed >> 32));
}

LT_HD uint64_t r64_of(const Rand4 &r) { return ((uint64_t)r.x0 << 32) | r.x1; }
LT_HD uint64_t m53_hi(const Rand4 &r) { return (((uint64_t)r.x0 << 32) | r.x1) >> 11; }
LT_HD uint64_t m53_of(const Rand4 &r) { return (((uint64_t)r.x2 << 32) | r.x3) >> 11; }

// m53 < thr as one 64-bit comparison: thr = floor(p 2^53) as x <= (thr << 11)
// - 1 on the unshifted words (thr <= 2^53; never for thr = 0).
struct Limit53 {
    uint64_t last;
    uint32_t some;  // thr > 0
};
inline Limit53 limit53(uint64_t thr) { return Limit53{(thr << 11) - 1u, thr != 0 ? 1u : 0u}; }
LT_HD bool below_hi(const Rand4 &r, const Limit53 &l) { return l.some && (((uint64_t)r.x0 << 32) | r.x1) <= l.last; }
LT_HD bool below(const Rand4 &r, const Limit53 &l) { return l.some && (((uint64_t)r.x2 << 32) | r.x3) <= l.last; }

// floor(p * 2^53) for a float probability widened to double.
inline uint64_t threshold53(float p)
{
    const double d = (double)p;
    if (!(d > 0.0)) return 0;
    if (d >= 1.0) return (uint64_t)1 << 53;
    return (uint64_t)(d * 9007199254740992.0);
}

// The smallest PPR stop probability taken.  A walk's length has 32 bits and is
// drawn until a draw stops it: at 2^-26 one of 2^32 walks is longer than 2^32
// with probability 2^32 e^-64 < 1e-18; far below, lengths would wrap, and under
// 2^-53, where floor(p 2^53) = 0, no draw would ever stop a walk.
constexpr float kMinStopProb = 1.0f / (1 << 26);

LT_HD float rcp_f32(float d)
{
#ifdef __CUDA_ARCH__
    return __frcp_rn(d);
#else
    return 1.0f / d;
#endif
}

// 1 / d with a relative error of at most 2^-23 (PTX rcp.approx)
LT_HD float rcp_approx_f32(float d)
{
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return r;
#else
    return 1.0f / d;
#endif
}

// x mod d for 0 < d <= 2^20 by folding: with m close below 2^32 / d, e = 2^32 -
// m d is congruent to 2^32 and below 2 d, so hi 2^32 + lo = hi e + lo (mod d).
// With d <= 2^20, e < 2^21: a fold leaves a high word of at most e, the next
// one of at most 2^10, the third x below 2^32 + 2^31 (a high word of at most
// 1), the fourth below 2^32; one multiplication by m then leaves less than 3 d.
//
// m: a single-precision reciprocal scaled down by 2^-22 (so that it never
// exceeds 2^32 / d; its relative error stays below 2^-21) and one Newton step
// in integers, after which floor(2^32 / d) - 1 <= m <= 2^32 / d.
//
// Most of it is multiply-adds: the walk kernels are bound by the integer ALU,
// which three native 32-bit remainders (d < 2^16) kept busy instead.
constexpr uint32_t kFoldMax = 1u << 20;

LT_HD uint32_t mod64_fold(uint32_t hi, uint32_t lo, uint32_t d)
{
    const uint32_t m0 = (uint32_t)(rcp_approx_f32((float)d) * 4294966272.0f);
    const uint32_t m = m0 + mulhi32(m0, 0u - m0 * d);
    const uint32_t e = 0u - m * d;
    uint64_t y = (uint64_t)hi * e + lo;
    y = (uint64_t)(uint32_t)(y >> 32) * e + (uint32_t)y;
    y = (uint64_t)(uint32_t)(y >> 32) * e + (uint32_t)y;
    const uint32_t w = (uint32_t)(y >> 32) * e + (uint32_t)y;
    uint32_t r = w - mulhi32(w, m) * d;
    // r < 3 d: the unsigned minimum takes the subtraction only where it does not wrap
    uint32_t t = r - d;
    r = t < r ? t : r;
    t = r - d;
    return t < r ? t : r;
}

// x mod d for 2^16 <= d < 2^32 (used above 2^20) without 64-bit division: reduce the high word
// (32-bit remainder), estimate the quotient of the remaining t = r1 2^32 + lo
// (t < d 2^32) in single precision, then correct in integers.  The estimate's
// relative error is below 2^-21, so after the first correction |r| < 1024 d;
// a second single-precision estimate of r / d (from r >> 16) leaves |r| < 3 d,
// which the final loops remove.  The result is exact whatever the rounding of
// the estimates.
LT_HD uint32_t mod64_large(uint64_t x, uint32_t d)
{
    const uint32_t hi = (uint32_t)(x >> 32), lo = (uint32_t)x;
    const uint32_t r1 = hi % d;
    const uint64_t t = ((uint64_t)r1 << 32) | lo;
    const float rd = rcp_f32((float)d);
    const float qf = ((float)r1 * 4294967296.0f + (float)lo) * rd;
    const uint32_t q = qf >= 4294967040.0f ? 0xFFFFFF00u : (qf <= 0.0f ? 0u : (uint32_t)qf);
    int64_t r = (int64_t)(t - (uint64_t)q * d);
    const int32_t c = (int32_t)floorf((float)(int32_t)(r >> 16) * 65536.0f * rd);
    r -= (int64_t)c * (int64_t)d;
    while (r < 0) r += d;
    while (r >= (int64_t)d) r -= d;
    return (uint32_t)r;
}

// r % n for the neighbour / vertex choice, without 64-bit division (which
// the compiler lowers through the FP64 pipe, slow on this part).  n fits 32
// bits on every graph the engine accepts (degree and V are below 2^32).
LT_HD uint64_t mod_u64(uint64_t r, uint64_t n)
{
    if ((n >> 32) == 0) {
        const uint32_t d = (uint32_t)n;
        return d <= kFoldMax ? mod64_fold((uint32_t)(r >> 32), (uint32_t)r, d) : mod64_large(r, d);
    }
    return r % n;
}

// r % n for an n known before the launch (the vertex count): inv =
// floor((2^64 - 1) / n) gives a quotient at most one too small.
struct ModN {
    uint64_t inv;
    uint32_t n;
};
inline ModN mod_n(uint32_t n) { return ModN{UINT64_MAX / n, n}; }
#ifdef __CUDACC__
// x / n for an x that n divides
__device__ __forceinline__ uint64_t div_exact(const ModN &m, uint64_t x)
{
    const uint64_t q = __umul64hi(x, m.inv);  // or one less than the quotient
    return q + (x - q * m.n ? 1u : 0u);
}
__device__ __forceinline__ uint32_t mod_by(const ModN &m, uint64_t x)
{
    const uint64_t rem = x - __umul64hi(x, m.inv) * m.n;
    return (uint32_t)(rem >= m.n ? rem - m.n : rem);
}
#endif

// PPR walks longer than this begin first in their pool: twice the mean
// length at stop threshold thr = floor(p 2^53).
inline uint32_t ppr_long_len(uint64_t thr)
{
    return thr ? (uint32_t)std::min(1e9, 2.0 * 9007199254740992.0 / (double)thr) + 1u : 0xFFFFFFFFu;
}

// PPR walk length (src/walk/SingleSource.h:11-18): step = 2, then one more
// for every draw with U > prob.
LT_HD uint32_t ppr_length(uint64_t seed, uint32_t run, uint64_t idx, uint64_t thr)
{
    uint32_t step = 2;
    for (uint32_t t = 0;; t++) {
        const Rand4 r = walk_draw(seed, t, kTagInit, run, idx);
        if (m53_hi(r) < thr) return step;
        step++;
        if (m53_of(r) < thr) return step;
        step++;
    }
}

// 16-bit lane l (0..7) of a Philox output, used by the RMAT generator.
LT_HD uint32_t lane16(const Rand4 &r, int l)
{
    const uint32_t w = (l >> 1) == 0 ? r.x0 : (l >> 1) == 1 ? r.x1 : (l >> 1) == 2 ? r.x2 : r.x3;
    return (l & 1) ? (w >> 16) : (w & 0xFFFFu);
}

}  // namespace lt
