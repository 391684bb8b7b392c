// rmat.cu -- seeded RMAT graph generator on the GPU.
//
// The reference reads its datasets from disk (tools/convert_from_txt.cc); the
// synthetic RMAT graphs stand in for them.  The generator is written so that
// the CSR comes out directly, without sorting an edge list:
//   1. the source of edge i is drawn bit by bit (level l uses 16-bit lane l
//      of Philox(ctr = (i lo, i hi, 0x10, l / 8)); bit = lane >= T_src) and
//      counted into out-degrees;  the multiset of sources is exactly that of
//      RMAT;
//   2. rowptr = exclusive scan of the out-degrees;
//   3. the k-th out-edge of u gets its destination from the RMAT conditional
//      given u's bits (lane l of Philox(ctr = (u, k, 0x11, l / 8)); bit =
//      lane >= (bit_l(u) ? T_d1 : T_d0)), so col is a pure function of (u, k);
//   4. vertices with no in- and no out-edges are removed keeping order
//      (tools/rm_isolated_vertices.cc:70-87).
// Every step is integer-only, so the CPU restatement produces the same bytes.
#include <cstdio>

#include "common.h"
#include "graph.h"
#include "lt_core.cuh"
#include "scan.cuh"

namespace lt {

namespace {

constexpr int kGenBlock = 256;

// The bits of 8 levels, most significant first, one 16-bit lane of r each:
// bit = lane >= threshold, t1 where the level's source bit (bit 7 - l of
// sbits) is set, else t0.
__device__ __forceinline__ uint32_t rmat_bits(const Rand4 &r, uint32_t sbits, uint32_t t0, uint32_t t1)
{
    uint32_t v = 0;
#pragma unroll
    for (int l = 0; l < 8; l++) v = (v << 1) | (lane16(r, l) >= ((sbits >> (7 - l)) & 1u ? t1 : t0) ? 1u : 0u);
    return v;
}

__device__ __forceinline__ uint32_t rmat_src(uint64_t seed, uint64_t i, int scale, uint32_t t_src)
{
    uint32_t v = 0;
    for (int l = 0; l < scale; l += 8) {
        const Rand4 r = philox4x32_10((uint32_t)i, (uint32_t)(i >> 32), kTagRmatSrc, (uint32_t)(l >> 3),
                                      (uint32_t)seed, (uint32_t)(seed >> 32));
        const int n = scale - l < 8 ? scale - l : 8;
        v = (v << n) | rmat_bits(r, 0u, t_src, t_src) >> (8 - n);
    }
    return v;
}

__device__ __forceinline__ uint32_t rmat_dst(uint64_t seed, uint32_t u, uint32_t k, int scale, uint32_t t_d0,
                                             uint32_t t_d1)
{
    uint32_t v = 0;
    for (int l = 0; l < scale; l += 8) {
        const Rand4 r =
            philox4x32_10(u, k, kTagRmatDst, (uint32_t)(l >> 3), (uint32_t)seed, (uint32_t)(seed >> 32));
        const int n = scale - l < 8 ? scale - l : 8;
        // the n source bits below the l already used, at the top of 8 bits
        const uint32_t sbits = ((u >> (scale - l - n)) << (8 - n)) & 0xFFu;
        v = (v << n) | rmat_bits(r, sbits, t_d0, t_d1) >> (8 - n);
    }
    return v;
}

// Out-degrees.  RMAT sources crowd the low ids (the top 8 levels are all zero
// for (a+b)^8 = 11 % of the edges, the lowest 32 ids alone draw 1.6 % at
// scale 20), and atomics on one line serialise in L2: the counters of the
// lowest kHotIds ids are kept per CTA in shared memory and added once at the
// end.  2^24 edges at scale 20: 440 -> 288 us, the time of the draws.
constexpr uint32_t kHotIds = 4096;

__global__ void __launch_bounds__(kGenBlock) degrees_kernel(uint64_t E, uint64_t seed, int scale, uint32_t t_src,
                                                            uint32_t *deg)
{
    __shared__ uint32_t hot[kHotIds];
    for (uint32_t i = threadIdx.x; i < kHotIds; i += kGenBlock) hot[i] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E; i += stride) {
        const uint32_t u = rmat_src(seed, i, scale, t_src);
        if (u < kHotIds)
            atomicAdd(&hot[u], 1u);
        else
            atomicAdd(&deg[u], 1u);
    }
    __syncthreads();
    // ids the graph does not have (a scale below 12) stay at zero
    for (uint32_t i = threadIdx.x; i < kHotIds; i += kGenBlock)
        if (hot[i]) atomicAdd(&deg[i], hot[i]);
}

// Column entries.  A warp fills kFillEdges consecutive edges at a time,
// whatever rows they belong to: the warp finds the rows of its first and last
// edge, and each lane finds its edge's row between them by a binary search of
// the cached offsets (the rows of 32 consecutive edges share their probes).
// Bound by the arithmetic of the draws (three Philox evaluations per edge at
// scale 20).  With one warp per 32 rows, the warp of the hub rows ran alone at
// the end (2^24 edges at scale 20: 17.4 ms); with 1024 edges per warp in
// windows of 32 rows, the warps of the sparse rows did (0.53 ms); this form
// takes 0.29 ms.
constexpr uint64_t kFillEdges = 512;

__global__ void __launch_bounds__(kGenBlock) fill_kernel(uint64_t V0, uint64_t E, const uint64_t *rowptr,
                                                         uint64_t seed, int scale, uint32_t t_d0, uint32_t t_d1,
                                                         uint32_t *col)
{
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x / 32);
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; w * kFillEdges < E; w += warps) {
        const uint64_t begin = w * kFillEdges, end = begin + kFillEdges < E ? begin + kFillEdges : E;
        const uint64_t r0 = warp_find_last(rowptr, 0, V0, begin), r1 = warp_find_last(rowptr, r0, V0, end - 1);
        for (uint64_t e = begin + lane; e < end; e += 32) {
            // the row of e: the largest u in [r0, r1] with rowptr[u] <= e
            uint32_t lo = (uint32_t)r0, n = (uint32_t)(r1 - r0 + 1);
            while (n > 1) {
                const uint32_t half = n / 2;
                if (__ldg(rowptr + lo + half) <= e) {
                    lo += half;
                    n -= half;
                } else {
                    n = half;
                }
            }
            col[e] = rmat_dst(seed, lo, (uint32_t)(e - __ldg(rowptr + lo)), scale, t_d0, t_d1);
        }
    }
}

__global__ void mark_present(uint64_t V0, const uint32_t *deg, uint32_t *present)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < V0; v += stride) present[v] = deg[v] > 0;
}

// Most targets are marked already: a look before the store keeps the hub
// vertices' lines from being written once per edge (2^24 edges at scale 20:
// 381 -> 46 us).
__global__ void mark_targets(uint64_t E, const uint32_t *col, uint32_t *present)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += stride) {
        const uint32_t v = col[e];
        if (present[v] == 0u) present[v] = 1u;
    }
}

__global__ void compact_rowptr(uint64_t V0, const uint32_t *present, const uint32_t *newid, const uint64_t *rowptr,
                               uint64_t *rowptr2)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= V0; v += stride) {
        if (v == V0)
            rowptr2[newid[V0]] = rowptr[V0];
        else if (present[v])
            rowptr2[newid[v]] = rowptr[v];
    }
}

__global__ void remap_col(uint64_t E, const uint32_t *newid, uint32_t *col)
{
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += stride) col[e] = newid[col[e]];
}

struct DevBufs {
    void *p[3] = {};
    ~DevBufs()
    {
        for (void *q : p)
            if (q) cudaFree(q);
    }
};

}  // namespace

uint32_t rmat_q16(double p) { return (uint32_t)(p * 65536.0 + 0.5); }

lt_status generate_rmat(int device, uint32_t scale, uint64_t E, double a, double b, double c, double d, uint64_t seed,
                        lt_graph &g)
{
    if (scale < 1 || scale > 31) return fail(LT_ERR_INVALID, "RMAT scale %u outside [1, 31]", scale);
    if (!(a >= 0 && b >= 0 && c >= 0 && d >= 0) || a + b <= 0 || c + d <= 0)
        return fail(LT_ERR_INVALID, "RMAT probabilities must be non-negative with a+b > 0 and c+d > 0");
    const uint32_t t_src = rmat_q16(a + b), t_d0 = rmat_q16(a / (a + b)), t_d1 = rmat_q16(c / (c + d));
    LT_CUDA_TRY(cudaSetDevice(device));
    const uint64_t V0 = 1ull << scale;
    int sms = 0;
    LT_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const int grid = sms * 8;
    cudaStream_t st = 0;

    DevBufs B;
    // one allocation for the per-vertex arrays (each costs a driver call of
    // some 80 us, and its release as much), u64 ones first
    const uint64_t tmp_n = scan_tmp_elems(V0 + 1);
    LT_CUDA_TRY(cudaMalloc(&B.p[0], 8 * (V0 + 1 + tmp_n) + 4 * (V0 + V0 + 1)));
    uint64_t *d_rowptr = (uint64_t *)B.p[0], *d_tmp = d_rowptr + V0 + 1;
    uint32_t *d_deg = (uint32_t *)(d_tmp + tmp_n), *d_newid = d_deg + V0;
    LT_CUDA_TRY(cudaMalloc(&B.p[1], 4 * (E ? E : 1)));
    uint32_t *d_col = (uint32_t *)B.p[1];

    LT_CUDA_TRY(cudaMemsetAsync(d_deg, 0, 4 * V0, st));
    degrees_kernel<<<grid, kGenBlock, 0, st>>>(E, seed, (int)scale, t_src, d_deg);
    LT_CUDA_TRY(cudaGetLastError());
    LT_CUDA_TRY((exclusive_scan<uint32_t, uint64_t>(d_deg, V0, d_rowptr, d_tmp, st)));
    fill_kernel<<<grid, kGenBlock, 0, st>>>(V0, E, d_rowptr, seed, (int)scale, t_d0, t_d1, d_col);
    LT_CUDA_TRY(cudaGetLastError());

    // isolated-vertex removal: present = out-degree > 0 or some in-edge.
    uint32_t *d_present = d_deg;  // reuse: deg is not needed after the flags are set
    mark_present<<<grid, kGenBlock, 0, st>>>(V0, d_deg, d_present);
    mark_targets<<<grid, kGenBlock, 0, st>>>(E, d_col, d_present);
    LT_CUDA_TRY(cudaGetLastError());
    uint32_t *d_tmp32 = (uint32_t *)d_tmp;
    LT_CUDA_TRY((exclusive_scan<uint32_t, uint32_t>(d_present, V0, d_newid, d_tmp32, st)));
    uint32_t V = 0;
    // page-locking the result's memory (2.2 ms for 64 MB) overlaps the kernels
    LT_TRY(host_alloc(g.col_buf, 4ull * E, true));
    LT_CUDA_TRY(cudaMemcpyAsync(&V, d_newid + V0, 4, cudaMemcpyDeviceToHost, st));
    LT_CUDA_TRY(cudaStreamSynchronize(st));
    LT_CUDA_TRY(cudaMalloc(&B.p[2], 8 * ((uint64_t)V + 1)));
    uint64_t *d_rowptr2 = (uint64_t *)B.p[2];
    compact_rowptr<<<grid, kGenBlock, 0, st>>>(V0, d_present, d_newid, d_rowptr, d_rowptr2);
    remap_col<<<grid, kGenBlock, 0, st>>>(E, d_newid, d_col);
    LT_CUDA_TRY(cudaGetLastError());

    g.V = V;
    g.E = E;
    LT_TRY(host_alloc(g.rowptr_buf, 8ull * ((uint64_t)V + 1), true));
    LT_CUDA_TRY(cudaMemcpyAsync(g.rowptr_mut(), d_rowptr2, 8ull * ((uint64_t)V + 1), cudaMemcpyDeviceToHost, st));
    LT_CUDA_TRY(cudaMemcpyAsync(g.col_mut(), d_col, 4ull * E, cudaMemcpyDeviceToHost, st));
    LT_CUDA_TRY(cudaStreamSynchronize(st));
    return LT_OK;
}

}  // namespace lt
