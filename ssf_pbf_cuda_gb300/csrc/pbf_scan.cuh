// Exclusive scan of per-cell counts in one thread-block cluster, shared by
// the step's scan and the allocation-free sort.
#pragma once
#include <cooperative_groups.h>
#include <cstdint>

#include "pbf_after.cuh"
#include "pbf_internal.h"

namespace pbf103 {

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v)
{
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// Each block (1024 threads) of the cluster holds a run of 1024 * R counts in
// registers, its total goes into every other block's shared memory, and after
// the cluster's barrier each block adds the totals before it.
// count(index) gives a count, out(index, offset, count) is called for every
// index below n, both by the thread of the block that holds the index; returns
// the sum of all counts.  A block's shared memory may be written from outside
// once the block runs, so the totals go out after a barrier of the cluster:
// the caller's (MET), or one that is arrived at here before the counts are
// requested and waited for after their warp scans.
template <uint32_t R, bool MET = false, class COUNT, class OUT>
__device__ __forceinline__ uint32_t cluster_scan(COUNT &&count, uint32_t n, OUT &&out)
{
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    __shared__ uint32_t ws[R][32], tot[32];
    const uint32_t rank = cluster.block_rank(), blocks = cluster.num_blocks();
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, base = rank * (1024u * R);
    if (!MET) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    uint32_t v[R], inc[R];
#pragma unroll
    for (uint32_t k = 0; k < R; ++k) {
        const uint32_t idx = base + k * 1024u + t;
        v[k] = idx < n ? count(idx) : 0u;
    }
#pragma unroll
    for (uint32_t k = 0; k < R; ++k) {
        inc[k] = warp_incl_scan(v[k]);
        if (lane == 31) ws[k][warp] = inc[k];
    }
    __syncthreads();
    if (!MET) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (warp == 0) {  // exclusive prefix of every (round, warp) total, rounds in order
        uint32_t carry = 0;
#pragma unroll
        for (uint32_t k = 0; k < R; ++k) {
            const uint32_t wv = ws[k][lane];
            const uint32_t wi = warp_incl_scan(wv);
            ws[k][lane] = carry + wi - wv;
            carry += __shfl_sync(0xffffffffu, wi, 31);
        }
        if (lane < blocks) *cluster.map_shared_rank(&tot[rank], lane) = carry;
    }
    cluster.sync();  // every block's totals are in; no block writes another's memory after it
    // every warp adds for itself, a block's total a lane: a block has 32 warps,
    // so each instruction here costs 8 cycles (a loop over the totals 1,300)
    static_assert(kScanClusterMax <= 32, "a total a lane");
    const uint32_t x = lane < blocks ? tot[lane] : 0u;
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < rank ? x : 0u);
    const uint32_t all = __reduce_add_sync(0xffffffffu, x);
#pragma unroll
    for (uint32_t k = 0; k < R; ++k) {
        const uint32_t idx = base + k * 1024u + t;
        if (idx < n) out(idx, before + ws[k][warp] + inc[k] - v[k], v[k]);
    }
    return all;
}

// R for n counts in a cluster of `blocks` blocks, 0 when they do not fit.
inline uint32_t cluster_scan_rounds(uint32_t n, uint32_t blocks)
{
    const uint32_t need = (n + blocks * 1024u - 1u) / (blocks * 1024u);
    for (uint32_t r = 1; r <= 16; r *= 2)
        if (need <= r) return r;
    return need <= kScanRoundsMax ? kScanRoundsMax : 0u;
}

// Launches fn (a kernel of 1024-thread blocks) as one cluster of `blocks`.
// AFTER: as launch_after does.
template <bool AFTER = false, class... A>
cudaError_t launch_cluster(void (*fn)(A...), uint32_t blocks, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(1024);
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = AFTER ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

// Whether fn may run as a cluster of kScanClusterMax blocks on the current
// device (beyond the portable size, so a device may have no room for it).
template <class... A>
bool allows_cluster(void (*fn)(A...))
{
    bool ok = cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kScanClusterMax);
    cfg.blockDim = dim3(1024);
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kScanClusterMax;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    ok = ok && cudaOccupancyMaxActiveClusters(&n, (const void *)fn, &cfg) == cudaSuccess && n > 0;
    if (!ok) cudaGetLastError();  // a refused attribute is an answer, not an error
    return ok;
}

}  // namespace pbf103
