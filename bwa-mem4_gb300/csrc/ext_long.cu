// ext_long.cu -- launches of the group-per-job extension kernel (ext_long.cuh): the query
// lengths the thread-per-job kernels cannot hold (their DP row lives in shared memory per
// thread), and, where the autotuner measures it faster, the longer buckets of the batched path.
//
// A call makes up to two launches per cell class: the first with the caller's ring size
// (enough for bands up to (R - 3) / 2 columns, or any band on queries of fewer than R
// columns), and a deferred launch over the jobs the first one set aside, a warp per job.
#include <cuda_runtime.h>

#include <algorithm>

#include "ext_long.cuh"
#include "kernels.h"

namespace bwacuda {

namespace {

constexpr int XL_C = 8;          // columns per lane per chunk
constexpr int XL_BLOCK = 128;    // threads per block of the first launch

template <bool W32, int L>
cudaError_t launch_first(const ExtLongLaunch &X, int nsm)
{
    auto kern = xl::ext_long_kernel<W32, L, XL_C>;
    const int groups = XL_BLOCK / L;
    // the largest ring up to the requested one whose block fits (jobs needing more are deferred)
    int ring = X.ring_cols;
    while (ring > XL_RING_MIN && (size_t)groups * xl::ring_words(ring, W32) * 4 > EXT_SMEM_BLOCK_MAX) ring >>= 1;
    const size_t smem = (size_t)groups * xl::ring_words(ring, W32) * 4;
    if (smem > EXT_SMEM_BLOCK_MAX) return cudaErrorInvalidValue;
    // process-wide per kernel: always the ceiling (see the persistent kernels)
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EXT_SMEM_BLOCK_MAX);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, XL_BLOCK, smem)) != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidValue;
    if (X.reserve_regs > 0 || X.reserve_threads > 0) {
        cudaFuncAttributes fa;
        if ((e = cudaFuncGetAttributes(&fa, kern)) != cudaSuccess) return e;
        const int regs_block = ((fa.numRegs * 32 + 255) / 256) * 256 * (XL_BLOCK / 32);
        const int cap_r = regs_block > 0 ? (X.sm_regs - X.reserve_regs) / regs_block : per_sm;
        const int cap_t = (X.sm_threads - X.reserve_threads) / XL_BLOCK;
        per_sm = std::max(1, std::min(per_sm, std::min(cap_r, cap_t)));
    }
    const size_t most = ((size_t)X.njobs * L + XL_BLOCK - 1) / XL_BLOCK;
    const uint32_t grid = (uint32_t)std::min<size_t>((size_t)per_sm * nsm, std::max<size_t>(most, 1));
    kern<<<grid, XL_BLOCK, smem, X.stream>>>(X.seq, X.jobs, X.order, X.bounds, X.part, X.part_min, X.counter, X.njobs,
                                            X.min_qlen, ring, X.defer, X.defer_count, W32 ? 0 : X.band, X.small, X.P,
                                            X.out, X.err, X.cells);
    return cudaGetLastError();
}

template <bool W32>
cudaError_t launch_first_lanes(const ExtLongLaunch &X, int nsm)
{
    if (X.lanes == 8) return launch_first<W32, 8>(X, nsm);
    if (X.lanes == 16) return launch_first<W32, 16>(X, nsm);
    return launch_first<W32, 32>(X, nsm);
}

template <bool W32>
cudaError_t launch_deferred(const ExtLongLaunch &X, const uint32_t *count, uint32_t *counter, uint32_t *counter_all,
                            int nsm)
{
    constexpr int TB = 32 * xl::DEFER_WARPS;
    auto kern = xl::ext_long_deferred_kernel<W32, XL_C>;
    const size_t smem = (size_t)xl::ring_words(W32 ? xl::RING_MAX_32 : xl::RING_MAX_16, W32) * 4;
    static_assert(xl::DEFER_WARPS * (xl::RING_MAX_16 / xl::DEFER_WARPS / 32) == xl::RING_MAX_16 / 32,
                  "the warps' rings fill the largest one's words");
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EXT_SMEM_BLOCK_MAX);
    if (e != cudaSuccess) return e;
    const uint32_t grid = (uint32_t)std::min<size_t>((size_t)nsm, std::max<size_t>(X.njobs, 1));
    kern<<<grid, TB, smem, X.stream>>>(X.seq, X.jobs, X.defer, count, counter, counter_all, X.njobs, X.small, X.P, X.out,
                                       X.err, X.cells);
    return cudaGetLastError();
}

}  // namespace

cudaError_t ext_long_launch(const ExtLongLaunch &X, bool w32, int nsm)
{
    return w32 ? launch_first_lanes<true>(X, nsm) : launch_first_lanes<false>(X, nsm);
}

cudaError_t ext_long_deferred_launch(const ExtLongLaunch &X, bool w32, uint32_t *work, int nsm)
{
    const uint32_t *count = work + XL_WORK_DCOUNT;
    return w32 ? launch_deferred<true>(X, count, work + XL_WORK_DCOUNTER32, work + XL_WORK_DCOUNTER32 + 1, nsm)
               : launch_deferred<false>(X, count, work + XL_WORK_DCOUNTER16, work + XL_WORK_DCOUNTER16 + 1, nsm);
}

int ext_long_ring_for_band(int w)
{
    long long need = 2LL * (w < 0 ? 0 : w) + 3;
    int r = XL_RING_MIN;
    while (r < need && r < XL_RING_FIRST_MAX) r <<= 1;
    return r;
}

}  // namespace bwacuda
