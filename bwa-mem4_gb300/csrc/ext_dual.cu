// ext_dual.cu -- the 8-bit length buckets of large batches, two jobs per thread (ext_dual.cuh).
#include <cuda_runtime.h>

#include <algorithm>

#include "ext_dual.cuh"
#include "kernels.h"
#include "persist.h"

namespace bwacuda {
namespace dual {

// Warps take 64 consecutive sorted jobs at a time from the bucket's counter, two neighbours a lane.
template <int TB, bool SYM>
__global__ void __launch_bounds__(TB)
ext_dual_kernel(const uint8_t *__restrict__ seq, const bwacuda_dev_ext_job *__restrict__ jobs,
                const uint32_t *__restrict__ order, uint32_t *__restrict__ table, const __grid_constant__ ExtParams P,
                int qcap, const __grid_constant__ DualMul mul, bwacuda_ext_result *__restrict__ out, uint32_t *__restrict__ err,
                unsigned long long *__restrict__ cells_total)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31;
    uint32_t *cw = reinterpret_cast<uint32_t *>(smem_raw) + tid;
    uint16_t *qs = reinterpret_cast<uint16_t *>(smem_raw + (size_t)thread_cells(qcap) * TB * 4) + tid;
    const uint32_t start = table[0], stop = table[1];
    uint32_t *counter = table + 2;
    unsigned long long ncells = 0;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(counter, 64u);
        base = __shfl_sync(0xffffffffu, base, 0) + start;
        if (base >= stop) break;
        const uint32_t k = base + 2u * (uint32_t)lane;
        if (k < stop) {
            const bool two = k + 1 < stop;
            const uint32_t ja = order[k], jb = two ? order[k + 1] : ja;
            const bwacuda_dev_ext_job JA = jobs[ja], JB = jobs[jb];
            const bool ok = JA.qlen >= 0 && JB.qlen >= 0 && JA.qlen + 1 <= qcap && JB.qlen + 1 <= qcap &&
                            ext_fits_u8(JA.qlen, JA.tlen, JA.h0, P.sc.max_sc) &&
                            ext_fits_u8(JB.qlen, JB.tlen, JB.h0, P.sc.max_sc);
            if (!ok) {
                atomicOr(err, ERR_RANGE);
            } else {
                bool bad = false;
                bwacuda_ext_result ra, rb;
                run_pair<TB, SYM>(cw, qs, seq, JA, JB, two, P, mul, bad, ncells, ra, rb);
                if (bad) atomicOr(err, ERR_BASE);
                out[ja] = ra;
                if (two) out[jb] = rb;
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ncells += __shfl_xor_sync(0xffffffffu, ncells, o);
    if (lane == 0 && ncells) atomicAdd(cells_total, ncells);
}

template <int TB>
cudaError_t launch(const PersistLaunch &L, const ExtBucketDef &d, uint32_t *table, int nsm)
{
    const size_t smem = thread_bytes(d.qcap) * TB;
    const bool sym = L.P.sc.o_del + L.P.sc.e_del == L.P.sc.o_ins + L.P.sc.e_ins;
    auto kern = sym ? ext_dual_kernel<TB, true> : ext_dual_kernel<TB, false>;
    // process-wide per kernel: always the ceiling (see the other persistent kernels)
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EXT_SMEM_BLOCK_MAX);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TB, smem)) != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidValue;
    if (L.reserve_regs > 0 || L.reserve_threads > 0) {
        cudaFuncAttributes fa;
        if ((e = cudaFuncGetAttributes(&fa, kern)) != cudaSuccess) return e;
        const int regs_block = ((fa.numRegs * 32 + 255) / 256) * 256 * (TB / 32);
        const int cap_r = regs_block > 0 ? (L.sm_regs - L.reserve_regs) / regs_block : per_sm;
        const int cap_t = (L.sm_threads - L.reserve_threads) / TB;
        per_sm = std::max(1, std::min(per_sm, std::min(cap_r, cap_t)));
    }
    kern<<<per_sm * nsm, TB, smem, L.stream>>>(L.seq, L.jobs, L.order, table, L.P, d.qcap, DualMul(), L.out, L.err, L.cells);
    return cudaGetLastError();
}

}  // namespace dual

cudaError_t ext_dual_launch(const PersistLaunch &L, const ExtBucketDef &d, uint32_t *table, int nsm)
{
    return dual::launch<64>(L, d, table, nsm);
}

}  // namespace bwacuda
