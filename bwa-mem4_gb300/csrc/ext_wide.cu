// ext_wide.cu -- the 32-bit jobs of a sorted small batch where they are many: the thread-per-job length
// buckets, all in one launch.
//
// Bound.  A thread's row takes 8 bytes a column of shared memory, so an SM holds few jobs and their
// latency sets the time.  The buckets' own kernels (ext_persist.cuh) fill the GPU bucket by bucket, but a
// small batch seldom has such a job, and eleven launches that find nothing took the band kernel beside
// them 3-10% (10,000 read pairs 380 -> 390-420 us).  One block an SM here walks the buckets, longest queries first, each with as many threads
// as its rows leave room for.  On 152 SMs, 150-base jobs: 10,000 in 0.88 ms (1.24 in the group-per-job
// kernel, 1.01 in the buckets' own), 20,000 in 1.64 (2.18, 1.91), 50,000 in 2.41 (5.00, 2.80).  The bucket
// bounds are searched here, a thread each: a kernel that did it for every small batch cost each of them
// 7-10 us, a tenth of a millisecond on a serving call of thirty small requests.
#include <cuda_runtime.h>

#include "ext_job.cuh"
#include "kernels.h"
#include "persist.h"

namespace bwacuda {
namespace {

constexpr int WIDE_TB = 512;

// Threads of a bucket: the most whose rows fit a block (0: none).
__device__ __forceinline__ int wide_threads(int qcap)
{
    int tb = WIDE_TB;
    while (tb >= 32 && ext_block_smem(qcap, tb, FmtI32::bytes) > EXT_SMEM_BLOCK_MAX) tb >>= 1;
    return tb >= 32 ? tb : 0;
}

// One bucket on the block's first TB threads.
template <int TB>
__device__ __forceinline__ void wide_bucket(unsigned char *smem, const uint8_t *__restrict__ seq,
                                            const bwacuda_dev_ext_job *__restrict__ jobs,
                                            const uint32_t *__restrict__ order, uint32_t start, uint32_t stop,
                                            uint32_t *__restrict__ counter, const ExtParams &P, int qcap, bwacuda_ext_result *__restrict__ out,
                                            uint32_t *__restrict__ err, unsigned long long &ncells)
{
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid >= TB) return;
    FmtI32::T *cell = reinterpret_cast<FmtI32::T *>(smem) + tid;
    uint32_t *qw = reinterpret_cast<uint32_t *>(reinterpret_cast<FmtI32::T *>(smem) + (size_t)qcap * TB) + tid;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(counter, 32u);
        base = __shfl_sync(0xffffffffu, base, 0) + start;
        if (base >= stop) break;
        const uint32_t k = base + lane;
        if (k < stop) {
            const uint32_t jid = order[k];
            const bwacuda_dev_ext_job J = jobs[jid];
            if (J.qlen < 0 || J.qlen + 1 > qcap) {
                atomicOr(err, ERR_RANGE);
            } else {
                bool bad = false;
                const bwacuda_ext_result r = ext_run_job<FmtI32, TB>(cell, qw, seq, J, P, bad, ncells);
                if (bad) atomicOr(err, ERR_BASE);
                out[jid] = r;
            }
        }
    }
}

__global__ void __launch_bounds__(WIDE_TB)
ext_wide_kernel(const uint8_t *__restrict__ seq, const bwacuda_dev_ext_job *__restrict__ jobs,
                const uint32_t *__restrict__ order, const uint32_t *__restrict__ keys, uint32_t n, uint32_t wide_min,
                const ExtBucketDef *__restrict__ defs, int nb, uint32_t *__restrict__ work,
                const __grid_constant__ ExtParams P, bwacuda_ext_result *__restrict__ out, uint32_t *__restrict__ err,
                unsigned long long *__restrict__ cells_total)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (work[XL_WORK_KINDS + 2] < wide_min) return;
    __shared__ uint32_t bounds[2][EXT_MAX_BUCKETS], first;
    if (threadIdx.x == 0) first = n;
    __syncthreads();
    if (threadIdx.x < 2 * EXT_MAX_BUCKETS) {  // a thread a search
        const int b = threadIdx.x % EXT_MAX_BUCKETS, hi = threadIdx.x / EXT_MAX_BUCKETS;
        if (b < nb && defs[b].cls == 2 && defs[b].kernel == 0) {
            const BucketKeys k = bucket_keys(defs[b]);
            const uint32_t at = lower_bound(keys, n, hi ? k.hi + 1u : k.lo);
            bounds[hi][b] = at;
            if (!hi) atomicMin(&first, at);
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) work[XL_WORK_WIDE_STOP] = first;
    unsigned long long ncells = 0;
    for (int b = nb - 1; b >= 0; --b) {
        const ExtBucketDef d = defs[b];
        if (d.cls != 2 || d.kernel != 0) continue;
        const uint32_t start = bounds[0][b], stop = bounds[1][b];
        uint32_t *counter = work + XL_WORK_WIDE_COUNTERS + b;
        if (start == stop) continue;
        switch (wide_threads(d.qcap)) {
#define WIDE_CASE(T) \
    case T: wide_bucket<T>(smem_raw, seq, jobs, order, start, stop, counter, P, d.qcap, out, err, ncells); break
            WIDE_CASE(512);
            WIDE_CASE(256);
            WIDE_CASE(128);
            WIDE_CASE(64);
            WIDE_CASE(32);
#undef WIDE_CASE
        default: if (threadIdx.x == 0) atomicOr(err, ERR_RANGE);
        }
        __syncthreads();  // the next bucket's rows lie over this one's
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ncells += __shfl_xor_sync(0xffffffffu, ncells, o);
    if ((threadIdx.x & 31) == 0 && ncells) atomicAdd(cells_total, ncells);
}

}  // namespace

static_assert(XL_WORK_WIDE_COUNTERS + EXT_MAX_BUCKETS <= XL_WORK_WORDS, "a work counter a bucket");

cudaError_t ext_wide_launch(const PersistLaunch &L, const uint32_t *keys, uint32_t n, uint32_t wide_min,
                            const ExtBucketDef *d_defs, int nb, uint32_t *work, int nsm)
{
    // process-wide per kernel: always the ceiling (see the persistent kernels)
    cudaError_t e = cudaFuncSetAttribute(ext_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EXT_SMEM_BLOCK_MAX);
    if (e != cudaSuccess) return e;
    ext_wide_kernel<<<nsm, WIDE_TB, EXT_SMEM_BLOCK_MAX, L.stream>>>(L.seq, L.jobs, L.order, keys, n, wide_min, d_defs, nb,
                                                                    work, L.P, L.out, L.err, L.cells);
    return cudaGetLastError();
}

}  // namespace bwacuda
