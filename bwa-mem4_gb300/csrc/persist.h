// persist.h -- interface of the batched (sorted, bucketed, persistent) extension path.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "common.cuh"

namespace bwacuda {

// One bucket: jobs of cell class `cls` (0 = 8-bit pairs, 1 = 16-bit, 2 = 32-bit)
// with qlen in [qlo, qhi], run with qcap cell columns per thread (kernel 0) or by the
// group-per-job kernel (kernel 1: the open-ended buckets, whose queries may exceed any
// thread's shared-memory row, and the buckets from the tuned query length up).
struct ExtBucketDef {
    int32_t cls;
    int32_t qlo, qhi;
    int32_t qcap;
    int32_t kernel;
};

constexpr int EXT_MAX_BUCKETS = 64;  // one thread each in the bucket-bounds kernel
constexpr int32_t EXT_QHI_OPEN = 1 << 30;  // qhi of a class's open-ended last bucket

// First and last sort key of a bucket: class, then query length (clamped at 1023) descending, then ten
// more bits.
struct BucketKeys {
    uint32_t lo, hi;
};
__device__ __forceinline__ BucketKeys bucket_keys(const ExtBucketDef &d)
{
    const uint32_t ql_hi = d.qhi > 1023 ? 1023u : (uint32_t)d.qhi;
    const uint32_t ql_lo = d.qlo > 1023 ? 1023u : (uint32_t)d.qlo;
    return {((uint32_t)d.cls << 20) | ((1023u - ql_hi) << 10), ((uint32_t)d.cls << 20) | ((1023u - ql_lo) << 10) | 1023u};
}
__device__ __forceinline__ uint32_t lower_bound(const uint32_t *a, uint32_t n, uint32_t v)
{
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

struct PersistLaunch {
    const uint8_t *seq;
    const bwacuda_dev_ext_job *jobs;
    const uint32_t *order;  // sorted job indices
    ExtParams P;
    bwacuda_ext_result *out;
    uint32_t *err;
    unsigned long long *cells;
    int grab;  // 32-job rounds a warp takes per work-counter grab
    cudaStream_t stream;
    // registers and threads per SM the persistent blocks leave free for kernels
    // that run beside them (0: fill the SM); sm_regs / sm_threads are the SM's
    int reserve_regs = 0, reserve_threads = 0;
    int sm_regs = 65536, sm_threads = 2048;
};

// long_qlo: buckets holding queries of this length or longer use the group-per-job kernel
// (INT_MAX: only the open-ended ones).
int ext_bucket_defs(ExtBucketDef *defs, int max_defs, int step, int long_qlo);
size_t ext_sort_temp_bytes(size_t n);
// the sort's own kernels prefer the maximum shared-memory carveout (once per device)
cudaError_t ext_sort_prefer_shared();
// Keys and radix sort: idx_out holds the job indices by class (at least min_cls), query length, target
// length and seed score, each descending.  n_to_16 puts 8-bit jobs whose query holds a code of 4 or more
// into the 16-bit class; with ug enabled the key kernel also settles ungapped hits (results written to
// out).  small (a small batch's parameters): the classes are the band kernel's jobs, the other 16-bit
// ones and the 32-bit ones, and their numbers are added to kinds[0 .. 3).
cudaError_t ext_sort_jobs(const bwacuda_dev_ext_job *jobs, size_t n, int max_sc, uint32_t min_cls, bool n_to_16,
                          const uint8_t *seq, const UngappedRule &ug, int zdrop, bwacuda_ext_result *out, uint32_t *keys_in,
                          uint32_t *keys_out, uint32_t *idx_in, uint32_t *idx_out, void *tmp, size_t tmp_bytes,
                          cudaStream_t s, const ExtParams *small = nullptr, uint32_t *kinds = nullptr);
// ext_sort_jobs and the bucket bounds; d_table holds 4 words per bucket (start, end, work counter,
// the band kernel's work counter).  pair_lanes false (gap costs too large for 16-bit lanes) keeps every
// job out of the 8-bit class.
cudaError_t ext_sort_and_bucket(const bwacuda_dev_ext_job *jobs, size_t n, int max_sc, bool pair_lanes, bool n_to_16,
                                const uint8_t *seq,
                                const UngappedRule &ug, int zdrop, bwacuda_ext_result *out, uint32_t *keys_in,
                                uint32_t *keys_out, uint32_t *idx_in, uint32_t *idx_out, void *tmp,
                                size_t tmp_bytes, const ExtBucketDef *d_defs, int nb, uint32_t *d_table,
                                cudaStream_t s);
// The 32-bit jobs of a sorted small batch (its sort keys and kinds) in their thread-per-job length buckets,
// all in one launch (ext_wide.cu), when there are wide_min or more of them: work[XL_WORK_WIDE_STOP] is then
// where those begin.
cudaError_t ext_wide_launch(const PersistLaunch &L, const uint32_t *keys, uint32_t n, uint32_t wide_min,
                            const ExtBucketDef *d_defs, int nb, uint32_t *work, int nsm);
// An 8-bit bucket with two jobs per thread (ext_dual.cuh): scorings of at most five letters.
cudaError_t ext_dual_launch(const PersistLaunch &L, const ExtBucketDef &d, uint32_t *d_bucket_table, int nsm);
// per-grab instantiations (ext_persist_g1.cu, _g2.cu, _g4.cu)
cudaError_t ext_persist_launch_g1(const PersistLaunch &L, const ExtBucketDef &d, uint32_t *table, int nsm, int tb);
cudaError_t ext_persist_launch_g2(const PersistLaunch &L, const ExtBucketDef &d, uint32_t *table, int nsm, int tb);
cudaError_t ext_persist_launch_g4(const PersistLaunch &L, const ExtBucketDef &d, uint32_t *table, int nsm, int tb);
cudaError_t ext_persist_launch(const PersistLaunch &L, const ExtBucketDef &d, uint32_t *d_bucket_table, int nsm,
                               int tb);

}  // namespace bwacuda
