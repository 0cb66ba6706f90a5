// kernels.h -- host-side launch interface of the device kernels.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "common.cuh"

namespace bwacuda {

// Largest shared memory of one extension block.  An SM holds 228 KB and reserves 1 KB per
// resident block, so a block of at most 225 KB still lets one small block (a gather, a
// length pass, another stream's kernel) run beside it; a 227 KB block would hold its SM
// alone, and a bucket launch of such blocks waits for every other kernel to leave an SM.
constexpr size_t EXT_SMEM_BLOCK_MAX = 225u * 1024u;

struct ExtLaunch {
    const uint8_t *seq;
    const bwacuda_dev_ext_job *jobs;
    const uint32_t *order;      // job index list, or nullptr for 0..n-1
    const uint32_t *count_ptr;  // device count overriding n, or nullptr
    size_t n;
    ExtParams P;
    int qcap;                   // >= max qlen + 1 over the launch
    int only_wide;              // wide launch: 1 = skip jobs that fit narrow cells;
                                // narrow launch: 2 = report wide jobs (no wide launch follows)
    int long_follows = 0;       // 1: jobs with qlen + 1 > qcap are left to a group-per-job launch
    bwacuda_ext_result *out;
    uint32_t *err;
    unsigned long long *cells;
    cudaStream_t stream;
};

cudaError_t ext_tpj_launch(const ExtLaunch &L, bool wide);
size_t ext_tpj_smem_limit_qcap(bool wide);

// Group-per-job extension of any query length (ext_long.cu, ext_long.cuh).  Every call site
// owns XL_WORK_WORDS device words, zeroed before its launches, and a deferred-job list of
// njobs entries.
constexpr int XL_WORK_DCOUNT = 0;                              // deferred jobs
constexpr int XL_WORK_DCOUNTER16 = 1, XL_WORK_DCOUNTER32 = 3;  // work counters of the deferred launches, two each
constexpr int XL_WORK_COUNTER16 = 5, XL_WORK_COUNTER32 = 6;    // work counters of unbucketed first launches
constexpr int XL_WORK_BAND = 7;                                // work counter of a small batch's band launch
// Of a sorted small batch: the jobs of its three kinds (the band kernel's, the other 16-bit ones, the
// 32-bit ones; they lie in this order), the work counter of a second launch over the 16-bit ones, where the
// 32-bit jobs of the length buckets begin and those buckets' work counters.
constexpr int XL_WORK_KINDS = 8, XL_WORK_COUNTER_MANY = 11, XL_WORK_WIDE_STOP = 12, XL_WORK_WIDE_COUNTERS = 16;
constexpr int XL_WORK_WORDS = 16 + 64;
constexpr int XL_LANES_DEFAULT = 16;  // lanes a job of the group-per-job kernel
constexpr int XL_RING_MIN = 256, XL_RING_FIRST_MAX = 4096;
constexpr int XL_RING_DEFAULT = 512;  // first-launch ring when the bands are not known on the host

enum { XL_PART_ALL = 0, XL_PART_LEFT, XL_PART_LEFT_MANY, XL_PART_WIDE };
struct ExtLongLaunch {
    const uint8_t *seq;
    const bwacuda_dev_ext_job *jobs;
    const uint32_t *order;   // job index list (nullptr: the identity)
    const uint32_t *bounds;  // [start, stop) of positions in order, device words (nullptr: [0, njobs))
    // other than XL_PART_ALL: bounds is work + XL_WORK_KINDS and the launch runs one kind of a small batch,
    // the other 16-bit jobs when there are fewer than part_min (LEFT) or that many (LEFT_MANY), or the
    // 32-bit ones, without those of the length buckets when there are part_min or more (WIDE)
    int part = 0;
    uint32_t part_min = 0;
    uint32_t *counter;       // zeroed work counter of the first launch
    uint32_t njobs;          // jobs of the call: bounds every position and job index
    int min_qlen;            // shorter jobs belong to another launch
    int lanes;               // lanes per job: 8, 16 or 32
    int ring_cols;           // first launch's ring columns per job (a power of two)
    ExtParams P;
    bwacuda_ext_result *out;
    uint32_t *err;
    unsigned long long *cells;
    uint32_t *defer;         // njobs entries: jobs set aside for the deferred launch
    uint32_t *defer_count;   // work + XL_WORK_DCOUNT
    int band = 0;  // 1: the band kernel runs beside this launch, which leaves it the jobs of band_takes
    // 1: a small batch, all of whose jobs come here: a negative target length is an empty target on the
    // queries that the length buckets run a thread each (EXT_TPJ_QLEN_MAX), as there
    int small = 0;
    int reserve_regs = 0, reserve_threads = 0, sm_regs = 65536, sm_threads = 2048;
    cudaStream_t stream;
};
constexpr int EXT_TPJ_QLEN_MAX = 1022;  // longest query of a thread-per-job bucket

cudaError_t ext_long_launch(const ExtLongLaunch &X, bool w32, int nsm);
// Batched calls of up to this many jobs per SM run without length buckets in the band kernel, and host calls of up
// to this many straight from the caller's arrays.  Device-resident calls on 152 SMs, microseconds
// (read pairs / mixed lengths):
//   jobs       sorted buckets   8 lanes (sorted)  16        32 lanes a job
//   1,024       521 / 1369                    188 / 337      166 / 267
//   2,048       551 / 1680                    201 / 347      203 / 303
//   8,192       732 / 1747      330 / 531     379 / 494      394 / 485
//   16,384      768 / 1795      402 / 630     610 / 719      620 / 682
//   32,768      784 / 1948      510 / 668    1061 / 1130    1088 / 1126
//   65,536      812 / 1972      847 / 910    1966 / 2015    2017 / 2039
//   131,072     907 / 2130     1597 / 1595
constexpr int EXT_SMALL_JOBS_PER_SM = 350;
// What the band kernel leaves of a small batch runs in the group-per-job kernels, except that 32-bit
// jobs from EXT_SMALL_WIDE_PER_SM per SM on get a thread each in the length buckets; the 16-bit ones get
// 8 lanes each from EXT_SMALL_LEFT8_PER_SM per SM on unless the option or the tuner set other lanes than
// the default.
// Microseconds on 152 SMs, buckets / 16 lanes / 8 lanes:
//   jobs      150 bases, 32-bit      300 bases, band 200     600 bases, band 150
//    3,500       990 /  505 /  568    1790 /   941 /  1131    3000 /  1964 /  2376
//   10,000       884 / 1317 / 1170    3240 /  2452 /  2317    5660 /  4981 /  4817
//   20,000      1640 / 2294 / 1921    4810 /  4435 /  3695   10070 /  9147 /  7614
//   50,000      2408 / 5300 / 4324    9490 / 10531 /  8213   25180 / 22002 / 17157
constexpr int EXT_SMALL_WIDE_PER_SM = 45;
constexpr int EXT_SMALL_LEFT8_PER_SM = 60;
constexpr int EXT_DIRECT_JOBS_PER_SM = 24;
// The band kernel (ext_band.cuh) with 8, 16 or 32 lanes a job over X's jobs that band_takes admits,
// when [start, stop) holds count_lo or more and fewer than count_hi; counter: a zeroed device word.
cudaError_t ext_band_launch(const ExtLongLaunch &X, int lanes, uint32_t *counter, uint32_t count_lo, uint32_t count_hi,
                            int nsm);
// A warp per job of a host job array the device reads in place; every job passed ext_band_direct_ok
// (and has non-negative lengths and valid slices).
bool ext_band_direct_ok(int qlen, int tlen, int h0, int max_sc);
cudaError_t ext_band_direct_launch(const bwacuda_ext_job *hjobs, uint32_t n, int w, const ExtParams &P,
                                   bwacuda_ext_result *hout, uint32_t *err, unsigned long long *cells, cudaStream_t s);
cudaError_t ext_long_deferred_launch(const ExtLongLaunch &X, bool w32, uint32_t *work, int nsm);
// First-launch ring for bands up to w (XL_RING_MIN .. XL_RING_FIRST_MAX columns).
int ext_long_ring_for_band(int w);

// Rescue (ksw_local_fwd / ksw_align2).  mode: 0 = batched_ksw_align2,
// 1 = scalar ksw_align2, 2 = forward pass only (per-job minsc / endsc).
constexpr size_t RESCUE_NPAIR_UNKNOWN = ~(size_t)0;
struct RescueLaunch {
    size_t npair = RESCUE_NPAIR_UNKNOWN;  // jobs of the launch whose values fit a byte, where the caller knows
    size_t beside = 0;  // jobs of the launches that run side by side, this one among them (0: it runs alone)
    const uint8_t *seq;
    const bwacuda_dev_rescue_job *jobs;
    const uint32_t *order;
    const uint32_t *count_ptr;
    size_t n;
    Scoring sc;
    int mode;
    int lanes;        // 0 = bwa's rule per job, else 16 or 8
    int minsc;        // modes 0 and 1
    int qcap;         // >= padded query length + 16
    int only_wide;    // as ExtLaunch::only_wide
    int pair_cols = 0;  // 32-bit wavefront: skip the jobs the paired wavefront of this many columns took
    uint2 *scratch;   // suboptimal-tracker entries
    const uint64_t *scratch_off;  // per job entry offset into scratch
    bwacuda_rescue_result *out_aln;
    bwacuda_fwd_result *out_fwd;
    uint32_t *err;
    cudaStream_t stream;
};

// Whether a rescue job runs in the two-jobs-per-group wavefront of `cols` columns
// (rescue_wf2.cuh): every value fits a byte (qlen * max_sc <= 255, on rows past a job's target too,
// which its lane goes on computing while the other job of the pair has rows) and the padded
// query of both passes (bwa's width rule, or lanes_fixed; the reverse pass may pad to 16) fits
// min(cols, 256) columns; the target has fewer than 2^20 rows (the kernel's row field).
__host__ __device__ inline bool rescue_pair_job_ok(int qlen, int tlen, int max_sc, int lanes_fixed, int cols)
{
    if (qlen < 0 || tlen < 0 || tlen >= (1 << 20) || max_sc < 1 || cols <= 0) return false;
    if ((long long)qlen * max_sc > 255) return false;
    const int ln = lanes_fixed ? lanes_fixed : ((long long)qlen * max_sc < 250 ? 16 : 8);
    const int p1 = (qlen + ln - 1) / ln * ln, p16 = (qlen + 15) / 16 * 16;
    const int need = p1 > p16 ? p1 : p16;
    return need <= (cols < 256 ? cols : 256);
}

cudaError_t rescue_tpj_launch(const RescueLaunch &L, bool wide);
cudaError_t rescue_wf_launch(const RescueLaunch &L, int qcap, int lanes);  // lanes per job: 8, 16 or 32
// The paired wavefront (two jobs per group of 4, 8 or 16 lanes) over the jobs rescue_pair_job_ok
// admits at its column count; *cols receives that count (0: no launch, the matrix or the
// queries do not suit it).
cudaError_t rescue_wf2_launch(const RescueLaunch &L, int qcap, int lanes, int *cols);
int rescue_wf_max_qpad();
size_t rescue_tpj_smem_limit_qcap(bool wide);
// Entries the suboptimal tracker may need for a target of tlen rows.
__host__ __device__ inline uint64_t rescue_scratch_entries(int tlen) { return (uint64_t)(tlen / 2 + 2); }
cudaError_t rescue_scratch_offsets(const bwacuda_dev_rescue_job *jobs, size_t n, uint64_t *off,
                                   void *tmp, size_t tmp_bytes, size_t *tmp_needed,
                                   cudaStream_t s);

}  // namespace bwacuda
