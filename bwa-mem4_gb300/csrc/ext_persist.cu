// ext_persist.cu -- the batched extension path: jobs are length-sorted on the
// device, cut into buckets by query length and cell width, and each bucket is
// run by a persistent kernel sized to fill the GPU at that bucket's shared
// memory footprint.  Warps pull 32 consecutive sorted jobs at a time from the
// bucket's work counter, so the jobs that share a warp have near-equal row
// counts and window widths (the SIMT analogue of the reference's length-sorted
// lane groups, crates/bwa-neon/src/matesw.rs:176-183).  Bucket kernels go out
// on several streams so one bucket's tail overlaps the next bucket's start.
// The whole sequence (keys, sort, bucket bounds, launches) depends only on
// device data, so it can be captured once into a CUDA graph and replayed.
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>

#include "common.cuh"
#include "ext_job.cuh"
#include "ext_long.cuh"
#include "kernels.h"
#include "persist.h"

namespace bwacuda {

namespace {

constexpr int EXT_KEY_BITS = 22;

// Cell class of a job: 0 = 8-bit pairs, 1 = 16-bit, 2 = 32-bit cells.
__device__ __forceinline__ uint32_t ext_cell_class(const bwacuda_dev_ext_job &J, int max_sc)
{
    if (ext_fits_u8(J.qlen, J.tlen, J.h0, max_sc)) return 0u;
    return ext_fits_i16(J.qlen, J.tlen, J.h0, max_sc) ? 1u : 2u;
}

// What sets the classes of a sorted small batch: the band of a job (on: such a batch).
struct SmallRule {
    int on, end_bonus, o_ins, e_ins, o_del, e_del;
};

// Class of a job in a small batch: 0 = the band kernel's, 1 = the other 16-bit ones, 2 = 32-bit.
__device__ __forceinline__ uint32_t ext_small_class(const bwacuda_dev_ext_job &J, int max_sc, const SmallRule &r)
{
    if (J.qlen < 0) return 1u;  // the group-per-job kernel flags it
    if (!ext_fits_i16(J.qlen, J.tlen, J.h0, max_sc)) return 2u;
    const int w = clamp_band(J.w < 0 ? 0 : J.w, J.qlen, max_sc, r.end_bonus, r.o_ins, r.e_ins, r.o_del, r.e_del);
    return xl::band_takes(J.qlen, w) ? 0u : 1u;
}

// Sort key of EXT_KEY_BITS: class, query length descending (clamped at 1023),
// target length descending in 32-row steps, seed score descending in steps of 4; the queries of 1023
// bases or more, whose rows the open-ended buckets' kernels run longest first with the jobs of a warp
// in step, by target length alone (32-row steps up to 32,736 rows; 20,000 jobs of 2-10 kb: 23.2 ms in
// 1024-row steps, whose warps held jobs of unequal length, 21.9 in these).  The
// seed score sets how far a row's live cells reach and how many rows live, so warps of equal scores
// run nearly equal windows: 4.2M read pairs 13.39 -> 12.4 ms, 1M mixed lengths 4.22 -> 3.84 ms with
// it.  Within a bucket the order sets only which jobs run together, never a result.
__device__ __forceinline__ uint32_t ext_sort_key(const bwacuda_dev_ext_job &J, uint32_t cls)
{
    const uint32_t ql = J.qlen < 0 ? 0u : (J.qlen > 1023 ? 1023u : (uint32_t)J.qlen);
    const uint32_t ts = J.tlen < 0 ? 0u : (uint32_t)J.tlen >> 5;
    if (ql == 1023u) return (cls << 20) | (1023u - (ts > 1023u ? 1023u : ts));
    const uint32_t tb = ts > 15u ? 15u : ts;
    const uint32_t hb = J.h0 < 0 ? 0u : (J.h0 > 255 ? 63u : (uint32_t)J.h0 >> 2);
    return (cls << 20) | ((1023u - ql) << 10) | ((15u - tb) << 6) | (63u - hb);
}

// ungapped_hit (crates/bwa-neon/src/batched.rs:602-697): the result of a job whose
// diagonal carries at most x mismatches, no N and no z-drop, or false ("run the DP").
__device__ bool ungapped_hit(const uint8_t *q, int qlen, const uint8_t *t, int tlen, int h0, const UngappedRule &u,
                             int zdrop, bwacuda_ext_result &r)
{
    if (qlen == 0 || h0 <= 0 || tlen < qlen || u.x < 0) return false;
    // mismatch columns; only the first 128 are representable (the reference's u128 bitmap)
    uint32_t mis[4] = {0u, 0u, 0u, 0u};
    int nmis = 0;
    for (int c = 0; c < qlen; ++c) {
        const uint32_t qb = q[c], tb = t[c];
        if (qb >= 4u || tb >= 4u) return false;
        if (qb != tb) {
            if (++nmis > u.x) return false;
            if (c >= 128) return false;
            mis[c >> 5] |= 1u << (c & 31);
        }
    }
    if (nmis == 0) {
        const int s = h0 + qlen * u.a;
        r.score = s; r.qle = qlen; r.tle = qlen; r.gtle = qlen; r.gscore = s; r.max_off = 0;
        return true;
    }
    if (qlen > 128) return false;
    int run = h0, best = h0, best_end = 0;
    for (int c = 0; c < qlen; ++c) {
        if (run == 0) continue;
        if (((mis[c >> 5] >> (c & 31)) & 1u) == 0u) run += u.a;
        else {
            run -= u.b;
            if (run < 0) run = 0;
        }
        if (run > best) { best = run; best_end = c + 1; }
        else if (zdrop > 0 && best - run > zdrop) return false;
    }
    if (run == 0) return false;
    r.score = best; r.qle = best_end; r.tle = best_end; r.gtle = qlen; r.gscore = run; r.max_off = 0;
    return true;
}

// Sort keys; with the ungapped rule on, jobs it settles get their result here
// and key class 3, which no bucket covers.
__global__ void ext_keys_kernel(const bwacuda_dev_ext_job *__restrict__ jobs, uint32_t n, int max_sc,
                                uint32_t min_cls, int n_to_16, const SmallRule small,
                                const uint8_t *__restrict__ seq, const UngappedRule ug, int zdrop,
                                bwacuda_ext_result *__restrict__ out, uint32_t *__restrict__ keys,
                                uint32_t *__restrict__ idx, uint32_t *__restrict__ kinds)
{
    uint32_t kind[3] = {0u, 0u, 0u};
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const bwacuda_dev_ext_job J = jobs[k];
        const uint32_t cls = small.on ? ext_small_class(J, max_sc, small) : max(ext_cell_class(J, max_sc), min_cls);
        uint32_t key = ext_sort_key(J, cls);
        if (small.on) ++kind[cls];
        bool settled = false;
        if (ug.enabled) {
            bwacuda_ext_result r;
            settled = ungapped_hit(seq + J.q_off, J.qlen, seq + J.t_off, J.tlen, J.h0, ug, zdrop, r);
            if (settled) {
                out[k] = r;
                key = 3u << 20;
            }
        }
        if (n_to_16 && !settled && key < (1u << 20) && J.qlen > 0) {  // an 8-bit job: any code of 4 or more?
            uint32_t any = 0u;
            for (int j = 0; j < J.qlen; j += 16) {
                uint32_t v[4];
                load16(seq + J.q_off, J.qlen, j, v);
                any |= v[0] | v[1] | v[2] | v[3];
            }
            if (any & 0xfcfcfcfcu) key |= 1u << 20;
        }
        keys[k] = key;
        idx[k] = k;
    }
    if (small.on) {
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            const uint32_t c = __reduce_add_sync(0xffffffffu, kind[x]);
            if ((threadIdx.x & 31u) == 0 && c) atomicAdd(kinds + x, c);
        }
    }
}

// Bucket b covers sorted keys [key_lo, key_hi]; writes its [start, end) and
// clears its work counter.  This kernel is the only writer of the bounds, and a lower bound over
// the n sorted keys lies in [0, n], so no persistent kernel reading them (in a stream launch or a
// graph replay, whose capture is keyed on the same n) can index past the order and job arrays.
__global__ void ext_bucket_bounds_kernel(const uint32_t *__restrict__ keys, uint32_t n,
                                         const ExtBucketDef *__restrict__ defs, int nb,
                                         uint32_t *__restrict__ table)
{
    const int b = threadIdx.x;
    if (b >= nb) return;
    const BucketKeys k = bucket_keys(defs[b]);
    table[b * 4 + 0] = lower_bound(keys, n, k.lo);
    table[b * 4 + 1] = lower_bound(keys, n, k.hi + 1);
    table[b * 4 + 2] = 0;  // work counter
    table[b * 4 + 3] = 0;  // work counter of the band kernel (open-ended buckets)
}

}  // namespace

// Query-length buckets of each cell class.  Below 257 columns the caps step by
// `step` (16, 32 or 64: the autotuner's bucket granularity); longer queries
// (16/32-bit cells only: an 8-bit job has h0 + min(qlen, tlen) * max_sc < 256)
// take fixed caps; the last bucket of a class is open-ended.
static const int kQcapLong[] = {385, 513, 769, EXT_TPJ_QLEN_MAX + 1};

static int max_qcap_of_class(int cls)
{
    if (cls == 0) return 257;  // bound < 256 forces min(qlen, tlen) < 256; longer queries meet short targets
    return (int)ext_tpj_smem_limit_qcap(cls == 2);
}

int ext_bucket_defs(ExtBucketDef *defs, int max_defs, int step, int long_qlo)
{
    if (step != 16 && step != 32 && step != 64) step = 32;
    int nb = 0;
    for (int cls = 0; cls < 3; ++cls) {
        int caps[32], nc = 0;
        for (int c = step + 1; c <= 257; c += step) caps[nc++] = c;
        const int nlong = cls == 0 ? 0 : (cls == 1 ? 4 : 3);  // 32-bit cells: up to 769 columns in one block
        for (int k = 0; k < nlong; ++k) caps[nc++] = kQcapLong[k];
        int lo = 0;
        for (int c = 0; c < nc && nb < max_defs; ++c) {
            ExtBucketDef d;
            d.cls = cls;
            d.qlo = lo;
            d.qhi = caps[c] - 1;
            d.qcap = caps[c];
            d.kernel = d.qhi >= long_qlo ? 1 : 0;  // the bucket holds queries of long_qlo or more
            defs[nb++] = d;
            lo = caps[c];
        }
        // the open-ended last class: every longer query up to the class's limit
        if (nb < max_defs) {
            ExtBucketDef d;
            d.cls = cls;
            d.qlo = lo;
            d.qhi = EXT_QHI_OPEN;
            d.qcap = cls == 0 ? (int)ext_tpj_smem_limit_qcap(false) : max_qcap_of_class(cls);
            d.kernel = 1;  // any query length
            defs[nb++] = d;
        }
    }
    return nb;
}

cudaError_t ext_sort_prefer_shared()
{
    // The bucket-bound kernel (one block, no shared memory) prefers the bucket kernels'
    // maximum shared-memory carveout.  The key kernel keeps the default: its blocks live for
    // one pass only, and with the ungapped rule it reads every job's bases through L1.
    return cudaFuncSetAttribute(ext_bucket_bounds_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                cudaSharedmemCarveoutMaxShared);
}

size_t ext_sort_temp_bytes(size_t n)
{
    size_t bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const uint32_t *)nullptr, (uint32_t *)nullptr,
                                    (const uint32_t *)nullptr, (uint32_t *)nullptr, (int)n, 0, EXT_KEY_BITS);
    return bytes;
}

cudaError_t ext_sort_jobs(const bwacuda_dev_ext_job *jobs, size_t n, int max_sc, uint32_t min_cls, bool n_to_16,
                          const uint8_t *seq, const UngappedRule &ug, int zdrop, bwacuda_ext_result *out, uint32_t *keys_in,
                          uint32_t *keys_out, uint32_t *idx_in, uint32_t *idx_out, void *tmp, size_t tmp_bytes,
                          cudaStream_t s, const ExtParams *small, uint32_t *kinds)
{
    if (n == 0) return cudaSuccess;
    SmallRule sr{};
    if (small)
        sr = SmallRule{1, small->end_bonus, small->sc.o_ins, small->sc.e_ins, small->sc.o_del, small->sc.e_del};
    uint32_t grid = (uint32_t)((n + 255) / 256);
    if (grid > 8192) grid = 8192;
    ext_keys_kernel<<<grid, 256, 0, s>>>(jobs, (uint32_t)n, max_sc, min_cls, n_to_16 ? 1 : 0, sr, seq, ug, zdrop, out,
                                         keys_in, idx_in, kinds);
    return cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, keys_in, keys_out, idx_in, idx_out, (int)n, 0, EXT_KEY_BITS, s);
}

cudaError_t ext_sort_and_bucket(const bwacuda_dev_ext_job *jobs, size_t n, int max_sc, bool pair_lanes, bool n_to_16,
                                const uint8_t *seq, const UngappedRule &ug, int zdrop, bwacuda_ext_result *out, uint32_t *keys_in,
                                uint32_t *keys_out, uint32_t *idx_in, uint32_t *idx_out, void *tmp,
                                size_t tmp_bytes, const ExtBucketDef *d_defs, int nb, uint32_t *d_table,
                                cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    const cudaError_t e = ext_sort_jobs(jobs, n, max_sc, pair_lanes ? 0u : 1u, n_to_16, seq, ug, zdrop, out, keys_in, keys_out,
                                        idx_in, idx_out, tmp, tmp_bytes, s);
    if (e != cudaSuccess) return e;
    ext_bucket_bounds_kernel<<<1, EXT_MAX_BUCKETS, 0, s>>>(keys_out, (uint32_t)n, d_defs, nb, d_table);
    return cudaGetLastError();
}

cudaError_t ext_persist_launch(const PersistLaunch &L, const ExtBucketDef &d, uint32_t *d_bucket_table, int nsm,
                               int tb)
{
    if (L.grab == 4) return ext_persist_launch_g4(L, d, d_bucket_table, nsm, tb);
    if (L.grab == 2) return ext_persist_launch_g2(L, d, d_bucket_table, nsm, tb);
    return ext_persist_launch_g1(L, d, d_bucket_table, nsm, tb);
}

}  // namespace bwacuda
