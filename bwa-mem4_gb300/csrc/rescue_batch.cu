// rescue_batch.cu -- rescue batches on the device: the survey that sizes a batch's launches, the
// launches by query-length class for ragged batches, and the host-buffer route whose jobs the
// device gathers itself.
//
// Ragged batches.  A register wavefront's columns are fixed at compile time, so a launch sized by
// its longest query computes the others' missing columns too, and a warp (16 jobs in 4-lane
// groups) steps to its longest target.  The survey adds up, over the batch, the columns and rows
// each job needs; where the unsorted launch would compute an eighth more than that, the jobs are
// radix-sorted by (column class, target length descending) and every class is launched with its
// own column count, the classes side by side on three more streams so that one class's last
// blocks run beside the next class's.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <new>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "kernels.h"
#include "runtime.h"

namespace bwacuda {

namespace {

constexpr int RC_CLASSES = 8;  // padded queries of up to 32, 64, 96, 128, 160, 192, 256 columns, and the longer ones
constexpr int RC_TLEN_MAX = 8191;

__host__ __device__ inline int rescue_class(int qlen)
{
    const int p = (qlen + 15) / 16 * 16;
    return p <= 192 ? (p <= 32 ? 0 : (p + 31) / 32 - 1) : (p <= 256 ? 6 : 7);
}

// Columns of a class (class 7: the batch's longest padded query).
__host__ __device__ inline int rescue_class_cols(int cls, int qmax)
{
    return cls < 6 ? 32 * (cls + 1) : (cls == 6 ? 256 : (qmax + 15) / 16 * 16);
}

// What the survey leaves in device memory (zeroed before it).
struct RescueStat {
    int32_t qmax, tmax;
    uint32_t bad;       // an invalid job (the host route: also a null slice with a length)
    uint32_t nwide;     // jobs whose values need 32-bit cells
    uint32_t not_u8, not_i16;  // some job leaves the reference's 8- / 16-bit batch width
    uint32_t hist[RC_CLASSES];
    uint32_t pairs[RC_CLASSES];  // those of a class whose values fit a byte
    unsigned long long useful;  // sum over jobs of class columns x target rows
    unsigned long long cells;   // sum of qlen x tlen
};

struct SurveyAcc {
    int qmax = 0, tmax = 0;
    uint32_t bad = 0, nwide = 0, not_u8 = 0, not_i16 = 0;
    unsigned long long useful = 0, cells = 0;
    __device__ __forceinline__ void job(int qlen, int tlen, int max_sc, uint32_t *hist_s)
    {
        qmax = max(qmax, qlen);
        tmax = max(tmax, tlen);
        const int cls = rescue_class(qlen);
        atomicAdd(hist_s + cls, 1u);
        if ((long long)qlen * max_sc <= 255) atomicAdd(hist_s + RC_CLASSES + cls, 1u);
        useful += (unsigned long long)rescue_class_cols(cls < 7 ? cls : 7, qlen) * (unsigned)tlen;
        cells += (unsigned long long)(unsigned)qlen * (unsigned)tlen;
        const long long top = (long long)min(qlen, tlen) * max_sc;
        nwide += !(top < 32768 && qlen + 32 < 65536);
        not_u8 |= !(top < 250 && qlen < 250);
        not_i16 |= !(top < 30000 && tlen < 30000);
    }
    // every thread of the block, once
    __device__ __forceinline__ void flush(RescueStat *st, const uint32_t *hist_s)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            useful += __shfl_xor_sync(0xffffffffu, useful, o);
            cells += __shfl_xor_sync(0xffffffffu, cells, o);
        }
        qmax = __reduce_max_sync(0xffffffffu, qmax);
        tmax = __reduce_max_sync(0xffffffffu, tmax);
        bad = __reduce_or_sync(0xffffffffu, bad);
        nwide = __reduce_add_sync(0xffffffffu, nwide);
        not_u8 = __reduce_or_sync(0xffffffffu, not_u8);
        not_i16 = __reduce_or_sync(0xffffffffu, not_i16);
        if ((threadIdx.x & 31) == 0) {
            atomicMax(&st->qmax, qmax);
            atomicMax(&st->tmax, tmax);
            if (bad) atomicOr(&st->bad, 1u);
            if (nwide) atomicAdd(&st->nwide, nwide);
            if (not_u8) atomicOr(&st->not_u8, 1u);
            if (not_i16) atomicOr(&st->not_i16, 1u);
            if (useful) atomicAdd(&st->useful, useful);
            if (cells) atomicAdd(&st->cells, cells);
        }
        __syncthreads();  // every thread's counts are in hist_s
        if (threadIdx.x < RC_CLASSES && hist_s[threadIdx.x]) {
            atomicAdd(st->hist + threadIdx.x, hist_s[threadIdx.x]);
            const uint32_t p = hist_s[RC_CLASSES + threadIdx.x];
            if (p) atomicAdd(st->pairs + threadIdx.x, p);
        }
    }
};

__device__ __forceinline__ uint16_t rescue_sort_key(int qlen, int tlen)
{
    const int t = tlen < RC_TLEN_MAX ? tlen : RC_TLEN_MAX;
    return (uint16_t)((rescue_class(qlen) << 13) | (RC_TLEN_MAX - t));
}

// Survey of device-resident jobs.
__global__ void rescue_survey_kernel(const bwacuda_dev_rescue_job *__restrict__ jobs, uint32_t n, int max_sc,
                                     RescueStat *__restrict__ st)
{
    __shared__ uint32_t hist_s[2 * RC_CLASSES];  // jobs of a class, and those whose values fit a byte
    if (threadIdx.x < 2 * RC_CLASSES) hist_s[threadIdx.x] = 0u;
    __syncthreads();
    SurveyAcc a;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int qlen = jobs[k].qlen, tlen = jobs[k].tlen;
        if (qlen < 0 || tlen < 0) a.bad = 1u;
        else a.job(qlen, tlen, max_sc, hist_s);
    }
    a.flush(st, hist_s);
}

__global__ void rescue_keys_kernel(const bwacuda_dev_rescue_job *__restrict__ jobs, uint32_t n,
                                   uint16_t *__restrict__ keys, uint32_t *__restrict__ idx)
{
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        keys[k] = rescue_sort_key(jobs[k].qlen, jobs[k].tlen);
        idx[k] = k;
    }
}

}  // namespace

// Work buffers of one launch sequence: [0] device-resident calls, [1], [2] the host route's chunks.
struct RescueWork {
    DevBuf stat, keys, idx, tmp;
    HostBuf h_stat;
};

struct RescueState {
    static constexpr int NSIDE = 3;
    cudaStream_t side[NSIDE] = {};
    cudaEvent_t fork = nullptr, join[NSIDE] = {}, last = nullptr;
    RescueWork work[3];
};

static int rescue_init(bwacuda_ctx *c)
{
    if (c->rescue) return BWACUDA_OK;
    RescueState *R = new (std::nothrow) RescueState();
    if (!R) return BWACUDA_ENOMEM;
    c->rescue = R;
    cudaError_t e = cudaEventCreateWithFlags(&R->fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&R->last, cudaEventDisableTiming);
    for (int x = 0; x < RescueState::NSIDE && e == cudaSuccess; ++x) {
        e = cudaStreamCreateWithFlags(&R->side[x], cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&R->join[x], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) {
        rescue_release(c);
        return cuda_status(e);
    }
    return BWACUDA_OK;
}

void rescue_release(bwacuda_ctx *c)
{
    RescueState *R = c->rescue;
    if (!R) return;
    for (int x = 0; x < RescueState::NSIDE; ++x) {
        if (R->side[x]) {
            cudaStreamSynchronize(R->side[x]);
            cudaStreamDestroy(R->side[x]);
        }
        if (R->join[x]) cudaEventDestroy(R->join[x]);
    }
    if (R->fork) cudaEventDestroy(R->fork);
    if (R->last) cudaEventDestroy(R->last);
    for (auto &w : R->work) {
        w.stat.release(); w.keys.release(); w.idx.release(); w.tmp.release(); w.h_stat.release();
    }
    delete R;
    c->rescue = nullptr;
}

namespace {

// The narrow launches of L's jobs (0 .. L.n-1, L.qcap from the survey): one launch, or one per
// column class over the sorted jobs.
cudaError_t rescue_launch_classes(bwacuda_ctx *c, RescueWork &W, const RescueStat &st, RescueLaunch L)
{
    // an unsorted launch computes the widest class's columns and the longest target for every job
    int top = RC_CLASSES - 1;
    while (top > 0 && st.hist[top] == 0) --top;
    const double all = (double)L.n * rescue_class_cols(top, st.qmax) * st.tmax;
    // below a warp of jobs per SM the launches' latency decides, not the padded work
    const bool sort = L.only_wide != 2 && c->rescue_kernel == BWACUDA_RESCUE_AUTO && L.n >= (size_t)c->nsm * 8 &&
                      all > 1.125 * (double)st.useful;
    if (!sort) {
        L.npair = 0;
        for (int b = 0; b < RC_CLASSES; ++b) L.npair += st.pairs[b];
        c->stats.kernel_launches += 1;
        return rescue_narrow_launch(c, L);
    }
    RescueState &R = *c->rescue;
    const uint32_t n = (uint32_t)L.n;
    size_t tb = 0;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, tb, (const uint16_t *)nullptr, (uint16_t *)nullptr,
                                                    (const uint32_t *)nullptr, (uint32_t *)nullptr, (int)n, 0, 16);
    const size_t n1 = ((size_t)n + 63) & ~(size_t)63;
    if (e == cudaSuccess) e = W.keys.ensure(n1 * 2 * 2);
    if (e == cudaSuccess) e = W.idx.ensure(n1 * 4 * 2);
    if (e == cudaSuccess) e = W.tmp.ensure(tb + 64);
    if (e != cudaSuccess) return e;
    uint16_t *k0 = static_cast<uint16_t *>(W.keys.p), *k1 = k0 + n1;
    uint32_t *i0 = static_cast<uint32_t *>(W.idx.p), *i1 = i0 + n1;
    cudaStream_t s = L.stream;
    const uint32_t grid = (uint32_t)std::min<size_t>((n + 255) / 256, (size_t)c->nsm * 8);
    rescue_keys_kernel<<<grid, 256, 0, s>>>(L.jobs, n, k0, i0);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cub::DeviceRadixSort::SortPairs(W.tmp.p, tb, k0, k1, i0, i1, (int)n, 0, 16, s)) != cudaSuccess) return e;
    if ((e = cudaEventRecord(R.fork, s)) != cudaSuccess) return e;
    for (int x = 0; x < RescueState::NSIDE; ++x)
        if ((e = cudaStreamWaitEvent(R.side[x], R.fork, 0)) != cudaSuccess) return e;
    // widest class first; the first on the caller's stream
    uint32_t at[RC_CLASSES + 1];
    at[0] = 0;
    for (int b = 0; b < RC_CLASSES; ++b) at[b + 1] = at[b] + st.hist[b];
    int nl = 0;
    for (int b = RC_CLASSES - 1; b >= 0 && e == cudaSuccess; --b) {
        if (!st.hist[b]) continue;
        RescueLaunch X = L;
        X.order = i1 + at[b];
        X.n = st.hist[b];
        X.npair = st.pairs[b];
        X.beside = n;
        X.qcap = std::min(L.qcap, rescue_class_cols(b, st.qmax) + 16);
        X.stream = nl % (RescueState::NSIDE + 1) ? R.side[nl % (RescueState::NSIDE + 1) - 1] : s;
        e = rescue_narrow_launch(c, X);
        ++nl;
    }
    c->stats.kernel_launches += 2 + (uint64_t)nl;
    for (int x = 0; x < RescueState::NSIDE; ++x) {  // joined on errors too: nothing runs on unseen
        cudaError_t ej = cudaEventRecord(R.join[x], R.side[x]);
        if (ej == cudaSuccess) ej = cudaStreamWaitEvent(s, R.join[x], 0);
        if (e == cudaSuccess) e = ej;
    }
    return e;
}

}  // namespace

// One piece of a device-resident rescue call (n <= the context's piece size): survey, tracker
// offsets, launches.
int rescue_device_piece(bwacuda_ctx *c, const uint8_t *d_seq, const bwacuda_dev_rescue_job *d_jobs, size_t n,
                        const Scoring &sc, int minsc, int mode, int lanes, bwacuda_rescue_result *d_out,
                        cudaStream_t s)
{
    int rc = rescue_init(c);
    if (rc) return rc;
    RescueState &R = *c->rescue;
    RescueWork &W = R.work[0];
    cudaError_t e;
    // the work buffers are the context's: a call on another stream waits for the last one's kernels
    if ((e = cudaStreamWaitEvent(s, R.last, 0)) != cudaSuccess) return cuda_status(e);
    if ((e = W.stat.ensure(sizeof(RescueStat))) != cudaSuccess) return cuda_status(e);
    if ((e = W.h_stat.ensure(sizeof(RescueStat) + 64)) != cudaSuccess) return cuda_status(e);
    RescueStat *d_st = static_cast<RescueStat *>(W.stat.p);
    size_t tmp_need = 0;
    rescue_scratch_offsets(d_jobs, n, nullptr, nullptr, 0, &tmp_need, s);
    if ((e = c->d_dev_aux.ensure(n * 8 + tmp_need + 64)) != cudaSuccess) return cuda_status(e);
    uint64_t *off = static_cast<uint64_t *>(c->d_dev_aux.p);
    void *tmp = static_cast<char *>(c->d_dev_aux.p) + n * 8;
    if ((e = cudaMemsetAsync(d_st, 0, sizeof(RescueStat), s)) != cudaSuccess) return cuda_status(e);
    rescue_survey_kernel<<<(uint32_t)std::min<size_t>((n + 255) / 256, (size_t)c->nsm * 4), 256, 0, s>>>(
        d_jobs, (uint32_t)n, sc.max_sc, d_st);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
    // tracker scratch: exclusive scan of per-job capacities, total read back to size the pool
    if ((e = rescue_scratch_offsets(d_jobs, n, off, tmp, tmp_need, nullptr, s)) != cudaSuccess) return cuda_status(e);
    char *h = static_cast<char *>(W.h_stat.p);
    RescueStat st;
    // total = off[n-1] + cap(n-1): read the last job's offset and tlen
    uint64_t *h_off = reinterpret_cast<uint64_t *>(h + sizeof(RescueStat));
    bwacuda_dev_rescue_job *h_job = reinterpret_cast<bwacuda_dev_rescue_job *>(h_off + 1);
    if ((e = cudaMemcpyAsync(h, d_st, sizeof(RescueStat), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return cuda_status(e);
    if ((e = cudaMemcpyAsync(h_off, off + n - 1, 8, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return cuda_status(e);
    if ((e = cudaMemcpyAsync(h_job, d_jobs + n - 1, sizeof(*h_job), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return cuda_status(e);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_status(e);
    memcpy(&st, h, sizeof(st));
    if (st.bad) return BWACUDA_EINVAL;  // a negative length would size the tracker scratch wrongly
    const int qcap = (st.qmax + 15) / 16 * 16 + 16;
    if ((size_t)qcap > rescue_tpj_smem_limit_qcap(false)) return BWACUDA_EUNSUPPORTED;
    const uint64_t total = *h_off + rescue_scratch_entries(h_job->tlen);
    if ((e = c->d_dev_scratch.ensure(total * sizeof(uint2) + 16)) != cudaSuccess) return cuda_status(e);
    RescueLaunch L;
    L.seq = d_seq;
    L.jobs = d_jobs;
    L.order = nullptr;
    L.count_ptr = nullptr;
    L.n = n;
    L.sc = sc;
    L.mode = mode;
    L.lanes = lanes;
    L.minsc = minsc;
    L.qcap = qcap;
    const bool wide_fits = (size_t)qcap <= rescue_tpj_smem_limit_qcap(true);
    L.only_wide = wide_fits ? 0 : 2;
    L.scratch = static_cast<uint2 *>(c->d_dev_scratch.p);
    L.scratch_off = off;
    L.out_aln = d_out;
    L.out_fwd = nullptr;
    L.err = reinterpret_cast<uint32_t *>(c->d_misc.p);
    L.stream = s;
    e = rescue_launch_classes(c, W, st, L);
    if (e == cudaSuccess && wide_fits && st.nwide) {
        L.only_wide = 1;
        e = rescue_tpj_launch(L, true);
        c->stats.kernel_launches += 1;
    }
    const cudaError_t er = cudaEventRecord(R.last, s);
    if (e == cudaSuccess) e = er;
    if (e != cudaSuccess) return cuda_status(e);
    c->stats.kernel_launches += 4;
    c->stats.rescue_jobs += n;
    c->dev_pending_stream = s;
    return BWACUDA_OK;
}

// ---------------------------------------------------------------- host buffers, gathered by the device

namespace {

constexpr int RG_THREADS = 128;
// Jobs per chunk of the host route: while a chunk's kernels run, the next one is planned and
// gathered on the other slot's stream.
constexpr size_t RG_CHUNK = size_t(1) << 17;

__device__ __forceinline__ void rescue_limits(const bwacuda_rescue_job &, bwacuda_dev_rescue_job &D)
{
    D.minsc = 0;
    D.endsc = 0;
}
__device__ __forceinline__ void rescue_limits(const bwacuda_fwd_job &J, bwacuda_dev_rescue_job &D)
{
    D.minsc = J.minsc;
    D.endsc = J.endsc;
}

// The only read of the caller's job array: every job is validated and surveyed, its reserve in the
// sequence buffer and its tracker entries sized, and its fields left in its device descriptor (the
// slice addresses in q_off / t_off; an invalid job empty).
template <typename JobT>
__global__ void __launch_bounds__(RG_THREADS) rescue_plan_kernel(const JobT *__restrict__ hjobs, uint32_t n, int max_sc,
                                                                 uint64_t *__restrict__ sizes,
                                                                 uint64_t *__restrict__ entries,
                                                                 bwacuda_dev_rescue_job *__restrict__ djobs,
                                                                 RescueStat *__restrict__ st)
{
    __shared__ uint32_t hist_s[2 * RC_CLASSES];  // jobs of a class, and those whose values fit a byte
    if (threadIdx.x < 2 * RC_CLASSES) hist_s[threadIdx.x] = 0u;
    __syncthreads();
    SurveyAcc a;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const JobT J = hjobs[k];
        const bool ok = J.qlen >= 0 && J.tlen >= 0 && (J.qlen == 0 || J.query != nullptr) &&
                        (J.tlen == 0 || J.target != nullptr) && J.qlen <= 65000;
        bwacuda_dev_rescue_job D;
        D.q_off = reinterpret_cast<uint64_t>(J.query);
        D.t_off = reinterpret_cast<uint64_t>(J.target);
        D.qlen = ok ? J.qlen : 0;
        D.tlen = ok ? J.tlen : 0;
        rescue_limits(J, D);
        djobs[k] = D;
        sizes[k] = ok ? 16ull * (slice_words(J.query, J.qlen) + slice_words(J.target, J.tlen)) : 0u;
        entries[k] = rescue_scratch_entries(D.tlen);
        if (ok) a.job(J.qlen, J.tlen, max_sc, hist_s);
        else a.bad = 1u;
    }
    a.flush(st, hist_s);
}

// A warp completes 32 jobs' descriptors and copies their slices (warp_gather_slices).
__global__ void __launch_bounds__(RG_THREADS) rescue_gather_kernel(uint32_t n, const uint64_t *__restrict__ offs,
                                                                   uint8_t *__restrict__ seq,
                                                                   bwacuda_dev_rescue_job *__restrict__ djobs)
{
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32u; k0 < n; k0 += gridDim.x * blockDim.x) {
        const uint32_t k = k0 + lane;
        uint64_t qa = 0, ta = 0, base = 0;
        uint32_t qw = 0, tw = 0;
        if (k < n) {
            bwacuda_dev_rescue_job D = djobs[k];
            base = offs[k];
            qa = D.q_off;
            ta = D.t_off;
            qw = slice_words(reinterpret_cast<const uint8_t *>(qa), D.qlen);
            tw = slice_words(reinterpret_cast<const uint8_t *>(ta), D.tlen);
            D.q_off = base + (qa & 15);
            D.t_off = base + 16ull * qw + (ta & 15);
            djobs[k] = D;
        }
        warp_gather_slices(qa & ~15ull, ta & ~15ull, base, qw, tw, seq);
    }
}

__global__ void __launch_bounds__(256) rescue_scatter_kernel(const uint32_t *__restrict__ src, size_t words,
                                                             uint32_t *__restrict__ dst)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < words; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

// One chunk on its slot's stream, up to the results in the caller's array.
template <typename JobT>
int rescue_host_chunk(bwacuda_ctx *c, int slot_i, const JobT *hj, size_t cn, const Scoring &sc, int minsc, int mode,
                      int lanes, void *out, RescueStat *total)
{
    Slot &sl = c->slot[slot_i];
    RescueWork &W = c->rescue->work[1 + slot_i];
    cudaStream_t s = sl.stream;
    cudaError_t e;
    const uint32_t n = (uint32_t)cn;
    const size_t osz = mode == 2 ? sizeof(bwacuda_fwd_result) : sizeof(bwacuda_rescue_result);
    size_t tb = 0;
    if ((e = cub::DeviceScan::ExclusiveSum(nullptr, tb, (const uint64_t *)nullptr, (uint64_t *)nullptr, (int)cn + 1)) !=
        cudaSuccess)
        return cuda_status(e);
    const size_t n1 = cn + 1;
    if ((e = W.stat.ensure(sizeof(RescueStat))) != cudaSuccess) return cuda_status(e);
    if ((e = W.h_stat.ensure(sizeof(RescueStat) + 64)) != cudaSuccess) return cuda_status(e);
    if ((e = sl.d_aux.ensure(n1 * 8 * 4 + tb + 64)) != cudaSuccess) return cuda_status(e);
    if ((e = sl.d_jobs.ensure(cn * sizeof(bwacuda_dev_rescue_job))) != cudaSuccess) return cuda_status(e);
    if ((e = sl.d_out.ensure(cn * osz)) != cudaSuccess) return cuda_status(e);
    RescueStat *d_st = static_cast<RescueStat *>(W.stat.p);
    uint64_t *sizes = static_cast<uint64_t *>(sl.d_aux.p), *entries = sizes + n1, *offs = entries + n1, *soff = offs + n1;
    void *tmp = soff + n1;
    bwacuda_dev_rescue_job *dj = static_cast<bwacuda_dev_rescue_job *>(sl.d_jobs.p);
    if ((e = cudaMemsetAsync(d_st, 0, sizeof(RescueStat), s)) != cudaSuccess) return cuda_status(e);
    if ((e = cudaMemsetAsync(sizes + cn, 0, 8, s)) != cudaSuccess) return cuda_status(e);
    if ((e = cudaMemsetAsync(entries + cn, 0, 8, s)) != cudaSuccess) return cuda_status(e);
    const uint32_t grid = (uint32_t)std::min<size_t>((cn + RG_THREADS - 1) / RG_THREADS, (size_t)c->nsm * 16);
    rescue_plan_kernel<JobT><<<grid, RG_THREADS, 0, s>>>(hj, n, sc.max_sc, sizes, entries, dj, d_st);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
    if ((e = cub::DeviceScan::ExclusiveSum(tmp, tb, sizes, offs, (int)cn + 1, s)) != cudaSuccess) return cuda_status(e);
    if ((e = cub::DeviceScan::ExclusiveSum(tmp, tb, entries, soff, (int)cn + 1, s)) != cudaSuccess) return cuda_status(e);
    char *h = static_cast<char *>(W.h_stat.p);
    uint64_t *h_tot = reinterpret_cast<uint64_t *>(h + sizeof(RescueStat));
    if ((e = cudaMemcpyAsync(h, d_st, sizeof(RescueStat), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return cuda_status(e);
    if ((e = cudaMemcpyAsync(h_tot, offs + cn, 8, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return cuda_status(e);
    if ((e = cudaMemcpyAsync(h_tot + 1, soff + cn, 8, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return cuda_status(e);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_status(e);
    RescueStat st;
    memcpy(&st, h, sizeof(st));
    if (st.bad) return BWACUDA_EINVAL;
    const int qcap = (st.qmax + 15) / 16 * 16 + 16;
    if ((size_t)qcap > rescue_tpj_smem_limit_qcap(st.nwide > 0)) return BWACUDA_EUNSUPPORTED;
    if ((e = sl.d_seq.ensure(h_tot[0] + 16)) != cudaSuccess) return cuda_status(e);
    if ((e = sl.d_scratch.ensure(h_tot[1] * sizeof(uint2) + 16)) != cudaSuccess) return cuda_status(e);
    rescue_gather_kernel<<<grid, RG_THREADS, 0, s>>>(n, offs, static_cast<uint8_t *>(sl.d_seq.p), dj);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
    RescueLaunch L;
    L.seq = static_cast<const uint8_t *>(sl.d_seq.p);
    L.jobs = dj;
    L.order = nullptr;
    L.count_ptr = nullptr;
    L.n = cn;
    L.sc = sc;
    L.mode = mode;
    L.lanes = lanes;
    L.minsc = minsc;
    L.qcap = qcap;
    L.only_wide = 0;
    L.scratch = static_cast<uint2 *>(sl.d_scratch.p);
    L.scratch_off = soff;
    L.out_aln = mode == 2 ? nullptr : static_cast<bwacuda_rescue_result *>(sl.d_out.p);
    L.out_fwd = mode == 2 ? static_cast<bwacuda_fwd_result *>(sl.d_out.p) : nullptr;
    L.err = reinterpret_cast<uint32_t *>(c->d_misc.p);
    L.stream = s;
    if ((e = rescue_launch_classes(c, W, st, L)) != cudaSuccess) return cuda_status(e);
    if (st.nwide) {
        L.only_wide = 1;
        if ((e = rescue_tpj_launch(L, true)) != cudaSuccess) return cuda_status(e);
        c->stats.kernel_launches += 1;
    }
    const size_t words = cn * (osz / 4);
    rescue_scatter_kernel<<<(uint32_t)std::min<size_t>((words + 255) / 256, (size_t)c->nsm * 8), 256, 0, s>>>(
        static_cast<const uint32_t *>(sl.d_out.p), words, static_cast<uint32_t *>(out));
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
    c->stats.kernel_launches += 5;
    total->not_u8 |= st.not_u8;
    total->not_i16 |= st.not_i16;
    total->cells += st.cells;
    return cuda_status(cudaEventRecord(sl.done, s));
}

template <typename JobT>
int rescue_batch_gather_t(bwacuda_ctx *c, const JobT *jobs, size_t n, const Scoring &sc, int minsc, int mode, int lanes,
                          void *out, bool *u8ok, bool *i16ok, uint64_t *cells)
{
    if (!c->pageable_access) return BWACUDA_EUNSUPPORTED;
    int rc = rescue_init(c);
    if (rc) return rc;
    const size_t osz = mode == 2 ? sizeof(bwacuda_fwd_result) : sizeof(bwacuda_rescue_result);
    const size_t CH = std::min(c->chunk_jobs, RG_CHUNK);
    RescueStat total{};
    bool busy[2] = {false, false};
    for (size_t c0 = 0, k = 0; c0 < n && rc == BWACUDA_OK; c0 += CH, ++k) {
        const int si = (int)(k & 1);
        if (busy[si]) {  // the slot's buffers are free once its last chunk's results are stored
            const cudaError_t e = cudaEventSynchronize(c->slot[si].done);
            if (e != cudaSuccess) { rc = cuda_status(e); break; }
        }
        const size_t cn = std::min(CH, n - c0);
        rc = rescue_host_chunk<JobT>(c, si, jobs + c0, cn, sc, minsc, mode, lanes, static_cast<char *>(out) + c0 * osz,
                                     &total);
        busy[si] = true;
    }
    for (int si = 0; si < 2; ++si) {  // errors included: nothing is left running
        const cudaError_t e = cudaStreamSynchronize(c->slot[si].stream);
        if (!rc) rc = cuda_status(e);
    }
    *u8ok = !total.not_u8;
    *i16ok = !total.not_i16;
    *cells = total.cells;
    return rc;
}

}  // namespace

int rescue_batch_gather(bwacuda_ctx *c, const bwacuda_rescue_job *jobs, size_t n, const Scoring &sc, int minsc, int mode,
                        int lanes, void *out, bool *u8ok, bool *i16ok, uint64_t *cells)
{
    return rescue_batch_gather_t(c, jobs, n, sc, minsc, mode, lanes, out, u8ok, i16ok, cells);
}
int rescue_batch_gather(bwacuda_ctx *c, const bwacuda_fwd_job *jobs, size_t n, const Scoring &sc, int minsc, int mode,
                        int lanes, void *out, bool *u8ok, bool *i16ok, uint64_t *cells)
{
    return rescue_batch_gather_t(c, jobs, n, sc, minsc, mode, lanes, out, u8ok, i16ok, cells);
}

}  // namespace bwacuda
