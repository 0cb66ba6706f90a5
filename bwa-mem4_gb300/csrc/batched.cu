// batched.cu -- host orchestration of the batched extension path: buffers,
// the bucket fan-out over several streams, CUDA-graph capture and replay of the
// whole device sequence, and the host-buffer pipeline that feeds it.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstring>
#include <vector>

#include "ext_job.cuh"
#include "kernels.h"
#include "persist.h"
#include "runtime.h"

namespace bwacuda {

// Bucket streams: FAN, or FAN_WIDE for calls below EXT_WIDE_JOBS_PER_SM jobs per SM.  There a bucket's
// time is its longest jobs' and it leaves most of an SM free, so the eight length classes run at once;
// above, the buckets fill the GPU one after another, and the long ones finish later when they share it
// from the start.  Device-resident, four streams / eight, microseconds, mixed lengths: 60,000 jobs
// 2010 / 1240, 120,000 1970 / 1310, 250,000 2110 / 1870, 500,000 2500 / 2770, 1M 3840 / 4340; read
// pairs: 250,000 1260 / 1120.  The others are created at their first use, and small batches, which have
// no buckets, never ask for them.  Created ones cost later calls nothing: 2M read pairs through host
// buffers 7.80 ms in a fresh context, 7.73-7.79 after calls that use eight.
constexpr int FAN = 4, FAN_WIDE = 8;
constexpr int EXT_WIDE_JOBS_PER_SM = 2200;
// Open-ended buckets: jobs per SM from which the band kernel gives a job 8 lanes, below it 32 (queries
// of 2-10 kb on 152 SMs: 1,000 jobs 9.6 / 6.5 ms, 2,400 jobs 9.8 / 9.8, 20,000 jobs 23.1 / 42.4; the 8 lanes 21.9 with the
// finer target steps of the sort key).
constexpr int BAND_LANES8_JOBS = 14;
// Two jobs a thread (ext_dual.cuh) from this many jobs per SM on, in the 8-bit buckets of up to this
// many columns (longer ones leave an SM too few of its warps).  Milliseconds on 152 SMs, one / two jobs
// a thread:        read pairs     mixed lengths    1% errors and N bases
//     131,072     0.87 / 0.92      1.89 / 2.09      0.94 / 1.45
//     524,288     2.01 / 1.79      2.46 / 2.66      2.17 / 2.29
//   1,048,576     3.43 / 3.14      4.09 / 4.00      3.96 / 3.90
//   4,194,304    12.63 / 11.26    14.95 / 13.40    14.42 / 13.90
constexpr int EXT_DUAL_JOBS_PER_SM = 5000;
constexpr int EXT_DUAL_QCAP = 129;

// Device work buffers of one in-flight batch.
struct BatchBufs {
    DevBuf keys_in, keys_out, idx_in, idx_out, tmp, table;
    DevBuf xl;  // group-per-job buckets: work words and the deferred-job list
    cudaStream_t fan[FAN_WIDE] = {};
    cudaEvent_t fork = nullptr, join[FAN_WIDE] = {};
    // graph cache for device-resident replays
    cudaGraphExec_t graph = nullptr;
    const void *g_seq = nullptr, *g_jobs = nullptr, *g_out = nullptr;
    const void *g_bufs[6] = {};  // work buffers the graph was captured with
    uint64_t g_gen = 0;          // tuning generation the graph was captured with
    size_t g_n = 0;
    cudaStream_t g_stream = nullptr;
    ExtParams g_P{};
    int nfan = 0;            // streams and join events that exist
    size_t call_jobs = 0;    // jobs of the whole call when the batch is one chunk of it
    int launched = 0;        // kernel launches of the last sequence enqueued (the sort counted as one)
    int g_launched = 0;      // of the captured one
    bool shapes = false;     // the autotuner's runs: length buckets with a job a thread whatever the batch
    int left = EXT_LEFT_16 | EXT_LEFT_32;  // what a small batch may hold besides the band kernel's jobs
    // per-SM room the bucket kernels leave for kernels running beside them
    int reserve_regs = 0, reserve_threads = 0;
    size_t jobs_cap = 0;  // jobs the work buffers are sized for (batched_enqueue, batched_reserve)
};

// Jobs to size a reused slot's work buffers for, n or more: they grow at least twofold (every
// regrowth frees a buffer, and cudaFree waits for the whole device, stalling the work of the
// other streams, e.g. the serving loop's other waves).
static size_t batched_grow_jobs(BatchBufs &bb, size_t n)
{
    if (n > bb.jobs_cap) bb.jobs_cap = std::max(n, bb.jobs_cap * 2);
    return bb.jobs_cap;
}

struct BatchedState {
    int nsm = 0;
    int sm_regs = 65536, sm_threads = 2048;
    int nb = 0;
    // tuning (set by bwacuda_autotune_extend or the options); gen changes with every setting
    int tb = 128;    // threads per block of the persistent kernels
    int grab = 1;    // 32-job rounds per work-counter grab
    int step = 32;   // query-length bucket width below 257 columns
    int long_qlo = INT_MAX;  // buckets from this query length up use the group-per-job kernel
    uint64_t gen = 1;
    ExtBucketDef defs[EXT_MAX_BUCKETS];
    DevBuf d_defs;
    BatchBufs bufs[3];  // [0], [1]: host-pipeline slots; [2]: device-resident calls
};

// The first `fan` bucket streams and their join events.
static cudaError_t fan_streams(BatchBufs &bb, int fan)
{
    for (; bb.nfan < fan; ++bb.nfan) {
        const int f = bb.nfan;
        cudaError_t e = bb.fan[f] ? cudaSuccess : cudaStreamCreateWithFlags(&bb.fan[f], cudaStreamNonBlocking);
        if (e == cudaSuccess && !bb.join[f]) e = cudaEventCreateWithFlags(&bb.join[f], cudaEventDisableTiming);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

static int batched_init(bwacuda_ctx *c)
{
    if (c->batched) return BWACUDA_OK;
    BatchedState *B = new (std::nothrow) BatchedState();
    if (!B) return BWACUDA_ENOMEM;
    cudaError_t e = cudaDeviceGetAttribute(&B->nsm, cudaDevAttrMultiProcessorCount, c->device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&B->sm_regs, cudaDevAttrMaxRegistersPerMultiprocessor, c->device);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&B->sm_threads, cudaDevAttrMaxThreadsPerMultiProcessor, c->device);
    if (e == cudaSuccess) e = ext_sort_prefer_shared();
    if (e != cudaSuccess) { delete B; return cuda_status(e); }
    B->nb = ext_bucket_defs(B->defs, EXT_MAX_BUCKETS, B->step, B->long_qlo);
    if ((e = B->d_defs.ensure(sizeof(B->defs))) != cudaSuccess) { delete B; return cuda_status(e); }
    if ((e = cudaMemcpy(B->d_defs.p, B->defs, sizeof(ExtBucketDef) * B->nb, cudaMemcpyHostToDevice)) != cudaSuccess) {
        delete B;
        return cuda_status(e);
    }
    for (auto &bb : B->bufs) {
        e = fan_streams(bb, FAN);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&bb.fork, cudaEventDisableTiming);
        if (e == cudaSuccess) e = bb.table.ensure(EXT_MAX_BUCKETS * 4 * sizeof(uint32_t));
        if (e != cudaSuccess) break;
    }
    c->batched = B;
    return cuda_status(e);
}

void batched_release(bwacuda_ctx *c)
{
    BatchedState *B = c->batched;
    if (!B) return;
    for (auto &bb : B->bufs) {
        if (bb.graph) cudaGraphExecDestroy(bb.graph);
        for (int f = 0; f < FAN_WIDE; ++f) {
            if (bb.fan[f]) cudaStreamSynchronize(bb.fan[f]);
        }
        for (int f = 0; f < FAN_WIDE; ++f) {
            if (bb.fan[f]) cudaStreamDestroy(bb.fan[f]);
            if (bb.join[f]) cudaEventDestroy(bb.join[f]);
        }
        if (bb.fork) cudaEventDestroy(bb.fork);
        bb.keys_in.release(); bb.keys_out.release(); bb.idx_in.release(); bb.idx_out.release();
        bb.tmp.release(); bb.table.release(); bb.xl.release();
    }
    B->d_defs.release();
    delete B;
    c->batched = nullptr;
}

int batched_set_block(bwacuda_ctx *c, int tb)
{
    int rc = batched_init(c);
    if (rc) return rc;
    c->batched->tb = tb;
    c->batched->gen++;
    return BWACUDA_OK;
}

int batched_set_grab(bwacuda_ctx *c, int grab)
{
    int rc = batched_init(c);
    if (rc) return rc;
    c->batched->grab = grab;
    c->batched->gen++;
    return BWACUDA_OK;
}

// New bucket boundaries; waits for in-flight batches (they read the old table).
int batched_set_bucket_step(bwacuda_ctx *c, int step)
{
    int rc = batched_init(c);
    if (rc) return rc;
    BatchedState *B = c->batched;
    if (B->step == step) return BWACUDA_OK;
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return cuda_status(e);
    B->step = step;
    B->nb = ext_bucket_defs(B->defs, EXT_MAX_BUCKETS, step, B->long_qlo);
    if ((e = cudaMemcpy(B->d_defs.p, B->defs, sizeof(ExtBucketDef) * B->nb, cudaMemcpyHostToDevice)) != cudaSuccess)
        return cuda_status(e);
    B->gen++;
    return BWACUDA_OK;
}

// Query length from which the buckets use the group-per-job kernel (INT_MAX: only the
// open-ended buckets); waits for in-flight batches like batched_set_bucket_step.
int batched_set_long(bwacuda_ctx *c, int long_qlo)
{
    int rc = batched_init(c);
    if (rc) return rc;
    BatchedState *B = c->batched;
    if (B->long_qlo == long_qlo) return BWACUDA_OK;
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return cuda_status(e);
    B->long_qlo = long_qlo;
    B->nb = ext_bucket_defs(B->defs, EXT_MAX_BUCKETS, B->step, long_qlo);
    if ((e = cudaMemcpy(B->d_defs.p, B->defs, sizeof(ExtBucketDef) * B->nb, cudaMemcpyHostToDevice)) != cudaSuccess)
        return cuda_status(e);
    B->gen++;
    return BWACUDA_OK;
}

int batched_get_long(bwacuda_ctx *c) { return c->batched ? c->batched->long_qlo : INT_MAX; }

// Lanes per job of the group-per-job kernel; a new value invalidates captured graphs.
int batched_set_long_lanes(bwacuda_ctx *c, int lanes)
{
    int rc = batched_init(c);
    if (rc) return rc;
    if (c->long_lanes != lanes) {
        c->long_lanes = lanes;
        c->batched->gen++;
    }
    return BWACUDA_OK;
}

// Band kernel on the open-ended buckets: 0 off, 1 with lanes a job by the bucket's jobs, 2 with 8; a new
// value invalidates captured graphs.
int batched_set_long_slide(bwacuda_ctx *c, int mode)
{
    int rc = batched_init(c);
    if (rc) return rc;
    if (c->long_slide != mode) {
        c->long_slide = mode;
        c->batched->gen++;
    }
    return BWACUDA_OK;
}

// Largest call that runs as a small batch; a new value invalidates captured graphs.
int batched_set_small(bwacuda_ctx *c, size_t jobs)
{
    int rc = batched_init(c);
    if (rc) return rc;
    if (c->small_jobs != jobs) {
        c->small_jobs = jobs;
        c->batched->gen++;
    }
    return BWACUDA_OK;
}

// Device-resident calls as the autotuner times them: the launch shapes it turns (threads per block, jobs
// per grab, bucket width, the group kernel's buckets) are those of the length buckets with a job a thread,
// so small batches run in buckets too and no bucket runs two jobs a thread.
void batched_set_shapes(bwacuda_ctx *c, bool on)
{
    c->batched->bufs[2].shapes = on;
    c->batched->gen++;
}

void batched_get_tuning(bwacuda_ctx *c, int *tb, int *grab, int *step)
{
    BatchedState *B = c->batched;
    *tb = B ? B->tb : 128;
    *grab = B ? B->grab : 1;
    *step = B ? B->step : 32;
}

// Bucket streams of a batch of n jobs.
static int batched_fan(const bwacuda_ctx *c, const BatchBufs &bb, size_t n, const ExtParams &P)
{
    if (batched_is_small(c, n, P) && ext_pair_lanes_ok(P.sc.o_del, P.sc.e_del, P.sc.o_ins, P.sc.e_ins)) return FAN;
    return std::max(n, bb.call_jobs) < (size_t)c->batched->nsm * EXT_WIDE_JOBS_PER_SM ? FAN_WIDE : FAN;
}

static cudaError_t ensure_bufs(BatchBufs &bb, size_t n, int fan = FAN)
{
    cudaError_t e;
    if ((e = fan_streams(bb, fan)) != cudaSuccess) return e;
    if ((e = bb.keys_in.ensure(n * 4 + 16)) != cudaSuccess) return e;
    if ((e = bb.keys_out.ensure(n * 4 + 16)) != cudaSuccess) return e;
    if ((e = bb.idx_in.ensure(n * 4 + 16)) != cudaSuccess) return e;
    if ((e = bb.idx_out.ensure(n * 4 + 16)) != cudaSuccess) return e;
    if ((e = bb.xl.ensure(((size_t)XL_WORK_WORDS + n) * 4 + 16)) != cudaSuccess) return e;
    return bb.tmp.ensure(ext_sort_temp_bytes(n) + 256);
}

// Whether a call of n jobs runs as a small batch (the ungapped rule is part of the sorted path).
bool batched_is_small(const bwacuda_ctx *c, size_t n, const ExtParams &P)
{
    return n <= c->small_jobs && !P.ug.enabled;
}

// A small batch: the band kernel over every job, and what it leaves (bb.left: 32-bit values, queries
// and bands past its window) in the group-per-job kernels or, where it is many 32-bit jobs, in their
// length buckets (EXT_SMALL_WIDE_PER_SM).  Thread-per-job buckets take 0.3-0.5 ms however few jobs they
// hold.  32 lanes a job below 8 jobs per SM, 16 below 20, else 8 (the times stand at
// EXT_SMALL_JOBS_PER_SM); with 8 the jobs are sorted first, longest first: the four jobs of a warp step to
// its longest, and 20,000 queries of 2-10 kb in caller order took 32.4 ms against 23.1.
static cudaError_t enqueue_small(bwacuda_ctx *c, BatchBufs &bb, const uint8_t *d_seq,
                                 const bwacuda_dev_ext_job *d_jobs, size_t n, const ExtParams &P,
                                 bwacuda_ext_result *d_out, cudaStream_t s, uint32_t *err, unsigned long long *cells)
{
    BatchedState *B = c->batched;
    uint32_t *work = static_cast<uint32_t *>(bb.xl.p);
    bb.launched = 1;  // the band kernel
    cudaError_t e = cudaMemsetAsync(work, 0, XL_WORK_WORDS * 4, s);
    if (e != cudaSuccess) return e;
    ExtLongLaunch X;
    X.seq = d_seq;
    X.jobs = d_jobs;
    X.order = nullptr;
    X.bounds = nullptr;
    X.njobs = (uint32_t)n;
    X.min_qlen = 0;
    X.lanes = c->long_lanes;
    X.ring_cols = XL_RING_DEFAULT;
    X.P = P;
    X.out = d_out;
    X.err = err ? err : reinterpret_cast<uint32_t *>(c->d_misc.p);
    X.cells = cells ? cells : reinterpret_cast<unsigned long long *>((char *)c->d_misc.p + 8);
    X.defer = work + XL_WORK_WORDS;
    X.defer_count = work + XL_WORK_DCOUNT;
    X.band = 1;
    X.small = 1;
    X.reserve_regs = bb.reserve_regs;
    X.reserve_threads = bb.reserve_threads;
    X.sm_regs = B->sm_regs;
    X.sm_threads = B->sm_threads;
    X.stream = s;
    const bool left8 = c->long_lanes == XL_LANES_DEFAULT && n >= (size_t)B->nsm * EXT_SMALL_LEFT8_PER_SM;
    const int lanes = n < (size_t)B->nsm * 8 ? 32 : (n < (size_t)B->nsm * 20 ? 16 : 8);
    uint32_t *keys = static_cast<uint32_t *>(bb.keys_out.p), *order = static_cast<uint32_t *>(bb.idx_out.p);
    uint32_t *kinds = work + XL_WORK_KINDS;
    if (lanes == 8) {
        if ((e = ext_sort_jobs(d_jobs, n, P.sc.max_sc, 0u, false, d_seq, P.ug, P.zdrop, d_out,
                               static_cast<uint32_t *>(bb.keys_in.p), keys, static_cast<uint32_t *>(bb.idx_in.p), order,
                               bb.tmp.p, bb.tmp.cap, s, &P, kinds)) != cudaSuccess)
            return e;
        X.order = order;
        bb.launched += 2;
    }
    if ((e = ext_band_launch(X, lanes, work + XL_WORK_BAND, 0u, UINT32_MAX, B->nsm)) != cudaSuccess) return e;
    // the group-per-job kernels: a kind of the sorted jobs, or every job in caller order
    X.bounds = X.order ? kinds : nullptr;
    if (bb.left & EXT_LEFT_16) {
        X.counter = work + XL_WORK_COUNTER16;
        X.part = X.order ? XL_PART_LEFT : XL_PART_ALL;
        X.part_min = left8 ? (uint32_t)(B->nsm * EXT_SMALL_LEFT8_PER_SM) : UINT32_MAX;
        if ((e = ext_long_launch(X, false, B->nsm)) != cudaSuccess) return e;
        bb.launched += 2;  // and the deferred launch
        if (left8) {
            ExtLongLaunch Y = X;
            Y.lanes = 8;
            Y.counter = work + XL_WORK_COUNTER_MANY;
            Y.part = XL_PART_LEFT_MANY;
            if ((e = ext_long_launch(Y, false, B->nsm)) != cudaSuccess) return e;
            ++bb.launched;
        }
    }
    if (bb.left & EXT_LEFT_32) {
        const uint32_t wide_min = (uint32_t)(B->nsm * EXT_SMALL_WIDE_PER_SM);
        if (X.order && n >= wide_min) {
            PersistLaunch L;
            L.seq = d_seq;
            L.jobs = d_jobs;
            L.order = order;
            L.P = P;
            L.out = d_out;
            L.err = X.err;
            L.cells = X.cells;
            L.grab = 1;
            L.stream = s;
            ++bb.launched;
            if ((e = ext_wide_launch(L, keys, (uint32_t)n, wide_min, static_cast<const ExtBucketDef *>(B->d_defs.p), B->nb,
                                     work, B->nsm)) != cudaSuccess)
                return e;
        }
        X.counter = work + XL_WORK_COUNTER32;
        X.part = X.order ? XL_PART_WIDE : XL_PART_ALL;
        X.part_min = wide_min;
        if ((e = ext_long_launch(X, true, B->nsm)) != cudaSuccess) return e;
        bb.launched += 2;
    }
    for (int w32 = 0; w32 < 2; ++w32)
        if ((bb.left & (w32 ? EXT_LEFT_32 : EXT_LEFT_16)) &&
            (e = ext_long_deferred_launch(X, w32 != 0, work, B->nsm)) != cudaSuccess)
            return e;
    return cudaSuccess;
}

// Enqueue the batched sequence for n device-resident jobs on stream s.
static cudaError_t enqueue_batched(bwacuda_ctx *c, BatchBufs &bb, const uint8_t *d_seq,
                                   const bwacuda_dev_ext_job *d_jobs, size_t n, const ExtParams &P,
                                   bwacuda_ext_result *d_out, cudaStream_t s, uint32_t *err = nullptr,
                                   unsigned long long *cells = nullptr)
{
    BatchedState *B = c->batched;
    const bool lanes = ext_pair_lanes_ok(P.sc.o_del, P.sc.e_del, P.sc.o_ins, P.sc.e_ins);
    if (lanes && !bb.shapes && batched_is_small(c, n, P))
        return enqueue_small(c, bb, d_seq, d_jobs, n, P, d_out, s, err, cells);
    const int fan = std::min(batched_fan(c, bb, n, P), bb.nfan);
    // two jobs a thread in the 8-bit buckets of large batches; not behind the ungapped closed form, which
    // leaves the buckets the jobs whose rows end apart, and few (4M jobs, two / one a thread: read pairs
    // with 1% errors 6.43 / 5.84 ms, mixed lengths 3.98 / 3.79; 8.4M read pairs 2.85 / 2.85)
    const bool dual = !P.ug.enabled && !bb.shapes && lanes && P.sc.m <= 5 && n >= (size_t)B->nsm * EXT_DUAL_JOBS_PER_SM;
    cudaError_t e = ext_sort_and_bucket(d_jobs, n, P.sc.max_sc, lanes, dual, d_seq, P.ug, P.zdrop, d_out,
                                        static_cast<uint32_t *>(bb.keys_in.p),
                                        static_cast<uint32_t *>(bb.keys_out.p), static_cast<uint32_t *>(bb.idx_in.p),
                                        static_cast<uint32_t *>(bb.idx_out.p), bb.tmp.p, bb.tmp.cap,
                                        static_cast<const ExtBucketDef *>(B->d_defs.p), B->nb,
                                        static_cast<uint32_t *>(bb.table.p), s);
    if (e != cudaSuccess) return e;
    bb.launched = 3;  // keys, sort, bounds
    uint32_t *work = static_cast<uint32_t *>(bb.xl.p);
    if ((e = cudaMemsetAsync(work, 0, XL_WORK_WORDS * 4, s)) != cudaSuccess) return e;
    if ((e = cudaEventRecord(bb.fork, s)) != cudaSuccess) return e;
    for (int f = 0; f < fan; ++f)
        if ((e = cudaStreamWaitEvent(bb.fan[f], bb.fork, 0)) != cudaSuccess) return e;
    // Group-per-job buckets (the open-ended ones take queries of any length) one after
    // another on the first stream, then the deferred launches over the jobs whose bands
    // needed a larger ring; empty buckets exit at once.
    ExtLongLaunch X;
    X.seq = d_seq;
    X.jobs = d_jobs;
    X.order = static_cast<const uint32_t *>(bb.idx_out.p);
    X.njobs = (uint32_t)n;
    X.min_qlen = 0;
    X.lanes = c->long_lanes;
    X.ring_cols = XL_RING_DEFAULT;
    X.P = P;
    X.out = d_out;
    X.err = err ? err : reinterpret_cast<uint32_t *>(c->d_misc.p);
    X.cells = cells ? cells : reinterpret_cast<unsigned long long *>((char *)c->d_misc.p + 8);
    X.defer = work + XL_WORK_WORDS;
    X.defer_count = work + XL_WORK_DCOUNT;
    X.reserve_regs = bb.reserve_regs;
    X.reserve_threads = bb.reserve_threads;
    X.sm_regs = B->sm_regs;
    X.sm_threads = B->sm_threads;
    X.stream = bb.fan[0];
    // the open-ended buckets of the 8- and 16-bit classes run the band kernel (bands up to
    // bwa-mem's default 100 and a column; wider ones stay with the group kernel): 8 lanes a job
    // from BAND_LANES8_JOBS jobs per SM on (BWACUDA_OPT_LONG_SLIDE 2: always), 32 below
    const bool use_band = c->long_slide && lanes;
    const uint32_t cut = c->long_slide == 2 ? 0u : (uint32_t)(B->nsm * BAND_LANES8_JOBS);
    bool long16 = false, long32 = false;
    for (int b = B->nb - 1; b >= 0; --b) {
        if (B->defs[b].kernel != 1) continue;
        uint32_t *tab = static_cast<uint32_t *>(bb.table.p) + 4 * b;
        X.bounds = tab;
        X.counter = tab + 2;
        const bool w32 = B->defs[b].cls == 2;
        X.band = use_band && !w32 && B->defs[b].qhi == EXT_QHI_OPEN;
        bb.launched += 1 + (X.band ? 1 + (cut != 0u) : 0);
        if (X.band) {  // one of the two runs the bucket, the other exits at once
            if ((e = ext_band_launch(X, 8, tab + 3, cut, UINT32_MAX, B->nsm)) != cudaSuccess) return e;
            if (cut && (e = ext_band_launch(X, 32, tab + 3, 1u, cut, B->nsm)) != cudaSuccess) return e;
        }
        if ((e = ext_long_launch(X, w32, B->nsm)) != cudaSuccess) return e;
        long16 |= !w32;
        long32 |= w32;
    }
    if (long16 && (e = ext_long_deferred_launch(X, false, work, B->nsm)) != cudaSuccess) return e;
    if (long32 && (e = ext_long_deferred_launch(X, true, work, B->nsm)) != cudaSuccess) return e;
    bb.launched += (int)long16 + (int)long32;
    PersistLaunch L;
    L.seq = d_seq;
    L.jobs = d_jobs;
    L.order = static_cast<const uint32_t *>(bb.idx_out.p);
    L.P = P;
    L.out = d_out;
    L.err = err ? err : reinterpret_cast<uint32_t *>(c->d_misc.p);
    L.cells = cells ? cells : reinterpret_cast<unsigned long long *>((char *)c->d_misc.p + 8);
    L.grab = B->grab;
    L.reserve_regs = bb.reserve_regs;
    L.reserve_threads = bb.reserve_threads;
    L.sm_regs = B->sm_regs;
    L.sm_threads = B->sm_threads;
    // thread-per-job buckets, largest first: they hold the long jobs
    for (int b = B->nb - 1, k = 1; b >= 0; --b) {
        if (B->defs[b].kernel == 1) continue;
        L.stream = bb.fan[k++ % fan];
        ++bb.launched;
        uint32_t *tab = static_cast<uint32_t *>(bb.table.p) + 4 * b;
        e = dual && B->defs[b].cls == 0 && B->defs[b].qcap <= EXT_DUAL_QCAP ? ext_dual_launch(L, B->defs[b], tab, B->nsm)
                                        : ext_persist_launch(L, B->defs[b], tab, B->nsm, B->tb);
        if (e != cudaSuccess) return e;
    }
    for (int f = 0; f < fan; ++f) {
        if ((e = cudaEventRecord(bb.join[f], bb.fan[f])) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(s, bb.join[f], 0)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

int extend_device_batched(bwacuda_ctx *c, const uint8_t *d_seq, const bwacuda_dev_ext_job *d_jobs, size_t n,
                          const ExtParams &P, bwacuda_ext_result *d_out, cudaStream_t s)
{
    int rc = batched_init(c);
    if (rc) return rc;
    BatchBufs &bb = c->batched->bufs[2];
    cudaError_t e = ensure_bufs(bb, n, batched_fan(c, bb, n, P));
    if (e != cudaSuccess) return cuda_status(e);
    // Replay a captured graph when the same batch comes back (same buffers, size,
    // scoring and stream); otherwise capture a new one.
    const void *bufs[6] = {bb.keys_in.p, bb.keys_out.p, bb.idx_in.p, bb.idx_out.p, bb.tmp.p, bb.table.p};
    const bool same = bb.graph && bb.g_seq == d_seq && bb.g_jobs == d_jobs && bb.g_out == d_out && bb.g_n == n &&
                      bb.g_stream == s && bb.g_gen == c->batched->gen && memcmp(bb.g_bufs, bufs, sizeof(bufs)) == 0 &&
                      memcmp(&bb.g_P, &P, sizeof(P)) == 0;
    if (!same && c->use_graphs) {
        if (bb.graph) {
            cudaGraphExecDestroy(bb.graph);
            bb.graph = nullptr;
        }
        cudaGraph_t g = nullptr;
        if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)) != cudaSuccess) return cuda_status(e);
        cudaError_t e2 = enqueue_batched(c, bb, d_seq, d_jobs, n, P, d_out, s);
        e = cudaStreamEndCapture(s, &g);
        if (e2 != cudaSuccess) { if (g) cudaGraphDestroy(g); return cuda_status(e2); }
        if (e != cudaSuccess) return cuda_status(e);
        e = cudaGraphInstantiate(&bb.graph, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) { bb.graph = nullptr; return cuda_status(e); }
        bb.g_seq = d_seq; bb.g_jobs = d_jobs; bb.g_out = d_out; bb.g_n = n; bb.g_stream = s; bb.g_P = P;
        bb.g_gen = c->batched->gen;
        bb.g_launched = bb.launched;
        memcpy(bb.g_bufs, bufs, sizeof(bufs));
    }
    if (c->use_graphs) {
        if ((e = cudaGraphLaunch(bb.graph, s)) != cudaSuccess) return cuda_status(e);
        bb.launched = bb.g_launched;
    } else if ((e = enqueue_batched(c, bb, d_seq, d_jobs, n, P, d_out, s)) != cudaSuccess) {
        return cuda_status(e);
    }
    c->stats.kernel_launches += (uint64_t)bb.launched;
    c->stats.ext_jobs += n;
    c->dev_pending_stream = s;
    return BWACUDA_OK;
}

int batched_prepare(bwacuda_ctx *c) { return batched_init(c); }
void batched_set_reserve(BatchBufs *bb, int regs, int threads)
{
    bb->reserve_regs = regs;
    bb->reserve_threads = threads;
}
void batched_set_call(BatchBufs *bb, size_t jobs) { bb->call_jobs = jobs; }
void batched_set_left(BatchBufs *bb, int left) { bb->left = left; }
BatchBufs *batched_slot_bufs(bwacuda_ctx *c, int slot) { return &c->batched->bufs[slot & 1]; }
int batched_nsm(bwacuda_ctx *c) { return c->batched->nsm; }
int batched_launched(const BatchBufs *bb) { return bb->launched; }

static cudaError_t bufs_streams(BatchBufs &bb)
{
    cudaError_t e = fan_streams(bb, FAN);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&bb.fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = bb.table.ensure(EXT_MAX_BUCKETS * 4 * sizeof(uint32_t));
    return e;
}

BatchBufs *batchbufs_create()
{
    BatchBufs *bb = new (std::nothrow) BatchBufs();
    if (!bb) return nullptr;
    if (bufs_streams(*bb) != cudaSuccess) {
        batchbufs_destroy(bb);
        return nullptr;
    }
    return bb;
}

void batchbufs_destroy(BatchBufs *bb)
{
    if (!bb) return;
    for (int f = 0; f < FAN_WIDE; ++f) {
        if (bb->fan[f]) cudaStreamSynchronize(bb->fan[f]);
        if (bb->fan[f]) cudaStreamDestroy(bb->fan[f]);
        if (bb->join[f]) cudaEventDestroy(bb->join[f]);
    }
    if (bb->fork) cudaEventDestroy(bb->fork);
    if (bb->graph) cudaGraphExecDestroy(bb->graph);
    bb->keys_in.release(); bb->keys_out.release(); bb->idx_in.release(); bb->idx_out.release();
    bb->tmp.release(); bb->table.release(); bb->xl.release();
    delete bb;
}

// The batched sequence on the caller's buffers (batched_prepare must have run).
cudaError_t batched_enqueue(bwacuda_ctx *c, BatchBufs *bb, const uint8_t *d_seq, const bwacuda_dev_ext_job *d_jobs,
                            size_t n, const ExtParams &P, bwacuda_ext_result *d_out, cudaStream_t s, uint32_t *err,
                            unsigned long long *cells)
{
    cudaError_t e = ensure_bufs(*bb, batched_grow_jobs(*bb, n), batched_fan(c, *bb, n, P));
    if (e != cudaSuccess) return e;
    return enqueue_batched(c, *bb, d_seq, d_jobs, n, P, d_out, s, err, cells);
}

// Work buffers of a slot for n jobs ahead of its first batch (the serving loop's wave slots).
cudaError_t batched_reserve(BatchBufs *bb, size_t n)
{
    cudaError_t e = ensure_bufs(*bb, n);
    if (e == cudaSuccess) bb->jobs_cap = std::max(bb->jobs_cap, n);
    return e;
}

// Host-buffer form: the plain path's packing pipeline, each chunk run batched.
int extend_batch_host_batched(bwacuda_ctx *c, const bwacuda_ext_job *jobs, size_t n, int m, const int8_t *mat,
                              const ExtParams &P, int w, bwacuda_ext_result *out)
{
    int rc = batched_init(c);
    if (rc) return rc;
    return extend_host_pipeline(c, jobs, n, m, mat, P, w, out, [c](int slot, const ExtChunkInfo &I, cudaStream_t s) {
        BatchBufs &bb = c->batched->bufs[slot];
        cudaError_t e = ensure_bufs(bb, I.n, batched_fan(c, bb, I.n, I.P));
        if (e == cudaSuccess) e = enqueue_batched(c, bb, I.d_seq, I.d_jobs, I.n, I.P, I.d_out, s);
        if (e == cudaSuccess) c->stats.kernel_launches += (uint64_t)bb.launched;
        return cuda_status(e);
    });
}


}  // namespace bwacuda
