// ext_band.cu -- launches of the band kernel (ext_band.cuh): a group of 8, 16 or 32 lanes per job.
//
// 8 lanes a job cost the fewest instructions a cell, so they run where the jobs fill the GPU; 32
// finish a job soonest.  Two forms: over device-resident jobs (the open-ended length buckets and
// small batches of any length), and straight over a caller's host job array, a warp per job, for
// the smallest host calls, where a gather and its plan would cost more than the jobs themselves.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "ext_band.cuh"
#include "kernels.h"

namespace bwacuda {
namespace band {

constexpr int TB = 64;

// Measured (GB300): 10,000 queries of 1,500 bases in 3.24 ms with 8 lanes a job (5.06 with 150
// registers and six blocks an SM before the bound, per-pair tests and selects, and chunk lengths
// known at run time only), ALU pipe 73%, 537 instructions a warp row of four jobs, half of them the
// fixed part; 20,000 queries of 2-10 kb 21.9 ms against 39.5 for a thread per job, whose longest warp
// set the time.  4 lanes a job: 14.1 against 14.7 ms on 60,000 of those 1,500-base jobs, but 29.8
// against 23.1 ms on the 2-10 kb ones (both in 1024-row sort steps), so it is not built.
template <int L>
__global__ void __launch_bounds__(TB, 10)
ext_band_kernel(const uint8_t *__restrict__ seq, const bwacuda_dev_ext_job *__restrict__ jobs,
                const uint32_t *__restrict__ order, const uint32_t *__restrict__ bounds,
                uint32_t *__restrict__ counter, uint32_t njobs, int min_qlen, uint32_t count_lo, uint32_t count_hi,
                const __grid_constant__ ExtParams P, bwacuda_ext_result *__restrict__ out,
                uint32_t *__restrict__ err, unsigned long long *__restrict__ cells_total)
{
    constexpr int G = 32 / L, JW = job_words<L>();
    extern __shared__ __align__(16) uint32_t smem_w[];
    const int lane = threadIdx.x & 31, k = lane & (L - 1), grp = lane / L;
    uint32_t *sm = smem_w + ((threadIdx.x >> 5) * G + grp) * JW;
    uint32_t start = 0, stop = njobs;
    if (bounds) {
        // device-written bounds, clamped to the launch's job count
        stop = min(bounds[1], njobs);
        start = min(bounds[0], stop);
    }
    const uint32_t count = stop - start;
    if (count < count_lo || count >= count_hi) return;  // another group width's launch
    const bool sym = P.sc.o_del + P.sc.e_del == P.sc.o_ins + P.sc.e_ins;
    unsigned long long ncells = 0;
    for (;;) {
        uint32_t b0 = 0;
        if (lane == 0) b0 = atomicAdd(counter, (uint32_t)G);
        b0 = __shfl_sync(FULL, b0, 0);
        if (b0 >= count) break;
        const uint32_t pos = start + b0 + (uint32_t)grp;
        bool act = pos < stop;
        uint32_t jid = 0;
        int w = 0;
        bwacuda_dev_ext_job J;
        J.q_off = 0; J.t_off = 0; J.qlen = 0; J.tlen = 0; J.h0 = 1; J.w = 0;
        if (act) {
            jid = order ? order[pos] : pos;
            act = jid < njobs;  // the group-per-job kernel flags an index past the jobs
            if (act) J = jobs[jid];
            // a negative target length: an empty target where a bucket's thread takes it so, else the
            // group-per-job kernel's to flag
            act = act && J.qlen >= 0 && (J.tlen >= 0 || J.qlen <= EXT_TPJ_QLEN_MAX) && J.qlen >= min_qlen &&
                  ext_fits_i16(J.qlen, J.tlen, J.h0, P.sc.max_sc);
            if (act) {
                w = clamp_band(J.w < 0 ? 0 : J.w, J.qlen, P.sc.max_sc, P.end_bonus, P.sc.o_ins, P.sc.e_ins,
                               P.sc.o_del, P.sc.e_del);
                act = xl::band_takes(J.qlen, w);
            }
        }
        if (!__any_sync(FULL, act)) continue;
        bool bad = false;
        const uint8_t *q = seq + J.q_off, *t = seq + J.t_off;
        const bwacuda_ext_result r =
            sym ? band_run<L, true>(sm, act, q, t, J.qlen, J.tlen, J.h0, w, P, bad, ncells)
                : band_run<L, false>(sm, act, q, t, J.qlen, J.tlen, J.h0, w, P, bad, ncells);
        if (bad) atomicOr(err, ERR_BASE);
        if (act && k == 0) out[jid] = r;
        __syncwarp();  // the next jobs overwrite the rows
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ncells += __shfl_xor_sync(FULL, ncells, o);
    if (lane == 0 && ncells) atomicAdd(cells_total, ncells);
}

// A warp per job of a caller's host array (host memory the device reads through the host page
// tables): the job record, both slices as whole aligned words (no word lies outside a page the
// slice occupies), the result back into the caller's array.  The host has checked every job
// (band_direct_ok).
__global__ void __launch_bounds__(TB)
ext_band_direct_kernel(const bwacuda_ext_job *__restrict__ hjobs, uint32_t n, int w_call,
                       const __grid_constant__ ExtParams P, int32_t *__restrict__ hout, uint32_t *__restrict__ err,
                       unsigned long long *__restrict__ cells_total)
{
    constexpr int JW = row_words<32>() + RAW_WORDS, MAXW = (RAW_WORDS + 31) / 32;
    extern __shared__ __align__(16) uint32_t smem_w[];
    const int lane = threadIdx.x & 31;
    const uint32_t jid = (blockIdx.x * TB + threadIdx.x) >> 5;
    if (jid >= n) return;
    uint32_t *sm = smem_w + (threadIdx.x >> 5) * JW;
    uint32_t *raw = sm + row_words<32>();
    const bwacuda_ext_job J = hjobs[jid];
    const uint64_t qa = reinterpret_cast<uint64_t>(J.query), ta = reinterpret_cast<uint64_t>(J.target);
    const int nq = J.qlen > 0 ? ((int)(qa & 3) + J.qlen + 3) >> 2 : 0;
    const int nt = J.tlen > 0 ? ((int)(ta & 3) + J.tlen + 3) >> 2 : 0;
    const uint32_t *qw = reinterpret_cast<const uint32_t *>(qa & ~3ull), *tw = reinterpret_cast<const uint32_t *>(ta & ~3ull);
    uint32_t v[MAXW];
#pragma unroll
    for (int u = 0; u < MAXW; ++u) {
        const int x = 32 * u + lane;
        v[u] = x < nq ? qw[x] : (x < nq + nt ? tw[x - nq] : 0u);
    }
#pragma unroll
    for (int u = 0; u < MAXW; ++u)
        if (32 * u + lane < nq + nt) raw[32 * u + lane] = v[u];
    __syncwarp();
    const uint8_t *q = reinterpret_cast<const uint8_t *>(raw) + (qa & 3);
    const uint8_t *t = reinterpret_cast<const uint8_t *>(raw + nq) + (ta & 3);
    const int w = clamp_band(w_call, J.qlen, P.sc.max_sc, P.end_bonus, P.sc.o_ins, P.sc.e_ins, P.sc.o_del, P.sc.e_del);
    const bool sym = P.sc.o_del + P.sc.e_del == P.sc.o_ins + P.sc.e_ins;
    bool bad = false;
    unsigned long long ncells = 0;
    const bwacuda_ext_result r = sym ? band_run<32, true>(sm, true, q, t, J.qlen, J.tlen, J.h0, w, P, bad, ncells)
                                     : band_run<32, false>(sm, true, q, t, J.qlen, J.tlen, J.h0, w, P, bad, ncells);
    if (bad) atomicOr(err, ERR_BASE);
    const int32_t f[6] = {r.score, r.qle, r.tle, r.gtle, r.gscore, r.max_off};
    int32_t mine = f[0];
#pragma unroll
    for (int x = 1; x < 6; ++x) mine = lane == x ? f[x] : mine;
    if (lane < 6) hout[(size_t)jid * 6 + lane] = mine;
    if (lane == 0 && ncells) atomicAdd(cells_total, ncells);
}

template <int L>
cudaError_t launch(const ExtLongLaunch &X, uint32_t *counter, uint32_t count_lo, uint32_t count_hi, int nsm)
{
    auto kern = ext_band_kernel<L>;
    size_t smem = (size_t)(TB / L) * job_words<L>() * 4;
    // process-wide per kernel: always the ceiling (see the persistent kernels)
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EXT_SMEM_BLOCK_MAX);
    // an SM keeps the shared-memory split of the first kernel placed on it while empty; these blocks
    // and the other extension kernels beside them want the largest
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, TB, smem)) != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidValue;
    if (X.reserve_regs > 0 || X.reserve_threads > 0) {
        cudaFuncAttributes fa;
        if ((e = cudaFuncGetAttributes(&fa, kern)) != cudaSuccess) return e;
        const int regs_block = ((fa.numRegs * 32 + 255) / 256) * 256 * (TB / 32);
        const int cap_r = regs_block > 0 ? (X.sm_regs - X.reserve_regs) / regs_block : per_sm;
        const int cap_t = (X.sm_threads - X.reserve_threads) / TB;
        per_sm = std::max(1, std::min(per_sm, std::min(cap_r, cap_t)));
    }
    const size_t most = ((size_t)X.njobs * L + TB - 1) / TB;
    const uint32_t grid = (uint32_t)std::min<size_t>((size_t)per_sm * nsm, most);
    if (grid == 0) return cudaSuccess;
    // a grid that does not fill the GPU is spread evenly: shared memory for just the blocks an SM
    // should hold (left to itself the block scheduler puts several on one SM with others idle:
    // 1,000 queries of 1,500 bases with 8 lanes a job 3.31 against 1.57 ms, 5,000 3.19 against 2.25)
    if (grid < (uint32_t)per_sm * (uint32_t)nsm) {
        const size_t want = (grid + nsm - 1) / nsm;
        smem = std::max(smem, EXT_SMEM_BLOCK_MAX / want - 2048);
    }
    kern<<<grid, TB, smem, X.stream>>>(X.seq, X.jobs, X.order, X.bounds, counter, X.njobs, X.min_qlen, count_lo, count_hi,
                                      X.P, X.out, X.err, X.cells);
    return cudaGetLastError();
}

}  // namespace band

cudaError_t ext_band_launch(const ExtLongLaunch &X, int lanes, uint32_t *counter, uint32_t count_lo, uint32_t count_hi,
                            int nsm)
{
    if (lanes == 8) return band::launch<8>(X, counter, count_lo, count_hi, nsm);
    if (lanes == 16) return band::launch<16>(X, counter, count_lo, count_hi, nsm);
    return band::launch<32>(X, counter, count_lo, count_hi, nsm);
}

bool ext_band_direct_ok(int qlen, int tlen, int h0, int max_sc)
{
    return qlen <= 256 && tlen <= 512 && ext_fits_i16(qlen, tlen, h0, max_sc);
}

cudaError_t ext_band_direct_launch(const bwacuda_ext_job *hjobs, uint32_t n, int w, const ExtParams &P,
                                   bwacuda_ext_result *hout, uint32_t *err, unsigned long long *cells, cudaStream_t s)
{
    using namespace band;
    const size_t smem = (size_t)(TB / 32) * (row_words<32>() + RAW_WORDS) * 4;  // below the 48 KB every launch may use
    ext_band_direct_kernel<<<(n * 32 + TB - 1) / TB, TB, smem, s>>>(hjobs, n, w, P, reinterpret_cast<int32_t *>(hout), err,
                                                                   cells);
    return cudaGetLastError();
}

}  // namespace bwacuda
