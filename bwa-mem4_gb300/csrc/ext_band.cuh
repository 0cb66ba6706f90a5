// ext_band.cuh -- banded seed extension (ksw_extend2, crates/bwa-extend/src/sw.rs:203-493) by a
// group of L lanes per job that splits every row, with the 16-bit pair cells of the thread-per-job
// form (ext_job.cuh, ext_run_job_i16p).
//
// What it is for.  A thread per job needs about a hundred thousand jobs to fill the GPU and walks
// a job's rows in hundreds of microseconds; small batches and long queries (a few thousand jobs of
// thousands of rows) leave most SMs idle that way.  Here a row costs about 20 instructions a column
// pair, split over the group, and a fixed part (two short scans and the band update), so a job's
// latency falls with L while the work per cell grows only by the fixed part.
//
// A row.  The job's row lives in shared memory as a window of WC columns [base, base + WC) that
// moves right SLIDE_K columns whenever the band has left the first ones; pair p holds columns 2p,
// 2p + 1 (relative to base): X = (H, H), Y = (E, E), S = the query's score selectors.  The row's
// pairs p0 .. plast are cut into L chunks of K pairs (K odd, so that the lanes' words fall into
// different banks; compile-time, one straight-line body per K), the last chunk ending at plast.
//   1. Per pair: M, the gap opens, E of the next row (stored at once), max(M, E), and F from the
//      chunk's own columns alone.
//   2. F entering a chunk is the maximum over the chunks to its left of what they pass on less the
//      columns between: a scan of log2(L) shuffles.  All F are at least 0, so the terms below 0
//      drop out as in the recurrence.
//   3. Per pair: H = max(max(M, E), own F, entering F), stored one column to the right; the row
//      maximum keeps the later column on ties.
// Columns left of beg hold H = E = 0 (the one the band drops is zeroed before the row; the ones the
// live-cell scan passes are zero already) and beg never decreases, so the pairs left of p0 that the
// leading lanes' chunks reach add nothing to M, E, F or the maximum and stay 0: no per-pair test.
// A chunk that lies left of p0 altogether is moved into the PAD zero words in front of the row.  S has
// PAD selectors of its own in front, of code 0 like those past the query: without their sign bytes a score
// of -65 or less reads as one near -32768, and a large gap open takes that around to a positive F.
// Column `end` in an odd last pair is masked to zero on the way in and out of the maximum; it then
// receives the sentinel (H of the last column, E = 0) by the ordinary stores.  The live-cell scans
// of the adaptive band (sw.rs:465-482) look at the first and last cell, and probe L columns at once
// from either end where one of them is dead.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"
#include "ext_job.cuh"
#include "ext_long.cuh"

namespace bwacuda {
namespace band {

using xl::FULL;
using xl::SLIDE_K;

constexpr int WC = xl::BAND_WC;          // window columns
constexpr int PAIRS = WC / 2 + 2;        // pair words of the window and the spare ones behind it
constexpr int BAND_PAIRS = (WC - 4) / 2 + 1;  // pairs of its widest row, an odd first column included
constexpr int KP = SLIDE_K / 2;
constexpr int RAW_WORDS = (256 + 512 + 32) / 4;  // staged bases of a job read in place (ext_band_direct_ok)
// Longest chunk: the window's widest row (xl::BAND_WC - 4 columns, an odd first one) in L chunks.
template <int L>
constexpr int kmax() { return L == 32 ? 5 : (L == 16 ? 9 : 17); }
static_assert(8 * kmax<8>() >= BAND_PAIRS && 16 * kmax<16>() >= BAND_PAIRS && 32 * kmax<32>() >= BAND_PAIRS,
              "every L holds every row of the window");
// Zero pairs in front of the row: a chunk reaches at most kmax - 1 pairs left of p0.
template <int L>
constexpr int pad() { return (kmax<L>() + 3) / 4 * 4; }
template <int L>
constexpr int row_words() { return 2 * (pad<L>() + PAIRS) + (pad<L>() + PAIRS + 1) / 2; }  // X, Y, S (16 bits a pair)
// Shared words of a job: L modulo 32, so that with odd chunk lengths the warp's 32 lanes hit 32 banks
// (lane k's word is k * K modulo L, each residue once; the jobs then differ by multiples of L).
template <int L>
constexpr int job_words() { return (row_words<L>() + 31 - L % 32) / 32 * 32 + L % 32; }

// Row -1 values of columns c, c + 1 (sw.rs:269-279), 0 past the query.
__device__ __forceinline__ uint32_t row_minus1_pair(int c, int qlen, int h0, int oe_ins, int e_ins)
{
    const int a = c <= qlen ? xl::row_minus1(c, h0, oe_ins, e_ins) : 0;
    const int b = c + 1 <= qlen ? xl::row_minus1(c + 1, h0, oe_ins, e_ins) : 0;
    return (uint32_t)a | ((uint32_t)b << 16);
}

// Score selectors of columns c, c + 1 (prmt selector bytes 0x80 | code * 0x11, code 0 past the query).
__device__ __forceinline__ uint16_t query_pair(const uint8_t *__restrict__ q, int qlen, int c)
{
    const uint32_t a = c < qlen ? q[c] & 7u : 0u, b = c + 1 < qlen ? q[c + 1] & 7u : 0u;
    return (uint16_t)(0x8080u | a * 0x11u | b * 0x1100u);
}

// Gap constants, each 16-bit value in both lanes.
struct BandGaps {
    uint32_t noe_ins2, noe_del2, ne_del2, ne_ins2, n2e_ins2, fsel2;
    int e_ins;
    __device__ __forceinline__ void init(const Scoring &sc)
    {
        e_ins = sc.e_ins;
        noe_ins2 = (uint32_t)(-(sc.o_ins + sc.e_ins) & 0xffff) * 0x10001u;
        noe_del2 = (uint32_t)(-(sc.o_del + sc.e_del) & 0xffff) * 0x10001u;
        ne_del2 = (uint32_t)(-sc.e_del & 0xffff) * 0x10001u;
        ne_ins2 = (uint32_t)(-sc.e_ins & 0xffff) * 0x10001u;
        n2e_ins2 = (uint32_t)(-2 * sc.e_ins & 0xffff) * 0x10001u;  // e_ins <= 16384: at least -32768
        fsel2 = 0x8000u | ((uint32_t)(-sc.e_ins & 0xffff) << 16);
    }
};

// One row of every group in the warp: lane k's chunk of K pairs from X, Y, S on.  lm masks the last
// pair's columns (lane L - 1).  Returns the lane's row-maximum key (H << 16) | chunk-relative column
// and the last pair's H in hend.
template <int L, int K, bool SYM>
__device__ __forceinline__ int32_t band_row(uint32_t *X, uint32_t *Y, const uint16_t *S, int k, uint32_t lm,
                                            uint32_t plo, uint32_t phi, const BandGaps &g, uint32_t &hend)
{
    uint32_t me2[K], fl2[K];
    uint32_t fv = 0u;
#pragma unroll
    for (int u = 0; u < K; ++u) {
        uint32_t hd2 = X[u], e2 = Y[u];
        if (u == K - 1) {
            hd2 &= lm;
            e2 &= lm;
        }
        const uint32_t s2 = prmt(plo, phi, S[u]);
        const uint32_t g2 = __viaddmin_u16x2(hd2, 0u, 0x00010001u) * 0x7fffu;  // zero diagonals: see ext_job.cuh
        const uint32_t M2 = __viaddmin_s16x2(hd2, s2, g2);
        const uint32_t ti2 = __viaddmax_s16x2_relu(M2, g.noe_ins2, 0u);
        const uint32_t td2 = SYM ? ti2 : __viaddmax_s16x2_relu(M2, g.noe_del2, 0u);
        Y[u] = __viaddmax_s16x2(e2, g.ne_del2, td2);
        me2[u] = __vimax_s16x2_relu(M2, e2);  // E is never negative
        fl2[u] = f_pair(fv, ti2, g.fsel2, g.ne_ins2);
    }
    // F entering the chunk: 2K columns a chunk
    int v = (int)(fv >> 16);
    const int dec = 2 * K * g.e_ins;
#pragma unroll
    for (int d = 1; d < L; d <<= 1) {
        const int o = __shfl_up_sync(FULL, v, d, L) - d * dec;
        if (k >= d) v = v > o ? v : o;
    }
    const int fs = __shfl_up_sync(FULL, v, 1, L);
    const int fin = k > 0 ? max(fs, 0) : 0, fin1 = max(fin - g.e_ins, 0);
    uint32_t run2 = (uint32_t)fin | ((uint32_t)fin1 << 16);
    // the last pair's H ahead of the others: the next lane's first store needs it
    const int fz = fin - (2 * K - 2) * g.e_ins, fz1 = fz - g.e_ins;
    hend = __vimax3_s16x2(me2[K - 1], fl2[K - 1], (uint32_t)max(fz, 0) | ((uint32_t)max(fz1, 0) << 16));
    uint32_t h1v = __shfl_up_sync(FULL, hend, 1, L);
    if (k == 0) h1v = 0u;
    int32_t key = 0;
#pragma unroll
    for (int u = 0; u < K; ++u) {
        const uint32_t h2 = u == K - 1 ? hend : __vimax3_s16x2(me2[u], fl2[u], run2);
        if (u + 2 < K) run2 = __viaddmax_s16x2_relu(run2, g.n2e_ins2, 0u);
        X[u] = prmt(h1v, h2, 0x5432u);  // H(i, j - 1) for the next row's diagonal
        const uint32_t hk = u == K - 1 ? h2 & lm : h2;
        const int32_t ka = (int32_t)prmt((uint32_t)(2 * u), hk, 0x5410u);
        const int32_t kb = (int32_t)((hk & 0xffff0000u) | (uint32_t)(2 * u + 1));
        key = __vimax3_s32(key, ka, kb);
        h1v = h2;
    }
    return key;
}

// Chunk lengths built for L lanes (all odd): the smallest that holds `need` pairs a lane.
template <int L>
__device__ __forceinline__ int chunk_len(int need)
{
    return L == 8 && need > 13 ? 17 : need | 1;
}

// band_row for the chunk length K (uniform over the warp).
template <int L, bool SYM>
__device__ __forceinline__ int32_t band_row_k(int K, uint32_t *X, uint32_t *Y, const uint16_t *S, int k, uint32_t lm,
                                              uint32_t plo, uint32_t phi, const BandGaps &g, uint32_t &hend)
{
#define BAND_CASE(KC) \
    case KC: return band_row<L, KC, SYM>(X, Y, S, k, lm, plo, phi, g, hend)
    if constexpr (L == 8) {
        switch (K) {
            BAND_CASE(1); BAND_CASE(3); BAND_CASE(5); BAND_CASE(7); BAND_CASE(9); BAND_CASE(11); BAND_CASE(13);
        default: return band_row<L, 17, SYM>(X, Y, S, k, lm, plo, phi, g, hend);
        }
    } else if constexpr (L == 16) {
        switch (K) {
            BAND_CASE(1); BAND_CASE(3); BAND_CASE(5); BAND_CASE(7);
        default: return band_row<L, 9, SYM>(X, Y, S, k, lm, plo, phi, g, hend);
        }
    } else {
        switch (K) {
            BAND_CASE(1); BAND_CASE(3);
        default: return band_row<L, 5, SYM>(X, Y, S, k, lm, plo, phi, g, hend);
        }
    }
#undef BAND_CASE
}

// One job per group of L lanes, the warp's groups in lockstep (act: this group has one).  The
// result is returned in every lane of the group.
template <int L, bool SYM>
__device__ __forceinline__ bwacuda_ext_result band_run(uint32_t *__restrict__ sm, bool act, const uint8_t *q,
                                                       const uint8_t *t, int qlen, int tlen, int h0, int w,
                                                       const ExtParams &P, bool &bad, unsigned long long &ncells)
{
    constexpr int PAD = pad<L>();
    const int lane = threadIdx.x & 31, k = lane & (L - 1);
    uint32_t *X = sm + PAD, *Y = X + PAIRS + PAD;
    uint16_t *S = reinterpret_cast<uint16_t *>(Y + PAIRS) + PAD;
    uint16_t *X16 = reinterpret_cast<uint16_t *>(X), *Y16 = reinterpret_cast<uint16_t *>(Y);
    const int m = P.sc.m;
    const int o_del = P.sc.o_del, e_del = P.sc.e_del, o_ins = P.sc.o_ins, e_ins = P.sc.e_ins;
    const int oe_ins = o_ins + e_ins;
    if (act) {
#pragma unroll 4
        for (int j = k; j < qlen; j += L) bad |= q[j] >= (uint32_t)m;
        for (int p = k; p < PAIRS; p += L) {
            X[p] = row_minus1_pair(2 * p, qlen, h0, oe_ins, e_ins);
            Y[p] = 0u;
            S[p] = query_pair(q, qlen, 2 * p);
        }
    }
    for (int p = k; p < PAD; p += L) {
        X[p - PAD] = 0u;
        Y[p - PAD] = 0u;
        S[p - PAD] = 0x8080u;
    }
    const bool moves = act && qlen + 4 > WC, any_moves = __any_sync(FULL, moves);
    uint32_t cells = 0;
    int base = 0;  // first column of the window, a multiple of SLIDE_K
    int best = h0, best_i = -1, best_j = -1, best_ie = -1, gscore = -1, max_off = 0;
    int beg = 0, end = qlen;
    TargetStream ts;
    ts.init(t, act ? tlen : 0);
    BandGaps g;
    g.init(P.sc);
    int h1c = h0 - (o_del + e_del);  // H(i, -1) before the clamp at 0
    for (int i = 0;; ++i, h1c -= e_del) {
        const bool run = act && i < tlen;
        if (!__any_sync(FULL, run)) break;
        if (any_moves) {
            const bool mv = run && moves && i - w - 1 - base >= SLIDE_K;
            if (__any_sync(FULL, mv)) {
                __syncwarp();
                if (mv) {
                    // a lane touches only pairs congruent to it modulo L (KP is a multiple of L): no
                    // lane reads a word that another one writes
                    for (int p = k; p < PAIRS; p += L) {
                        const bool keep = p + KP < PAIRS;
                        X[p] = keep ? X[p + KP] : row_minus1_pair(base + SLIDE_K + 2 * p, qlen, h0, oe_ins, e_ins);
                        Y[p] = keep ? Y[p + KP] : 0u;
                        S[p] = keep ? S[p + KP] : query_pair(q, qlen, base + SLIDE_K + 2 * p);
                    }
                    base += SLIDE_K;
                }
                __syncwarp();
            }
        }
        uint32_t tc = 0;
        if (run) {
            tc = ts.next();
            bad |= tc >= (uint32_t)m;
            tc &= 7u;
            if (beg < i - w) {  // the band drops one column a row
                if (k == 0) {
                    X16[beg - base] = 0;
                    Y16[beg - base] = 0;
                }
                beg = i - w;
            }
            end = min(min(end, i + w + 1), qlen);
        }
        const uint32_t plo = P.sc.prof[tc][0], phi = P.sc.prof[tc][1];
        const int h1 = beg == 0 ? max(h1c, 0) : 0;
        const int ncol = run && end > beg ? end - beg : 0;
        const int rb = beg - base, re = end - base;
        const int p0 = rb >> 1, plast = (re - 1) >> 1;
        const int np = ncol > 0 ? plast - p0 + 1 : 0;
        // chunk length of the warp's longest row (at most kmax: the window bounds np)
        const int K = chunk_len<L>((int)__reduce_max_sync(FULL, (unsigned)(np + L - 1) / L));
        __syncwarp();
        const uint32_t lm = k == L - 1 && (re & 1) ? 0xffffu : 0xffffffffu;
        int pl = plast + 1 - (L - k) * K;             // the lane's first pair
        if (np == 0 || pl + K <= p0) pl = -PAD;       // nothing of the row: zeros, which stay zero
        uint32_t hend;
        int32_t rowkey;
        uint32_t *Xl = X + pl, *Yl = Y + pl;
        const uint16_t *Sl = S + pl;
        rowkey = band_row_k<L, SYM>(K, Xl, Yl, Sl, k, lm, plo, phi, g, hend);
        if ((rowkey >> 16) > 0) rowkey += 2 * pl;  // chunk-relative to window-relative columns
        else rowkey = 0;
        int hl = np > 0 ? (re & 1 ? (int)(hend & 0xffffu) : (int)(hend >> 16)) : h1;
        if (k == L - 1 && np > 0 && !(re & 1)) {  // sentinel column end (sw.rs:418-419)
            X16[re] = (uint16_t)hl;
            Y16[re] = 0;
        }
        hl = __shfl_sync(FULL, hl, L - 1, L);
        rowkey = xl::group_max<L>(rowkey);
        __syncwarp();
        bool scan = false;
        uint32_t fb = 0u;
        if (run) {
            cells += (uint32_t)ncol;
            if (k == 0 && beg == 0) X16[0] = (uint16_t)h1;  // H(i, -1) is column 0's next diagonal
            fb = beg == 0 ? (uint32_t)h1 : X16[rb];
            fb |= Y16[rb];
            const int jf = end > beg ? end : beg;
            if (jf == qlen && gscore <= hl) {  // later row wins ties (sw.rs:424-427)
                best_ie = i;
                gscore = hl;
            }
            const int rmax = rowkey >> 16;
            const int mj = (rowkey & 0xffff) + base;
            if (rmax == 0) {
                act = false;
            } else if (rmax > best) {
                best = rmax;
                best_i = i;
                best_j = mj;
                const int off = mj > i ? mj - i : i - mj;
                if (off > max_off) max_off = off;
            } else if (P.zdrop > 0) {  // sw.rs:440-456
                if (i - best_i > mj - best_j) {
                    if (best - rmax - ((i - best_i) - (mj - best_j)) * e_del > P.zdrop) act = false;
                } else if (best - rmax - ((mj - best_j) - (i - best_i)) * e_ins > P.zdrop) {
                    act = false;
                }
            }
            scan = act;
        }
        // adaptive band (sw.rs:465-482): first live column of [beg, end), last of [beg, end]
        int lo = beg, hi = end;
        bool sl = scan && fb == 0u, sh = scan && hl == 0;
        if (__any_sync(FULL, sl || sh)) {
            if (sl) lo = end;
            if (sh) hi = beg - 1;
            __syncwarp();
            for (int off = 0; __any_sync(FULL, sl || sh); off += L) {
                const int a = beg + off + k, b = end - off - k;
                const bool la = sl && a < end && (X16[a - base] | Y16[a - base]) != 0;
                const bool lb = sh && b >= beg && (X16[b - base] | Y16[b - base]) != 0;
                constexpr uint32_t GM = L == 32 ? 0xffffffffu : (1u << (L & 31)) - 1u;
                const uint32_t ma = (__ballot_sync(FULL, la) >> (lane & ~(L - 1))) & GM;
                const uint32_t mb = (__ballot_sync(FULL, lb) >> (lane & ~(L - 1))) & GM;
                if (sl) {
                    if (ma) lo = beg + off + __ffs((int)ma) - 1;
                    sl = ma == 0u && beg + off + L < end;
                }
                if (sh) {
                    if (mb) hi = end - off - (__ffs((int)mb) - 1);
                    sh = mb == 0u && end - off - L >= beg;
                }
            }
        }
        if (scan) {
            beg = lo;
            if (hi < beg) hi = beg - 1;  // the reference's scan for hi stops at the new beg - 1
            end = min(hi + 2, qlen);
        }
    }
    if (k == 0) ncells += cells;  // a job's cells fit 32 bits: tlen rows of at most WC
    bwacuda_ext_result r;
    r.score = best;
    r.qle = best_j + 1;
    r.tle = best_i + 1;
    r.gtle = best_ie + 1;
    r.gscore = gscore;
    r.max_off = max_off;
    return r;
}

}  // namespace band
}  // namespace bwacuda
