// ext_dual.cuh -- two banded seed extensions (ksw_extend2, crates/bwa-extend/src/sw.rs:203-493) per
// thread in 8-bit cells: job A in the low 16-bit lane of every register, job B in the high one.
//
// Bound.  The 8-bit buckets are bound by the ALU pipe.  With two columns of one job in the lanes
// (ext_run_job_u8p) F has to cross the lanes, a permute and two add-maxima a column pair, and a cell
// word takes two permutes to pack: 14.5 ALU instructions for two cells.  With a job per lane F passes
// from column to column in one instruction, one permute packs the word (H_A, E_A, H_B, E_B) and rows
// have no odd first or last column: 10.5 for two cells, and one instruction on the multiply pipe.
//
// The two jobs come from neighbouring places of the sort (class, query length, target length, h0), so
// their windows [beg, end) nearly agree.  A row runs over the union:
//  - left of a job's beg its cells are H = E = 0 (the one the band drops is zeroed before the row, the
//    ones the live-cell scan passed are zero already) and nothing reads them again, so the other job's
//    columns there need no test: zeros stay zeros;
//  - right of a job's end its cells are stale values the adaptive band may read back, so the row's
//    last columns go through four a step with masks that keep an ended job's bytes.
// A finished job's lane runs on as garbage (scored -128, so that it stays in a byte) and is never read.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"
#include "ext_job.cuh"

namespace bwacuda {
namespace dual {

// One job of the pair: its state over the rows.
struct Side {
    int qlen, tlen, h0, w;
    int beg, end, best, best_i, best_j, best_ie, gscore, max_off;
    bool act;
    __device__ __forceinline__ void init(const bwacuda_dev_ext_job &J, const ExtParams &P, bool on)
    {
        qlen = J.qlen;
        tlen = J.tlen;
        h0 = J.h0;
        w = clamp_band(J.w < 0 ? 0 : J.w, qlen, P.sc.max_sc, P.end_bonus, P.sc.o_ins, P.sc.e_ins, P.sc.o_del,
                       P.sc.e_del);
        beg = 0;
        end = qlen;
        best = h0;
        best_i = best_j = best_ie = gscore = -1;
        max_off = 0;
        act = on && tlen > 0;
    }
    // After row i: hl = H of its last column, key = its row maximum (H << 8) | column.
    __device__ __forceinline__ void row(int i, int hl, uint32_t key, const ExtParams &P)
    {
        const int jf = end > beg ? end : beg;
        if (jf == qlen && gscore <= hl) {  // later row wins ties (sw.rs:424-427)
            best_ie = i;
            gscore = hl;
        }
        const int rmax = (int)(key >> 8), mj = (int)(key & 0xffu);
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
                if (best - rmax - ((i - best_i) - (mj - best_j)) * P.sc.e_del > P.zdrop) act = false;
            } else if (best - rmax - ((mj - best_j) - (i - best_i)) * P.sc.e_ins > P.zdrop) {
                act = false;
            }
        }
    }
    __device__ __forceinline__ bwacuda_ext_result result() const
    {
        bwacuda_ext_result r;
        r.score = best;
        r.qle = best_j + 1;
        r.tle = best_i + 1;
        r.gtle = best_ie + 1;
        r.gscore = gscore;
        r.max_off = max_off;
        return r;
    }
};

struct DualMul {
    uint32_t k128 = 128u, k256 = 256u;
};

// Gap constants, each 16-bit value in both lanes.
struct Gaps {
    uint32_t noe_ins2, noe_del2, ne_del2, ne_ins2;
    uint32_t k128, k256;  // multipliers the compiler does not see: as constants the guard and the keys would
                          // become shifts of the ALU pipe
};

// N consecutive columns of a row for both jobs, from cell c, selector q and column jj on; keys: the
// largest (H << 8) | column of each job.  Phase by phase over the columns: warps are few here and issue
// in order, so independent instructions go back to back and only F and the keys are chained.  ENDS:
// the columns may pass a job's end (nend2 = -end of each): from there on its cells and key stay, and
// hl2 keeps the H of its last column.
template <int TB, bool SYM, int N, bool ENDS>
__device__ __forceinline__ void columns(uint32_t *c, const uint16_t *q, uint32_t jj, const Gaps &g, uint32_t pa,
                                        uint32_t pb, uint32_t nend2, uint32_t &f2, uint32_t &h1v, uint32_t &key2,
                                        uint32_t &hl2)
{
    uint32_t wv[N], M[N], ti[N], en[N], h[N];
#pragma unroll
    for (int u = 0; u < N; ++u) wv[u] = c[u * TB];
#pragma unroll
    for (int u = 0; u < N; ++u) M[u] = q[u * TB];
#pragma unroll
    for (int u = 0; u < N; ++u) M[u] = prmt(pa, pb, M[u]);
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const uint32_t hd2 = wv[u] & 0x00ff00ffu;
        h[u] = prmt(wv[u], 0u, 0x4341u);                       // E(i, j)
        M[u] = __viaddmin_s16x2(hd2, M[u], hd2 * g.k128);     // hd ? hd + s : <= 0, see ext_run_job_u8p
    }
#pragma unroll
    for (int u = 0; u < N; ++u) ti[u] = __viaddmax_s16x2_relu(M[u], g.noe_ins2, 0u);
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const uint32_t td = SYM ? ti[u] : __viaddmax_s16x2_relu(M[u], g.noe_del2, 0u);
        en[u] = __viaddmax_s16x2(h[u], g.ne_del2, td);
    }
#pragma unroll
    for (int u = 0; u < N; ++u) {
        h[u] = __vimax3_s16x2(M[u], h[u], f2);  // H(i, j)
        f2 = __viaddmax_s16x2(f2, g.ne_ins2, ti[u]);
    }
    if constexpr (ENDS) {
        // ti: all ones in the lanes whose column lies before the job's end
#pragma unroll
        for (int u = 0; u < N; ++u)
            ti[u] = prmt(__viaddmax_s16x2((jj + (uint32_t)u) * 0x10001u, nend2, 0x80008000u), 0u, 0xbb99u);
#pragma unroll
        for (int u = 0; u < N; ++u) {
            const uint32_t w = prmt(u ? h[u - 1] : h1v, en[u], 0x6240u);
            c[u * TB] = (w & ti[u]) | (wv[u] & ~ti[u]);
        }
        h1v = h[N - 1];
#pragma unroll
        for (int u = 0; u < N; ++u) hl2 = (h[u] & ti[u]) | (hl2 & ~ti[u]);
#pragma unroll
        for (int u = 0; u < N; ++u) h[u] = (h[u] & ti[u]) * g.k256 + (uint32_t)u * 0x10001u;
    } else {
        // the new words: H(i, j - 1) and E(i + 1, j) of each job
#pragma unroll
        for (int u = 0; u < N; ++u) c[u * TB] = prmt(u ? h[u - 1] : h1v, en[u], 0x6240u);
        h1v = h[N - 1];
#pragma unroll
        for (int u = 0; u < N; ++u) h[u] = h[u] * g.k256 + (uint32_t)u * 0x10001u;
    }
    // keys (H << 8) | u by multiply-adds, their maximum, then the columns' start in one add-max.  H is at
    // most 255 and the column below 256, so nothing carries from one part or lane to the next: a real
    // cell's H by the class's bound, a masked lane's is 0, and a lane without columns in this row scores
    // -128 everywhere, which adds to nothing.
    static_assert(N == 4 || N == 8, "key maxima");
    uint32_t k = __vimax3_u16x2(h[0], h[1], h[2]);
    if constexpr (N == 4) k = __vimax3_u16x2(k, h[3], h[3]);
    else k = __vimax3_u16x2(__vimax3_u16x2(__vimax3_u16x2(k, h[3], h[4]), h[5], h[6]), h[7], h[7]);
    key2 = __viaddmax_u16x2(k, jj * 0x10001u, key2);
}

template <int TB, bool SYM>
__device__ __forceinline__ void run_pair(uint32_t *__restrict__ cw, uint16_t *__restrict__ qs,
                                         const uint8_t *__restrict__ seq, const bwacuda_dev_ext_job &JA,
                                         const bwacuda_dev_ext_job &JB, bool two, const ExtParams &P, const DualMul &mul,
                                         bool &bad, unsigned long long &ncells, bwacuda_ext_result &ra,
                                         bwacuda_ext_result &rb)
{
    const int m = P.sc.m;
    const int o_del = P.sc.o_del, e_del = P.sc.e_del, o_ins = P.sc.o_ins, e_ins = P.sc.e_ins;
    const int oe_del = o_del + e_del, oe_ins = o_ins + e_ins;
    Side A, B;
    A.init(JA, P, true);
    B.init(JB, P, two);
    const int qmax = A.qlen > B.qlen ? A.qlen : B.qlen;
    // prmt selectors: A's score and its sign, B's and its sign (no query of this class holds a code of 4 or
    // more: the sort keeps those in the 16-bit class, which checks them); alphabets of fewer than four
    // letters are checked here
    const uint32_t letters = m < 4 ? (uint32_t)m : 4u;
    for (int j = 0; j < qmax; j += 16) {
        uint32_t va[4], vb[4];
        load16(seq + JA.q_off, A.qlen, j, va);
        load16(seq + JB.q_off, B.qlen, j, vb);
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const uint32_t a = (va[u >> 2] >> (8 * (u & 3))) & 0xffu, b = (vb[u >> 2] >> (8 * (u & 3))) & 0xffu;
            bad |= a >= letters || b >= letters;
            if (j + u < qmax) qs[(size_t)(j + u) * TB] = (uint16_t)(0xC480u + (a & 3u) * 0x11u + (b & 3u) * 0x1100u);
        }
    }
    // row -1 (sw.rs:269-279), E = 0; 0 past a query
    {
        int ha = A.h0, hb = B.h0;
        for (int j = 0; j <= qmax; ++j) {
            cw[(size_t)j * TB] = (j <= A.qlen ? (uint32_t)ha : 0u) | (j <= B.qlen ? (uint32_t)hb << 16 : 0u);
            const int d = j == 0 ? oe_ins : e_ins;
            ha = ha > d ? ha - d : 0;
            hb = hb > d ? hb - d : 0;
        }
    }
    Gaps g;
    g.noe_ins2 = (uint32_t)(-oe_ins & 0xffff) * 0x10001u;
    g.noe_del2 = (uint32_t)(-oe_del & 0xffff) * 0x10001u;
    g.ne_del2 = (uint32_t)(-e_del & 0xffff) * 0x10001u;
    g.ne_ins2 = (uint32_t)(-e_ins & 0xffff) * 0x10001u;
    g.k128 = mul.k128;
    g.k256 = mul.k256;
    TargetStream ta, tb;
    ta.init(seq + JA.t_off, A.act ? A.tlen : 0);
    tb.init(seq + JB.t_off, B.act ? B.tlen : 0);
    uint8_t *cb = reinterpret_cast<uint8_t *>(cw);
    for (int i = 0;; ++i) {
        A.act = A.act && i < A.tlen;
        B.act = B.act && i < B.tlen;
        if (!A.act && !B.act) break;
        uint32_t ca = 0, cbt = 0;
        if (A.act) {
            ca = ta.next();
            if (A.beg < i - A.w) {  // the band drops one column a row
                *reinterpret_cast<uint16_t *>(cb + (size_t)A.beg * TB * 4) = 0;
                A.beg = i - A.w;
            }
            A.end = min(min(A.end, i + A.w + 1), A.qlen);
        }
        if (B.act) {
            cbt = tb.next();
            if (B.beg < i - B.w) {
                *reinterpret_cast<uint16_t *>(cb + (size_t)B.beg * TB * 4 + 2) = 0;
                B.beg = i - B.w;
            }
            B.end = min(min(B.end, i + B.w + 1), B.qlen);
        }
        bad |= ca >= (uint32_t)m || cbt >= (uint32_t)m;
        ca &= 7u;
        cbt &= 7u;
        const int h1a = A.act && A.beg == 0 ? max(A.h0 - (o_del + e_del * (i + 1)), 0) : 0;
        const int h1b = B.act && B.beg == 0 ? max(B.h0 - (o_del + e_del * (i + 1)), 0) : 0;
        // a job without columns in this row (it ends with it), or done: no bounds of its own
        const bool ea = A.act && A.end > A.beg, eb = B.act && B.end > B.beg;
        const uint32_t pa = ea ? P.sc.prof[ca][0] : 0x80808080u, pb = eb ? P.sc.prof[cbt][0] : 0x80808080u;
        uint32_t key2 = 0u, h1v = (uint32_t)h1a | ((uint32_t)h1b << 16);
        int hla = h1a, hlb = h1b;
        if (ea || eb) {
            const int lo = ea && eb ? min(A.beg, B.beg) : (ea ? A.beg : B.beg);
            const int e1 = ea && eb ? min(A.end, B.end) : (ea ? A.end : B.end);
            const int e2 = ea && eb ? max(A.end, B.end) : e1;
            uint32_t f2 = 0u;
            uint32_t *c = cw + (size_t)lo * TB;
            const uint16_t *q = qs + (size_t)lo * TB;
            int j = lo;
            uint32_t hl2 = 0u;
            for (; j + 8 <= e1; j += 8) {
                columns<TB, SYM, 8, false>(c, q, (uint32_t)j, g, pa, pb, 0u, f2, h1v, key2, hl2);
                c += 8 * TB;
                q += 8 * TB;
            }
            // the rest, to the later end, four columns a step with each job's end masked
            hl2 = h1v;
            const uint32_t nend2 = ((uint32_t)(ea ? -A.end : -e2) & 0xffffu) | ((uint32_t)(eb ? -B.end : -e2) << 16);
            for (; j < e2; j += 4) {
                columns<TB, SYM, 4, true>(c, q, (uint32_t)j, g, pa, pb, nend2, f2, h1v, key2, hl2);
                c += 4 * TB;
                q += 4 * TB;
            }
            hla = (int)(hl2 & 0xffffu);
            hlb = (int)(hl2 >> 16);
            // sentinel column end (sw.rs:418-419): H = H(i, end - 1), E = 0
            if (ea) *reinterpret_cast<uint16_t *>(cb + (size_t)A.end * TB * 4) = (uint16_t)hla;
            if (eb) *reinterpret_cast<uint16_t *>(cb + (size_t)B.end * TB * 4 + 2) = (uint16_t)hlb;
        }
        if (A.act) {
            ncells += ea ? (unsigned long long)(A.end - A.beg) : 0u;
            A.row(i, ea ? hla : h1a, ea ? key2 & 0xffffu : 0u, P);
            if (A.act) {  // adaptive band (sw.rs:465-482)
                int lo = A.beg, hi = A.end;
                while (lo < A.end && *reinterpret_cast<const uint16_t *>(cb + (size_t)lo * TB * 4) == 0) ++lo;
                A.beg = lo;
                while (hi >= lo && *reinterpret_cast<const uint16_t *>(cb + (size_t)hi * TB * 4) == 0) --hi;
                A.end = min(hi + 2, A.qlen);
            }
        }
        if (B.act) {
            ncells += eb ? (unsigned long long)(B.end - B.beg) : 0u;
            B.row(i, eb ? hlb : h1b, eb ? key2 >> 16 : 0u, P);
            if (B.act) {
                int lo = B.beg, hi = B.end;
                while (lo < B.end && *reinterpret_cast<const uint16_t *>(cb + (size_t)lo * TB * 4 + 2) == 0) ++lo;
                B.beg = lo;
                while (hi >= lo && *reinterpret_cast<const uint16_t *>(cb + (size_t)hi * TB * 4 + 2) == 0) --hi;
                B.end = min(hi + 2, B.qlen);
            }
        }
    }
    ra = A.result();
    rb = B.result();
}

// Cells of a thread (the masked columns of a row's last step may lie up to three past the longest query)
// and its shared memory: a word a cell and a 16-bit selector a column.
__host__ __device__ inline int thread_cells(int qcap) { return qcap + 3; }
__host__ __device__ inline size_t thread_bytes(int qcap)
{
    return (size_t)thread_cells(qcap) * 4 + (size_t)((thread_cells(qcap) + 3) & ~3) * 2;
}

}  // namespace dual
}  // namespace bwacuda
