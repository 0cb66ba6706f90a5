// global_tag.cuh -- ksw_global2 (crates/bwa-extend/src/sw.rs:561-740) two alignments per thread, with
// the direction of every cell carried in its value.
//
// Bound.  The DP is integer work (ALU pipe).  The pair kernel of global.cu takes the direction of a
// cell from eight predicates of four maxima, about twenty instructions a cell; here the direction
// rides in the low bits of the values, so that the maxima themselves select it:
//   values are 4 v + tag, tag 3 for M, 1 for E, 0 for F: H = max(M, E, F) prefers M over E over F on
//   ties, as the reference's comparisons do, and its low bits name the winner;
//   E(i+1, j) = max(E - e, M - (o + e)) and F likewise: the open term carries M's tag 3, the extension
//   E's 1 or F's 0, so open wins ties (the reference extends only when strictly better).
// A job of the pair sits in each 16-bit lane of every register (A low, B high), so one DPX instruction
// updates a cell of each and F passes from column to column without a lane shuffle: ten ALU
// instructions for two cells, the rest (tag removal, direction nibbles) on the multiply pipe.
//
// Band storage.  Slot b of the band is column j = i + b - wl of row i: H(i, j) overwrites H(i-1, j-1),
// the diagonal it needed, and E(i+1, j) is stored at b and read at b + 1 of the next row's diagonal
// order, so nothing moves.  Two rows go through at a time: at column j row i (slot s) and row i + 1
// (slot s - 1) share the query column, row i + 1 takes H(i, j-1) and E(i+1, j) from registers, and the
// slots are read and written once for both.
//
// Borders.  H and E outside the band are NEG, below every reachable value by more than any garbage
// chain can add (tag_rule).  Column -1 is a column like the others whose E starts at -(o + e) and
// extends row by row: H(i, -1) follows.  Steps of the first group left of column -1, steps right of the
// band or the query and rows past the target compute garbage that flows only right and down, except E,
// which slot s + 1 passes to step s: the two slots right of the band are reset to NEG after every two
// rows.  Jobs whose band does not hold the corner run in the other kernels (tag_ok), so the traceback
// stays inside cells the DP reached.
//
// Directions: a nibble a cell (H's tag, bit 2: E opened, bit 3: F opened), eight steps a word, and the
// words of two rows and two jobs as one 16-byte store, laid out warp by warp:
// z4[(row pair * ng + step / 8) * 32 + lane].  A warp's stores are 512 consecutive bytes, and so are
// the loads of the traceback, whose lanes walk the same rows.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"
#include "ext_job.cuh"

namespace bwacuda {
namespace gtag {

constexpr int NEG = -7200;       // in units of a score point
constexpr int MAX_OE = 60;       // o + e of either gap
constexpr int MAX_ENTRY = 31;    // |matrix entry|: 4 v + 3 fits a signed byte
constexpr int LOW_LIMIT = 6800;  // reachable values stay above -LOW_LIMIT
constexpr int HIGH_LIMIT = 8000;
constexpr int MAX_BAND = 128;    // columns left / right of the diagonal, and MAX_QLEN: a warp's rows fit an SM
constexpr int MAX_QLEN = 2000;   // whatever the widest bands and longest queries of a launch
constexpr int LEFT_PAD = 16;     // query selectors left of column 0 (garbage steps of the first group)

struct TagRule {
    int ok, mn, mx, oe, e;  // mn = -min entry (>= 0), mx = max entry (>= 0), oe / e: the larger of the gaps'
    // 2, 4, 16 and -1: multipliers the compiler does not see, so that tag removal and direction nibbles
    // stay multiply-adds (as constants they become shifts and adds of the ALU pipe, which bounds this)
    int single = 0;  // one alignment a thread (batches that leave most SMs' slots empty)
    uint32_t k2 = 2u, k4 = 4u, k16 = 16u, km1 = 0xffffffffu;
};

__host__ __device__ inline int band_left(int w, int tlen) { return w < tlen - 1 ? w : tlen - 1; }
__host__ __device__ inline int band_right(int w, int qlen) { return w < qlen - 1 ? w : qlen - 1; }
// Steps of a row pair and their groups of eight; slots of the band buffer (a dummy slot in front, the
// two reset slots and the last group's garbage behind).
__host__ __device__ inline int steps(int wl, int wr) { return wl + wr + 2; }
__host__ __device__ inline int groups(int wl, int wr) { return (steps(wl, wr) + 7) >> 3; }
__host__ __device__ inline int slots(int wl, int wr) { return 8 * groups(wl, wr) + 3; }
__host__ __device__ inline int sel_count(int qlen, int wl, int wr) { (void)wl; (void)wr; return qlen + LEFT_PAD + 16; }

// Whether an alignment of these sizes fits the tagged 16-bit values: every reachable value is at least
// that of the path "one gap, then the diagonal", and one more gap open below it (E and F).
__host__ __device__ inline bool tag_ok(int qlen, int tlen, int w, const TagRule &r)
{
    if (!r.ok || qlen < 1 || tlen < 1 || w < 0 || qlen > MAX_QLEN || tlen > MAX_QLEN) return false;
    const int d = qlen > tlen ? qlen - tlen : tlen - qlen;
    if (d > w) return false;
    const int mnl = qlen < tlen ? qlen : tlen;
    const int wl = band_left(w, tlen), wr = band_right(w, qlen), wm = wl > wr ? wl : wr;
    if (wm > MAX_BAND) return false;
    if ((long long)r.mn * (mnl + 12) + 3LL * r.oe + (long long)r.e * (wm + 12) > LOW_LIMIT) return false;
    return (long long)r.mx * (mnl + 12) <= HIGH_LIMIT;
}

// Shared memory of a thread (both its alignments): band slots {H, E} and a byte a query column.  Shared
// memory sets how many warps an SM holds (7 of 150 bp reads with 16-bit selectors, 8 with bytes; 4 and
// 5 of 250 bp), and rebuilding the selector costs one ALU instruction for four cells.
__host__ __device__ inline size_t thread_bytes(int wl, int wr, int qlen)
{
    return (size_t)slots(wl, wr) * 8 + (size_t)((sel_count(qlen, wl, wr) + 3) & ~3);
}

// Query column of both alignments as a byte: A's profile byte 0..3 in the low nibble (4: N), B's 4..7 in
// the high one (0: N).
__device__ __forceinline__ uint32_t column_code(uint32_t a, uint32_t b)
{
    return (a == 4u ? 4u : a & 3u) | (b == 4u ? 0u : (4u + (b & 3u)) << 4);
}
constexpr uint32_t PAD_COLUMN = 0x40u;

// The prmt selector of a column: per alignment its byte and the sign of it.
__device__ __forceinline__ uint32_t column_sel(uint32_t c) { return c * 0x11u + 0x8080u + (c & 0xf0u) * 0xffu; }

__device__ __forceinline__ uint32_t both(int v) { return ((uint32_t)v & 0xffffu) * 0x10001u; }

// Directions of eight steps as they gather: four steps a 16-bit lane, then the words.
struct Row {
    uint32_t f;         // F, tag 0
    uint32_t acc, acc0; // nibbles of the open and the closed four steps
};

struct TagGaps {
    uint32_t noe_del, noe_ins, ne_del, ne_ins;
    uint32_t k2, k4, k16, km1;
};

// One cell of each alignment: hd the diagonal's H (tag 0), e its E (tag 1), s2 the scores 4 s + 3.
// Returns H with tag 0 in h, E of the next row with tag 1 in en.
template <bool SYM>
__device__ __forceinline__ void cell(uint32_t hd, uint32_t e, uint32_t s2, const TagGaps &g, Row &r, uint32_t &h,
                                     uint32_t &en)
{
    constexpr uint32_t MIN2 = 0x80008000u;
    const uint32_t m = __viaddmax_s16x2(hd, s2, MIN2);
    const uint32_t ht = __vimax3_s16x2(m, e, r.f);
    const uint32_t mo = __viaddmax_s16x2(m, g.noe_del, MIN2);
    const uint32_t mi = SYM ? mo : __viaddmax_s16x2(m, g.noe_ins, MIN2);
    const uint32_t er = __viaddmax_s16x2(e, g.ne_del, mo);
    const uint32_t fr = __viaddmax_s16x2(r.f, g.ne_ins, mi);
    const uint32_t th = ht & 0x00030003u, te = er & 0x00020002u, tf = fr & 0x00020002u;
    r.f = fr & 0xfffcfffcu;
    h = th * g.km1 + ht;   // ht - th: lanes hold their own tags, no borrow between them
    en = te * g.km1 + er;  // 3 -> 1 (opened), 1 -> 1 (extended)
    r.acc = r.acc * g.k16 + (tf * g.k4 + (te * g.k2 + th));
}

// s2 with the query's N columns put right.
__device__ __forceinline__ uint32_t fix_n(uint32_t s2, uint32_t c, uint32_t n2)
{
    const uint32_t mk = ((c & 0x4u) ? 0xffffu : 0u) | ((c & 0x40u) ? 0u : 0xffff0000u);
    return (s2 & ~mk) | (n2 & mk);
}

// A thread's two alignments: whether they share a pass (equal bands, and the larger sizes still fit),
// and the sizes of the pass.
struct PairGeo {
    bool dual;
    int q, t, w, wl, wr;
};
__host__ __device__ inline PairGeo pair_geo(int q0, int t0, int w0, bool has1, int q1, int t1, int w1, const TagRule &r)
{
    PairGeo g;
    const int q = q0 > q1 ? q0 : q1, t = t0 > t1 ? t0 : t1;
    g.dual = !r.single && has1 && w0 == w1 && tag_ok(q, t, w0, r);
    g.q = g.dual ? q : q0;
    g.t = g.dual ? t : t0;
    g.w = w0;
    g.wl = band_left(g.w, g.t);
    g.wr = band_right(g.w, g.q);
    return g;
}

// The directions of sixty-four consecutive sorted alignments (a warp's pairs): how they lie; where is
// the running sum of the groups' bytes.
struct WarpGroup {
    uint32_t pos;       // first sorted position
    uint16_t count;     // alignments, at most 64
    uint16_t ng;        // groups of eight steps a row pair holds
};

// Two rows of both alignments at columns of steps [8 g0, 8 g1 + 8).  P: slot 0 of the thread's band
// buffer (stride TB), S: selectors at the column of step 8 g0.  LAST: the row pair holds an alignment's
// last row, whose H at its last column (step ca / cb, row ra / rb of the pair) is the score.
template <int TB, bool SYM, bool SLOW, bool LAST>
__device__ __forceinline__ void two_rows(uint2 *P, const uint8_t *S, int g0, int g1, const TagGaps &gp, uint32_t pa0,
                                         uint32_t pb0, uint32_t pa1, uint32_t pb1, uint32_t n0, uint32_t n1,
                                         uint4 *z, int ncomp, int comp, int ca, int ra, int cb, int rb, int &sa, int &sb)
{
    Row r0, r1;
    r0.f = r1.f = both(4 * NEG);
    uint32_t hp = both(4 * NEG);  // H of the first row at the column before
    uint2 *X = P + (ptrdiff_t)(8 * g0) * TB;
    uint32_t xh = X[0].x;
    for (int g = g0; g <= g1; ++g) {
        // a group's loads together, ahead of its stores (to the compiler they may alias, so it orders
        // each load behind the stores before it: one shared-memory latency a step otherwise)
        uint2 xv[8];
        uint32_t sv0[8], sv1[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) xv[u] = X[(u + 1) * TB];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t c = S[u * TB];
            sv0[u] = c;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t c = sv0[u], sel = column_sel(c);
            sv0[u] = prmt(pa0, pb0, sel);
            sv1[u] = prmt(pa1, pb1, sel);
            if (SLOW) {
                sv0[u] = fix_n(sv0[u], c, n0);
                sv1[u] = fix_n(sv1[u], c, n1);
            }
        }
        r0.acc = r1.acc = 0u;
        r0.acc0 = r1.acc0 = 0u;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            uint32_t h0, h1, e0, e1;
            cell<SYM>(xh, xv[u].y, sv0[u], gp, r0, h0, e0);
            cell<SYM>(hp, e0, sv1[u], gp, r1, h1, e1);
            X[(u - 1) * TB] = make_uint2(h1, e1);
            hp = h0;
            xh = xv[u].x;
            if (LAST) {
                const int st = 8 * g + u;
                if (st == ca) sa = (int)(int16_t)((ra ? h1 : h0) & 0xffffu) >> 2;
                if (st == cb) sb = (int)(rb ? h1 : h0) >> 18;
            }
            if (u == 3) {
                r0.acc0 = r0.acc;
                r1.acc0 = r1.acc;
                r0.acc = r1.acc = 0u;
            }
        }
        const uint32_t a0 = prmt(r0.acc0, r0.acc, 0x5410u), b0 = prmt(r0.acc0, r0.acc, 0x7632u);
        const uint32_t a1 = prmt(r1.acc0, r1.acc, 0x5410u), b1 = prmt(r1.acc0, r1.acc, 0x7632u);
        if (ncomp == 2) {
            z[(size_t)g * 32] = make_uint4(a0, b0, a1, b1);
        } else {  // one alignment in both lanes
            uint32_t *zw = reinterpret_cast<uint32_t *>(z + (size_t)g * 32) + comp;
            zw[0] = a0;
            zw[2] = a1;
        }
        X += 8 * TB;
        S += 8 * TB;
    }
}

// The DP of sorted alignments [start, start + count): a thread takes positions 2t and 2t + 1, or in
// single mode one position; group gbase + t / 32 holds their directions.  Where a pair does not match,
// a thread of the grid's first half takes the second one (the others of that half leave at once): one
// thread after the other doubled the latency of a small batch.  ncig[k] = done marks a finished alignment for the traceback.
// Measured (GB300, 500,000 reads of 100 / 150 / 250 bp through host buffers): the call 8.08 -> 4.30 ms
// against the predicate pair kernel; the grid's first half for the pairs that do not match: 14,000
// alignments 1.32 -> 0.84 ms, 50,000 1.45 -> 1.00, 200,000 2.03 -> 1.74, 500,000 3.76 -> 3.65.  About 40 instructions, 18 of them ALU, for a step's four cells;
// ALU pipe 43-57%, bound by the warps shared memory leaves (1.0 a scheduler at 250 bp, 1.7 at 150 bp).
template <int TB, bool SYM, typename JobT>
__global__ void __launch_bounds__(TB, 384 / TB)
tag_kernel(const uint8_t *__restrict__ seq, const JobT *__restrict__ jobs, const uint32_t *__restrict__ order,
           uint32_t start, uint32_t count, const __grid_constant__ Scoring sc, const __grid_constant__ TagRule rule,
           int max_slots, int max_sel, const WarpGroup *__restrict__ wgroups, const uint64_t *__restrict__ zoffs,
           uint32_t gbase, uint8_t *__restrict__ z,
           int32_t *__restrict__ score_out, int32_t *__restrict__ ncig_out, int done, uint32_t range_flag,
           uint32_t *__restrict__ err, unsigned long long *__restrict__ cells_total)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t pt[8], nt[8];  // per target code: scores 4 s + 3 of query codes 0..3, and of N
    if (threadIdx.x < 8) {
        uint32_t v = 0;
        const int t = threadIdx.x;
        for (int q = 0; q < 4; ++q) {
            const int sv = (int)(int8_t)((sc.prof[t][0] >> (8 * q)) & 0xffu);
            v |= ((uint32_t)(4 * sv + 3) & 0xffu) << (8 * q);
        }
        pt[t] = v;
        nt[t] = (uint32_t)(4 * (int)(int8_t)(sc.prof[t][1] & 0xffu) + 3) & 0xffffu;
    }
    __syncthreads();
    const bool rest = !rule.single && blockIdx.x < gridDim.x / 2;
    const uint32_t blk = rule.single || rest ? blockIdx.x : blockIdx.x - gridDim.x / 2;
    const uint32_t tid = blk * TB + threadIdx.x, t = rule.single ? tid >> 1 : tid;
    if ((rule.single ? tid : 2 * t) >= count) return;
    uint2 *P = reinterpret_cast<uint2 *>(smem_raw) + TB + threadIdx.x;  // slot 0; slot -1 takes garbage
    uint8_t *S0 = reinterpret_cast<uint8_t *>(reinterpret_cast<uint2 *>(smem_raw) + (size_t)max_slots * TB) + threadIdx.x;
    const bool has1 = 2 * t + 1 < count;
    const uint32_t k0 = order[start + 2 * t], k1 = has1 ? order[start + 2 * t + 1] : k0;
    const JobT A0 = jobs[k0], B0 = jobs[k1];
    const PairGeo first = pair_geo(A0.qlen, A0.tlen, A0.w, has1, B0.qlen, B0.tlen, B0.w, rule);
    if (rest && (first.dual || !has1)) return;
    const WarpGroup wg = wgroups[gbase + (t >> 5)];
    uint4 *zw = reinterpret_cast<uint4 *>(z + (zoffs[gbase + (t >> 5)] - zoffs[0])) + (t & 31u);
    TagGaps gp;
    gp.noe_del = both(-4 * (sc.o_del + sc.e_del));
    gp.noe_ins = both(-4 * (sc.o_ins + sc.e_ins));
    gp.ne_del = both(-4 * sc.e_del);
    gp.ne_ins = both(-4 * sc.e_ins);
    gp.k2 = rule.k2;
    gp.k4 = rule.k4;
    gp.k16 = rule.k16;
    gp.km1 = rule.km1;
    unsigned long long ncells = 0;
    bool bad = false;
    const int pass = rule.single ? (int)(tid & 1u) : (int)rest;
    const uint32_t ka = pass ? k1 : k0, kb = first.dual ? k1 : ka;
    const JobT A = pass ? B0 : A0, B = first.dual ? B0 : A;
    const PairGeo g = first.dual ? first : pair_geo(A.qlen, A.tlen, A.w, false, A.qlen, A.tlen, A.w, rule);
    const int Q = g.q, T = g.t, wl = g.wl, wr = g.wr, SN = steps(wl, wr);
    if (slots(wl, wr) > max_slots || sel_count(Q, wl, wr) > max_sel || groups(wl, wr) > wg.ng) {
        atomicOr(err, range_flag);  // the host sizes these from the launch's alignments
        ncig_out[ka] = 0;
        ncig_out[kb] = 0;
        return;
    }
    const uint8_t *qa = seq + A.q_off, *qb = seq + B.q_off;
    bool slow = false;
    for (int x = 0; x < LEFT_PAD; ++x) S0[x * TB] = (uint8_t)PAD_COLUMN;
    for (int j = 0; j < Q + 16; j += 16) {
        uint32_t va[4], vb[4];
        load16(qa, A.qlen, j, va);
        load16(qb, B.qlen, j, vb);
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const uint32_t ca = (va[u >> 2] >> (8 * (u & 3))) & 0xffu, cb = (vb[u >> 2] >> (8 * (u & 3))) & 0xffu;
            bad |= ca >= (uint32_t)sc.m || cb >= (uint32_t)sc.m;
            slow |= ca == 4u || cb == 4u;
            if (j + u < Q + 16) S0[(LEFT_PAD + j + u) * TB] = (uint8_t)column_code(ca, cb);
        }
    }
    // before row 0: H(-1, j - 1) and E(0, j - 1) at slot wl + j; column -1's E opens the leading
    // deletion
    const uint32_t neg_h = both(4 * NEG), neg_e = both(4 * NEG + 1);
    const int ns = slots(wl, wr);
    for (int b = -1; b < ns - 1; ++b) {
        const int j = b - wl;
        uint2 v = make_uint2(neg_h, neg_e);
        if (j == 0) v = make_uint2(0u, both(-4 * (sc.o_del + sc.e_del) + 1));
        else if (j > 0 && j <= wr) v.x = both(-4 * (sc.o_ins + sc.e_ins * j));
        P[(ptrdiff_t)b * TB] = v;
    }
    TargetStream ta, tb;
    ta.init(seq + A.t_off, A.tlen);
    tb.init(seq + B.t_off, B.tlen);
    int sa = 0, sb = 0;
    for (int i = 0; i < T; i += 2) {
        uint32_t c[4];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            c[2 * x] = i + x < A.tlen ? ta.next() : 0u;
            c[2 * x + 1] = i + x < B.tlen ? tb.next() : 0u;
            bad |= c[2 * x] >= (uint32_t)sc.m || c[2 * x + 1] >= (uint32_t)sc.m;
        }
        const uint32_t pa0 = pt[c[0] & 7u], pb0 = pt[c[1] & 7u], pa1 = pt[c[2] & 7u], pb1 = pt[c[3] & 7u];
        const int g0 = (wl - i - 1 > 0 ? wl - i - 1 : 0) >> 3;
        const int last = min(SN - 1, Q - 1 - i + wl);
        const int g1 = last >> 3;
        const uint8_t *S = S0 + (ptrdiff_t)(8 * g0 + i - wl + LEFT_PAD) * TB;
        uint4 *zr = zw + (size_t)(i >> 1) * wg.ng * 32;
        const int ncomp = first.dual ? 2 : 1;
        const bool fa = (A.tlen - 1) >> 1 == i >> 1, fb = (B.tlen - 1) >> 1 == i >> 1;
        const int ca = fa ? A.qlen - 1 - i + wl : -1, cb = fb ? B.qlen - 1 - i + wl : -1;
        const int ra = (A.tlen - 1) & 1, rb = (B.tlen - 1) & 1;
        if (slow) {
            const uint32_t n0 = nt[c[0] & 7u] | (nt[c[1] & 7u] << 16), n1 = nt[c[2] & 7u] | (nt[c[3] & 7u] << 16);
            two_rows<TB, SYM, true, true>(P, S, g0, g1, gp, pa0, pb0, pa1, pb1, n0, n1, zr, ncomp, pass, ca, ra, cb,
                                          rb, sa, sb);
        } else if (fa || fb) {
            two_rows<TB, SYM, false, true>(P, S, g0, g1, gp, pa0, pb0, pa1, pb1, 0u, 0u, zr, ncomp, pass, ca, ra, cb,
                                           rb, sa, sb);
        } else {
            two_rows<TB, SYM, false, false>(P, S, g0, g1, gp, pa0, pb0, pa1, pb1, 0u, 0u, zr, ncomp, pass, -1, 0, -1,
                                            0, sa, sb);
        }
        // nothing right of the band may pass an E back into it
        P[(ptrdiff_t)(wl + wr + 1) * TB] = make_uint2(neg_h, neg_e);
        P[(ptrdiff_t)(wl + wr + 2) * TB] = make_uint2(neg_h, neg_e);
    }
    score_out[ka] = sa;
    ncig_out[ka] = done;
    if (first.dual) {
        score_out[kb] = sb;
        ncig_out[kb] = done;
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        if (x == 1 && !first.dual) break;
        // sum over rows of min(i + w + 1, qlen) - max(i - w, 0)
        const long long q = x ? B.qlen : A.qlen, tl = x ? B.tlen : A.tlen, w = g.w;
        const long long n1 = q - w < 0 ? 0 : (q - w < tl ? q - w : tl), lft = tl - 1 - w > 0 ? tl - 1 - w : 0;
        ncells += (unsigned long long)(n1 * (w + 1) + n1 * (n1 - 1) / 2 + (tl - n1) * q - lft * (lft + 1) / 2);
    }
    if (bad) atomicOr(err, ERR_BASE);
    if (ncells) atomicAdd(cells_total, ncells);
}

}  // namespace gtag
}  // namespace bwacuda
