"""The band kernel's row storage (csrc/ext_band.cuh) on the CPU: its window, its lanes' chunks of column pairs
and what each row reads, masks and writes, restated and checked against ksw_extend2
(crates/bwa-extend/src/sw.rs:203-493, the oracle).

The kernel keeps a job's row in PAIRS column pairs from column `base` on, behind PAD zero pairs, and moves the
window right by 64 columns before a row whose band has left the first ones.  A row's pairs p0 .. plast are cut
into L chunks of K pairs, the last one ending at plast, so that the leading chunks reach up to L K pairs left of
plast: pairs between p0 - K and p0 hold columns left of the band, and a chunk left of p0 altogether is moved to
the zeros in front of the row.  The restatement runs the recurrence on that storage and checks, row by row, that
every pair lies in the storage, that everything left of the band's first column is zero before and after, and, at
the end, that the result is the oracle's: a column that entered the window with anything but its row -1 value, or
a stale cell lost by a move, would change it."""
import numpy as np
import pytest

import oracle
from test_slide_window_cpu import _cases

WC, SLIDE = 272, 64
PAIRS = WC // 2 + 2
KMAX = {8: 17, 16: 9, 32: 5}


def band_takes(qlen, w):
    return qlen + 4 <= WC or 2 * w + 5 + SLIDE <= WC


def chunk_len(lanes, need):
    return 17 if lanes == 8 and need > 13 else need | 1


def band_extend(q, t, h0, mat, m, o_del, e_del, o_ins, e_ins, w, end_bonus, zdrop, lanes, rng, early=0):
    """The kernel's result for one job, and how often its window moved (early: columns too soon)."""
    q, t, qlen = np.asarray(q), np.asarray(t), len(q)
    mat = np.asarray(mat).reshape(m, m).astype(np.int64)
    oe_del, oe_ins = o_del + e_del, o_ins + e_ins
    w = oracle.clamp_band(w, qlen, int(mat.max()), end_bonus, o_ins, e_ins, o_del, e_del)
    assert band_takes(qlen, w)
    pad = (KMAX[lanes] + 3) // 4 * 4

    def row_minus1(c):
        if c > qlen:
            return 0
        return h0 if c == 0 else max(h0 - oe_ins - (c - 1) * e_ins, 0)

    def fill(lo, hi, base):  # columns base + lo .. base + hi as they enter the window
        X[off + lo:off + hi] = [row_minus1(base + c) for c in range(lo, hi)]
        Y[off + lo:off + hi] = 0
        S[off + lo:off + hi] = [q[base + c] if base + c < qlen else 0 for c in range(lo, hi)]

    off = 2 * pad  # array index of the window's first column
    X, Y, S = (np.zeros(off + 2 * PAIRS, np.int64) for _ in range(3))
    base, moved = 0, 0
    fill(0, 2 * PAIRS, 0)
    moves = qlen + 4 > WC
    best, best_i, best_j, best_ie, gscore, max_off = h0, -1, -1, -1, -1, 0
    beg, end = 0, qlen
    for i in range(len(t)):
        if moves and i - w - 1 - base >= SLIDE - early:
            for a in (X, Y, S):
                a[off:-SLIDE] = a[off + SLIDE:].copy()
            fill(2 * PAIRS - SLIDE, 2 * PAIRS, base + SLIDE)
            base += SLIDE
            moved += 1
        if beg < i - w:  # the band drops one column a row
            assert i - w == beg + 1 and beg >= base
            X[off + beg - base] = Y[off + beg - base] = 0
            beg = i - w
        end = min(end, i + w + 1, qlen)
        h1 = max(h0 - (o_del + e_del * (i + 1)), 0) if beg == 0 else 0
        rb, re = beg - base, end - base
        assert rb >= 0 and re < 2 * PAIRS  # every column of the row and the sentinel lie in the window
        hl, rmax, mj = h1, 0, -1
        if end > beg:
            p0, plast = rb >> 1, (re - 1) >> 1
            need = -(-(plast - p0 + 1) // lanes)
            K = chunk_len(lanes, need)
            if rng.random() < 0.3:  # a longer row beside this one sets the warp's chunks
                K = chunk_len(lanes, min(KMAX[lanes], need + int(rng.integers(0, 4))))
            assert K <= KMAX[lanes]
            used = [k for k in range(lanes) if plast + 1 - (lanes - k) * K + K > p0]
            assert K <= pad  # a lane with nothing of the row stays in the zeros in front
            first = plast + 1 - (lanes - used[0]) * K
            assert first >= -pad and first > p0 - K
            lo, hi = off + 2 * first, off + 2 * (plast + 1)
            assert hi <= len(X)
            assert not X[lo:off + rb].any() and not Y[lo:off + rb].any()  # left of the band
            hd, e = X[lo:hi].copy(), Y[lo:hi].copy()
            if re & 1:  # column end, in the last pair, is masked
                hd[-1] = e[-1] = 0
            M = np.where(hd != 0, hd + mat[t[i], S[lo:hi]], 0)
            ti, td = np.maximum(M - oe_ins, 0), np.maximum(M - oe_del, 0)
            Y[lo:hi] = np.maximum(e - e_del, td)
            idx = np.arange(hi - lo)
            F = np.zeros(hi - lo, np.int64)  # f = max(f - e_ins, max(M - oe_ins, 0)) from column to column
            F[1:] = np.maximum(np.maximum.accumulate(ti + (idx + 1) * e_ins)[:-1] - idx[1:] * e_ins, 0)
            H = np.maximum(np.maximum(M, e), F)
            X[lo], X[lo + 1:hi] = 0, H[:-1]
            if re & 1:
                H[-1] = 0  # and out of the maximum
            assert not X[lo:off + rb].any() and not Y[lo:off + rb].any()
            hl = int(H[off + re - 1 - lo])
            if not re & 1:
                X[off + re], Y[off + re] = hl, 0
            rmax = int(H.max())
            if rmax > 0:  # the later column on ties
                mj = int(np.nonzero(H == rmax)[0][-1]) + lo - off + base
                assert beg <= mj < end
        if beg == 0:
            X[off] = h1
        if max(beg, end) == qlen and gscore <= hl:
            best_ie, gscore = i, hl
        if rmax == 0:
            break
        if rmax > best:
            best, best_i, best_j = rmax, i, mj
            max_off = max(max_off, abs(mj - i))
        elif zdrop > 0:
            if i - best_i > mj - best_j:
                if best - rmax - ((i - best_i) - (mj - best_j)) * e_del > zdrop:
                    break
            elif best - rmax - ((mj - best_j) - (i - best_i)) * e_ins > zdrop:
                break
        live = (X[off + rb:off + re + 1] | Y[off + rb:off + re + 1]) != 0
        ahead, behind = np.nonzero(live[:-1])[0], np.nonzero(live)[0]
        lo_c = beg + int(ahead[0]) if len(ahead) else end
        hi_c = max(beg + int(behind[-1]) if len(behind) else beg - 1, lo_c - 1)
        beg, end = lo_c, min(hi_c + 2, qlen)
    return (best, best_j + 1, best_i + 1, best_ie + 1, gscore, max_off), moved


def _check(cases, lanes, mat, m, gaps, end_bonus, h0_scale=1, early=0):
    o_del, e_del, o_ins, e_ins = gaps
    rng = np.random.default_rng(lanes)
    moved = 0
    for q, t, h0, w, zdrop in cases:
        h0 *= h0_scale
        got, k = band_extend(q, t, h0, mat, m, o_del, e_del, o_ins, e_ins, w, end_bonus, zdrop, lanes, rng, early)
        want = oracle.extend2(np.array(q, np.uint8), np.array(t, np.uint8), h0, mat, o_del, e_del, o_ins, e_ins, w,
                              end_bonus, zdrop)
        assert got == tuple(want), (got, want, len(q), len(t), h0, w, zdrop)
        moved += k
    return moved


def _long_cases(seed, n):
    """Queries longer than the window, its widest bands among them."""
    rng = np.random.default_rng(seed)
    for _ in range(n):
        ql = int(rng.integers(269, 900))
        t = rng.integers(0, 4, ql + int(rng.integers(-40, 120)))
        q = np.resize(t, ql).copy()
        q[rng.random(ql) < rng.choice([0.01, 0.05])] ^= 1
        cut = int(rng.integers(0, ql))
        if rng.random() < 0.5:  # an indel
            q = np.concatenate([q[:cut], rng.integers(0, 4, int(rng.integers(1, 30))), q[cut:]])[:ql]
        yield q.tolist(), t.tolist(), int(rng.choice([5, 60, 400])), int(rng.choice([1, 40, 99, 100, 101])), 100


@pytest.mark.parametrize("lanes", [8, 16, 32])
def test_rows_on_the_window(lanes):
    mat = oracle.scmat()
    assert _check(_cases(100 + lanes, 120), lanes, mat, 5, (6, 1, 6, 1), 5) > 0
    assert _check(_long_cases(200 + lanes, 40), lanes, mat, 5, (6, 1, 6, 1), 5) > 100
    _check(_cases(7, 60), lanes, oracle.scmat(2, 3), 5, (5, 2, 4, 3), 0, h0_scale=3)


def test_a_wrong_move_is_noticed():
    """The check itself: a window that moves while the band still holds one of its first columns."""
    with pytest.raises(AssertionError):
        _check(_long_cases(300, 20), 8, oracle.scmat(), 5, (6, 1, 6, 1), 5, early=1)
