"""ksw_global2's tagged kernel (csrc/global_tag.cuh: two alignments a thread, directions in the values'
low bits) at the edges of what it takes, against the oracle, bit-exact on the score and every CIGAR
run: bands that just hold the corner, one-base queries and targets, group and row-pair remainders,
neighbours of equal bands and different lengths, N bases, the largest bands and scorings on both sides
of its limits."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture
def gctx(ctx):
    ctx.set_option(B.OPT_HOST_GATHER, B.GATHER_DEVICE)
    try:
        ctx.ksw_global2_batch(B.JobSet.from_lists([[0, 1]], [[0, 1]], w=[3]))
    except B.BwaCudaError as e:
        ctx.set_option(B.OPT_HOST_GATHER, B.GATHER_AUTO)
        assert e.code == B.EUNSUPPORTED
        pytest.skip("device cannot read pageable host memory")
    yield ctx
    ctx.set_option(B.OPT_HOST_GATHER, B.GATHER_AUTO)


def _check(ctx, js, mat=None, o_del=6, e_del=1, o_ins=6, e_ins=1):
    mat = oracle.scmat() if mat is None else mat
    sc, offs, words = ctx.ksw_global2_batch(js, mat, o_del, e_del, o_ins, e_ins)
    wsc, woffs, wwords = oracle.global2_batch(js, mat, o_del, e_del, o_ins, e_ins)
    bad = np.nonzero(sc != wsc)[0]
    assert len(bad) == 0, (f"{len(bad)} scores differ, first job {bad[0]} qlen={js.qlen[bad[0]]} "
                           f"tlen={js.tlen[bad[0]]} w={js.w[bad[0]]}: {sc[bad[0]]} vs {wsc[bad[0]]}")
    assert np.array_equal(offs, woffs)
    assert np.array_equal(words, wwords)


# batches of fewer alignments than a warp per SM run one a thread, larger ones in pairs
def _pairs(rng, lens, diffs, ws, n, n_rate=0.0, sub=0.03):
    qs, ts, wl = [], [], []
    for k in range(n):
        ql = int(lens[k % len(lens)])
        tl = max(1, ql + int(rng.choice(diffs)))
        t = rng.integers(0, 4, tl).astype(np.uint8)
        q = rng.integers(0, 4, ql).astype(np.uint8)
        ln = min(ql, tl)
        if k % 5:
            q[:ln] = t[:ln]
            q[:ln][rng.random(ln) < sub] ^= 1
            for _ in range(int(rng.integers(0, 4))):  # indels that keep the length
                p = int(rng.integers(0, ql))
                q = (np.insert(q, p, int(rng.integers(0, 4)))[:ql] if rng.random() < 0.5
                     else np.append(np.delete(q, p), int(rng.integers(0, 4))))
        q = q.astype(np.uint8)
        if n_rate:
            q[rng.random(ql) < n_rate] = 4
            t[rng.random(tl) < n_rate] = 4
        qs.append(q)
        ts.append(t)
        wl.append(abs(tl - ql) + int(rng.choice(ws)))
    return B.JobSet.from_lists(qs, ts, w=wl)


@pytest.mark.parametrize("n", [1, 65, 3000, 20000])
def test_short_and_remainder_lengths(gctx, n):
    rng = np.random.default_rng(1)
    _check(gctx, _pairs(rng, (1, 2, 3, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 64, 65), (-6, -2, -1, 0, 0, 1, 2, 7),
                        (0, 1, 2, 3, 7, 8, 30, 100), n))


@pytest.mark.parametrize("n", [1500, 9001])
def test_read_lengths_with_n(gctx, n):
    rng = np.random.default_rng(2)
    _check(gctx, _pairs(rng, (100, 101, 150, 151, 250), (-3, -1, 0, 0, 0, 2, 5), (0, 1, 3, 20, 40), n, n_rate=0.002))


@pytest.mark.parametrize("n", [520, 6000])
def test_largest_bands_and_lengths(gctx, n):
    rng = np.random.default_rng(3)
    _check(gctx, _pairs(rng, (126, 127, 128, 129, 130, 131, 200, 300, 500, 640, 641, 750), (-5, 0, 4),
                        (60, 110, 119, 123, 124, 125, 126, 127, 128, 129, 200), n))


def test_equal_bands_of_different_lengths(gctx):
    """One band for every job: neighbours of different lengths share a thread."""
    rng = np.random.default_rng(4)
    js = _pairs(rng, tuple(range(20, 60)), (-4, -1, 0, 0, 3), (0,), 8000)
    js.w = np.full(len(js), 9, np.int32)
    _check(gctx, js)


def _mat(a, b, n):
    m = np.full(25, n, dtype=np.int8)
    for r in range(4):
        for c in range(4):
            m[r * 5 + c] = a if r == c else -b
    return m


@pytest.mark.parametrize("mat,gaps", [
    (_mat(1, 4, -1), (5, 2, 8, 1)), (_mat(2, 3, 0), (5, 2, 5, 2)), (_mat(31, 31, -31), (1, 1, 1, 1)),
    (_mat(32, 4, -1), (6, 1, 6, 1)), (_mat(1, 32, -1), (6, 1, 6, 1)), (_mat(1, 4, 1), (0, 1, 0, 1)),
    (_mat(5, 4, -3), (40, 20, 59, 1)), (_mat(1, 4, -1), (41, 20, 60, 1)), (_mat(1, 4, -1), (100, 3, 90, 5))])
def test_scorings_on_both_sides_of_the_limits(gctx, mat, gaps):
    rng = np.random.default_rng(5)
    js = _pairs(rng, (1, 8, 40, 100, 150, 260), (-5, -1, 0, 0, 2, 6), (0, 2, 10, 40), 6000, n_rate=0.002)
    _check(gctx, js, mat, *gaps)


def test_random_matrix(gctx):
    rng = np.random.default_rng(6)
    mat = rng.integers(-31, 32, 25).astype(np.int8)
    _check(gctx, _pairs(rng, (9, 50, 120), (-3, 0, 3), (0, 5, 20), 600, n_rate=0.01), mat, 3, 2, 4, 1)


def test_corner_outside_the_band_next_to_tagged_jobs(gctx):
    rng = np.random.default_rng(7)
    js = _pairs(rng, (10, 60, 150), (-20, -3, 0, 0, 15), (0, 3, 12), 1200)
    cut = np.arange(len(js)) % 4 == 0
    js.w = np.where(cut & (np.abs(js.qlen - js.tlen) > 0), np.abs(js.qlen - js.tlen) - 1, js.w).astype(np.int32)
    try:
        _check(gctx, js)
    except B.BwaCudaError as e:  # the reference's own traceback leaves its matrix on such a job
        assert e.code == B.EUNSUPPORTED
        keep = ~cut | (js.qlen == js.tlen)
        _check(gctx, js.take(np.nonzero(keep)[0]))


def test_chunks(gctx):
    gctx.set_option(B.OPT_CHUNK_JOBS, 300)
    try:
        _check(gctx, B.synth_global(5003, seed=8))
    finally:
        gctx.set_option(B.OPT_CHUNK_JOBS, 1 << 20)


def test_invalid_base(gctx):
    js = B.synth_global(500, seed=9)
    js.seq[js.t_off[123] + 7] = 5
    with pytest.raises(B.BwaCudaError) as e:
        gctx.ksw_global2_batch(js)
    assert e.value.code == B.EBASE
    _check(gctx, B.synth_global(500, seed=9))
