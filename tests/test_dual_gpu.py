"""The 8-bit buckets of large batches, two jobs a thread (csrc/ext_dual.cuh), against the oracle, bit-exact
on every field: neighbours of different lengths, bands, seed scores and ends, values up to the class's
limit, queries with N (kept from this kernel by the sort), odd counts and other scorings."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu

N_JOBS = 152 * 5000 + 1  # the least batch that runs this way on 152 SMs, and odd


def _jobs(n, seed, sub=0.02, n_rate=0.0005, qmax=128, wmax=100):
    """Short jobs laid out flat: queries copied from their targets with substitutions, a share with a
    shifted copy (an indel), a share unrelated; seed scores up to the class's limit of 255."""
    rng = np.random.default_rng(seed)
    edges = np.array([0, 1, 2, 3, 4, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128])
    ql = np.where(rng.random(n) < 0.5, rng.choice(edges, n), rng.integers(1, qmax + 1, n)).clip(0, qmax)
    tl = np.maximum(0, ql + rng.integers(-10, 12, n))
    tl = np.where(rng.random(n) < 0.02, rng.integers(0, 3, n), tl)
    sizes = np.empty(2 * n, np.int64)
    sizes[0::2], sizes[1::2] = ql, tl
    offs = np.zeros(2 * n + 1, np.int64)
    np.cumsum(sizes, out=offs[1:])
    qo, to = offs[0:-1:2].copy(), offs[1:-1:2].copy()
    seq = rng.integers(0, 4, offs[-1]).astype(np.uint8)
    job = np.repeat(np.arange(n), ql)
    j = np.arange(len(job)) - np.repeat(np.cumsum(ql) - ql, ql)
    kind = rng.random(n)
    shift = np.where((kind > 0.6) & (kind < 0.75), rng.integers(1, 4, n), 0)
    src = j + np.where(j > ql[job] // 2, shift[job], 0)
    ok = (src < tl[job]) & (kind[job] < 0.9)
    seq[qo[job[ok]] + j[ok]] = seq[to[job[ok]] + src[ok]]
    hit = rng.random(len(job)) < sub
    seq[qo[job[hit]] + j[hit]] = (seq[qo[job[hit]] + j[hit]] + rng.integers(1, 4, int(hit.sum()))) & 3
    if n_rate:
        seq[rng.random(len(seq)) < n_rate] = 4
    top = 255 - np.minimum(ql, tl)
    h0 = np.where(rng.random(n) < 0.3, top, rng.integers(1, np.maximum(2, top + 1)))
    h0 = np.where(rng.random(n) < 0.1, rng.integers(1, 20, n), h0)
    w = rng.choice([0, 1, 3, 10, 50, wmax], n)
    return B.JobSet(seq, qo, to, ql.astype(np.int32), tl.astype(np.int32), h0.astype(np.int32), w.astype(np.int32))


def _device(ctx, js, **kw):
    import torch

    d_seq = torch.from_numpy(js.seq).cuda()
    d_jobs = torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda()
    d_out = torch.zeros(len(js) * 24, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    sc = ctx.scoring(**{k: v for k, v in kw.items() if k in ("o_del", "e_del", "o_ins", "e_ins", "mat")})
    ctx.extend_device(d_seq.data_ptr(), d_jobs.data_ptr(), len(js), d_out.data_ptr(), sc,
                      end_bonus=kw.get("end_bonus", 5), zdrop=kw.get("zdrop", 100))
    ctx.sync()
    return d_out.cpu().numpy().view(B.EXT_RES)


@pytest.mark.parametrize("kw", [dict(), dict(o_del=4, e_del=2, o_ins=7, e_ins=1, zdrop=20),
                                dict(o_del=0, e_del=1, o_ins=0, e_ins=1, zdrop=0)])
def test_edges(kw):
    js = _jobs(N_JOBS, seed=3)
    want, cells = oracle.extend_batch(js, **kw)
    with B.Context(0) as ctx:
        got = _device(ctx, js, **kw)
        bad = np.nonzero(got != want)[0]
        assert len(bad) == 0, (f"{len(bad)} differ; first job {bad[0]} qlen={js.qlen[bad[0]]} tlen={js.tlen[bad[0]]} "
                               f"h0={js.h0[bad[0]]} w={js.w[bad[0]]}: {got[bad[0]]} vs {want[bad[0]]}")
        assert ctx.stats()["ext_cells"] == cells


def test_match_score_two_and_random_matrix():
    js = _jobs(N_JOBS, seed=5, qmax=60)
    js.h0 = np.minimum(js.h0, 255 - 2 * np.minimum(js.qlen, js.tlen)).clip(1).astype(np.int32)
    mats = [oracle.scmat(2, 3), np.random.default_rng(1).integers(-6, 3, 25).astype(np.int8)]
    with B.Context(0) as ctx:
        for mat in mats:
            want, _ = oracle.extend_batch(js, mat)
            assert np.array_equal(_device(ctx, js, mat=mat), want)


def test_read_pairs_host_call():
    js = B.synth_ext(2, 1_900_001, seed=12)  # the last chunk of the call runs two jobs a thread
    want, cells = oracle.extend_batch(js)
    with B.Context(0) as ctx:
        assert np.array_equal(ctx.extend_batch(js), want)
        assert ctx.stats()["ext_cells"] == cells
