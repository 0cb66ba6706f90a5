"""Base codes past the scoring's alphabet fail a call whatever its size: alphabets of one to five letters,
a bad code in a query or in a target, through every extension route (a warp per job, lane groups, length
buckets, two jobs a thread)."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu


def _jobs(n, m, seed):
    """Short jobs of m letters, most queries copies of their targets with substitutions."""
    rng = np.random.default_rng(seed)
    ql = rng.integers(1, 25, n)
    tl = ql + rng.integers(1, 9, n)
    sizes = np.empty(2 * n, np.int64)
    sizes[0::2], sizes[1::2] = ql, tl
    offs = np.zeros(2 * n + 1, np.int64)
    np.cumsum(sizes, out=offs[1:])
    qo, to = offs[0:-1:2].copy(), offs[1:-1:2].copy()
    seq = rng.integers(0, m, offs[-1]).astype(np.uint8)
    job = np.repeat(np.arange(n), ql)
    j = np.arange(len(job)) - np.repeat(np.cumsum(ql) - ql, ql)
    copy = rng.random(len(job)) < 0.97
    seq[qo[job[copy]] + j[copy]] = seq[to[job[copy]] + j[copy]]
    h0 = rng.integers(1, 60, n)
    return B.JobSet(seq, qo, to, ql.astype(np.int32), tl.astype(np.int32), h0.astype(np.int32),
                    np.full(n, 100, np.int32))


def _mat(m):
    mat = np.full((m, m), -4, np.int8)
    np.fill_diagonal(mat, 1)
    return mat.reshape(-1)


def _device(ctx, js, mat, m):
    import torch

    d_seq = torch.from_numpy(js.seq).cuda()
    d_jobs = torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda()
    d_out = torch.zeros(len(js) * 24, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ctx.extend_device(d_seq.data_ptr(), d_jobs.data_ptr(), len(js), d_out.data_ptr(), ctx.scoring(mat, m=m))
    ctx.sync()  # reports bad codes
    return d_out.cpu().numpy().view(B.EXT_RES)


# lane groups, length buckets, two jobs a thread (from 5,000 jobs per SM of 152)
@pytest.mark.parametrize("n", [3000, 60000, 152 * 5000 + 1])
@pytest.mark.parametrize("m", [1, 2, 3, 4])
def test_codes_past_the_alphabet(m, n):
    js = _jobs(n, m, seed=m)
    mat = _mat(m)
    want, _ = oracle.extend_batch(js, mat, m=m)
    k = n // 2
    one = js.take([k])  # by itself: a warp straight from the caller's arrays
    with B.Context(0) as ctx:
        assert np.array_equal(_device(ctx, js, mat, m), want)
        assert np.array_equal(ctx.extend_batch(one, mat, m=m), want[k:k + 1])
        for at in (js.q_off[k], js.t_off[k]):  # the target's first base is read by every job
            keep = js.seq[at]
            js.seq[at] = m
            for call in (lambda: _device(ctx, js, mat, m), lambda: ctx.extend_batch(js.take([k]), mat, m=m)):
                with pytest.raises(B.BwaCudaError) as e:
                    call()
                assert e.value.code == B.EBASE
            js.seq[at] = keep
        assert np.array_equal(_device(ctx, js, mat, m), want)
