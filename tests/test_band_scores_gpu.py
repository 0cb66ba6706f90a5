"""The band kernel (csrc/ext_band.cuh) at the ends of its scores and gap costs: matrix entries down to -128,
where a score without its sign reads as one near -32768, with gap costs up to the 16-bit lanes' limit of
16384, for every number of lanes a job, against the oracle."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu


def _jobs(n, seed, w=None):
    rng = np.random.default_rng(seed)
    qs, ts = [], []
    for k in range(n):
        ql = int(rng.integers(1, 200))
        t = rng.integers(0, 4, ql + int(rng.integers(0, 60))).astype(np.uint8)
        q = t[:ql].copy()
        q[rng.random(ql) < 0.1] ^= 1
        qs.append(q)
        ts.append(t)
    ws = rng.choice([0, 1, 5, 40, 100, 101], n) if w is None else np.full(n, w)
    return B.JobSet.from_lists(qs, ts, rng.integers(1, 200, n), ws)


def _matrix(low, seed):
    rng = np.random.default_rng(seed)
    mat = rng.integers(low, 30, (5, 5)).astype(np.int8)
    mat[rng.random((5, 5)) < 0.3] = low
    np.fill_diagonal(mat[:4, :4], rng.choice([low, 3, 9], 4))
    mat[3, 3] = 7
    return mat.reshape(-1)


@pytest.mark.parametrize("gaps", [(6, 1, 129, 1), (4656, 1, 11937, 132), (16383, 1, 16000, 384), (0, 16384, 16383, 1)])
@pytest.mark.parametrize("low", [-65, -100, -128])
def test_large_costs(low, gaps):
    import torch

    with B.Context(0) as ctx:
        for n in (1, 40, 900, 2000, 4500):  # 32 lanes a job, 16 and 8
            mat = _matrix(low, n)
            js = _jobs(n, n - low)
            want, _ = oracle.extend_batch(js, mat, *gaps)
            bufs = [torch.from_numpy(js.seq).cuda(), torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda(),
                    torch.zeros(n * 24, dtype=torch.uint8, device="cuda")]
            torch.cuda.synchronize()
            ctx.extend_device(bufs[0].data_ptr(), bufs[1].data_ptr(), n, bufs[2].data_ptr(), ctx.scoring(mat, *gaps))
            ctx.sync()
            assert np.array_equal(bufs[2].cpu().numpy().view(B.EXT_RES), want), n
            js = _jobs(n, n, 100)  # straight from the caller's arrays up to 24 jobs per SM
            assert np.array_equal(ctx.extend_batch(js, mat, *gaps), oracle.extend_batch(js, mat, *gaps)[0]), n
