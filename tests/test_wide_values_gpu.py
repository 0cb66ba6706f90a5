"""Extensions whose seed scores reach to the end of a 32-bit integer, in batches of every size: the small
ones run in the group-per-job kernel (csrc/ext_long.cuh), whose F terms must not leave the integer where
the values themselves do not; against the oracle, bit-exact on every field."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu


def _jobs(n, seed, qmax, w):
    rng = np.random.default_rng(seed)
    qs, ts, h0s = [], [], []
    for k in range(n):
        ql = int(rng.integers(1, qmax + 1))
        t = rng.integers(0, 4, ql + int(rng.integers(0, 60))).astype(np.uint8)
        q = t[:ql].copy()
        q[rng.random(ql) < 0.03] ^= 1
        if k % 3 == 0 and ql > 8:  # an indel
            q = np.insert(q, ql // 2, [1, 2])[:ql] if k % 2 else np.append(np.delete(q, ql // 2), 0)
        qs.append(q.astype(np.uint8))
        ts.append(t)
        # the largest: a full-length match ends at 2^31 - 1
        h0s.append(int([33000, 1 << 24, (1 << 24) + 12345, 10 ** 9, 2 ** 31 - 1 - ql, 50][k % 6]))
    return B.JobSet.from_lists(qs, ts, h0s, w)


@pytest.mark.parametrize("kw", [dict(), dict(o_del=11, e_del=3, o_ins=2, e_ins=5, zdrop=30),
                                dict(o_del=6, e_del=9000, o_ins=6, e_ins=16000, zdrop=0)])
@pytest.mark.parametrize("n,qmax,w", [(12, 300, 3), (600, 130, 100), (600, 400, 200), (4000, 130, 100)])
def test_values_to_the_end_of_int(n, qmax, w, kw):
    import torch

    js = _jobs(n, n + w, qmax, w)
    want, _ = oracle.extend_batch(js, **kw)
    with B.Context(0) as ctx:
        for small in (None, 0):  # as such a batch runs by itself, and in length buckets
            if small is not None:
                ctx.set_option(B.OPT_SMALL_BATCH, small)
            assert np.array_equal(ctx.extend_batch(js, w=w, **kw), want)
            d_seq = torch.from_numpy(js.seq).cuda()
            d_jobs = torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda()
            d_out = torch.zeros(n * 24, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            sc = ctx.scoring(**{k: v for k, v in kw.items() if k != "zdrop"})
            ctx.extend_device(d_seq.data_ptr(), d_jobs.data_ptr(), n, d_out.data_ptr(), sc, zdrop=kw.get("zdrop", 100))
            ctx.sync()
            assert np.array_equal(d_out.cpu().numpy().view(B.EXT_RES), want)
