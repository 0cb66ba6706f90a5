"""Which wavefront a rescue batch of a size and a range of lengths runs, where two jobs a group do not pay: short
queries, batches that hold a few jobs past a byte, ragged ones; each with its results against the oracle."""
import numpy as np
import pytest

import bwacuda as B
import oracle
from kernel_trace import kernels

pytestmark = pytest.mark.gpu


def _jobs(n, qmin, qmax, seed=1, tl_add=150):
    rng = np.random.default_rng(seed)
    qs, ts = [], []
    for _ in range(n):
        ql = int(rng.integers(qmin, qmax + 1))
        t = rng.integers(0, 4, ql + tl_add).astype(np.uint8)
        at = int(rng.integers(0, tl_add))
        q = t[at:at + ql].copy()
        q[rng.random(ql) < 0.02] ^= 1
        qs.append(q)
        ts.append(t)
    return B.JobSet.from_lists(qs, ts)


# jobs per SM of 152: pairs from 24 on up to 128 columns, from 20 up to 208, from 16 above, from 100 when a few
# jobs do not fit a byte; the last two sort into column classes, where it is 16 and 32
@pytest.mark.parametrize("n,qmin,qmax,a,pairs", [
    (152 * 24 - 1, 36, 36, 1, False), (152 * 24, 36, 36, 1, True), (152 * 20 - 1, 150, 150, 1, False),
    (152 * 20, 150, 150, 1, True), (152 * 16 - 1, 250, 250, 1, False), (152 * 16, 250, 250, 1, True),
    (3000, 240, 256, 1, False), (152 * 100, 240, 256, 1, True), (3000, 150, 150, 2, False),
    (3000, 110, 130, 2, False), (4000, 20, 250, 1, False)])
def test_shapes(n, qmin, qmax, a, pairs):
    js = _jobs(n, qmin, qmax)
    mat = oracle.scmat(a, 4)
    want, _ = oracle.align2_batch(js, mat, minsc=19, max_sc=a)
    with B.Context(0) as ctx:
        call = lambda: ctx.ksw_align2_batch(js, mat, minsc=19, max_sc=a)  # noqa: E731
        assert np.array_equal(call(), want)
        names = kernels(call)
        if names is not None:
            assert any("rescue_wf2_kernel" in x for x in names) == pairs
        ctx.set_option(B.OPT_HOST_GATHER, B.GATHER_HOST)
        assert np.array_equal(call(), want)
