"""The forward pass alone, whose jobs stop at their own end score: which wavefront runs a batch of which size,
and its results against the oracle on either side of the sizes where that changes."""
import numpy as np
import pytest

import bwacuda as B
import oracle
from kernel_trace import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 2500, 3000, 5000, 152 * 200 - 1, 152 * 200])
def test_forward_batches(n):
    js = B.synth_rescue(n, seed=n)
    rng = np.random.default_rng(n)
    minsc = rng.integers(0, 60, n).astype(np.int32)
    endsc = rng.choice([1, 40, 100, 100000], n).astype(np.int32)
    want = oracle.local_fwd_batch(js, minsc, endsc)
    want = want[0] if isinstance(want, tuple) else want
    with B.Context(0) as ctx:
        assert np.array_equal(ctx.ksw_local_fwd_batch(js, minsc, endsc), want)
        names = kernels(lambda: ctx.ksw_local_fwd_batch(js, minsc, endsc))
        if names is not None:  # two jobs a group from 200 per SM (of 152) on
            assert any("rescue_wf2_kernel" in x for x in names) == (n >= 152 * 200)
            assert any("rescue_wf_kernel" in x for x in names)
