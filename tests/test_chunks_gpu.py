"""The host-fed extension's split of a batch into chunks (csrc/ats.cu): sizes at the edges where the
last chunk joins or halves, with the default ramp and with a small chunk limit, against the oracle."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu

RAMP = 131072  # the first chunk of the default ramp; the next is 9/4 of it


@pytest.fixture(scope="module")
def batch():
    js = B.synth_ext(1, RAMP + RAMP * 9 // 4 + RAMP * 2 + 1, seed=31)
    return js, oracle.extend_batch(js)[0]


@pytest.fixture(scope="module")
def ctx():
    c = B.Context(0)
    c.set_option(B.OPT_EXT_PATH, B.PATH_BATCHED)
    c.set_option(B.OPT_SMALL_BATCH, 0)
    yield c
    c.close()


@pytest.mark.parametrize("chunk,n", [
    (1 << 20, RAMP), (1 << 20, RAMP + 1), (1 << 20, RAMP * 3 // 2 - 1), (1 << 20, RAMP * 3 // 2),
    (1 << 20, RAMP + RAMP * 9 // 4 + 1), (1 << 20, RAMP + RAMP * 9 // 4 + RAMP * 2 + 1),
    (RAMP, RAMP * 3 // 2 - 1), (4099, 4099), (4099, 4100), (4099, 4099 * 3 // 2), (4099, 4099 * 3 // 2 + 1),
    (4099, 4099 * 3 - 1), (1, 5), (63, 64 * 3 + 1)])
def test_every_job_once(ctx, batch, chunk, n):
    js, want = batch
    ctx.set_option(B.OPT_CHUNK_JOBS, chunk)
    sub = js.take(np.arange(n))
    ctx.reset_stats()
    got = ctx.extend_batch(sub)
    assert np.array_equal(got, want[:n])
    assert ctx.stats()["ext_jobs"] == n
