"""The kernel_launches statistic against the kernels a call launches (the device's own trace): small batches,
length buckets, captured and replayed graphs, host calls, the retry rounds and the CIGAR stage."""
import numpy as np
import pytest

import bwacuda as B
from kernel_trace import kernels

pytestmark = pytest.mark.gpu


def _device_call(ctx, js):
    import torch

    bufs = [torch.from_numpy(js.seq).cuda(), torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda(),
            torch.zeros(len(js) * 24, dtype=torch.uint8, device="cuda")]
    torch.cuda.synchronize()

    def call():
        ctx.extend_device(bufs[0].data_ptr(), bufs[1].data_ptr(), len(js), bufs[2].data_ptr())
        ctx.sync()
        return bufs

    return call


def _check(ctx, call, sorts):
    """sorts: the sorts of the call, library kernels that count as one each (the offset scans do not count)."""
    call()  # buffers, and the graph of a device call
    names = kernels(call)
    if names is None:
        pytest.skip("no kernel trace")
    ctx.reset_stats()
    call()
    assert ctx.stats()["kernel_launches"] == len([n for n in names if not n.startswith("cub::")]) + sorts, names


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("small", [True, False], ids=["small", "buckets"])
@pytest.mark.parametrize("n", [1, 1000, 4000, 12000])
def test_device_calls(n, small, graphs):
    js = B.synth_ext(2, n, seed=n)
    with B.Context(0) as ctx:
        ctx.set_option(B.OPT_GRAPHS, graphs)
        if not small:
            ctx.set_option(B.OPT_SMALL_BATCH, 0)
        _check(ctx, _device_call(ctx, js), 1 if not small or n >= 4000 else 0)


@pytest.mark.parametrize("n", [1, 2000, 6000])
def test_host_calls(n):
    js = B.synth_ext(2, n, seed=n)
    with B.Context(0) as ctx:
        # straight from the caller's arrays up to 24 jobs per SM; else the plan's lengths, gather and scatter
        _check(ctx, lambda: ctx.extend_batch(js), 1 if n > 24 * 152 else 0)


def test_retry_rounds():
    js = B.synth_ext(2, 1000, seed=8)
    with B.Context(0) as ctx:
        ctx.set_option(B.OPT_HOST_GATHER, B.GATHER_HOST)
        _check(ctx, lambda: ctx.extend_batch_retry(js, None, 2, w=3), 0)


@pytest.mark.parametrize("n", [300, 6000])
@pytest.mark.parametrize("w", [20, 200], ids=["tagged", "untagged"])
def test_cigar_stage(w, n):
    rng = np.random.default_rng(n)
    ts = [rng.integers(0, 4, 150).astype(np.uint8) for _ in range(n)]
    js = B.JobSet.from_lists(ts, ts, None, w)
    with B.Context(0) as ctx:
        call = lambda: ctx.ksw_global2_batch(js)  # noqa: E731
        _check(ctx, call, 1)
        # no more launches than before there was a tagged kernel: 16 at 300 alignments, 21 at 6,000, whose
        # sort is six kernels instead of one
        assert len(kernels(call, library=True)) <= (16 if n == 300 else 21)
