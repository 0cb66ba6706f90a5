"""Lengths of device-resident extension jobs, which no host check sees: a negative query length fails the call
and a negative target length is an empty target, in a batch of any size and of any cell width."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu


def _call(ctx, js):
    import torch

    bufs = [torch.from_numpy(js.seq).cuda(), torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda(),
            torch.zeros(len(js) * 24, dtype=torch.uint8, device="cuda")]
    torch.cuda.synchronize()
    ctx.extend_device(bufs[0].data_ptr(), bufs[1].data_ptr(), len(js), bufs[2].data_ptr())
    ctx.sync()
    return bufs[2].cpu().numpy().view(B.EXT_RES)


@pytest.mark.parametrize("small", [True, False], ids=["small", "buckets"])
@pytest.mark.parametrize("n", [5, 2000, 4000, 12000])
def test_negative_lengths(n, small):
    js = B.synth_ext(1, n, seed=n)
    js.h0 = js.h0.copy()
    js.h0[::3] = 33000  # 32-bit cells
    js.w = np.where(np.arange(n) % 2 == 0, 300, 100).astype(np.int32)
    empty = np.arange(n) % 5 == 1
    js.tlen = np.where(empty, 0, js.tlen).astype(np.int32)
    want, _ = oracle.extend_batch(js)
    js.tlen = np.where(empty, -1 - np.arange(n) % 7, js.tlen).astype(np.int32)
    with B.Context(0) as ctx:
        if not small:
            ctx.set_option(B.OPT_SMALL_BATCH, 0)
        assert np.array_equal(_call(ctx, js), want)
        keep = js.qlen[n // 2]
        js.qlen[n // 2] = -3
        with pytest.raises(B.BwaCudaError) as e:
            _call(ctx, js)
        assert e.value.code == B.EUNSUPPORTED
        js.qlen[n // 2] = keep
        assert np.array_equal(_call(ctx, js), want)
