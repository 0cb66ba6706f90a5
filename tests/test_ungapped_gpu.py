"""The ungapped closed form ahead of the DP in batches large enough for the kernel of two jobs a thread:
results against the oracle, N bases included, and which kernel runs the jobs it leaves."""
import numpy as np
import pytest

import bwacuda as B
import oracle
from kernel_trace import kernels

pytestmark = pytest.mark.gpu


def _device(ctx, js):
    import torch

    bufs = [torch.from_numpy(js.seq).cuda(), torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda(),
            torch.zeros(len(js) * 24, dtype=torch.uint8, device="cuda")]
    torch.cuda.synchronize()

    def run():
        ctx.extend_device(bufs[0].data_ptr(), bufs[1].data_ptr(), len(js), bufs[2].data_ptr())
        ctx.sync()
        return bufs[2]

    return run


@pytest.mark.parametrize("cfg", [1, 2, 3])
def test_large_batches(cfg):
    js = B.synth_ext(cfg, 152 * 5000 + 7, seed=40 + cfg)  # past the size that runs two jobs a thread
    rng = np.random.default_rng(cfg)
    js.seq[rng.integers(0, len(js.seq), len(js) // 40)] = 4
    want, _ = oracle.extend_batch(js)
    with B.Context(0) as ctx:
        ctx.set_option(B.OPT_UNGAPPED, 1)
        assert np.array_equal(_device(ctx, js)().cpu().numpy().view(B.EXT_RES), want)


def test_jobs_left_by_the_closed_form_run_one_a_thread():
    """Two jobs a thread suit the many like jobs of a large batch, not the few that the closed form leaves."""
    js = B.synth_ext(2, 152 * 5000 + 7, seed=3)
    with B.Context(0) as ctx:
        run = _device(ctx, js)
        names = kernels(run)
        if names is None:
            pytest.skip("no kernel trace")
        assert any("ext_dual_kernel" in n for n in names)
        ctx.set_option(B.OPT_UNGAPPED, 1)
        names = kernels(run)
        assert any("ext_persist_pair_kernel" in n for n in names)
        assert not any("ext_dual_kernel" in n for n in names)
