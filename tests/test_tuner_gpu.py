"""What the autotuner times: launch shapes that its candidates' kernels have, whatever the sample's size."""
import numpy as np
import pytest

import bwacuda as B
import oracle
from kernel_trace import kernels

pytestmark = pytest.mark.gpu


def test_extension_candidates_run_the_kernels_they_shape():
    import torch

    js = B.synth_ext(2, 20000, seed=5)  # a batch of this size by itself runs without length buckets
    want, _ = oracle.extend_batch(js)
    d_seq = torch.from_numpy(js.seq).cuda()
    d_jobs = torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda()
    d_out = torch.zeros(len(js) * 24, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with B.Context(0) as ctx:
        t = {}

        def call():
            ctx.extend_device(d_seq.data_ptr(), d_jobs.data_ptr(), len(js), d_out.data_ptr())
            ctx.sync()

        names = kernels(lambda: t.update(ctx.autotune_extend(d_seq.data_ptr(), d_jobs.data_ptr(), len(js))))
        assert t["candidates"] == 45 and t["ext_gcups"] > 0
        if names is not None:
            for tb in (32, 64, 128, 256):
                for grab in (1, 2, 4):
                    assert any(f"ext_persist_pair_kernel<{tb}, {grab}, false>" in n for n in names), (tb, grab)
            # and calls run as before
            names = kernels(call)
            assert any("ext_band_kernel" in n for n in names)
            assert not any("ext_persist_pair_kernel" in n for n in names)
        call()
        assert np.array_equal(d_out.cpu().numpy().view(B.EXT_RES), want)


def test_a_copied_tuning_leaves_an_unset_rescue_shape_unset():
    """get_tuning says whether the rescue shape is a setting: copying one context's tuning to another does
    not pin the other to one job per group."""
    js = B.synth_rescue(16384, seed=3)

    def copy(src, dst):
        t = src.tuning()
        dst.set_option(B.OPT_PERSIST_BLOCK, t["persist_block"])
        dst.set_option(B.OPT_RESCUE_KERNEL, t["rescue_kernel"])
        if not t["rescue_auto"]:
            dst.set_option(B.OPT_RESCUE_LANES, t["rescue_lanes"])
            dst.set_option(B.OPT_RESCUE_PAIR, t["rescue_pair"])

    with B.Context(0) as a, B.Context(0) as b, B.Context(0) as c:
        assert a.tuning()["rescue_auto"] == 1
        copy(a, b)
        assert b.tuning() == a.tuning()
        names = kernels(lambda: b.ksw_align2_batch(js))
        assert names is None or any("rescue_wf2_kernel" in n for n in names)  # pairs at this size
        a.set_option(B.OPT_RESCUE_LANES, 32)
        assert a.tuning()["rescue_auto"] == 0
        copy(a, c)
        assert (c.tuning()["rescue_auto"], c.tuning()["rescue_lanes"], c.tuning()["rescue_pair"]) == (0, 32, 0)
