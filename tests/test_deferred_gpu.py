"""Jobs whose band needs a larger ring than the group-per-job kernel's first launch holds (the deferred
launch of csrc/ext_long.cu): bands at the edges of every ring, both cell widths in one call, few jobs and
more than a launch has warps, against the oracle; and that a small batch of them takes no longer than the
same batch in length buckets."""
import time

import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu


def _jobs(n, qlens, ws, seed, h0=(20, 60), tl_add=60):
    """Jobs laid out flat: queries copied from their targets with substitutions."""
    rng = np.random.default_rng(seed)
    ql = rng.choice(np.asarray(qlens), n)
    tl = ql + tl_add
    sizes = np.empty(2 * n, np.int64)
    sizes[0::2], sizes[1::2] = ql, tl
    offs = np.zeros(2 * n + 1, np.int64)
    np.cumsum(sizes, out=offs[1:])
    qo, to = offs[0:-1:2].copy(), offs[1:-1:2].copy()
    seq = rng.integers(0, 4, offs[-1]).astype(np.uint8)
    job = np.repeat(np.arange(n), ql)
    j = np.arange(len(job)) - np.repeat(np.cumsum(ql) - ql, ql)
    base = seq[to[job] + j]
    hit = rng.random(len(job)) < 0.01
    seq[qo[job] + j] = np.where(hit, base ^ 1, base)
    return B.JobSet(seq, qo, to, ql.astype(np.int32), tl.astype(np.int32),
                    rng.integers(h0[0], h0[1] + 1, n).astype(np.int32), rng.choice(np.asarray(ws), n).astype(np.int32))


class _Device:
    def __init__(self, ctx, js):
        import torch

        self.ctx, self.n, self.torch = ctx, len(js), torch
        self.seq = torch.from_numpy(js.seq).cuda()
        self.jobs = torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda()
        self.out = torch.zeros(len(js) * 24, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def __call__(self):
        self.ctx.extend_device(self.seq.data_ptr(), self.jobs.data_ptr(), self.n, self.out.data_ptr())
        self.ctx.sync()

    def result(self):
        self()
        return self.out.cpu().numpy().view(B.EXT_RES)

    def best_ms(self, reps=5):
        self()
        best = 1e9
        for _ in range(reps):
            t0 = time.perf_counter()
            self()
            best = min(best, time.perf_counter() - t0)
        return best * 1e3


# 2w + 3 against rings of 512, 1024 (32-bit cells) and 2048 columns, and beyond them
@pytest.mark.parametrize("n", [1, 33, 300, 3500])
@pytest.mark.parametrize("long", [False, True], ids=["q500-1022", "q1500-4500"])
def test_ring_edges(n, long):
    qlens = [1500, 2047, 2048, 2300, 4500] if long else [500, 511, 512, 600, 1022]
    if long and n > 300:
        n = 160  # rows of the oracle
    js = _jobs(n, qlens, [254, 255, 510, 511, 1022, 1023, 1500], seed=n, tl_add=20)
    js.h0[::3] = 33000  # 32-bit cells
    want, cells = oracle.extend_batch(js)
    with B.Context(0) as ctx:
        assert np.array_equal(_Device(ctx, js).result(), want)
        assert ctx.stats()["ext_cells"] == cells
        ctx.set_option(B.OPT_SMALL_BATCH, 0)
        ctx.set_option(B.OPT_LONG_QLEN, 1)  # every bucket in the group kernel
        assert np.array_equal(_Device(ctx, js).result(), want)


def _times(js):
    with B.Context(0) as ctx:
        d = _Device(ctx, js)
        small = d.best_ms()
        ctx.set_option(B.OPT_SMALL_BATCH, 0)
        return small, d.best_ms()


@pytest.mark.parametrize("n", [300, 2000])
def test_small_batches_of_deferred_jobs_take_no_longer(n):
    js = _jobs(n, np.arange(700, 901), [300], seed=1, tl_add=300)
    small, buckets = _times(js)
    assert small < 1.1 * buckets, (small, buckets)
