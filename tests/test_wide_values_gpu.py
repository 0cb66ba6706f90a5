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


def _flat(n, qlens, seed, tl_add=40, w=100):
    """Jobs laid out flat: queries copied from their targets with substitutions."""
    rng = np.random.default_rng(seed)
    ql = rng.choice(np.asarray(qlens), n)
    sizes = np.empty(2 * n, np.int64)
    sizes[0::2], sizes[1::2] = ql, ql + tl_add
    offs = np.zeros(2 * n + 1, np.int64)
    np.cumsum(sizes, out=offs[1:])
    qo, to = offs[0:-1:2].copy(), offs[1:-1:2].copy()
    seq = rng.integers(0, 4, offs[-1]).astype(np.uint8)
    job = np.repeat(np.arange(n), ql)
    j = np.arange(len(job)) - np.repeat(np.cumsum(ql) - ql, ql)
    base = seq[to[job] + j]
    seq[qo[job] + j] = np.where(rng.random(len(job)) < 0.02, base ^ 1, base)
    return B.JobSet(seq, qo, to, ql.astype(np.int32), (ql + tl_add).astype(np.int32),
                    rng.integers(20, 60, n).astype(np.int32), np.full(n, w, np.int32))


class _Device:
    def __init__(self, ctx, js):
        import torch

        self.ctx, self.n = ctx, len(js)
        self.seq = torch.from_numpy(js.seq).cuda()
        self.jobs = torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda()
        self.out = torch.zeros(self.n * 24, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def run(self):
        self.ctx.extend_device(self.seq.data_ptr(), self.jobs.data_ptr(), self.n, self.out.data_ptr())
        self.ctx.sync()

    def result(self):
        self.out.zero_()
        self.run()
        return self.out.cpu().numpy().view(B.EXT_RES)

    def best_ms(self, reps=6):
        import time

        self.run()
        best = 1e9
        for _ in range(reps):
            t0 = time.perf_counter()
            self.run()
            best = min(best, time.perf_counter() - t0)
        return best * 1e3


# 45 jobs per SM of 152: fewer 32-bit jobs run in the group-per-job kernel, more a thread each by length
@pytest.mark.parametrize("nwide", [0, 1, 152 * 45 - 1, 152 * 45, 152 * 45 + 1, 9001])
def test_wide_jobs_among_others_in_a_small_batch(nwide):
    n = 9001
    js = _flat(n, [1, 2, 30, 64, 65, 128, 129, 256, 257, 300, 512, 513, 768, 769, 800, 1100], seed=nwide + 1)
    pick = np.random.default_rng(4).permutation(n)[:nwide]
    js.h0[pick] = 33000
    js.w[::7] = 150
    want, cells = oracle.extend_batch(js)
    with B.Context(0) as ctx:
        d = _Device(ctx, js)
        for _ in range(2):  # captured and replayed
            ctx.reset_stats()
            assert np.array_equal(d.result(), want)
            assert ctx.stats()["ext_cells"] == cells
        ctx.set_option(B.OPT_GRAPHS, 0)
        assert np.array_equal(d.result(), want)


@pytest.mark.parametrize("gather", [B.GATHER_DEVICE, B.GATHER_HOST], ids=["devgather", "hostpack"])
@pytest.mark.parametrize("nwide", [0, 1, 7000])
@pytest.mark.parametrize("w", [100, 150])
def test_host_call_with_and_without_jobs_the_band_kernel_leaves(w, nwide, gather):
    """The device gather counts what the band kernel leaves, and the call launches only what that needs."""
    js = _flat(9001, [30, 100, 250] if w == 100 else [30, 100, 300], seed=w, w=w)
    js.h0[:nwide] = 33000
    want, cells = oracle.extend_batch(js)
    with B.Context(0) as ctx:
        ctx.set_option(B.OPT_HOST_GATHER, gather)
        ctx.reset_stats()
        assert np.array_equal(ctx.extend_batch(js, w=w), want)
        assert ctx.stats()["ext_cells"] == cells


@pytest.mark.parametrize("n,qlen,w,h0", [(20000, 150, 100, 33000), (50000, 150, 100, 33000), (50000, 300, 200, 40)])
def test_small_batches_left_by_the_band_kernel_take_no_longer(n, qlen, w, h0):
    js = _flat(n, [qlen], seed=2, tl_add=100, w=w)
    js.h0[:] = h0
    with B.Context(0) as ctx:
        d = _Device(ctx, js)
        small = d.best_ms()
        ctx.set_option(B.OPT_SMALL_BATCH, 0)
        buckets = d.best_ms()
    assert small < 1.05 * buckets, (small, buckets)


def test_serving_waves_with_and_without_such_jobs():
    """Small requests through the serving loop, whose waves launch what their requests' jobs may need."""
    with B.Context(0) as ctx:
        ctx.server_start(hbm_budget_bytes=256 << 20, max_waves=2)
        try:
            reqs = []
            for k in range(24):
                n = [1, 40, 700, 3500, 9500][k % 5]
                js = _flat(n, [30, 100, 250] if k % 2 else [30, 268, 269, 300, 1100], seed=k, w=[100, 150][k // 2 % 2])
                if k % 3 == 0:
                    js.h0[n // 2:] = 33000
                reqs.append((ctx.submit_extend(js, w=int(js.w[0])), js))
            for rid, js in reqs:
                assert np.array_equal(ctx.wait(rid)[0], oracle.extend_batch(js)[0])
        finally:
            ctx.server_stop()
