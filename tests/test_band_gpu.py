"""The band kernel (csrc/ext_band.cuh: a group of lanes splits every row of an extension) against the
oracle, bit-exact on every field: small batches straight from the caller's arrays and on the device,
with 8, 16 and 32 lanes a job, next to jobs it leaves to the group-per-job kernels, and the sorted
buckets on the same jobs."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu

EDGE_Q = (0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 100, 131, 200, 255, 256, 257, 264, 268, 269, 300)


def _jobs(n, seed, wmax=120, long_share=0.0):
    rng = np.random.default_rng(seed)
    qs, ts, h0s, ws = [], [], [], []
    for k in range(n):
        ql = int(EDGE_Q[k % len(EDGE_Q)]) if rng.random() >= long_share else int(rng.integers(400, 3000))
        tl = max(0, ql + int(rng.integers(-20, 110))) if k % 9 else int(rng.integers(0, 4))
        t = rng.integers(0, 4, tl).astype(np.uint8)
        q = rng.integers(0, 4, ql).astype(np.uint8)
        ln = min(ql, tl)
        if k % 4:
            q[:ln] = t[:ln]
            q[:ln][rng.random(ln) < 0.02] ^= 1
            if k % 3 == 0 and ql > 10:  # an indel near the middle
                q = np.insert(q, ql // 2, [2, 1])[:ql] if k % 2 else np.append(np.delete(q, ql // 2), 0)
            if k % 8 == 1 and ql > 20:  # an error-dense tail: z-drop and dying rows
                tail = q[ql // 2:]
                tail[rng.random(len(tail)) < 0.4] ^= 2
        if k % 11 == 0 and ql:
            q[int(rng.integers(0, ql))] = 4
        if k % 13 == 0 and tl:
            t[int(rng.integers(0, tl))] = 4
        qs.append(q.astype(np.uint8))
        ts.append(t)
        h0s.append(int(rng.choice([1, 2, 7, 19, 60, 150, 400, 30000 if k % 50 == 0 else 30])))
        ws.append(int(rng.choice([0, 1, 2, 5, 20, 100, 101, 102, wmax])))
    return B.JobSet.from_lists(qs, ts, h0s, np.array(ws))


def _uniform_w(js, w):
    return B.JobSet(js.seq, js.q_off, js.t_off, js.qlen, js.tlen, js.h0, np.full(len(js), w, np.int32))


@pytest.fixture
def fresh():
    with B.Context(0) as ctx:
        yield ctx


def _device(ctx, js, **kw):
    import torch

    d_seq = torch.from_numpy(js.seq).cuda()
    d_jobs = torch.from_numpy(js.dev_ext_jobs().view(np.uint8)).cuda()
    d_out = torch.zeros(len(js) * 24, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    sc = ctx.scoring(**{k: v for k, v in kw.items() if k in ("o_del", "e_del", "o_ins", "e_ins", "mat")})
    ctx.extend_device(d_seq.data_ptr(), d_jobs.data_ptr(), len(js), d_out.data_ptr(), sc,
                      end_bonus=kw.get("end_bonus", 5), zdrop=kw.get("zdrop", 100))
    ctx.sync()
    return d_out.cpu().numpy().view(B.EXT_RES)


SCORINGS = [dict(), dict(o_del=4, e_del=2, o_ins=7, e_ins=1, zdrop=20), dict(o_del=0, e_del=1, o_ins=0, e_ins=1, zdrop=0),
            dict(o_del=11, e_del=3, o_ins=2, e_ins=5, end_bonus=0, zdrop=60)]


@pytest.mark.parametrize("kw", SCORINGS)
@pytest.mark.parametrize("n", [2, 5, 700, 2000, 4500])
def test_device_small_batches(fresh, n, kw):
    """Up to 700 jobs: 32 lanes a job; 2,000: 16; 4,500: 8."""
    js = _jobs(n, seed=n + 1, wmax=300)
    want, cells = oracle.extend_batch(js, **kw)
    fresh.reset_stats()
    assert np.array_equal(_device(fresh, js, **kw), want)
    assert fresh.stats()["ext_cells"] == cells
    fresh.set_option(B.OPT_SMALL_BATCH, 0)
    assert np.array_equal(_device(fresh, js, **kw), want)


@pytest.mark.parametrize("gather", [B.GATHER_DEVICE, B.GATHER_HOST], ids=["devgather", "hostpack"])
@pytest.mark.parametrize("w", [0, 3, 100, 300])
def test_host_small_batches(fresh, gather, w):
    """Up to 24 jobs per SM straight from the caller's arrays where every query fits; the job of 257
    or more columns sends the call through the gather."""
    fresh.set_option(B.OPT_HOST_GATHER, gather)
    js = _uniform_w(_jobs(1500, seed=77), w)
    want, cells = oracle.extend_batch(js)
    fresh.reset_stats()
    assert np.array_equal(fresh.extend_batch(js, w=w), want)
    assert fresh.stats()["ext_cells"] == cells
    short = js.take(np.nonzero((js.qlen <= 256) & (js.tlen <= 512) & (js.h0 < 30000))[0])
    want, cells = oracle.extend_batch(short)
    fresh.reset_stats()
    assert np.array_equal(fresh.extend_batch(short, w=w), want)
    st = fresh.stats()
    assert st["ext_cells"] == cells and st["ext_jobs"] == len(short)
    for k in (0, 3, 14, 15):  # single jobs: every alignment of the slices
        one = short.take([k])
        assert np.array_equal(fresh.extend_batch(one, w=w), want[k:k + 1])


def test_long_jobs_in_a_small_batch(fresh):
    js = _jobs(900, seed=5, wmax=500, long_share=0.5)
    want, cells = oracle.extend_batch(js)
    fresh.reset_stats()
    assert np.array_equal(_device(fresh, js), want)
    assert fresh.stats()["ext_cells"] == cells


@pytest.mark.parametrize("mode", [1, 2])
def test_long_buckets(fresh, mode):
    """The open-ended buckets: 32 lanes a job (few jobs) and 8 (forced)."""
    fresh.set_option(B.OPT_SMALL_BATCH, 0)
    fresh.set_option(B.OPT_LONG_SLIDE, mode)
    rng = np.random.default_rng(8)
    qs, ts, ws = [], [], []
    for k in range(300):
        ql = int(rng.integers(1000, 2500))
        t = rng.integers(0, 4, ql + 110).astype(np.uint8)
        q = t[:ql].copy()
        q[rng.random(ql) < 0.01] ^= 1
        if k % 3 == 0:
            q = np.insert(q, ql // 3, [0, 1, 2])
        qs.append(q)
        ts.append(t[:int(rng.integers(30, 200))] if k % 7 == 0 else t)
        ws.append(int(rng.choice([1, 7, 40, 100, 101, 102])))
    js = B.JobSet.from_lists(qs, ts, rng.integers(1, 200, 300), np.array(ws))
    want, cells = oracle.extend_batch(js)
    fresh.reset_stats()
    assert np.array_equal(_device(fresh, js), want)
    assert fresh.stats()["ext_cells"] == cells


def test_invalid_jobs(fresh):
    js = _uniform_w(_jobs(300, seed=6), 100)
    js.h0 = js.h0.copy()
    js.h0[17] = 0
    with pytest.raises(B.BwaCudaError) as e:
        fresh.extend_batch(js)
    assert e.value.code == B.EINVAL
    js.h0[17] = 5
    k = int(np.nonzero(js.qlen > 5)[0][3])
    js.seq[js.q_off[k] + 2] = 6
    with pytest.raises(B.BwaCudaError) as e:
        fresh.extend_batch(js)
    assert e.value.code == B.EBASE
    js.seq[js.q_off[k] + 2] = 1
    want, _ = oracle.extend_batch(js)
    assert np.array_equal(fresh.extend_batch(js), want)
