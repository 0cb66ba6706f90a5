"""Rescue batches by size and raggedness: the launch shape each batch size picks, the launches by
column class of ragged batches, and the host-buffer route whose jobs the device gathers, against
the oracle, bit-exact on every field."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu

# column-class edges, queries past the 8-bit and the 256-column limits, empty ones
EDGES = (0, 1, 15, 16, 17, 31, 32, 33, 64, 65, 96, 97, 128, 129, 150, 160, 161, 192, 193, 250, 255, 256, 257, 300, 520)


def _ragged(n, seed, qlens=EDGES, tmax=420):
    rng = np.random.default_rng(seed)
    qs, ts = [], []
    for k in range(n):
        ql = int(qlens[k % len(qlens)])
        tl = int(rng.integers(0, tmax)) if k % 7 else int(rng.integers(0, 3))
        t = rng.integers(0, 4, tl).astype(np.uint8)
        q = rng.integers(0, 4, ql).astype(np.uint8)
        ln = min(ql, tl)
        if k % 5 and ln:  # a planted copy with substitutions and, on some jobs, an insertion
            at = int(rng.integers(0, tl - ln + 1))
            q[:ln] = t[at:at + ln]
            q[:ln][rng.random(ln) < 0.03] ^= 1
            if k % 3 == 0:
                q = np.insert(q, ql // 2, 2)[:ql]
        if k % 11 == 0 and ql:
            q[int(rng.integers(0, ql))] = 4
        if k % 13 == 0 and tl:
            t[int(rng.integers(0, tl))] = 4
        qs.append(q)
        ts.append(t)
    perm = rng.permutation(n)
    return B.JobSet.from_lists([qs[i] for i in perm], [ts[i] for i in perm])


@pytest.fixture(params=[B.GATHER_DEVICE, B.GATHER_HOST], ids=["devgather", "hostpack"])
def fresh(request):
    """A context of its own: no option and no tuning has set a rescue shape."""
    with B.Context(0) as ctx:
        ctx.set_option(B.OPT_HOST_GATHER, request.param)
        yield ctx


@pytest.mark.parametrize("n", [1, 31, 1300, 2500, 5000, 20000])
def test_host_batch_by_size(fresh, n):
    js = _ragged(n, seed=n)
    want, _ = oracle.align2_batch(js, minsc=19)
    assert np.array_equal(fresh.ksw_align2_batch(js, minsc=19), want)


def test_chunks_and_all_modes(fresh):
    js = _ragged(4000, seed=9)
    fresh.set_option(B.OPT_CHUNK_JOBS, 1500)
    want, _ = oracle.align2_batch(js, minsc=19)
    assert np.array_equal(fresh.ksw_align2_batch(js, minsc=19), want)
    want, _ = oracle.align2_batch(js, minsc=19, mode=1)
    assert np.array_equal(fresh.ksw_align2_scalar_batch(js, minsc=19), want)
    rng = np.random.default_rng(3)
    minsc = rng.integers(0, 60, len(js)).astype(np.int32)
    endsc = rng.integers(20, 200, len(js)).astype(np.int32)
    want = oracle.local_fwd_batch(js, minsc, endsc)
    want = want[0] if isinstance(want, tuple) else want
    assert np.array_equal(fresh.ksw_local_fwd_batch(js, minsc, endsc), want)


@pytest.mark.parametrize("scoring", [dict(o_del=6, e_del=1, o_ins=6, e_ins=1), dict(o_del=5, e_del=2, o_ins=9, e_ins=1)])
def test_device_resident_ragged(fresh, scoring):
    import torch

    js = _ragged(3000, seed=17)
    sc = fresh.scoring(**scoring)
    d_seq = torch.from_numpy(js.seq).cuda()
    d_jobs = torch.from_numpy(js.dev_res_jobs().view(np.uint8)).cuda()
    for mode in (0, 1):
        d_out = torch.zeros(len(js) * 28, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        fresh.ksw_align2_device(d_seq.data_ptr(), d_jobs.data_ptr(), len(js), d_out.data_ptr(), sc, minsc=19, mode=mode)
        fresh.sync()
        want, _ = oracle.align2_batch(js, minsc=19, mode=mode, **scoring)
        assert np.array_equal(d_out.cpu().numpy().view(B.ALN_RES), want)


def test_invalid_jobs(fresh):
    js = _ragged(2000, seed=23, qlens=(100, 150))
    js.qlen[1234] = -1
    with pytest.raises(B.BwaCudaError) as e:
        fresh.ksw_align2_batch(js)
    assert e.value.code == B.EINVAL
    js = _ragged(2000, seed=23, qlens=(100, 150))
    js.seq[js.q_off[77] + 3] = 5
    with pytest.raises(B.BwaCudaError) as e:
        fresh.ksw_align2_batch(js)
    assert e.value.code == B.EBASE
    js = _ragged(2000, seed=23, qlens=(100, 150))  # and the context still works
    want, _ = oracle.align2_batch(js, minsc=19)
    assert np.array_equal(fresh.ksw_align2_batch(js, minsc=19), want)


@pytest.mark.parametrize("max_sc", [1, 2])
def test_matrix_above_max_sc(fresh, max_sc):
    """Entries above the caller's max_sc take scores past what its width rule promises."""
    js = _ragged(3000, seed=31, qlens=(40, 100, 150, 240))
    mat = oracle.scmat(3, 4)
    want, _ = oracle.align2_batch(js, mat, minsc=19, max_sc=max_sc)
    assert want["score"].max() > 255
    assert np.array_equal(fresh.ksw_align2_batch(js, mat, minsc=19, max_sc=max_sc), want)


@pytest.mark.parametrize("a,b", [(1, 4), (2, 3)])
def test_pairs_whose_targets_end_apart(fresh, a, b):
    """Long queries against short and long targets in turn: a job's lane computes rows past its target
    while its neighbour has rows."""
    rng = np.random.default_rng(41)
    qs, ts = [], []
    for k in range(3000):
        t = rng.integers(0, 4, 400 if k & 1 else int(rng.integers(1, 60))).astype(np.uint8)
        unit = rng.integers(0, 4, int(rng.integers(1, 4))).astype(np.uint8)
        q = np.resize(unit, 250 // a)  # repeats: rows past the target keep matching
        t[:min(len(t), 60)] = np.resize(unit, min(len(t), 60))
        qs.append(q)
        ts.append(t)
    js = B.JobSet.from_lists(qs, ts)
    mat = oracle.scmat(a, b)
    want, _ = oracle.align2_batch(js, mat, minsc=19, max_sc=a)
    assert np.array_equal(fresh.ksw_align2_batch(js, mat, minsc=19, max_sc=a), want)
