"""The serving loop's admission gather (csrc/server.cu): codes are checked while the slices are copied as
aligned 16-byte words, so only the slice's own bytes of its first and last words may count."""
import numpy as np
import pytest

import bwacuda as B
import oracle

pytestmark = pytest.mark.gpu


def _jobs(kind):
    """Slices of 0 .. 70 bases at every alignment, all other bytes 255 (no valid code)."""
    rng = np.random.default_rng(5)
    lens = [1, 2, 3, 4, 5, 14, 15, 16, 17, 18, 31, 32, 33, 47, 48, 49, 64, 70]
    ql, tl, qo, to, at = [], [], [], [], 0
    for k in range(400):
        q, t = lens[k % len(lens)], lens[(k // 3) % len(lens)]
        if kind == "extend" and k % 37 == 0:
            q = 0
        if kind == "extend" and k % 41 == 0:
            t = 0
        at += int(rng.integers(1, 24))
        qo.append(at)
        at += q + int(rng.integers(1, 24))
        to.append(at)
        at += t
        ql.append(q)
        tl.append(t)
    seq = np.full(at + 64, 255, np.uint8)
    for o, n in list(zip(qo, ql)) + list(zip(to, tl)):
        seq[o:o + n] = rng.integers(0, 5, n)
    n = len(ql)
    return B.JobSet(seq, np.array(qo, np.int64), np.array(to, np.int64), np.array(ql, np.int32),
                    np.array(tl, np.int32), np.full(n, 20, np.int32), np.full(n, 100, np.int32))


@pytest.mark.parametrize("kind", ["extend", "rescue"])
def test_only_the_slices_bytes_count(ctx, kind):
    js = _jobs(kind)
    submit = ctx.submit_extend if kind == "extend" else lambda j: ctx.submit_rescue(j, minsc=20)
    ctx.server_start(hbm_budget_bytes=64 << 20, max_waves=2)
    try:
        out = ctx.wait(submit(js))[0]
        want = oracle.extend_batch(js)[0] if kind == "extend" else oracle.align2_batch(js, minsc=20)[0]
        assert np.array_equal(out, want)
        spots = []
        for k in range(0, 400, 29):
            for o, n in ((js.q_off[k], js.qlen[k]), (js.t_off[k], js.tlen[k])):
                if n:
                    spots += [o, o + n - 1, o + n // 2]
        rng = np.random.default_rng(6)
        for p in spots:
            old = js.seq[p]
            js.seq[p] = rng.choice([5, 6, 127, 128, 255])
            with pytest.raises(B.BwaCudaError) as e:
                ctx.wait(submit(js))
            assert e.value.code == B.EBASE
            js.seq[p] = old
        assert np.array_equal(ctx.wait(submit(js))[0], want)
    finally:
        ctx.server_stop()
