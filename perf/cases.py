"""Workloads of the Smith-Waterman engine, each one call a program makes through its public entry points.

The sizes are those of the repository's benchmark and tests (2 x 150 bp read pairs, mixed read
lengths and bands, 150 bp mates against 750 bp windows, CIGAR-stage alignments, 2-10 kb queries,
mixed serving requests) from one job to millions.  Host-buffer calls go through the C entry points
with the job and result arrays the caller holds, as a C or Rust program makes them; device calls
take jobs resident in HBM.  One context serves every call of a program; its options are the
defaults except where a case names one.
"""
import atexit
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bwa-mem4_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import bwacuda as B  # noqa: E402

# DP cells per extension job and bases per job of the synthetic workloads (the kernels' own counter):
# 1 = 1% substitutions, qlen 1-120; 2 = read pairs; 3 = mixed read lengths, bands 50 / 100 / 200
_EXT_CELLS = {1: 5700, 2: 5260, 3: 5650}
_EXT_BASES = {1: 221, 2: 211, 3: 231}
# operations of a DP cell: extension 9, rescue and global alignment 10
_OPS_EXT, _OPS_LOCAL = 9, 10

_SCORING = (6, 1, 6, 1)  # o_del, e_del, o_ins, e_ins: bwa-mem's defaults
_END_BONUS, _ZDROP, _MINSC, _MIN_SEED = 5, 100, 20, 19


def listed():
    return [
        # one seed extension through SwBackend::extend: pure call latency
        {"name": "extend_one", "kind": "extend", "qlen": 100},
        # one worker thread's small batch of read-pair extensions
        {"name": "extend_batch_1k", "kind": "extend_batch", "jobs": 1000, "workload": 2, "ungapped": False},
        # the benchmark's first configuration: 20,000 jobs with 1% substitutions and N bases
        {"name": "extend_batch_20k", "kind": "extend_batch", "jobs": 20000, "workload": 1, "ungapped": False},
        # a large chunk of read pairs through host buffers, transfers included
        {"name": "extend_batch_2m", "kind": "extend_batch", "jobs": 2097152, "workload": 2, "ungapped": False},
        # read pairs resident in HBM: the headline workload
        {"name": "extend_device_4m", "kind": "extend_device", "jobs": 4194304, "workload": 2},
        # mixed read lengths and per-job bands, an odd count
        {"name": "extend_device_mixed_1m", "kind": "extend_device", "jobs": 1000003, "workload": 3},
        # queries of 2-10 kb (long reads)
        {"name": "extend_device_long_20k", "kind": "extend_long", "jobs": 20000, "qmin": 2000, "qmax": 10000},
        # mate rescue of 150 bp mates in 750 bp windows resident in HBM
        {"name": "rescue_device_256k", "kind": "rescue_device", "jobs": 262144, "qmin": 150, "qmax": 150,
         "tmin": 750, "tmax": 750},
        # mate rescue through host buffers with ragged mates and windows
        {"name": "rescue_batch_50k", "kind": "rescue_batch", "jobs": 50000, "qmin": 100, "qmax": 250,
         "tmin": 300, "tmax": 1400},
        # mate rescue with the windows fetched from the reference held in HBM
        {"name": "rescue_windows_100k", "kind": "windows", "jobs": 100000},
        # the CIGAR stage: global alignment with traceback
        {"name": "cigar_500k", "kind": "cigar", "jobs": 500000},
        # a burst of mixed requests through the serving loop
        {"name": "serve_mixed_24", "kind": "serve", "requests": 24, "jmin": 1000, "jmax": 131072},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["extend", "extend_batch", "extend_batch", "extend_device", "extend_device", "retry",
                       "extend_long", "rescue_device", "rescue_batch", "windows", "cigar", "cigar", "serve"])
    if kind == "extend":
        return {"kind": kind, "qlen": rng.randint(1, 120)}
    if kind == "extend_batch":
        return {"kind": kind, "jobs": _logint(rng, 64, 2000000), "workload": rng.choice([1, 2, 3]),
                "ungapped": rng.random() < 0.3}
    if kind == "extend_device":
        return {"kind": kind, "jobs": _logint(rng, 1000, 4000000), "workload": rng.choice([1, 2, 3])}
    if kind == "retry":
        # the band-doubling loop at bwa-mem's band and at narrow ones, where jobs go round again
        return {"kind": kind, "jobs": _logint(rng, 1000, 500000), "workload": rng.choice([1, 2]),
                "w": rng.choice([3, 8, 100])}
    if kind == "extend_long":
        qmin = rng.randint(300, 4000)
        return {"kind": kind, "jobs": _logint(rng, 64, 16000), "qmin": qmin, "qmax": qmin + rng.randint(0, 6000)}
    if kind in ("rescue_device", "rescue_batch"):
        qmin, tmin = rng.randint(50, 150), rng.randint(200, 700)
        return {"kind": kind, "jobs": _logint(rng, 256, 200000), "qmin": qmin,
                "qmax": qmin + rng.choice([0, rng.randint(1, 100)]), "tmin": tmin,
                "tmax": tmin + rng.choice([0, rng.randint(1, 700)])}
    if kind == "windows":
        return {"kind": kind, "jobs": _logint(rng, 1000, 200000)}
    if kind == "cigar":
        return {"kind": kind, "jobs": _logint(rng, 256, 700000)}
    return {"kind": "serve", "requests": rng.randint(4, 32), "jmin": 1000, "jmax": _logint(rng, 4000, 131072)}


# ---------------------------------------------------------------- contexts a program keeps

_contexts = {}


def _context(key="default"):
    """A program's context: made once, used by every call."""
    if key not in _contexts:
        ctx = B.Context(0)
        if key == "ungapped":
            ctx.set_option(B.OPT_UNGAPPED, 1)
        if key == "serve":
            ctx.server_start(hbm_budget_bytes=1 << 30, max_waves=3, max_requests=4096)
        _contexts[key] = ctx
    return _contexts[key]


@atexit.register
def _close():
    for key, ctx in _contexts.items():
        if key == "serve":
            ctx.server_stop()
        ctx.close()
    _contexts.clear()


# ---------------------------------------------------------------- inputs

def _offsets(ql, tl):
    """Offsets of the queries and targets laid out job after job, and the total."""
    sizes = torch.stack([ql, tl], 1).reshape(-1)
    ends = sizes.cumsum(0)
    starts = ends - sizes
    return starts[0::2], starts[1::2], int(ends[-1])


def _planted(ql, tl, at, sub, unrelated, n_rate, g):
    """Random bases for every job, each query a copy of its target from position `at` on with
    substitutions at rate `sub`; a share `unrelated` of the jobs keeps a random query."""
    dev = ql.device
    q_off, t_off, total = _offsets(ql, tl)
    seq = torch.randint(0, 4, (total,), dtype=torch.uint8, device=dev, generator=g)
    starts = ql.cumsum(0) - ql
    job = torch.repeat_interleave(torch.arange(len(ql), device=dev), ql)
    j = torch.arange(len(job), device=dev) - starts[job]
    base = seq[t_off[job] + at[job] + j]
    hit = torch.rand(len(job), device=dev, generator=g) < sub
    other = torch.randint(1, 4, (len(job),), dtype=torch.uint8, device=dev, generator=g)
    base = torch.where(hit, (base + other) & 3, base)
    keep = torch.rand(len(ql), device=dev, generator=g) < unrelated
    dst = q_off[job] + j
    seq[dst] = torch.where(keep[job], seq[dst], base)
    if n_rate:
        seq[torch.rand(total, device=dev, generator=g) < n_rate] = 4
    return seq, q_off, t_off


def _lengths(lo, hi, n, g):
    return torch.randint(lo, hi + 1, (n,), device="cuda", generator=g)


def _jobset(seq, q_off, t_off, ql, tl, h0, w):
    to = lambda x, t: x.cpu().numpy().astype(t)  # noqa: E731
    return B.JobSet(seq.cpu().numpy(), to(q_off, np.int64), to(t_off, np.int64), to(ql, np.int32), to(tl, np.int32),
                    to(h0, np.int32), to(w, np.int32))


def _rescue_jobs(case, seed):
    n = case["jobs"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    ql = _lengths(case["qmin"], case["qmax"], n, g)
    tl = torch.maximum(_lengths(case["tmin"], case["tmax"], n, g), ql)
    at = (torch.rand(n, device="cuda", generator=g) * (tl - ql + 1)).long().clamp_(max=tl - ql)
    seq, q_off, t_off = _planted(ql, tl, at, 0.005, 0.10, 0.0002, g)
    one = torch.ones_like(ql)
    return _jobset(seq, q_off, t_off, ql, tl, one, one * 0)


def _long_jobs(case, seed):
    n = case["jobs"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    ql = _lengths(case["qmin"], case["qmax"], n, g)
    tl = ql + 100
    seq, q_off, t_off = _planted(ql, tl, torch.zeros_like(ql), 0.01, 0.0, 0.0, g)
    return _jobset(seq, q_off, t_off, ql, tl, _lengths(20, 60, n, g), torch.full_like(ql, 100))


def _bytes_on_gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()


def _on_device(state, js, jobs, fields):
    state["seq"], state["jobs"] = torch.from_numpy(js.seq).cuda(), _bytes_on_gpu(jobs)
    state["out"] = torch.zeros((len(js), fields), dtype=torch.int32, device="cuda")
    return state


def _vp(a):
    return C.c_void_p(a.ctypes.data)


def _check(rc, what):
    if rc != B.OK:
        raise B.BwaCudaError(rc, what)


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case, "ctx": _context(), "mat": B.scmat()}
    n = case.get("jobs", 1)
    state["n"] = n
    if kind == "extend":
        # a read-pair style job of the wanted query length
        g = torch.Generator(device="cuda").manual_seed(seed)
        ql = torch.full((1,), case["qlen"], dtype=torch.int64, device="cuda")
        seq, q_off, t_off = _planted(ql, ql + 100, torch.zeros_like(ql), 0.002, 0.0, 0.0, g)
        js = _jobset(seq, q_off, t_off, ql, ql + 100, _lengths(19, 60, 1, g), torch.full_like(ql, 100))
        state.update(js=js, q=js.query(0).copy(), t=js.target(0).copy(), h0=int(js.h0[0]),
                     out=np.zeros((1, 6), np.int32))
    elif kind in ("extend_batch", "retry"):
        if case.get("ungapped"):
            state["ctx"] = _context("ungapped")
        js = B.synth_ext(case["workload"], n, seed=seed)
        state.update(js=js, jobs=B.Context._host_jobs(js, B.EXT_JOB), out=np.zeros((n, 6), np.int32))
        if kind == "retry":
            state["prev"] = np.where(np.arange(n) % 2 == 0, -1, js.h0).astype(np.int32)
            state["w_used"] = np.zeros(n, np.int32)
    elif kind in ("extend_device", "extend_long"):
        js = _long_jobs(case, seed) if kind == "extend_long" else B.synth_ext(case["workload"], n, seed=seed)
        _on_device(state, js, js.dev_ext_jobs(), 6)
    elif kind == "rescue_device":
        js = _rescue_jobs(case, seed)
        _on_device(state, js, js.dev_res_jobs(), 7)
    elif kind == "rescue_batch":
        js = _rescue_jobs(case, seed)
        state.update(js=js, jobs=B.Context._host_jobs(js, B.RES_JOB), out=np.zeros((n, 7), np.int32))
    elif kind == "windows":
        # one genome per program; the requests change
        if "windows" not in _contexts:
            ctx = B.Context(0)
            ctx.ref_set(B.RescueWindows(1, seed=1))
            _contexts["windows"] = ctx
        rw = B.RescueWindows(n, seed=1)
        g = np.random.default_rng(seed)
        order = g.permutation(n)
        rw.mates = np.ascontiguousarray(rw.mates[order])
        flip = g.random(rw.mates.shape) < 0.005
        rw.mates[flip] = (rw.mates[flip] + 1) & 3
        for name in ("orient", "anchor_rb", "anchor_rid"):
            setattr(rw, name, np.ascontiguousarray(getattr(rw, name)[order]))
        state.update(ctx=_contexts["windows"], rw=rw, reqs=rw.requests(), out=np.zeros(n, dtype=B.WINDOW_RES))
    elif kind == "cigar":
        js = B.synth_global(n, seed=seed)
        jobs = np.zeros(n, dtype=B.GLOBAL_JOB)
        jobs["query"] = js.seq.ctypes.data + js.q_off.astype(np.uint64)
        jobs["target"] = js.seq.ctypes.data + js.t_off.astype(np.uint64)
        jobs["qlen"], jobs["tlen"], jobs["w"] = js.qlen, js.tlen, js.w
        state.update(js=js, jobs=jobs, score=np.zeros(n, np.int32), offs=np.zeros(n + 1, np.uint64),
                     words=np.zeros(4 * n + 64, np.uint32))  # 1.15 runs per job on this workload
    elif kind == "serve":
        rng = np.random.default_rng(seed)
        state["ctx"] = _context("serve")
        requests, at = [], 0
        plan = _serve_plan(case)
        pool = {2: B.synth_ext(2, sum(e for e, _, c, _ in plan if c == 2) + 1, seed=seed),
                3: B.synth_ext(3, sum(e for e, _, c, _ in plan if c == 3) + 1, seed=seed)}
        nres = sum(r for _, r, _, _ in plan)
        pool["r"] = B.synth_rescue(nres + 1, seed=seed)
        arrays = {2: B.Context._host_jobs(pool[2], B.EXT_JOB), 3: B.Context._host_jobs(pool[3], B.EXT_JOB),
                  "r": B.Context._host_jobs(pool["r"], B.RES_JOB)}
        used = {2: 0, 3: 0, "r": 0}
        for k in rng.permutation(len(plan)):
            ne, nr, cfg, w = plan[k]
            requests.append((arrays[cfg].ctypes.data + used[cfg] * B.EXT_JOB.itemsize, ne,
                             arrays["r"].ctypes.data + used["r"] * B.RES_JOB.itemsize, nr, w, at))
            used[cfg] += ne
            used["r"] += nr
            at += ne * B.EXT_RES.itemsize + nr * B.ALN_RES.itemsize
        state.update(pool=pool, arrays=arrays, requests=requests, out=np.zeros(at // 4, np.int32),
                     sc=B.Context.scoring())
    else:
        raise ValueError(kind)
    return state


def _serve_plan(case):
    """Per request: extension jobs, rescue jobs, workload, band (sizes log-uniform, fixed by the case)."""
    rng = np.random.default_rng(case["requests"] * 1000003 + case["jmax"])
    plan = []
    for k in range(case["requests"]):
        n = int(np.exp(rng.uniform(np.log(case["jmin"]), np.log(case["jmax"]))))
        nr = int(n * (0.0 if k % 5 == 0 else rng.uniform(0.05, 0.4)))
        cfg = 2 + int(rng.integers(0, 2))
        plan.append((n - nr, nr, cfg, 100 if cfg == 2 else int(rng.choice([50, 100, 200]))))
    return plan


# ---------------------------------------------------------------- one pass

def run(state):
    kind, ctx, n, L = state["kind"], state["ctx"], state["n"], B.lib()
    mat = _vp(state["mat"])
    if kind == "extend":
        _check(L.bwacuda_extend(ctx.h, _vp(state["q"]), len(state["q"]), _vp(state["t"]), len(state["t"]), 5, mat,
                                *_SCORING, 100, _END_BONUS, _ZDROP, state["h0"], _vp(state["out"])), kind)
        return state["out"]
    if kind == "extend_batch":
        _check(L.bwacuda_extend_batch(ctx.h, _vp(state["jobs"]), n, 5, mat, *_SCORING, 100, _END_BONUS, _ZDROP,
                                      _vp(state["out"])), kind)
        return state["out"]
    if kind == "retry":
        _check(L.bwacuda_extend_batch_retry(ctx.h, _vp(state["jobs"]), n, 5, mat, *_SCORING, state["case"]["w"],
                                            _END_BONUS, _ZDROP, 2, _vp(state["prev"]), _vp(state["out"]),
                                            _vp(state["w_used"])), kind)
        return [state["out"], state["w_used"]]
    if kind in ("extend_device", "extend_long"):
        ctx.extend_device(state["seq"].data_ptr(), state["jobs"].data_ptr(), n, state["out"].data_ptr())
        ctx.sync()  # waits for the results and reports bad input
        return state["out"]
    if kind == "rescue_device":
        ctx.ksw_align2_device(state["seq"].data_ptr(), state["jobs"].data_ptr(), n, state["out"].data_ptr(),
                              minsc=_MINSC)
        ctx.sync()
        return state["out"]
    if kind == "rescue_batch":
        _check(L.bwacuda_ksw_align2_batch(ctx.h, _vp(state["jobs"]), n, 5, mat, *_SCORING, _MINSC, 1,
                                          _vp(state["out"])), kind)
        return state["out"]
    if kind == "windows":
        _check(L.bwacuda_mate_rescue_windows(ctx.h, _vp(state["reqs"]), n, 5, mat, *_SCORING, _MINSC, 1, _MIN_SEED,
                                             _vp(state["out"])), kind)
        return {f: state["out"][f] for f in state["out"].dtype.names}
    if kind == "cigar":
        words = state["words"]
        _check(L.bwacuda_ksw_global2_batch(ctx.h, _vp(state["jobs"]), n, 5, mat, *_SCORING, _vp(state["score"]),
                                           _vp(state["offs"]), _vp(words), len(words)), kind)
        return [state["score"], state["offs"].view(np.int64), words.view(np.int32)]
    ids = []
    for ep, ne, rp, nr, w, _ in state["requests"]:
        rid = C.c_uint64()
        _check(L.bwacuda_server_submit_mixed(ctx.h, C.c_void_p(ep), ne, C.c_void_p(rp), nr, C.byref(state["sc"]), w,
                                             _END_BONUS, _ZDROP, _MINSC, 1, C.byref(rid)), "submit")
        ids.append(rid)
    for rid, req in zip(ids, state["requests"]):
        _check(L.bwacuda_server_wait(ctx.h, rid, C.c_void_p(state["out"].ctypes.data + req[5]), -1, None), "wait")
    return state["out"]


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    kind, n = case["kind"], case.get("jobs", 1)
    if kind == "extend":
        rows = case["qlen"] + 100
        return {"bytes": case["qlen"] + rows + 24, "flops": _OPS_EXT * case["qlen"] * rows // 2}
    if kind in ("extend_batch", "extend_device", "retry"):
        cells = _EXT_CELLS[case["workload"]]
        if case.get("ungapped") and case["workload"] != 1:
            cells = cells * 3 // 100  # the closed form settles 97% of the read-pair jobs
        if case.get("w", 100) < 100:
            cells = min(cells, 160 * (2 * case["w"] + 1))
        return {"bytes": n * (_EXT_BASES[case["workload"]] + 32 + 24), "flops": _OPS_EXT * cells * n}
    if kind == "extend_long":
        q = (case["qmin"] + case["qmax"]) // 2
        return {"bytes": n * (2 * q + 100 + 32 + 24), "flops": _OPS_EXT * n * q * 200}
    if kind in ("rescue_device", "rescue_batch", "windows"):
        q = (case["qmin"] + case["qmax"]) // 2 if "qmin" in case else 150
        t = (case["tmin"] + case["tmax"]) // 2 if "tmin" in case else 750
        return {"bytes": n * ((q + t if "tmin" in case else q + t // 4) + 32 + 28), "flops": _OPS_LOCAL * n * q * t}
    if kind == "cigar":
        return {"bytes": n * (311 + 40 + 20), "flops": _OPS_LOCAL * n * 12900}
    plan = _serve_plan(case)
    ne, nr = sum(p[0] for p in plan), sum(p[1] for p in plan)
    return {"bytes": ne * 280 + nr * 960, "flops": _OPS_EXT * ne * 5400 + _OPS_LOCAL * nr * 150 * 750}


def exact(case, seed):
    """Every output is a whole number."""
    return None
