"""The length buckets (BWACUDA_OPT_SMALL_BATCH 0) on batches that by themselves would run without them: the
tests of the persistent kernels, their launch shapes and cell widths, the group-per-job kernel on shorter
buckets, the retry rounds and concurrent callers, each on a context whose every batch is sorted into buckets,
and the kernels that a call then launches."""
import numpy as np
import pytest

import bwacuda as B
import oracle
import test_concurrency_gpu as TC
import test_extend_gpu as TE
import test_long_gpu as TL
import test_retry_gpu as TR
from kernel_trace import kernels

pytestmark = pytest.mark.gpu

HOSTPACK, DEVGATHER = (B.PATH_BATCHED, B.GATHER_HOST), (B.PATH_BATCHED, B.GATHER_DEVICE)
SCORINGS = [(1, 4, 6, 1, 6, 1, 5, 100), (2, 3, 5, 2, 4, 3, 0, 40), (1, 1, 0, 1, 0, 1, 9, 0), (3, 5, 11, 1, 7, 2, 1, 200),
            (1, 4, 6, 1, 6, 1, 5, 1), (1, 4, 16383, 1, 16000, 384, 5, 100), (2, 4, 30000, 3000, 17000, 5, 5, 100)]


@pytest.fixture
def bctx():
    with B.Context(0) as ctx:
        ctx.set_option(B.OPT_EXT_PATH, B.PATH_BATCHED)
        ctx.set_option(B.OPT_SMALL_BATCH, 0)
        yield ctx


@pytest.fixture(scope="module")
def classes():
    """Jobs of all three cell widths and every bucket, and their results."""
    a, b = B.synth_ext(3, 9000, seed=14), TL.long_jobs(300, 257, 1100, 100, seed=3)
    js = B.JobSet(np.concatenate([a.seq, b.seq]), np.concatenate([a.q_off, b.q_off + len(a.seq)]),
                  np.concatenate([a.t_off, b.t_off + len(a.seq)]),
                  *[np.concatenate([getattr(a, f), getattr(b, f)]) for f in ("qlen", "tlen", "h0", "w")])
    js.h0 = js.h0.copy()
    js.h0[::3] += 300  # 16-bit cells
    js.h0[::5] = 33000  # 32-bit cells
    return js, oracle.extend_batch(js)[0]


@pytest.mark.parametrize("step", [16, 32, 64])
@pytest.mark.parametrize("grab", [1, 2, 4])
@pytest.mark.parametrize("block", [32, 64, 128, 256])
def test_launch_shapes(bctx, classes, block, grab, step):
    js, want = classes
    bctx.set_option(B.OPT_PERSIST_BLOCK, block)
    bctx.set_option(B.OPT_GRAB, grab)
    bctx.set_option(B.OPT_BUCKET_STEP, step)
    outs = []
    names = kernels(lambda: outs.extend(TE._device_run(bctx, js, B.PATH_BATCHED, reps=2)))  # captured, replayed
    for got in outs:
        assert np.array_equal(got, want)
    if names is not None:
        for kernel in (f"ext_persist_pair_kernel<{block}, {grab}, false>", f"ext_persist_pair_kernel<{block}, {grab}, true>",
                       f"ext_persist_kernel<FmtI32, {block}, {grab}>"):
            assert any(kernel in n for n in names), kernel


@pytest.mark.parametrize("scoring", SCORINGS)
def test_cell_classes(bctx, scoring):
    TE.test_pair_cell_classes_swept(bctx, scoring)


@pytest.mark.parametrize("path", [HOSTPACK, DEVGATHER], ids=["hostpack", "devgather"])
def test_wide_cells(bctx, path):
    js = [None]
    names = kernels(lambda: js.append(TE.test_wide_cells_for_large_scores(bctx, path)))
    assert names is None or any("ext_persist_kernel<FmtI32" in n for n in names)


@pytest.mark.parametrize("path", [HOSTPACK, DEVGATHER], ids=["hostpack", "devgather"])
def test_streams_and_workloads(bctx, path):
    TE.test_batch_streams_through_both_paths(bctx, path)
    TE.test_workload_mixed_lengths_and_bands(bctx, path)
    TE.test_edge_cases(bctx, path)
    TE.test_invalid_inputs_fail_loudly(bctx, path)
    TE.test_invalid_job_in_a_later_chunk(bctx, path)


def test_long_queries_short_targets(bctx):
    for scoring in SCORINGS[:2]:
        TE.test_long_queries_short_targets(bctx, scoring)


def test_device_calls(bctx):
    TE.test_device_entry_equals_oracle(bctx, B.PATH_BATCHED)
    TE.test_device_batch_in_pieces(bctx, B.PATH_BATCHED)


def test_feeds_agree(bctx):
    TE.test_chunked_pipeline_boundaries(bctx)
    TE.test_device_gather_equals_host_packing(bctx)


@pytest.mark.parametrize("lanes", [8, 16, 32])
@pytest.mark.parametrize("qlo", [1, 129])
def test_group_kernel_on_shorter_buckets(bctx, qlo, lanes):
    names = kernels(lambda: TL.test_knobs_route_shorter_buckets(bctx, lanes, qlo))
    assert names is None or any(f"ext_long_kernel<false, {lanes}, 8>" in n for n in names)


@pytest.mark.parametrize("lanes", [8, 32])
def test_gate_stream_through_group_kernel(bctx, lanes):
    TL.test_gate_stream_through_group_kernel(bctx, lanes)


@pytest.mark.parametrize("slide", [0, 1, 2])
def test_open_ended_buckets(bctx, slide):
    """0: the group-per-job kernel alone; 1, 2: the band kernel, 32 and 8 lanes a job at this size."""
    bctx.set_option(B.OPT_LONG_SLIDE, slide)
    for case in (TL.test_long_queries_16bit, TL.test_long_queries_mixed_with_read_pairs, TL.test_long_queries_32bit_cells,
                 TL.test_long_queries_short_targets, TL.test_other_scorings):
        case(bctx)
    for w in (99, 101, 102, 300, 3000):
        TL._check(bctx, TL.long_jobs(30, 1030, 4000, w, seed=40 + w), w)


def test_retry_rounds(bctx):
    for w0, tries in ((100, 2), (8, 2), (3, 4), (0, 2)):
        for route in (B.GATHER_HOST, B.GATHER_AUTO):
            TR.test_host_retry_matches_run_side(bctx, route, w0, tries)
    for piece in (1 << 30, 7001):
        TR.test_device_retry_per_job_bands(bctx, piece)


def test_threads_on_one_context(bctx):
    TC.test_threads_share_one_context(bctx, B.PATH_BATCHED)
