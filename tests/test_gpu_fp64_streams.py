"""FP64 schedules built on one stream and read on others.

A schedule's arrays come from the memory pool of torch's current stream, are
filled on the evaluation's stream and kept for evaluations on any stream.  The
tests put a pause (a device-side sleep) where an order is needed: before the fill
kernels, before the work that used the memory last, and before a reader whose
schedule is dropped.  Results are the tensor-core path's own, bit for bit (its
sums are integers)."""

import gc

import pytest

from helpers import plan_and_view
from volumential_gb300 import _lib
from volumential_gb300 import workloads as W
from volumential_gb300.batched import MixedSchedule, _held

pytestmark = pytest.mark.gpu

PAUSE = 40_000_000      # clocks, about 20 ms


@pytest.fixture
def problem(cuda):
    torch = cuda
    w = W.uniform_workload("streams", 3, 3, 4, seed=81)
    plan, view, keep = plan_and_view(w)
    c = torch.from_numpy(w.coefs[0]).cuda()
    want = torch.empty_like(c)
    for _ in range(2):
        plan.eval_fp64(view, c, want, stream=0, keep=keep)
    plan.raise_on_status(0)
    assert view.fp64_schedules[1][1] is not None
    torch.cuda.synchronize()
    return plan, view, keep, c, want


def _forget(view):
    """The view as new: its schedules dropped."""
    del view._fp64_known, view.fp64_schedules


def test_a_schedule_is_complete_when_another_stream_gets_it(problem, cuda, monkeypatch):
    torch = cuda
    plan, view, keep, c, want = problem
    lib = _lib.lib()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    fill = lib.vl1_schedule_build_fill

    def late(*args):
        with torch.cuda.stream(a):
            torch.cuda._sleep(PAUSE)
        return fill(*args)

    monkeypatch.setattr(lib, "vl1_schedule_build_fill", late)
    _forget(view)
    outs = [torch.zeros_like(c) for _ in range(3)]
    torch.cuda.synchronize()
    plan.eval_fp64(view, c, outs[0], stream=a.cuda_stream, keep=keep)   # seen
    plan.eval_fp64(view, c, outs[1], stream=a.cuda_stream, keep=keep)   # built
    plan.eval_fp64(view, c, outs[2], stream=b.cuda_stream, keep=keep)
    b.synchronize()
    assert torch.equal(outs[2], want)
    a.synchronize()
    assert torch.equal(outs[1], want)
    plan.raise_on_status(0)


def test_the_fill_waits_for_the_memorys_last_user(problem, cuda):
    """The arrays take over blocks that the current stream still writes."""
    torch = cuda
    plan, view, keep, c, want = problem
    s = view.fp64_schedules[1][1]
    sizes = [t.numel() for t in (s.tile_rows, s.tile_key_start, s.key_ids, s.key_xrow)]
    _forget(view)
    del s
    gc.collect()
    a = torch.cuda.Stream()
    outs = [torch.zeros_like(c) for _ in range(2)]
    plan.eval_fp64(view, c, outs[0], stream=a.cuda_stream, keep=keep)
    torch.cuda.synchronize()
    blocks = [torch.empty(n, dtype=torch.int32, device="cuda") for n in sizes for _ in range(2)]
    torch.cuda._sleep(PAUSE)
    for t in blocks:
        t.fill_(-1)
    del blocks, t
    plan.eval_fp64(view, c, outs[1], stream=a.cuda_stream, keep=keep)
    torch.cuda.synchronize()
    assert torch.equal(outs[1], want)
    for _ in range(2):
        plan.eval_fp64(view, c, outs[1], stream=a.cuda_stream, keep=keep)
    torch.cuda.synchronize()
    assert torch.equal(outs[1], want)
    plan.raise_on_status(0)


@pytest.mark.parametrize("capturing", [False, True])
def test_a_dropped_schedule_outlives_its_readers(problem, cuda, capturing):
    torch = cuda
    plan, view, keep, c, want = problem
    s = view.fp64_schedules[1][1]
    sizes = [t.numel() for t in (s.tile_rows, s.tile_key_start, s.key_ids, s.key_xrow, s.items)]
    del s
    a = torch.cuda.Stream()
    out, other = torch.zeros_like(c), torch.zeros_like(c)
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(PAUSE)
    plan.eval_fp64(view, c, out, stream=a.cuda_stream, keep=keep)
    if capturing:       # dropped while a stream is being captured
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, capture_error_mode="thread_local"):
            other.fill_(3.0)
            _forget(view)
            gc.collect()
        g.replay()
    else:
        _forget(view)
        gc.collect()
    blocks = [torch.empty(n, dtype=torch.int32, device="cuda").fill_(-1) for n in sizes
              for _ in range(2)]
    a.synchronize()
    assert torch.equal(out, want)
    if capturing:
        torch.cuda.synchronize()
        assert torch.equal(other, torch.full_like(c, 3.0))
    del blocks
    plan.raise_on_status(0)


def test_many_streams(problem, cuda):
    """More streams than a schedule notes readers of, then other schedules:
    nothing stays behind."""
    torch = cuda
    plan, view, keep, c, want = problem
    s = view.fp64_schedules[1][1]
    assert isinstance(s, MixedSchedule)
    outs = []
    for _ in range(80):
        st = torch.cuda.Stream()
        out = torch.zeros_like(c)
        st.wait_stream(torch.cuda.current_stream())
        plan.eval_fp64(view, c, out, stream=st.cuda_stream, keep=keep)
        outs.append(out)
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
    _forget(view)
    del s
    gc.collect()
    assert not _held


def test_capture_of_a_stream_that_is_not_current(problem, cuda):
    """The evaluation's stream is captured while torch's current stream is
    another: no schedule is built (that would end the capture), the graph
    replays the per-box kernel."""
    torch = cuda
    plan, view, keep, c, want = problem
    ref = torch.empty_like(c)
    plan.eval_fp64(view, c, ref, stream=0)
    _forget(view)
    a, out = torch.cuda.Stream(), torch.zeros_like(c)
    plan.eval_fp64(view, c, out, stream=a.cuda_stream, keep=keep)      # seen
    torch.cuda.synchronize()
    out.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(a):
        g.capture_begin(capture_error_mode="thread_local")
        with torch.cuda.stream(torch.cuda.default_stream()):
            plan.eval_fp64(view, c, out, stream=a.cuda_stream, keep=keep)
        g.capture_end()
    torch.cuda.synchronize()
    assert torch.count_nonzero(out) == 0
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    plan.eval_fp64(view, c, out, stream=a.cuda_stream, keep=keep)
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    plan.raise_on_status(0)
