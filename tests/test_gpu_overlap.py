"""Kernels that start beside the last blocks of the one before them.

The digit passes and the tensor-core kernels are launched with programmatic
overlap.  Calls queued without a host wait, with inputs that change between
them on the stream, must give what each gives alone, bit for bit, in order of
the stream: on one stream, on two at once, and replayed from a graph.
"""

import numpy as np
import pytest

from helpers import plan_and_view
from volumential_gb300 import workloads as W
from volumential_gb300.batched import MixedSchedule, eval_mixed
from volumential_gb300.plan import as_device_tensor

pytestmark = pytest.mark.gpu

CASES = {
    "2d": lambda: W.uniform_workload("ov2", 2, 5, 4, seed=31, nrhs=6),
    "3d": lambda: W.uniform_workload("ov3", 3, 3, 4, seed=32, nrhs=2),
}


def _setup(torch, name):
    w = CASES[name]()
    plan, view, keep = plan_and_view(w)
    c = as_device_tensor(np.ascontiguousarray(w.coefs))
    # right-hand sides of very different scales: a pass that read the last
    # call's exponents or digits would show
    return w, plan, view, keep, [c, c * 2.0 ** -37, -c * 2.0 ** 90, c.flip(0) * 3.0]


def _run(torch, path, plan, view, keep, coefs, out):
    stream = torch.cuda.current_stream().cuda_stream
    if path == "mixed":
        eval_mixed(plan, view, coefs, out, stream=stream, nrhs=coefs.shape[0], keep=keep)
    else:
        plan.eval_fp64(view, coefs, out, stream=stream, nrhs=coefs.shape[0], keep=keep)


@pytest.mark.parametrize("path", ["mixed", "fp64"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_calls_queued_back_to_back(cuda, name, path):
    torch = cuda
    w, plan, view, keep, sets = _setup(torch, name)
    alone = []
    for c in sets:
        for _ in range(3):   # the FP64 rule builds its schedule when a tree comes again
            out = torch.empty_like(c)
            _run(torch, path, plan, view, keep, c, out)
            torch.cuda.synchronize()
        alone.append(out)
    buf = torch.empty_like(sets[0])
    outs = [torch.full_like(buf, float("nan")) for _ in range(40)]
    for i, out in enumerate(outs):
        buf.copy_(sets[i % 4])
        _run(torch, path, plan, view, keep, buf, out)
        buf.fill_(float("nan"))   # after the call, on its stream
    torch.cuda.synchronize()
    plan.raise_on_status(torch.cuda.current_stream().cuda_stream)
    for i, out in enumerate(outs):
        assert torch.equal(out, alone[i % 4]), i


def test_two_streams_at_once(cuda):
    torch = cuda
    w, plan, view, keep, sets = _setup(torch, "3d")
    nrhs = sets[0].shape[0]
    main = torch.cuda.current_stream().cuda_stream
    alone = []
    for c in sets[:2]:
        out = torch.empty_like(c)
        eval_mixed(plan, view, c, out, stream=main, nrhs=nrhs, keep=keep)
        alone.append(out)
    torch.cuda.synchronize()
    import ctypes as C

    from volumential_gb300 import _lib
    lib = _lib.lib()
    streams = [torch.cuda.Stream() for _ in range(2)]
    scheds = [MixedSchedule(plan, view, keep, nrhs, main) for _ in range(2)]
    torch.cuda.synchronize()
    outs = [[torch.empty_like(sets[0]) for _ in range(15)] for _ in range(2)]
    for k in range(15):
        for i in range(2):
            _lib.check(lib.vl1_eval_mixed(
                plan.handle, C.byref(view), C.byref(scheds[i].c_struct), sets[i].data_ptr(), nrhs,
                outs[i][k].data_ptr(), scheds[i].workspace.data_ptr(),
                scheds[i].workspace.numel(), C.c_void_p(streams[i].cuda_stream)),
                "vl1_eval_mixed")
    torch.cuda.synchronize()
    plan.raise_on_status(main)
    for i in range(2):
        for out in outs[i]:
            assert torch.equal(out, alone[i])


def test_replayed_from_a_graph(cuda):
    torch = cuda
    w, plan, view, keep, sets = _setup(torch, "2d")
    nrhs = sets[0].shape[0]
    alone = []
    for c in sets:
        out = torch.empty_like(c)
        _run(torch, "mixed", plan, view, keep, c, out)
        alone.append(out)
    torch.cuda.synchronize()
    buf, out = sets[0].clone(), torch.empty_like(sets[0])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _run(torch, "mixed", plan, view, keep, buf, out)
    for i in list(range(4)) * 3:
        buf.copy_(sets[i])
        out.fill_(float("nan"))
        g.replay()
        assert torch.equal(out, alone[i])
