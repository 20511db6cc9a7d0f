"""The persistent tensor-core kernel: several work items per CTA.

Every CTA of a launch takes work items until none is left, its pipeline, its
exact buffers and its row data running on from item to item.  The cases have
many more items than CTAs (short ones, so that one item's first unit follows
the last of the one before; rounds that end inside an item; one and two column
chunks; splits), compare with the FP64 path, and check that repeated calls
give the same bits.  Tolerances: sums of digit products that keep ~2^-38 of
the largest products, as for the other tests of this path.
"""

import gc

import numpy as np
import pytest

from helpers import plan_and_view, rel_l2
from volumential_gb300 import workloads as W
from volumential_gb300.batch import BatchProblem, MixedBatch
from volumential_gb300.batched import eval_mixed, get_schedule
from volumential_gb300.kernels import HelmholtzKernel
from volumential_gb300.plan import as_device_tensor

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _collect():
    """Leave no device tensors in reference cycles for later memory checks."""
    yield
    gc.collect()

TOL_MIXED = 1e-9


def _mixed(torch, w, plan, view, keep, coefs, nrhs, cap=None):
    stream = torch.cuda.current_stream().cuda_stream
    odt = torch.complex128 if plan.complex_table else torch.float64
    outs = []
    for _ in range(2):
        out = torch.full((nrhs, w.n_points), float("nan"), dtype=odt, device="cuda")
        eval_mixed(plan, view, coefs, out, stream=stream, nrhs=nrhs, keep=keep,
                   max_keys_per_item=cap)
        plan.raise_on_status(stream)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    return outs[0]


def _fp64(torch, plan, view, coefs, like):
    out = torch.full_like(like, float("nan"))
    stream = torch.cuda.current_stream().cuda_stream
    for r in range(like.shape[0]):
        plan.eval_fp64(view, coefs[r], out[r], stream=stream)
    plan.raise_on_status(stream)
    return out


CASES = {
    # 2D q = 3: one 16-column chunk, 9 one-unit keys (3 rounds) per tile
    "2d-q3": lambda: W.uniform_workload("mp1", 2, 5, 3, seed=61, nrhs=90),
    # complex 2D q = 5: 50 of 64 columns, real and imaginary parts interleaved
    "2d-q5-complex": lambda: W.uniform_workload(
        "mp2", 2, 5, 5, seed=62, kernel=HelmholtzKernel(2), complex_table=True, nrhs=50),
    # complex 2D q = 4: 32 of 32 columns, two CTAs per SM
    "2d-q4-complex": lambda: W.uniform_workload(
        "mp3", 2, 5, 4, seed=63, kernel=HelmholtzKernel(2), complex_table=True, nrhs=85),
    # 3D q = 5: two column chunks of 64, four units per key
    "3d-q5": lambda: W.uniform_workload("mp4", 3, 3, 5, seed=64, nrhs=41),
}


@pytest.mark.parametrize("cap", [None, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_many_items_per_cta(cuda, name, cap):
    torch = cuda
    w = CASES[name]()
    if w.tables is not None and name.endswith("complex"):
        w.tables = W.synthetic_tables(2, w.q, w.kernel, seed=7, complex_values=True,
                                      source_box_extent=w.tree.root_extent / 32)
    plan, view, keep = plan_and_view(w)
    nrhs = w.coefs.shape[0]
    coefs = as_device_tensor(np.ascontiguousarray(w.coefs))
    got = _mixed(torch, w, plan, view, keep, coefs, nrhs, cap)
    stream = torch.cuda.current_stream().cuda_stream
    sched = get_schedule(plan, view, keep, nrhs, stream, cap)
    geo = plan.mixed_geometry()
    n_items = max(sched.n_items, sched.n_tiles) * (geo["np"] // geo["nch"])
    per_sm = 1 if geo["nch"] >= 64 else 2
    n_sm = torch.cuda.get_device_properties(0).multi_processor_count
    assert n_items > (1 if cap is None else 2) * per_sm * n_sm
    want = _fp64(torch, plan, view, coefs, got).cpu().numpy()
    got = got.cpu().numpy()
    for r in range(nrhs):
        assert rel_l2(got[r], want[r]) <= TOL_MIXED


@pytest.mark.parametrize("ctas", [1, 7, 0])
def test_capped_batch_launch_runs_every_item(cuda, ctas):
    """A batch launch of few CTAs walks all items of two problems."""
    torch = cuda
    ws = [W.uniform_workload("mb1", 2, 4, 4, seed=66, nrhs=3),
          W.adaptive_workload("mb2", 2, 4, tol=1e-2, max_level=5, min_level=2, seed=67)]
    probs, wants = [], []
    for w in ws:
        plan, view, keep = plan_and_view(w)
        nrhs = w.coefs.shape[0]
        coefs = as_device_tensor(np.ascontiguousarray(w.coefs))
        out = torch.full((nrhs, w.n_points), float("nan"), dtype=torch.float64, device="cuda")
        probs.append(BatchProblem(plan, view, keep, coefs, out, nrhs))
        wants.append(_fp64(torch, plan, view, coefs, out).cpu().numpy())
    batch = MixedBatch(probs, max_keys_per_item=2, ctas_per_launch=ctas)
    for _ in range(2):
        for p in probs:
            p.out.fill_(float("nan"))
        batch.eval()
        batch.raise_on_status()
        for p, want in zip(probs, wants):
            got = p.out.cpu().numpy()
            for r in range(len(want)):
                assert rel_l2(got[r], want[r]) <= TOL_MIXED


def test_items_with_large_tails(cuda):
    """Items of more than 2^14 source points convert their tails the general
    way; cut into short items they take the other one."""
    torch = cuda
    w = W.adaptive_workload("mt", 3, 6, tol=3e-2, max_level=5, min_level=2, seed=68)
    plan, view, keep = plan_and_view(w)
    coefs = as_device_tensor(np.ascontiguousarray(w.coefs))
    whole = _mixed(torch, w, plan, view, keep, coefs, 1, 1 << 30)
    stream = torch.cuda.current_stream().cuda_stream
    kp = plan.mixed_geometry()["kp"]
    assert get_schedule(plan, view, keep, 1, stream, 1 << 30).max_keys_per_item * kp > 1 << 14
    cut = _mixed(torch, w, plan, view, keep, coefs, 1, 5)
    assert get_schedule(plan, view, keep, 1, stream, 5).max_keys_per_item * kp < 1 << 14
    want = _fp64(torch, plan, view, coefs, whole).cpu().numpy()
    whole, cut = whole.cpu().numpy(), cut.cpu().numpy()
    assert rel_l2(whole[0], want[0]) <= TOL_MIXED
    assert rel_l2(cut[0], want[0]) <= TOL_MIXED


def test_subnormal_and_zero_results(cuda):
    """Results below the normal range are rounded as FP64 rounds them: within
    the path's accuracy and one unit of the subnormal spacing."""
    torch = cuda
    w = W.uniform_workload("ms", 2, 3, 3, seed=69, nrhs=2)
    plan, view, keep = plan_and_view(w)
    c = np.ascontiguousarray(w.coefs)
    want = _fp64(torch, plan, view, as_device_tensor(c), torch.empty(
        c.shape, dtype=torch.float64, device="cuda")).cpu().numpy()
    scale = 2.0 ** -1030 / np.abs(want[0]).max()   # powers of two keep the digits
    scale = 2.0 ** np.floor(np.log2(scale))
    tiny = c.copy()
    tiny[0] *= scale
    tiny[1] = 0.0
    got = _mixed(torch, w, plan, view, keep, as_device_tensor(tiny), 2).cpu().numpy()
    assert np.all(got[1] == 0.0)
    err = np.abs(got[0] / scale - want[0]).max()
    assert np.abs(got[0]).max() < 2.0 ** -1022 and np.abs(got[0]).max() > 0.0
    # the densities themselves are subnormal: half a spacing of 2^-1074 each
    bound = TOL_MIXED * np.abs(want[0]).max() + 2.0 ** -1074 / scale * (1 + w.n_points)
    assert err <= bound
