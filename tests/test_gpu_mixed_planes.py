"""Density digit planes: the FP64 multiply-add against the integer shifts.

The plane pass takes a row's digits by one FP64 multiply-add when its scale
exponent is moderate, and rows of one box together when all of a group are
right-hand sides of that box.  Scaling the densities of a right-hand side by a
power of two scales its results by the same power exactly on either path, so
a call whose exponents lie far below that range (integer shifts, rows taken
singly) must give the same bits as the one with moderate exponents, with the
same schedule.
"""

import gc

import numpy as np
import pytest

from helpers import plan_and_view
from volumential_gb300 import workloads as W
from volumential_gb300.batched import eval_mixed
from volumential_gb300.plan import as_device_tensor

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _collect():
    """Leave no device tensors in reference cycles for later memory checks."""
    yield
    gc.collect()


def _mixed(torch, w, plan, view, keep, coefs):
    nrhs = coefs.shape[0]
    stream = torch.cuda.current_stream().cuda_stream
    out = torch.full((nrhs, w.n_points), float("nan"), dtype=torch.float64, device="cuda")
    eval_mixed(plan, view, as_device_tensor(np.ascontiguousarray(coefs)), out, stream=stream,
               nrhs=nrhs, keep=keep)
    plan.raise_on_status(stream)
    return out.cpu().numpy()


@pytest.mark.parametrize("dim,q", [(2, 3), (2, 5), (3, 3), (3, 4)])
@pytest.mark.parametrize("nrhs", [1, 31, 32, 37])
def test_planes_agree_over_scales_and_groups(cuda, dim, q, nrhs):
    torch = cuda
    w = W.adaptive_workload("pl", dim, q, tol=3e-2, max_level=4, min_level=2, seed=91)
    plan, view, keep = plan_and_view(w)
    rng = np.random.default_rng(92)
    base = np.asarray(w.coefs[0])
    # the first density with the largest magnitudes at the very scale bound
    # (one below a power of two), ties of the last digit, zeros and signs
    c = base[None, :] * rng.uniform(-1.0, 1.0, (nrhs, w.n_points))
    c /= np.abs(c).max(axis=1, keepdims=True) * (1.0 + 2.0 ** -52)
    tie = rng.integers(0, w.n_points, (nrhs, 40))
    np.put_along_axis(c, tie, (rng.integers(-2 ** 20, 2 ** 20, tie.shape) + 0.5) * 2.0 ** -39, 1)
    np.put_along_axis(c, rng.integers(0, w.n_points, (nrhs, 20)), 0.0, 1)
    c[:, 0] = 1.0 - 2.0 ** -53
    want = _mixed(torch, w, plan, view, keep, c)
    # far below the moderate range: integer shifts for every row
    far = _mixed(torch, w, plan, view, keep, c * 2.0 ** -920)
    assert np.array_equal(far * 2.0 ** 460 * 2.0 ** 460, want)


@pytest.mark.parametrize("gap", [0, 3])
@pytest.mark.parametrize("dim,level,q,nrhs", [(2, 4, 3, 5), (2, 4, 5, 33), (3, 2, 3, 4)])
def test_scales_of_scattered_boxes(cuda, dim, level, q, nrhs, gap):
    """Boxes in another order than their points, or with unused values between
    them, have the scale exponents of their own points only."""
    torch = cuda
    from volumential_gb300.plan import tree_view_from_arrays

    w = W.uniform_workload("sc", dim, level, q, seed=93, nrhs=nrhs)
    plan, view, keep = plan_and_view(w)
    rng = np.random.default_rng(94)
    nq, n = q ** dim, w.n_points
    want = _mixed(torch, w, plan, view, keep, w.coefs)
    # leaf i's points move to block place[i], blocks `gap` values apart
    place = rng.permutation(n // nq)
    if gap:
        place = np.arange(n // nq)   # in order, but not adjacent
    stride = nq + gap
    total = stride * (n // nq)
    counts = keep["src_counts"].cpu().numpy()
    starts = keep["src_starts"].cpu().numpy()
    new = starts.copy()
    new[counts > 0] = place[starts[counts > 0] // nq] * stride
    pos = (place[:, None] * stride + np.arange(nq)[None, :]).reshape(-1)
    modes = np.zeros(total, dtype=np.int32)
    modes[pos] = keep["smode"].cpu().numpy()
    coefs = np.full((nrhs, total), 1e200)
    coefs[:, pos] = w.coefs
    v2, k2 = tree_view_from_arrays(
        target_boxes=keep["target_boxes"], neighbor_source_boxes_starts=keep["starts"],
        neighbor_source_boxes_lists=keep["lists"], box_centers=keep["centers"],
        box_levels=keep["levels"], box_source_starts=new,
        box_source_counts_nonchild=counts, box_target_starts=new,
        box_target_counts_nonchild=counts, source_mode_ids=modes, target_point_ids=modes,
        root_extent=w.tree.root_extent)
    out = torch.full((nrhs, total), 7.0, dtype=torch.float64, device="cuda")
    eval_mixed(plan, v2, as_device_tensor(coefs), out,
               stream=torch.cuda.current_stream().cuda_stream, nrhs=nrhs, keep=k2)
    plan.raise_on_status(torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    assert np.array_equal(got[:, pos], want)
    rest = np.ones(total, dtype=bool)
    rest[pos] = False
    assert np.all(got[:, rest] == 7.0)
