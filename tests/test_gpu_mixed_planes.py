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
