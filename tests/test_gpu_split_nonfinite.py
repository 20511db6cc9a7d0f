"""Infinite and NaN weights in the split remainder sum: a target whose own
weight is not finite does not see it when self pairs are excluded, by the
tables of R as by the per-pair kernel.

The per-pair kernel runs when a tree has fewer than 512 target boxes or when its
points are no template; here one point of a far box is moved by more than the
template test's bound and less than any tolerance."""

import numpy as np
import pytest

from helpers import plan_and_view, rel_l2
from volumential_gb300 import workloads as W
from volumential_gb300.helmholtz_split import (max_neighbor_distance, series_terms,
                                               split_correction)
from volumential_gb300.kernels import LaplaceKernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,level,q", [(2, 5, 3), (3, 3, 2)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("exclude", [True, False])
def test_own_weight(cuda, dim, level, q, value, cplx, exclude):
    import torch

    w = W.uniform_workload("split_n", dim, level, q, seed=24, kernel=LaplaceKernel(dim))
    _, view, _keep = plan_and_view(w)
    k = 20.0 if dim == 2 else 9.0
    n = series_terms(dim, k, max_neighbor_distance(w.tree))
    wts = w.coefs[0] * w.tree.weights * (1.0 + 0.5j if cplx else 1.0)
    i = w.n_points // 3
    wts[i] = value
    moved = w.tree.targets.copy()
    moved[0, -1] += 1e-11                   # per-pair kernel

    def run(points):
        return split_correction(view, torch.from_numpy(np.ascontiguousarray(points)).cuda(),
                                torch.from_numpy(wts).cuda(), k, n,
                                exclude_self=exclude).cpu().numpy()

    got, ref = run(w.tree.targets), run(moved)
    assert np.isfinite(ref[i]) == exclude
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    fine = np.isfinite(ref)
    assert 0 < fine.sum() < fine.size and rel_l2(got[fine], ref[fine]) <= 1e-9
