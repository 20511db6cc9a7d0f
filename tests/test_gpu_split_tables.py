"""The split remainder sum on trees of many boxes, where R is read from tables
by relative position: against the CPU restatement on uniform and adaptive
trees, real and complex weights and wave numbers, with and without the self
pairs; the general kernel takes over when the points are no template.

Tolerance 1e-12 relative l2, as for the per-pair sum (FP64 sums of at most a
few thousand terms; the points' own rounding changes R by less)."""

import numpy as np
import pytest

from helpers import plan_and_view, rel_l2
from oracle import split_oracle as SO
from volumential_gb300 import workloads as W
from volumential_gb300.helmholtz_split import (max_neighbor_distance, series_terms,
                                               split_correction)
from volumential_gb300.kernels import LaplaceKernel

pytestmark = pytest.mark.gpu


def _sum(w, weights, k, points=None, exclude=True):
    import torch

    _, view, keep = plan_and_view(w)
    pts = torch.from_numpy(np.ascontiguousarray(w.tree.targets if points is None
                                                else points)).cuda()
    n = series_terms(w.dim, k, max_neighbor_distance(w.tree))
    out = split_correction(view, pts, torch.from_numpy(np.ascontiguousarray(weights)).cuda(), k,
                           n, exclude_self=exclude)
    return out.cpu().numpy()


def _ref(w, weights, k, points=None, exclude=True):
    tr, tree = w.traversal, w.tree
    return SO.split_sum(w.dim, k, tree.targets if points is None else points,
                        np.asarray(weights, dtype=np.complex128), tr.target_boxes,
                        tr.neighbor_source_boxes_starts, tr.neighbor_source_boxes_lists,
                        tree.box_target_starts, tree.box_target_counts_nonchild,
                        exclude_self=exclude)


@pytest.mark.parametrize("dim,level,q,k,cw", [(2, 5, 2, 20.0, False), (2, 5, 3, 7.5, True),
                                              (2, 5, 2, 3.0 + 1.0j, False),
                                              (3, 3, 2, 9.0, False), (3, 3, 2, 4.0 + 0.5j, True)])
@pytest.mark.parametrize("exclude", [True, False])
def test_uniform_trees(cuda, dim, level, q, k, cw, exclude):
    w = W.uniform_workload("split_t", dim, level, q, seed=21, kernel=LaplaceKernel(dim))
    wts = w.coefs[0] * w.tree.weights * ((1.0 + 0.3j) if cw else 1.0)
    assert len(w.traversal.target_boxes) >= 512
    assert rel_l2(_sum(w, wts, k, exclude=exclude), _ref(w, wts, k, exclude=exclude)) <= 1e-12


@pytest.mark.parametrize("dim,q,tol,level", [(2, 3, 0.02, 6), (3, 2, 0.02, 5)])
def test_adaptive_trees(cuda, dim, q, tol, level):
    w = W.adaptive_workload("split_a", dim, q, tol=tol, max_level=level, seed=22)
    assert len(w.traversal.target_boxes) >= 512
    wts = w.coefs[0] * w.tree.weights
    assert rel_l2(_sum(w, wts, 11.0), _ref(w, wts, 11.0)) <= 1e-12


def test_moved_points_take_the_general_kernel(cuda):
    w = W.uniform_workload("split_m", 2, 5, 3, seed=23, kernel=LaplaceKernel(2))
    pts = w.tree.targets.copy()
    pts[0, 1000] += 1e-5               # one point off its box's template
    wts = w.coefs[0] * w.tree.weights
    got, ref = _sum(w, wts, 20.0, points=pts), _ref(w, wts, 20.0, points=pts)
    assert rel_l2(got, ref) <= 1e-12
    assert rel_l2(_sum(w, wts, 20.0), ref) > 1e-12    # the move is seen
