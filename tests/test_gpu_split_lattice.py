"""The split remainder sum reads R by relative position only on trees whose
centres lie on their lattice; it uses the points alone otherwise.

The oracle forms every distance from the points.  Tolerance 1e-12 relative l2,
as for the per-pair sum."""

import numpy as np
import pytest

from helpers import plan_and_view, rel_l2
from oracle import split_oracle as SO
from volumential_gb300 import workloads as W
from volumential_gb300.helmholtz_split import (max_neighbor_distance, series_terms,
                                               split_correction)
from volumential_gb300.kernels import LaplaceKernel

pytestmark = pytest.mark.gpu


def _check(w, view, pts, k, weights=None):
    import torch

    wts = w.coefs[0] * w.tree.weights if weights is None else weights
    tr, tree = w.traversal, w.tree
    assert len(tr.target_boxes) >= 512
    n = series_terms(w.dim, k, max_neighbor_distance(tree))
    got = split_correction(view, torch.from_numpy(pts).cuda(), torch.from_numpy(wts).cuda(), k,
                           n).cpu().numpy()
    ref = SO.split_sum(w.dim, k, pts, wts.astype(np.complex128), tr.target_boxes,
                       tr.neighbor_source_boxes_starts, tr.neighbor_source_boxes_lists,
                       tree.box_target_starts, tree.box_target_counts_nonchild)
    assert rel_l2(got, ref) <= 1e-12


@pytest.mark.parametrize("dim,level,q", [(2, 5, 3), (3, 3, 2)])
@pytest.mark.parametrize("shift", [1e-5, 1e-9, 1e-13])
def test_a_box_off_the_lattice(cuda, dim, level, q, shift):
    """One box's centre and points moved together, by parts of its size."""
    w = W.uniform_workload("lat", dim, level, q, seed=31, kernel=LaplaceKernel(dim))
    _, view, keep = plan_and_view(w)
    i = len(w.traversal.target_boxes) // 2
    box = int(w.traversal.target_boxes[i])
    s0 = int(w.tree.box_target_starts[box])
    d = shift * w.tree.root_extent * 0.5 ** level
    pts = w.tree.targets.copy()
    pts[0, s0:s0 + q ** dim] += d
    keep["centers"][0, box] += d          # the array that the view points to
    _check(w, view, pts, 20.0 if dim == 2 else 9.0)


@pytest.mark.parametrize("dim,level,q", [(2, 5, 3), (3, 3, 2)])
def test_rounded_centres(cuda, dim, level, q):
    """Centres rounded to 32 bits (boxes of a domain that is no power of two),
    the points around the rounded centres."""
    w = W.uniform_workload("lat32", dim, level, q, seed=32, kernel=LaplaceKernel(dim), a=-0.3,
                           b=0.4)
    _, view, keep = plan_and_view(w)
    c = keep["centers"]
    c32 = c.float().double()
    delta = (c32 - c).cpu().numpy()
    assert np.abs(delta).max() > 0.0
    c.copy_(c32)
    box_of = np.empty(w.n_points, dtype=np.int64)
    nq = q ** dim
    for b in w.traversal.target_boxes:
        s = int(w.tree.box_target_starts[b])
        box_of[s:s + nq] = b
    _check(w, view, np.ascontiguousarray(w.tree.targets + delta[:, box_of]),
           20.0 if dim == 2 else 9.0)


@pytest.mark.parametrize("dim,level,q", [(2, 5, 3), (3, 3, 2)])
@pytest.mark.parametrize("factor", [1e-4, 1e-9])
def test_root_extent_that_does_not_fit(cuda, dim, level, q, factor):
    w = W.uniform_workload("lat_e", dim, level, q, seed=33, kernel=LaplaceKernel(dim))
    _, view, _keep = plan_and_view(w)
    view.root_extent *= 1.0 + factor
    _check(w, view, np.ascontiguousarray(w.tree.targets), 20.0 if dim == 2 else 9.0)


@pytest.mark.parametrize("a,b", [(-0.5, 0.5), (0.1, 0.8), (1000.1, 1000.8)])
def test_trees_on_their_lattice(cuda, a, b):
    """Ordinary trees, near the origin and far from it, keep the tables'
    accuracy (the points' rounding moves R by the same amount in both sums)."""
    w = W.uniform_workload("lat_o", 2, 5, 3, seed=34, kernel=LaplaceKernel(2), a=a, b=b)
    _, view, _keep = plan_and_view(w)
    wts = np.random.default_rng(3).standard_normal(w.n_points) * w.tree.weights
    import torch

    pts = np.ascontiguousarray(w.tree.targets)
    n = series_terms(2, 20.0, max_neighbor_distance(w.tree))
    got = split_correction(view, torch.from_numpy(pts).cuda(), torch.from_numpy(wts).cuda(), 20.0,
                           n).cpu().numpy()
    tr, tree = w.traversal, w.tree
    ref = SO.split_sum(2, 20.0, pts, wts.astype(np.complex128), tr.target_boxes,
                       tr.neighbor_source_boxes_starts, tr.neighbor_source_boxes_lists,
                       tree.box_target_starts, tree.box_target_counts_nonchild)
    # coordinates rounded at 2^-53 of |x|: distances off by that over the spacing
    tol = 1e-12 + 1e-12 * max(abs(a), abs(b))
    assert rel_l2(got, ref) <= tol
