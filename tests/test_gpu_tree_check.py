"""Every index bound of a tree view raises when broken, and the edges of the
accepted ranges pass (``vl1_tree_check``)."""

import numpy as np
import pytest

from volumential_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _arrays(w):
    import torch

    tr, tree = w.traversal, w.tree
    local = tree.box_local_mode_ids()
    dev = lambda a, dt=torch.int32: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dt)  # noqa
    return dict(
        target_boxes=dev(tr.target_boxes),
        neighbor_source_boxes_starts=dev(tr.neighbor_source_boxes_starts),
        neighbor_source_boxes_lists=dev(tr.neighbor_source_boxes_lists),
        box_centers=dev(tree.box_centers, torch.float64),
        box_levels=dev(tree.box_levels, torch.uint8),
        box_source_starts=dev(tree.box_target_starts),
        box_source_counts_nonchild=dev(tree.box_target_counts_nonchild),
        box_target_starts=dev(tree.box_target_starts),
        box_target_counts_nonchild=dev(tree.box_target_counts_nonchild),
        source_mode_ids=dev(local), target_point_ids=dev(local), root_extent=tree.root_extent)


@pytest.fixture(scope="module")
def w():
    return W.uniform_workload("check", 2, 4, 3, seed=31)


@pytest.mark.parametrize("name,index,value", [
    ("target_boxes", 3, -1), ("target_boxes", -1, "nboxes"),
    ("neighbor_source_boxes_starts", 0, 1), ("neighbor_source_boxes_starts", -1, "nnz+1"),
    ("neighbor_source_boxes_starts", 5, 0), ("neighbor_source_boxes_lists", 0, -1),
    ("neighbor_source_boxes_lists", -1, "nboxes"), ("box_levels", -1, 61),
    ("box_source_starts", -1, -1), ("box_source_starts", -1, "npart"),
    ("box_target_starts", -1, -1), ("box_target_starts", -1, "npart"),
    ("box_source_counts_nonchild", -1, -1), ("box_source_counts_nonchild", -1, 10),
    ("box_target_counts_nonchild", -1, -2), ("box_target_counts_nonchild", -1, 10)])
def test_broken_bounds_raise(cuda, w, name, index, value):
    from volumential_gb300.plan import tree_view_from_arrays

    a = _arrays(w)
    sizes = {"nboxes": a["box_levels"].numel(), "npart": a["source_mode_ids"].numel(),
             "nnz+1": a["neighbor_source_boxes_lists"].numel() + 1}
    a[name][index] = sizes.get(value, value)
    with pytest.raises(ValueError):
        tree_view_from_arrays(**a)


def test_edges_of_the_ranges_pass(cuda, w):
    from volumential_gb300.plan import tree_view_from_arrays

    a = _arrays(w)
    empty = (a["box_source_counts_nonchild"] == 0).nonzero()[0]
    a["box_source_starts"][empty] = -7       # unused: the box has no sources
    a["box_target_starts"][empty] = 10 ** 6
    a["box_levels"][empty] = 60
    tree_view_from_arrays(**a)
