"""Sorted box keys of trees of every depth.

The tree builder sorts the boxes' keys by as many bits as the deepest level
needs, and finds the levels' first boxes on the device.  Trees refined towards
one corner (one box of a level splits), the root alone and trees with an empty
range of levels must equal the host builder's arrays and list 1.
"""

import itertools

import numpy as np
import pytest

from test_gpu_treebuild import _same_tree
from volumential_gb300.tree_build import (
    build_list1_traversal,
    build_list1_traversal_device,
    build_tree_from_leaves,
    build_tree_from_leaves_device,
)

pytestmark = pytest.mark.gpu


def _corner_leaves(dim, depth, corner):
    """Leaves by level: the box at `corner` splits down to `depth`."""
    kids = np.array(list(itertools.product((0, 1), repeat=dim)), dtype=np.int64)
    leaves, box = {}, np.zeros((1, dim), dtype=np.int64)
    for lev in range(depth):
        children = 2 * box + kids
        pick = np.all(children % 2 == corner, axis=1)
        leaves[lev + 1] = children[~pick]
        box = children[pick]
    leaves[depth] = np.concatenate([leaves[depth], box]) if depth else box
    return leaves


@pytest.mark.parametrize("corner", [0, 1])
@pytest.mark.parametrize("dim,depth", [(2, 0), (3, 0), (2, 1), (3, 1), (2, 4), (3, 3), (2, 8),
                                       (2, 9), (3, 8)])
def test_trees_towards_a_corner(cuda, dim, depth, corner):
    leaves = _corner_leaves(dim, depth, corner)
    lv = np.concatenate([np.full(len(c), l, np.uint8) for l, c in leaves.items()])
    co = np.concatenate(list(leaves.values()))
    order = np.random.default_rng(depth).permutation(len(lv))
    host = build_tree_from_leaves({k: v.copy() for k, v in leaves.items()}, dim=dim, q_order=2)
    dev = build_tree_from_leaves_device(lv[order], co[order], dim=dim, q_order=2, balance=True)
    _same_tree(host, dev)
    hc, dc = build_list1_traversal(host), build_list1_traversal_device(dev)
    assert np.array_equal(hc.neighbor_source_boxes_lists, dc.neighbor_source_boxes_lists)
    assert np.array_equal(hc.neighbor_source_boxes_starts, dc.neighbor_source_boxes_starts)
