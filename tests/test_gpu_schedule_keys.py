"""Schedules of plans with many keys, and of few that occur.

The device builder counts keys in shared memory up to 8192 of them and in
global memory beyond, and sorts only the words of the keys that occur.  Either
side of both lines must give the box order of the host restatement.
"""

import ctypes as C

import numpy as np
import pytest

from helpers import plan_and_view
from test_gpu_schedule import _device_order
from volumential_gb300 import _lib
from volumential_gb300 import workloads as W
from volumential_gb300.batched import MixedSchedule

pytestmark = pytest.mark.gpu


def _uniform(n_tables):
    return W.uniform_workload("sk", 2, 4, 1, seed=11, n_tables=n_tables)


def _adaptive(n_tables):
    w = W.adaptive_workload("sa", 2, 2, tol=1e-3, max_level=7, min_level=2, seed=12,
                            n_terms=8, width_range=(0.02, 0.1))
    w.tables = W.make_tables("synthetic", 2, 2, w.kernel, n_tables=n_tables,
                             source_box_extent=w.tree.root_extent)
    return w


CASES = {
    "one-table": lambda: _uniform(1),            # 9 of 33 keys: one word
    "two-words": lambda: _adaptive(3),           # up to 99 keys
    "shared-memory-edge": lambda: _uniform(248),   # 8184 keys
    "global-counts": lambda: _uniform(249),        # 8217 keys
    "global-counts-adaptive": lambda: _adaptive(260),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_order_of_boxes(cuda, name):
    torch = cuda
    w = CASES[name]()
    plan, view, keep = plan_and_view(w)
    stream = torch.cuda.current_stream().cuda_stream
    K = plan.n_tables * plan.n_cases
    tr = w.traversal
    starts = np.asarray(tr.neighbor_source_boxes_starts, dtype=np.int64)
    n_tb = len(starts) - 1
    keys = torch.empty(int(starts[-1]), dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().vl1_classify_pairs(plan.handle, C.byref(view), keys.data_ptr(),
                                             C.c_void_p(stream)), "vl1_classify_pairs")
    keys = keys.cpu().numpy().astype(np.int64)
    dev = MixedSchedule(plan, view, keep, 1, stream, packing="device", workspace=False)
    rows = dev.tile_rows.cpu().numpy().reshape(-1, 128)
    order = _device_order(keys, starts, n_tb, K)
    # tiles are groups of 128 boxes in that order (themselves longest first)
    want = {tuple(order[t:t + 128]) for t in range(0, n_tb, 128)}
    got = {tuple(r[r >= 0]) for r in rows}
    assert got == want
    # each tile's keys are those of its boxes
    pair_box = np.repeat(np.arange(n_tb), np.diff(starts))
    ks = dev.tile_key_start.cpu().numpy()
    ids = dev.key_ids.cpu().numpy()
    for t, r in enumerate(rows):
        assert np.array_equal(ids[ks[t]:ks[t + 1]],
                              np.unique(keys[np.isin(pair_box, r[r >= 0])]))


@pytest.mark.parametrize("count,modes,what", [
    (9, list(range(9)), None), (9, list(range(8)) + [7], "distinct"),
    (9, list(range(8)) + [9], "distinct"), (9, [-1] + list(range(1, 9)), "distinct")])
def test_mode_checks(cuda, count, modes, what):
    """One box's mode ids in range and distinct, or refused."""
    torch = cuda
    w = W.uniform_workload("sm", 2, 2, 3, seed=13)
    plan, view, keep = plan_and_view(w)
    stream = torch.cuda.current_stream().cuda_stream
    changed = keep["smode"].clone()
    changed[5 * 9:6 * 9] = torch.tensor(modes, dtype=torch.int32, device="cuda")
    view.source_mode_ids = changed.data_ptr()
    try:
        if what is None:
            MixedSchedule(plan, view, keep, 1, stream, packing="device", workspace=False)
        else:
            with pytest.raises(ValueError, match=what):
                MixedSchedule(plan, view, keep, 1, stream, packing="device", workspace=False)
    finally:
        view.source_mode_ids = keep["smode"].data_ptr()
