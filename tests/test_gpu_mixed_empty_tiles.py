"""Work items without units (tiles whose target boxes have empty lists) between
ordinary ones in the persistent mixed kernel: every CTA walks several of them in
a row.  The ordinary rows agree with the FP64 kernel at the path's 1e-9, the
others are zero, and no wait runs out."""

import ctypes as C

import numpy as np
import pytest

from helpers import plan_and_view, rel_l2
from volumential_gb300 import _lib
from volumential_gb300 import plan as plan_module
from volumential_gb300 import workloads as W
from volumential_gb300.batched import get_schedule
from volumential_gb300.plan import tree_view_from_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,level,q,nrhs", [(2, 7, 2, 32), (2, 6, 6, 32), (3, 4, 4, 16)])
@pytest.mark.parametrize("run", [1, 2, 5, 40])     # empty items in a row
def test_empty_items_between_ordinary_ones(cuda, dim, level, q, nrhs, run):
    torch = cuda
    w = W.uniform_workload("empty", dim, level, q, seed=95)
    plan, view, keep = plan_and_view(w)
    st = w.traversal.neighbor_source_boxes_starts.astype(np.int64)
    n_tb = len(st) - 1
    keep_list = np.arange(n_tb) % 4 == 0               # three quarters get no list
    counts = np.where(keep_list, np.diff(st), 0)
    lists = np.concatenate([w.traversal.neighbor_source_boxes_lists[st[i]:st[i + 1]]
                            for i in np.flatnonzero(keep_list)])
    args = dict(zip(plan_module._VIEW_ARGS, (keep[k] for k in plan_module._VIEW_KEYS)))
    args["neighbor_source_boxes_starts"] = np.concatenate([[0], np.cumsum(counts)])
    args["neighbor_source_boxes_lists"] = lists
    v, k = tree_view_from_arrays(root_extent=view.root_extent, **args)
    c = torch.from_numpy(np.random.default_rng(7).standard_normal((nrhs, w.n_points))).cuda()
    ref, out = torch.empty_like(c), torch.full_like(c, float("nan"))
    plan.eval_fp64(v, c, ref, stream=0, nrhs=nrhs)
    sched = get_schedule(plan, v, k, nrhs, 0)
    items = sched.items_np
    n_keys = items[:, 2] - items[:, 1]
    full, empty = np.flatnonzero(n_keys > 0), np.flatnonzero(n_keys == 0)
    assert len(empty) > 2 * len(full)
    order, e = [], 0
    for i in full:
        order += [i, *empty[e:e + run]]
        e = min(e + run, len(empty))
    order += list(empty[e:])
    assert sorted(order) == list(range(len(items)))
    sched.items.copy_(torch.from_numpy(np.ascontiguousarray(items[order])))
    _lib.check(_lib.lib().vl1_eval_mixed(
        plan.handle, C.byref(v), C.byref(sched.c_struct), c.data_ptr(), nrhs, out.data_ptr(),
        sched.workspace.data_ptr(), sched.workspace.numel(), C.c_void_p(0)), "vl1_eval_mixed")
    plan.raise_on_status(0)
    got, want = out.cpu().numpy(), ref.cpu().numpy()
    assert rel_l2(got, want) <= 1e-9
    assert np.all(got[want == 0.0] == 0.0)
    sched.items.copy_(torch.from_numpy(items))         # (cached)
