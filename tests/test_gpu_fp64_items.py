"""Work items that are too long for the FP64 tensor-core path: refused by the
status word, their tiles not written (the sums of the last digits could leave
their 32 bits)."""

import ctypes as C

import numpy as np
import pytest

from helpers import plan_and_view, rel_l2
from volumential_gb300 import _lib
from volumential_gb300 import workloads as W
from volumential_gb300.batched import MixedSchedule

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("whole_tiles", [False, True])
def test_long_items_are_refused(cuda, whole_tiles):
    torch = cuda
    w = W.adaptive_workload("items", 3, 6, tol=0.3, max_level=4, seed=91)
    plan, view, keep = plan_and_view(w)
    cap = int(_lib.lib().vl1_eval_fp64_item_keys(plan.handle))
    c = torch.from_numpy(w.coefs).cuda()
    ref = torch.empty_like(c)
    plan.eval_fp64(view, c, ref, stream=0)

    def tiles(keys):
        s = MixedSchedule(plan, view, keep, 1, 0, max_keys_per_item=keys, workspace=False)
        assert (s.max_keys_per_item > cap) == (keys > cap)
        if whole_tiles and keys > cap:      # one item per tile, in the kernel
            s.c_struct.n_items = s.c_struct.n_splits = s.c_struct.n_slots = 0
            s.c_struct.items = None
        out = torch.full_like(c, float("nan"))
        _lib.check(_lib.lib().vl1_eval_fp64_tiles(
            plan.handle, C.byref(view), C.byref(s.c_struct), c.data_ptr(), _lib.VL1_REAL64, 1,
            out.data_ptr(), C.c_void_p(0)), "vl1_eval_fp64_tiles")
        torch.cuda.synchronize()
        return out.cpu().numpy()

    got = tiles(1 << 30)
    with pytest.raises(_lib.VL1Error) as e:
        plan.raise_on_status(0)
    assert e.value.code == _lib.VL1_E_ARG
    assert np.isnan(got).any()
    r = ref.cpu().numpy()
    fine = ~np.isnan(got)                   # shorter tiles are evaluated
    assert not fine.any() or rel_l2(got[fine], r[fine]) <= 1e-12
    got = tiles(cap)
    plan.raise_on_status(0)
    assert rel_l2(got, r) <= 1e-12


@pytest.mark.parametrize("dim,level,q,cplx", [(2, 6, 3, False), (3, 3, 4, True)])
def test_tiles_without_pairs(cuda, dim, level, q, cplx):
    """Target boxes with empty lists: their tiles have no keys and their rows
    are zero."""
    from volumential_gb300 import plan as plan_module
    from volumential_gb300.plan import tree_view_from_arrays

    torch = cuda
    w = W.uniform_workload("items_e", dim, level, q, seed=92)
    plan, view, keep = plan_and_view(w)
    st = w.traversal.neighbor_source_boxes_starts.astype(np.int64)
    full = np.arange(len(st) - 1) % 4 == 0
    args = dict(zip(plan_module._VIEW_ARGS, (keep[k] for k in plan_module._VIEW_KEYS)))
    args["neighbor_source_boxes_starts"] = np.concatenate(
        [[0], np.cumsum(np.where(full, np.diff(st), 0))])
    args["neighbor_source_boxes_lists"] = np.concatenate(
        [w.traversal.neighbor_source_boxes_lists[st[i]:st[i + 1]] for i in np.flatnonzero(full)])
    v, k = tree_view_from_arrays(root_extent=view.root_extent, **args)
    c = torch.from_numpy(np.random.default_rng(9).standard_normal(w.n_points)).cuda()
    c = c * (1.0 + 2.0j) if cplx else c
    ref, out = torch.empty_like(c), torch.full_like(c, float("nan"))
    plan.eval_fp64(v, c, ref, stream=0)
    s = MixedSchedule(plan, v, k, 2 if cplx else 1, 0, workspace=False, split_scratch=False)
    assert (np.diff(s.key_start_np) == 0).any()
    _lib.check(_lib.lib().vl1_eval_fp64_tiles(
        plan.handle, C.byref(v), C.byref(s.c_struct), c.data_ptr(),
        _lib.VL1_COMPLEX128 if cplx else _lib.VL1_REAL64, 1, out.data_ptr(), C.c_void_p(0)),
        "vl1_eval_fp64_tiles")
    plan.raise_on_status(0)
    got, want = out.cpu().numpy(), ref.cpu().numpy()
    assert rel_l2(got, want) <= 1e-12
    assert (want == 0.0).any() and np.all(got[want == 0.0] == 0.0)
