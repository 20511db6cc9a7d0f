"""The FP64 schedules that a tree view keeps: one per plan and row count, so
that plans which alternate on one tree all leave the per-box kernel.

Both kernels are FP64-accurate (a few units of 2^-53 of the sums' magnitude), so
they agree to 1e-13 relative l2."""

import gc
import weakref

import numpy as np
import pytest

from helpers import plan_and_view, rel_l2, wrangler_for
from volumential_gb300 import batched
from volumential_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _second_plan(w, factor):
    """A plan of ``w``'s tables times ``factor``."""
    wr, tr = wrangler_for(w), w.traversal
    payload = wr.get_payload(w.kernel)
    kw = wr._near_field_kwargs(payload, tr.target_boxes, tr.neighbor_source_boxes_starts,
                               tr.neighbor_source_boxes_lists, None)
    names = ("mode_nmlz_combined", "case_indices", "encoding_base", "encoding_shift",
             "table_root_extent", "table_starting_level")
    return wr.near_field_evaluator(w.kernel, payload).get_plan(
        table_data_combined=kw["table_data_combined"] * factor, cache=False,
        **{n: kw[n] for n in names}, **{n: kw[n] for n in kw if n.startswith("arithmetic_")})


def test_two_plans_alternate_on_one_view(cuda):
    torch = cuda
    w = W.uniform_workload("two", 3, 3, 4, seed=61)      # modelled time below 1.5 ms
    plan, view, keep = plan_and_view(w)
    plans = [plan, _second_plan(w, 3.0)]
    c = torch.from_numpy(w.coefs[0]).cuda()
    out, ref = torch.empty_like(c), torch.empty_like(c)
    for _ in range(4):
        taken = []
        for p in plans:
            p.eval_fp64(view, c, out, stream=0, keep=keep)
            p.eval_fp64(view, c, ref, stream=0)
            assert rel_l2(out.cpu().numpy(), ref.cpu().numpy()) <= 1e-13
            taken.append(view.fp64_schedules[1])
    assert all(t[1] is not None for t in taken)
    assert [t[0] == p for t, p in zip(taken, plans)] == [True, True]


def test_a_failed_build_is_tried_again(cuda, monkeypatch):
    """Out of memory while the schedule is built: this call goes per box, the
    next one builds it."""
    torch = cuda
    w = W.uniform_workload("oom", 3, 3, 4, seed=62)
    plan, view, keep = plan_and_view(w)
    c = torch.from_numpy(w.coefs[0]).cuda()
    out, ref = torch.empty_like(c), torch.empty_like(c)
    plan.eval_fp64(view, c, ref, stream=0)
    plan.eval_fp64(view, c, out, stream=0, keep=keep)    # seen once
    calls = []
    init = batched.MixedSchedule.__init__

    def fails_once(self, *a, **k):
        calls.append(1)
        if len(calls) == 1:
            raise torch.OutOfMemoryError("CUDA out of memory (planted)")
        init(self, *a, **k)

    monkeypatch.setattr(batched.MixedSchedule, "__init__", fails_once)
    plan.eval_fp64(view, c, out, stream=0, keep=keep)
    assert torch.equal(out, ref)
    for _ in range(2):
        plan.eval_fp64(view, c, out, stream=0, keep=keep)
        assert rel_l2(out.cpu().numpy(), ref.cpu().numpy()) <= 1e-13
    assert view.fp64_schedules[1][1] is not None and len(calls) == 2


def test_other_errors_while_building_are_raised(cuda, monkeypatch):
    torch = cuda
    w = W.uniform_workload("err", 3, 3, 4, seed=63)
    plan, view, keep = plan_and_view(w)
    c = torch.from_numpy(w.coefs[0]).cuda()
    out = torch.empty_like(c)
    plan.eval_fp64(view, c, out, stream=0, keep=keep)

    def fails(self, *a, **k):
        raise RuntimeError("CUDA error: planted")

    monkeypatch.setattr(batched.MixedSchedule, "__init__", fails)
    with pytest.raises(RuntimeError, match="planted"):
        plan.eval_fp64(view, c, out, stream=0, keep=keep)


def test_schedules_go_with_their_views(cuda):
    """FP64 evaluations of many trees keep no tree longer than the view cache
    does, and nothing in the mixed path's schedule cache."""
    from volumential_gb300 import plan as plan_module
    from volumential_gb300.plan import tree_view_from_arrays

    torch = cuda
    w = W.uniform_workload("many_trees", 3, 3, 4, seed=64)
    plan, view, keep = plan_and_view(w)
    c = torch.from_numpy(w.coefs[0]).cuda()
    out = torch.empty_like(c)
    before = len(batched._cache)
    seen = []
    for _ in range(20):
        k = {n: t.clone() for n, t in keep.items()}
        args = dict(zip(plan_module._VIEW_ARGS, (k[n] for n in plan_module._VIEW_KEYS)))
        for _ in range(2):
            v, kk = tree_view_from_arrays(root_extent=view.root_extent, **args)
            plan.eval_fp64(v, c, out, stream=0, keep=kk)
        assert v.fp64_schedules[1][1] is not None
        seen.append(weakref.ref(k["lists"]))
        del v, kk, k, args
    plan.raise_on_status(0)
    assert len(batched._cache) == before
    gc.collect()
    assert sum(r() is not None for r in seen) <= 8


def test_schedules_do_not_keep_plans(cuda):
    torch = cuda
    w = W.uniform_workload("plan_ref", 3, 3, 4, seed=65)
    _, view, keep = plan_and_view(w)
    c = torch.from_numpy(w.coefs[0]).cuda()
    out = torch.empty_like(c)
    p = _second_plan(w, 2.0)
    for _ in range(2):
        p.eval_fp64(view, c, out, stream=0, keep=keep)
    assert view.fp64_schedules[1][1] is not None
    torch.cuda.synchronize()
    ref = weakref.ref(p)
    del p
    gc.collect()
    assert ref() is None
    plan, _, _ = plan_and_view(w)
    for _ in range(3):                 # another plan, perhaps at the same address
        plan.eval_fp64(view, c, out, stream=0, keep=keep)
    want = torch.empty_like(c)
    plan.eval_fp64(view, c, want, stream=0)
    assert rel_l2(out.cpu().numpy(), np.asarray(want.cpu())) <= 1e-13
