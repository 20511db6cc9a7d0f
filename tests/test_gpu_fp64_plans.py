"""The FP64 schedules that a tree view keeps: one per plan and row count, so
that plans which alternate on one tree all leave the per-box kernel.

Both kernels are FP64-accurate (a few units of 2^-53 of the sums' magnitude), so
they agree to 1e-13 relative l2."""

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
