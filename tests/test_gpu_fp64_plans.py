"""The FP64 schedules that a tree view keeps: one per plan and row count, so
that plans which alternate on one tree all leave the per-box kernel.

Both kernels are FP64-accurate (a few units of 2^-53 of the sums' magnitude), so
they agree to 1e-13 relative l2."""

import pytest

from helpers import plan_and_view, rel_l2, wrangler_for
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
