"""FP64 evaluations with a NaN in the table: the targets that read the value get
NaN, all others their sums, as the per-box kernel gives them.

The fixed-point digits of the tensor-core path cannot hold a NaN, so such a
plan stays with the per-box kernel.  Equality is exact where both results come
from that kernel."""

import ctypes as C

import numpy as np
import pytest

from helpers import plan_and_view, wrangler_for
from volumential_gb300 import _lib
from volumential_gb300 import workloads as W
from volumential_gb300.batched import get_schedule
from volumential_gb300.kernels import HelmholtzKernel

pytestmark = pytest.mark.gpu


def _plan(w, change):
    """A plan of ``w`` whose table values went through ``change``."""
    wr, tr = wrangler_for(w), w.traversal
    payload = wr.get_payload(w.kernel)
    kw = wr._near_field_kwargs(payload, tr.target_boxes, tr.neighbor_source_boxes_starts,
                               tr.neighbor_source_boxes_lists, None)
    table = kw["table_data_combined"].copy()
    change(table)
    names = ("mode_nmlz_combined", "case_indices", "encoding_base", "encoding_shift",
             "table_root_extent", "table_starting_level")
    return wr.near_field_evaluator(w.kernel, payload).get_plan(
        table_data_combined=table, cache=False, **{n: kw[n] for n in names},
        **{n: kw[n] for n in kw if n.startswith("arithmetic_")})


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("at", [(0, 0), (24, 3)])     # (source, target) of a block
def test_nan_in_a_table(cuda, cplx, at):
    torch = cuda
    kernel = dict(kernel=HelmholtzKernel(2), complex_table=True) if cplx else {}
    w = W.uniform_workload("nan_t", 2, 6, 5, seed=41, **kernel)
    clean, view, keep = plan_and_view(w)
    keys = torch.empty(keep["lists"].numel(), dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().vl1_classify_pairs(clean.handle, C.byref(view), keys.data_ptr(),
                                             C.c_void_p(0)), "vl1_classify_pairs")
    torch.cuda.synchronize()
    entry = int(clean.orbit_index_map()[0][int(keys[0]) % clean.n_cases][at])

    def change(t):
        t[0, entry] = complex(1.0, np.nan) if cplx else np.nan

    plan = _plan(w, change)
    c = torch.from_numpy(w.coefs[0]).cuda()
    dtype = torch.complex128 if cplx else torch.float64
    new = lambda: torch.full(c.shape, 7.0, dtype=dtype, device="cuda")  # noqa
    ref, got, tiles = new(), new(), new()
    plan.eval_fp64(view, c, ref, stream=0)
    ref = ref.cpu().numpy()
    assert 0 < np.isnan(ref).sum() < ref.size
    for _ in range(3):
        plan.eval_fp64(view, c, got, stream=0, keep=keep)
    plan.raise_on_status(0)
    assert np.array_equal(got.cpu().numpy(), ref, equal_nan=True)
    sched = get_schedule(plan, view, keep, 1, 0)
    _lib.check(_lib.lib().vl1_eval_fp64_tiles(
        plan.handle, C.byref(view), C.byref(sched.c_struct), c.data_ptr(), _lib.VL1_REAL64, 1,
        tiles.data_ptr(), C.c_void_p(0)), "vl1_eval_fp64_tiles")
    assert np.array_equal(tiles.cpu().numpy(), ref, equal_nan=True)


def test_nan_in_an_unused_case(cuda):
    """A NaN where no pair of the tree reads it changes nothing."""
    torch = cuda
    w = W.uniform_workload("nan_u", 2, 6, 5, seed=42)
    _, view, keep = plan_and_view(w)
    c = torch.from_numpy(w.coefs[0]).cuda()
    ref, got = torch.empty_like(c), torch.empty_like(c)
    clean = _plan(w, lambda t: None)
    clean.eval_fp64(view, c, ref, stream=0)
    n = clean._host["table"].shape[1]
    # an entry of a case outside the uniform tree's list: found by trying a few
    for entry in range(n - 1, 0, -(n // 16)):
        plan = _plan(w, lambda t, e=entry: t.__setitem__((0, e), np.nan))
        for _ in range(3):
            plan.eval_fp64(view, c, got, stream=0, keep=keep)
        per_box = torch.empty_like(c)
        plan.eval_fp64(view, c, per_box, stream=0)
        assert np.array_equal(got.cpu().numpy(), per_box.cpu().numpy(), equal_nan=True)
        if torch.equal(per_box, ref):
            return
    pytest.fail("every tried entry is read by the tree")
