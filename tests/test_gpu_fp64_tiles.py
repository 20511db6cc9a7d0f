"""FP64 evaluation on the tensor cores (``vl1_eval_fp64_tiles``) against the C
oracle: the sizes where its tiles, units and column chunks end, real and
complex tables and densities, permuted modes, densities over many decades,
non-finite densities, and the rule that chooses the path.

Tolerance: an FP64 sum of n terms is off by at most about n ulps of its terms'
absolute sum; list 1 has at most a few thousand terms, so 1e-12 relative l2,
and 1e-11 of the box's largest value per target box, hold for both the oracle
and the kernel."""

import ctypes as C

import numpy as np
import pytest

from helpers import (FIXED, LAP2, LAP3, PER_LEVEL, oracle_eval, oracle_for_workload,
                     plan_and_view, rel_l2)
from volumential_gb300 import workloads as W
from volumential_gb300.kernels import HelmholtzKernel

pytestmark = pytest.mark.gpu


def _tiles(w, coefs, keep_change=None):
    """[nrhs, N] result of the tensor-core path."""
    import torch

    from volumential_gb300 import _lib
    from volumential_gb300.batched import get_schedule
    from volumential_gb300.plan import tree_view_from_arrays  # noqa: F401

    plan, view, keep = plan_and_view(w)
    c = torch.from_numpy(np.ascontiguousarray(coefs)).cuda()
    nrhs = c.shape[0]
    cplx = plan.complex_table or c.is_complex()
    out = torch.full(c.shape, 7.0, dtype=torch.complex128 if cplx else torch.float64,
                     device="cuda")
    cap = int(_lib.lib().vl1_eval_fp64_item_keys(plan.handle))
    sched = get_schedule(plan, view, keep, nrhs * (2 if c.is_complex() else 1), 0,
                         max_keys_per_item=min(cap, keep_change or cap))
    _lib.check(_lib.lib().vl1_eval_fp64_tiles(
        plan.handle, C.byref(view), C.byref(sched.c_struct), c.data_ptr(),
        _lib.VL1_COMPLEX128 if c.is_complex() else _lib.VL1_REAL64, nrhs, out.data_ptr(),
        C.c_void_p(0)), "vl1_eval_fp64_tiles")
    plan.raise_on_status(0)
    return out.cpu().numpy()


def _oracle(w, policy, coefs):
    prob = oracle_for_workload(w, policy)
    rows = []
    for c in coefs:
        if np.iscomplexobj(c):
            rows.append(oracle_eval(prob, w, np.ascontiguousarray(c.real))
                        + 1j * oracle_eval(prob, w, np.ascontiguousarray(c.imag)))
        else:
            rows.append(oracle_eval(prob, w, c))
    return np.stack(rows)


def _check(w, got, ref):
    nq = w.q ** w.dim
    assert rel_l2(got, ref) <= 1e-12
    g, r = (x.reshape(x.shape[0], -1, nq) for x in (got, ref))
    scale = np.abs(r).max(-1)
    assert np.all(np.abs(g - r).max(-1) <= 1e-11 * scale)


# q^dim 1 .. 256: below, at and above one unit of 16 source points, one and
# several column chunks of 16, 32 and 64
@pytest.mark.parametrize("dim,level,q", [(2, 2, 1), (2, 3, 2), (2, 3, 4), (2, 3, 5), (2, 2, 6),
                                         (2, 1, 8), (2, 1, 16), (3, 2, 2), (3, 2, 3), (3, 2, 4),
                                         (3, 1, 5), (3, 1, 6)])
@pytest.mark.parametrize("nrhs,complex_coefs", [(1, False), (3, True)])
def test_sizes(cuda, dim, level, q, nrhs, complex_coefs):
    w = W.uniform_workload("tiles", dim, level, q, seed=11, nrhs=nrhs)
    c = w.coefs + 1j * np.roll(w.coefs, 5, axis=1) if complex_coefs else w.coefs
    _check(w, _tiles(w, c), _oracle(w, LAP2 if dim == 2 else LAP3, c))


@pytest.mark.parametrize("dim,level,q", [(2, 3, 5), (2, 3, 4), (3, 2, 3), (3, 1, 5)])
@pytest.mark.parametrize("complex_coefs", [False, True])
def test_complex_tables_per_level(cuda, dim, level, q, complex_coefs):
    w = W.uniform_workload("tiles_h", dim, level, q, seed=12, kernel=HelmholtzKernel(dim),
                           complex_table=True, n_tables=level + 1)
    for i, t in enumerate(w.tables):       # table levels of very different magnitude
        t.data[:] *= 10.0 ** (-3 * i)
    c = w.coefs + 1j * np.roll(w.coefs, 3, axis=1) if complex_coefs else w.coefs
    _check(w, _tiles(w, c), _oracle(w, PER_LEVEL, c))


@pytest.mark.parametrize("dim,tol,policy", [(2, 0.05, LAP2), (3, 0.3, LAP3)])
def test_adaptive_trees_and_split_tiles(cuda, dim, tol, policy):
    w = W.adaptive_workload("tiles_a", dim, 3, tol=tol, max_level=5 if dim == 2 else 4, seed=13)
    ref = _oracle(w, policy, w.coefs)
    for cap in (None, 3, 1):               # whole tiles, and key ranges of 3 and 1 keys
        _check(w, _tiles(w, w.coefs, cap), ref)


@pytest.mark.parametrize("dim,policy", [(2, LAP2), (3, LAP3)])
def test_magnitudes(cuda, dim, policy):
    """Neighbouring boxes up to six decades apart (digit shifts), the domain
    over 200 decades, values near the ends of the FP64 range."""
    w = W.uniform_workload("tiles_m", dim, 3 if dim == 2 else 2, 3, seed=14)
    nq, x = 3 ** dim, w.tree.targets[0]
    boxes = np.repeat(10.0 ** np.random.default_rng(1).uniform(-3, 3, w.n_points // nq), nq)
    rows = np.stack([w.coefs[0] * boxes, w.coefs[0] * 10.0 ** (100 * np.sin(2 * np.pi * x)),
                     w.coefs[0] * 1e300, np.where(x < 0, 0.0, w.coefs[0])])
    for r in rows:
        got, ref = _tiles(w, r[None]), _oracle(w, policy, r[None])
        s = np.abs(ref).max()
        g, f = (v.reshape(-1, nq) / s for v in (got, ref))
        scale = np.abs(f).max(-1)
        assert np.all(np.abs(g - f).max(-1) <= 1e-11 * scale)


@pytest.mark.parametrize("complex_coefs", [False, True])
def test_non_finite_densities(cuda, complex_coefs):
    """Targets with an infinite or NaN source get what the per-box kernel
    gives them, the others their finite sums."""
    import torch

    w = W.uniform_workload("tiles_n", 2, 3, 5, seed=15)
    c = w.coefs.copy()
    c[0, 3], c[0, 700], c[0, 701] = np.inf, np.nan, -np.inf
    if complex_coefs:
        c = c + 1j * w.coefs
    plan, view, keep = plan_and_view(w)
    ct = torch.from_numpy(np.ascontiguousarray(c)).cuda()
    ref = torch.empty_like(ct)
    plan.eval_fp64(view, ct, ref, stream=0)
    ref, got = ref.cpu().numpy(), _tiles(w, c)
    parts = ((got.real, ref.real), (got.imag, ref.imag)) if complex_coefs else ((got, ref),)
    for g, r in parts:
        assert np.array_equal(np.isnan(g), np.isnan(r))
        assert np.array_equal(g[np.isinf(r)], r[np.isinf(r)])
        fine = np.isfinite(r)
        assert 0 < fine.sum() < r.size and rel_l2(g[fine], r[fine]) <= 1e-12


def test_permuted_modes_partial_boxes_and_errors(cuda):
    """Box-local modes in any order, boxes with fewer points than modes, and a
    mode outside the box, which raises as in the per-box kernel."""
    import torch

    from volumential_gb300.plan import tree_view_from_arrays

    w = W.uniform_workload("tiles_p", 3, 2, 4, seed=16)
    plan, view, keep = plan_and_view(w)
    nq, rng = 64, np.random.default_rng(2)
    n = w.n_points

    def views(smode, tmode, counts):
        k = dict(target_boxes=keep["target_boxes"], neighbor_source_boxes_starts=keep["starts"],
                 neighbor_source_boxes_lists=keep["lists"], box_centers=keep["centers"],
                 box_levels=keep["levels"], box_source_starts=keep["src_starts"],
                 box_source_counts_nonchild=counts, box_target_starts=keep["tgt_starts"],
                 box_target_counts_nonchild=counts, root_extent=view.root_extent)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()  # noqa
        return tree_view_from_arrays(source_mode_ids=dev(smode), target_point_ids=dev(tmode), **k)

    perm = np.concatenate([rng.permutation(nq) for _ in range(n // nq)])
    counts = keep["src_counts"].clone()
    counts[counts > 0] -= (torch.arange(int((counts > 0).sum()), device="cuda") % 3).to(
        counts.dtype)
    c = torch.from_numpy(w.coefs).cuda()
    v, k = views(perm, np.concatenate([rng.permutation(nq) for _ in range(n // nq)]), counts)
    ref, got = torch.zeros_like(c), torch.zeros_like(c)
    plan.eval_fp64(v, c, ref, stream=0)
    for _ in range(2):                     # the second call of a tree gets a schedule
        plan.eval_fp64(v, c, got, stream=0, keep=k)
    plan.raise_on_status(0)
    assert v.fp64_schedules[1][1] is not None
    assert rel_l2(got.cpu().numpy(), ref.cpu().numpy()) <= 1e-12
    bad = perm.copy()
    bad[5] = nq
    v, k = views(perm, bad, counts)
    for _ in range(2):
        plan.eval_fp64(v, c, got, stream=0, keep=k)
        with pytest.raises(ValueError):
            plan.raise_on_status(0)
    dup = perm.copy()                      # no schedule: stays with the per-box kernel
    dup[1] = dup[0]
    v, k = views(dup, perm, counts)
    plan.eval_fp64(v, c, ref, stream=0)
    for _ in range(2):
        plan.eval_fp64(v, c, got, stream=0, keep=k)
    plan.raise_on_status(0)
    assert v.fp64_schedules[1] == (plan, None)
    assert np.array_equal(got.cpu().numpy(), ref.cpu().numpy())


def test_graph_capture_and_other_streams(cuda):
    """Under capture the call is the per-box kernel's; on a stream of its own
    the scratch follows the stream."""
    import torch

    w = W.uniform_workload("tiles_s", 3, 2, 4, seed=17)
    plan, view, keep = plan_and_view(w)
    c = torch.from_numpy(w.coefs).cuda()
    ref, out = torch.zeros_like(c), torch.zeros_like(c)
    plan.eval_fp64(view, c, ref, stream=0)
    for _ in range(2):
        plan.eval_fp64(view, c, out, stream=0, keep=keep)
    torch.cuda.synchronize()
    outs = [torch.zeros_like(c) for _ in range(4)]
    for o in outs:
        s = torch.cuda.Stream()
        plan.eval_fp64(view, c, o, stream=s.cuda_stream, keep=keep)
    torch.cuda.synchronize()
    for o in outs:
        assert torch.equal(o, out)         # integer sums: the same bits every time
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.eval_fp64(view, c, out, stream=torch.cuda.current_stream().cuda_stream, keep=keep)
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)


def test_fixed_table_policy_uses_the_same_sums(cuda):
    w = W.uniform_workload("tiles_f", 2, 4, 5, seed=18, kernel=HelmholtzKernel(2),
                           complex_table=True)
    w.tables = W.synthetic_tables(2, 5, w.kernel, seed=3, source_box_extent=1.0 / 16,
                                  complex_values=True)
    _check(w, _tiles(w, w.coefs), _oracle(w, FIXED, w.coefs))
