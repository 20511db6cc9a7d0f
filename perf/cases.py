"""The list-1 evaluations, builds and corrections whose times are tracked.

Each case is one piece of work that a program using this package asks of it
through its public entry points; ``run`` does one pass of it.  The kinds:

* ``call``: ``NearFieldFromCSR.__call__`` on device arrays, one right-hand
  side (the reference's evaluator call, in its default FP64 precision or with
  ``list1_precision="mixed"``);
* ``drive``: ``drive_volume_fmm(list1_only=True)``, the whole call of a user
  of the reference, on the host arrays of a tree;
* ``many``: ``FPNDExpansionWrangler.eval_direct_batched``, many right-hand
  sides of one tree;
* ``batch``: ``MixedBatch.eval``, problems of different depth, order and
  right-hand side count in one set of launches;
* ``remesh``: what a step of an adaptive computation does: the tree and its
  list 1 built on the device from new leaves, then one evaluation;
* ``split``: the Helmholtz split mode's list-1 correction of a wrangler;
* ``table``: a near-field table built by Duffy quadrature.

Near-field tables of the evaluation kinds are filled from a closed form with
the symmetry, sign pattern and decay of the kernels' own tables (a regularised
Green's function times quadrature weights), so that ``exact`` can form the
dense interaction blocks by itself.
"""

import functools
import math

import numpy as np
import torch

DENSITY_TERMS = 12


# {{{ the cases

def listed():
    return [
        # a small 2D solve of the kind the examples and tests run: latency
        dict(name="call_lap2d_l3_q3", kind="call", kernel="laplace", dim=2, q=3, level=3,
             precision="fp64"),
        # the plain 2D configuration: uniform level 5, q = 4, 16,384 points
        dict(name="call_lap2d_l5_q4", kind="call", kernel="laplace", dim=2, q=4, level=5,
             precision="fp64"),
        # 2D Helmholtz, complex table and density, q = 5, 102,400 points
        dict(name="call_helm2d_l6_q5", kind="call", kernel="helmholtz", dim=2, q=5, level=6,
             precision="fp64", complex_density=True),
        # the plain 3D configuration: adaptive octree, q = 4, ~1.5M points
        dict(name="call_lap3d_adaptive_q4", kind="call", kernel="laplace", dim=3, q=4,
             level=6, mesh=2006, tol=1e-3, precision="fp64"),
        # the same solve in the mixed-precision mode
        dict(name="call_lap3d_adaptive_q4_mixed", kind="call", kernel="laplace", dim=3, q=4,
             level=6, mesh=2006, tol=1e-3, precision="mixed"),
        # a whole driver call, odd point count per box (q = 5: 125 nodes)
        dict(name="drive_lap3d_l4_q5", kind="drive", kernel="laplace", dim=3, q=5, level=4),
        # several right-hand sides in FP64, 27 points per box
        dict(name="many_lap3d_l4_q3_8rhs", kind="many", kernel="laplace", dim=3, q=3, level=4,
             nrhs=8, precision="fp64"),
        # the batched 2D Helmholtz configuration: 256 densities, complex table
        dict(name="many_helm2d_l6_q5_256rhs_mixed", kind="many", kernel="helmholtz", dim=2,
             q=5, level=6, nrhs=256, precision="mixed"),
        # uneven problems in one batch: levels, orders and rhs counts differ
        dict(name="batch_lap3d_uneven", kind="batch", dim=3, problems="2/3/5 3/4/12 3/5/3 "
             "4/3/17 4/4/6 4/5/9 5/3/2 5/4/1"),
        # one step of an adaptive computation: new tree, list 1, evaluation
        dict(name="remesh_lap3d_q4_mixed", kind="remesh", kernel="laplace", dim=3, q=4,
             level=6, mesh=2006, tol=1e-3, precision="mixed"),
        # the Helmholtz split mode's remainder on the 2D Helmholtz tree, k = 20
        dict(name="split_helm2d_l6_q5", kind="split", dim=2, q=5, level=6, k=20.0),
        # the 3D Laplace table of the plain 3D configuration, default orders
        dict(name="table_lap3d_q4", kind="table", kernel="laplace", dim=3, q=4),
    ]


def draw(rng):
    kind = rng.choice(["call", "call", "call", "drive", "many", "many", "batch", "remesh",
                       "split", "table"])
    dim = rng.choice([2, 3])
    q = rng.choice([2, 3, 4, 5, 6]) if dim == 2 else rng.choice([2, 3, 4, 5])
    level = rng.randint(2, 7) if dim == 2 else rng.randint(1, 5 if q <= 3 else 4)
    kernel = rng.choice(["laplace", "laplace", "helmholtz"])
    precision = rng.choice(["fp64", "mixed"])
    jitter = rng.randint(1, 1 << 20)
    if kind == "call":
        c = dict(kind=kind, kernel=kernel, dim=dim, q=q, level=level, precision=precision)
        if rng.random() < 0.5:
            c["complex_density"] = True
        if kernel == "laplace" and rng.random() < 0.6:
            c.update(mesh=jitter, tol=10.0 ** rng.uniform(-3, -1))
        return c
    if kind == "drive":
        return dict(kind=kind, kernel="laplace", dim=dim, q=q, level=min(level, 6 if dim == 2
                                                                          else 4),
                    mesh=jitter, tol=10.0 ** rng.uniform(-3, -1))
    if kind == "many":
        points = (2 ** dim) ** level * q ** dim
        nrhs = int(2 ** rng.uniform(1, max(1.0, min(7.0, math.log2(2.0e7 / points)))))
        if precision == "fp64":
            nrhs = min(nrhs, 11)
        return dict(kind=kind, kernel=kernel, dim=dim, q=q, level=level, nrhs=nrhs,
                    precision=precision)
    if kind == "batch":
        parts = []
        for _ in range(rng.randint(2, 9)):
            pq = rng.choice([3, 4, 5])
            parts.append("%d/%d/%d" % (rng.randint(1, 4), pq, rng.randint(1, 19)))
        return dict(kind=kind, dim=3, problems=" ".join(parts))
    if kind == "remesh":
        return dict(kind=kind, kernel="laplace", dim=dim, q=q, level=min(level + 1, 7 if dim == 2
                                                                         else 5),
                    mesh=jitter, tol=10.0 ** rng.uniform(-3, -1), precision=precision)
    if kind == "split":
        return dict(kind=kind, dim=dim, q=q if dim == 2 else min(q, 4), level=min(level, 6 if
                    dim == 2 else 3), k=round(rng.uniform(1.0, 30.0), 3))
    kernel = rng.choice(["laplace", "helmholtz"])
    return dict(kind=kind, kernel=kernel, dim=dim, q=rng.choice([2, 3]) if dim == 3
                else rng.randint(2, 5), regular=rng.randint(8, 20), radial=rng.randint(21, 61))

# }}}


# {{{ densities and tables

def _mixture(seed, dim, lo=0.02, hi=0.1):
    """Centres, widths and amplitudes of a seeded sum of Gaussians."""
    rng = np.random.default_rng(seed)
    n = DENSITY_TERMS
    return (rng.uniform(-0.5, 0.5, size=(n, dim)),
            np.exp(rng.uniform(math.log(lo), math.log(hi), size=n)), rng.standard_normal(n))


def _evaluate(mixture, points):
    """The sum of Gaussians at ``points`` [dim, ...] (a CUDA tensor)."""
    out = torch.zeros(points.shape[1:], dtype=torch.float64, device=points.device)
    for c, w, a in zip(*mixture):
        r2 = sum((points[i] - float(c[i])) ** 2 for i in range(points.shape[0]))
        out += float(a) * torch.exp(r2 * (-1.0 / float(w) ** 2))
    return out


def _densities(seed, points, nrhs, complex_valued=False):
    dim = points.shape[0]
    rows = [_evaluate(_mixture(1000003 * seed + r, dim), points) for r in range(nrhs)]
    if complex_valued:
        rows = [torch.complex(x, _evaluate(_mixture(1000003 * seed + 500009 + r, dim), points))
                for r, x in enumerate(rows)]
    return torch.stack(rows)


def _gauss(q):
    x, w = np.polynomial.legendre.leggauss(q)
    return 0.5 * (x + 1.0), 0.5 * w


def _nodes(dim, q):
    """Tensor nodes [q^dim, dim] and weights [q^dim] of the unit box."""
    x, w = _gauss(q)
    grids = np.meshgrid(*([x] * dim), indexing="ij")
    wgrids = np.meshgrid(*([w] * dim), indexing="ij")
    return (np.stack([g.ravel() for g in grids], axis=1),
            np.prod(np.stack([g.ravel() for g in wgrids]), axis=0))


def _table_values(kernel, dim, q, extent, k, sources, weights, targets):
    """Interaction values of the closed form: source nodes and weights of the
    unit box, targets in the source box's unit coordinates (broadcast over
    leading axes; numpy arrays or torch tensors), box extent ``extent``."""
    xp = torch if torch.is_tensor(targets) else np
    r2 = ((targets - sources) ** 2).sum(-1) + (0.3 / q) ** 2
    r = extent * xp.sqrt(r2)
    g = 1.0 / (4.0 * math.pi * r) if dim == 3 else -xp.log(r) / (2.0 * math.pi)
    g = g * (weights * extent ** dim)
    if kernel == "laplace":
        return g
    return g * (xp.cos(k * r) + 1j * xp.sin(k * r))


HELMHOLTZ_K = 20.0


def _kernel(case):
    from volumential_gb300.kernels import HelmholtzKernel, LaplaceKernel

    return (LaplaceKernel if case["kernel"] == "laplace" else HelmholtzKernel)(case["dim"])


def _table_extent(case):
    # Laplace: one canonical table at the root extent; Helmholtz: the table
    # of the tree's level
    return 1.0 if case["kernel"] == "laplace" else 0.5 ** case["level"]


@functools.lru_cache(maxsize=None)
def _table(kernel_name, dim, q, extent):
    from volumential_gb300.kernels import HelmholtzKernel, LaplaceKernel
    from volumential_gb300.nearfield_potential_table import NearFieldInteractionTable

    knl = (LaplaceKernel if kernel_name == "laplace" else HelmholtzKernel)(dim)
    t = NearFieldInteractionTable(
        q, dim=dim, sumpy_kernel=knl, source_box_extent=extent,
        dtype=np.float64 if kernel_name == "laplace" else np.complex128)
    info = t._get_invariant_entry_info()
    ids = np.asarray(info["entry_ids"], dtype=np.int64)
    nq = q ** dim
    case_ids, s, p = ids // (nq * nq), (ids % (nq * nq)) // nq, ids % nq
    targets = np.moveaxis(t.get_case_target_points(), 0, -1) / extent   # [case, point, dim]
    src, w = _nodes(dim, q)
    t.set_reduced_table_data(ids, _table_values(kernel_name, dim, q, extent, HELMHOLTZ_K,
                                                src[s], w[s], targets[case_ids, p]))
    if dim == 2:
        t.build_normalizer_table()
    return t

# }}}


# {{{ meshes and wranglers

@functools.lru_cache(maxsize=None)
def _mesh(dim, q, level, mesh, tol):
    """Traversal (host arrays) and leaves of a uniform tree, or with ``mesh``
    of the tree refined to at most ``level`` where that seed's Gaussian sum
    varies by more than ``tol`` over a leaf."""
    from volumential_gb300 import tree_build as tb

    if mesh is None:
        tree = tb.build_uniform_tree(dim, level, q)
    elif mesh == 2006 and dim == 3:
        from volumential_gb300.workloads import random_gaussian_mixture

        mix = random_gaussian_mixture(np.random.default_rng(mesh), 3, 16, (0.01, 0.08))
        tree = _refined(tb, dim, q, level, tol, (mix.centers, mix.widths, mix.amps))
    else:
        tree = _refined(tb, dim, q, level, tol, _mixture(mesh, dim))
    trav = tb.build_list1_traversal_device(tree)
    lv = torch.from_numpy(np.ascontiguousarray(tree.box_levels[tree.leaf_boxes])).cuda()
    co = torch.from_numpy(np.ascontiguousarray(tree.box_coords[tree.leaf_boxes])).cuda()
    return trav, lv, co


def _refined(tb, dim, q, level, tol, mixture):
    def refine(nodes):
        v = _evaluate(mixture, nodes)
        return (v.amax(-1) - v.amin(-1)) > tol

    return tb.build_adaptive_tree_device(dim, q, refine, max_level=level,
                                         min_level=min(2, level))


def _traversal(case):
    return _mesh(case["dim"], case["q"], case["level"], case.get("mesh"), case.get("tol"))


@functools.lru_cache(maxsize=None)
def _wrangler_of(items):
    from volumential_gb300.expansion_wrangler_fpnd import (
        FPNDExpansionWrangler, FPNDTreeIndependentDataForWrangler)
    from volumential_gb300.kernels import HelmholtzKernel

    case = dict(items)
    trav = _traversal(case)[0]
    extra = {}
    if case["kind"] == "split":
        knl = HelmholtzKernel(case["dim"])
        table = _table("laplace", case["dim"], case["q"], 1.0)
        extra = dict(self_extra_kwargs=None, kernel_extra_kwargs={"k": case["k"]})
    else:
        knl = _kernel(case)
        table = _table(case["kernel"], case["dim"], case["q"], _table_extent(case))
    dtype = np.complex128 if knl.is_complex_valued else np.float64
    wr = FPNDExpansionWrangler(
        FPNDTreeIndependentDataForWrangler(target_kernels=[knl]), trav, [table], dtype=dtype,
        quad_order=case["q"], **extra)
    return wr, knl, trav


def _wrangler(case):
    return _wrangler_of(tuple(sorted((k, v) for k, v in case.items() if k != "name")))


TREE_ARRAYS = ("target_boxes", "neighbor_source_boxes_starts", "neighbor_source_boxes_lists",
               "box_centers", "box_levels", "box_source_starts", "box_source_counts_nonchild",
               "box_target_starts", "box_target_counts_nonchild", "source_mode_ids",
               "target_point_ids")


def _table_arguments(payload):
    """The table, case and symmetry arguments of ``NearFieldFromCSR.__call__``."""
    info = payload["reconstruction_info"]
    return dict(
        case_indices=payload["case_indices"], encoding_base=payload["base"],
        encoding_shift=payload["shift"], mode_nmlz_combined=payload["mode_nmlz"],
        exterior_mode_nmlz_combined=payload["exterior_mode_nmlz"],
        table_data_combined=payload["table_data"],
        table_root_extent=payload["table_root_extent"],
        table_starting_level=payload["table_starting_level"],
        arithmetic_case_orbit_ranks=info["case_orbit_ranks"],
        arithmetic_case_axis_perm=info["case_axis_perm"],
        arithmetic_case_axis_sign=info["case_axis_sign"],
        arithmetic_case_axis_group=info["case_axis_group"],
        arithmetic_case_value_offsets=info["case_value_offsets"],
        arithmetic_axis_sign_power=info["axis_sign_power"],
        arithmetic_axis_direction_signs=info["axis_direction_signs"],
        arithmetic_direction_sign_axis=info["direction_sign_axis"])


def _tree_arguments(trav, nq):
    """The tree and list-1 arguments as new device tensors."""
    tree = trav.tree

    def dev(a, dtype):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=dtype)).cuda()

    starts = dev(tree.box_target_starts, np.int32)
    counts = dev(tree.box_target_counts_nonchild, np.int32)
    local = torch.arange(nq, dtype=torch.int32, device="cuda").repeat(tree.ntargets // nq)
    return dict(
        target_boxes=dev(trav.target_boxes, np.int32),
        neighbor_source_boxes_starts=dev(trav.neighbor_source_boxes_starts, np.int32),
        neighbor_source_boxes_lists=dev(trav.neighbor_source_boxes_lists, np.int32),
        box_centers=dev(tree.box_centers, np.float64), box_levels=dev(tree.box_levels, np.uint8),
        box_source_starts=starts, box_source_counts_nonchild=counts,
        box_target_starts=starts.clone(), box_target_counts_nonchild=counts.clone(),
        source_mode_ids=local, target_point_ids=local.clone(), root_extent=tree.root_extent)


def _points(trav):
    return torch.from_numpy(np.ascontiguousarray(trav.tree.targets)).cuda()


def _batch_problems(case):
    return [tuple(int(x) for x in p.split("/")) for p in case["problems"].split()]

# }}}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "table":
        rng = np.random.default_rng(seed)
        return dict(kind=kind, case=case, extent=float(rng.uniform(0.5, 2.0)),
                    k=float(rng.uniform(1.0, 30.0)))
    if kind == "batch":
        return _prepare_batch(case, seed)
    wr, knl, trav = _wrangler(case)
    nq = case["q"] ** case["dim"]
    points = _points(trav)
    rhs = _densities(seed, points, case.get("nrhs", 1), case.get("complex_density", False))
    state = dict(kind=kind, case=case, wrangler=wr, traversal=trav, densities=rhs)
    if kind in ("call", "remesh"):
        payload = wr.get_payload(knl)
        state["evaluator"] = wr.near_field_evaluator(
            knl, payload, {"list1_precision": case["precision"]})
        state["table_arguments"] = _table_arguments(payload)
        state["tree_arguments"] = _tree_arguments(trav, nq)
        state["result"] = torch.empty(
            trav.tree.ntargets, device="cuda",
            dtype=torch.complex128 if knl.is_complex_valued or rhs.is_complex()
            else torch.float64)
    if kind == "remesh":
        _, lv, co = _traversal(case)
        state["leaves"] = (lv.clone(), co.clone())
    if kind in ("drive", "split"):
        weights = torch.from_numpy(np.ascontiguousarray(trav.tree.weights)).cuda()
        state["weighted"] = rhs[0] * weights
    return state


def _prepare_batch(case, seed):
    from volumential_gb300.batch import BatchProblem, MixedBatch, problem_arrays
    from volumential_gb300.kernels import LaplaceKernel
    from volumential_gb300.workloads import Workload

    problems, plans = [], {}
    for i, (level, q, nrhs) in enumerate(_batch_problems(case)):
        trav = _mesh(3, q, level, None, None)[0]
        w = Workload("problem%d" % i, 3, q, LaplaceKernel(3), trav,
                     [_table("laplace", 3, q, 1.0)], np.zeros((nrhs, 0)), seed)
        plan, view, keep = problem_arrays(w, plan=plans.get(q), cache=False)
        plans[q] = plan
        rhs = _densities(97 * seed + i, _points(trav), nrhs)
        problems.append(BatchProblem(plan, view, keep, rhs.reshape(-1).contiguous(),
                                     torch.empty_like(rhs).reshape(-1), nrhs))
    return dict(kind="batch", case=case, problems=problems, batch=MixedBatch(problems))


def run(state):
    kind = state["kind"]
    if kind == "call":
        out, _ = state["evaluator"](None, result=state["result"],
                                    mode_coefs=state["densities"][0],
                                    **state["tree_arguments"], **state["table_arguments"])
        return out
    if kind == "drive":
        from volumential_gb300.volume_fmm import drive_volume_fmm

        return drive_volume_fmm(state["traversal"], state["wrangler"], state["weighted"],
                                state["densities"][0], list1_only=True)
    if kind == "many":
        trav = state["traversal"]
        outs, _ = state["wrangler"].eval_direct_batched(
            trav.target_boxes, trav.neighbor_source_boxes_starts,
            trav.neighbor_source_boxes_lists, state["densities"],
            precision=state["case"]["precision"])
        return outs[0]
    if kind == "batch":
        state["batch"].eval()
        return [p.out for p in state["problems"]]
    if kind == "remesh":
        return _run_remesh(state)
    if kind == "split":
        trav = state["traversal"]
        out, _ = state["wrangler"].eval_direct_helmholtz_split_correction(
            trav.target_boxes, trav.neighbor_source_boxes_starts,
            trav.neighbor_source_boxes_lists, state["weighted"],
            src_func=state["densities"][0])
        return out[0]
    return _run_table(state)


def _run_remesh(state):
    from volumential_gb300.tree_build import (
        build_list1_traversal_device, build_tree_from_leaves_device)

    case = state["case"]
    tree = build_tree_from_leaves_device(*state["leaves"], dim=case["dim"], q_order=case["q"],
                                         as_numpy=False)
    trav = build_list1_traversal_device(tree, as_numpy=False)
    local = state["tree_arguments"]
    out, _ = state["evaluator"](
        None, result=state["result"], mode_coefs=state["densities"][0],
        target_boxes=trav.target_boxes,
        neighbor_source_boxes_starts=trav.neighbor_source_boxes_starts,
        neighbor_source_boxes_lists=trav.neighbor_source_boxes_lists,
        box_centers=tree.box_centers, box_levels=tree.box_levels,
        box_source_starts=tree.box_target_starts,
        box_source_counts_nonchild=tree.box_target_counts_nonchild,
        box_target_starts=tree.box_target_starts,
        box_target_counts_nonchild=tree.box_target_counts_nonchild,
        source_mode_ids=local["source_mode_ids"], target_point_ids=local["target_point_ids"],
        root_extent=tree.root_extent, **state["table_arguments"])
    return {"potential": out, "points": tree.targets,
            "lists": trav.neighbor_source_boxes_lists}


def _run_table(state):
    from volumential_gb300.nearfield_potential_table import NearFieldInteractionTable

    case = state["case"]
    knl = _kernel(case)
    table = NearFieldInteractionTable(
        case["q"], dim=case["dim"], sumpy_kernel=knl, source_box_extent=state["extent"],
        dtype=np.complex128 if knl.is_complex_valued else np.float64)
    kw = {"k": state["k"]} if knl.is_complex_valued else {}
    table.build_table_via_duffy_radial(regular_quad_order=case.get("regular", 20),
                                       radial_quad_order=case.get("radial", 61), **kw)
    return table.get_reduced_table_data()[1]


# {{{ work

def _pairs(trav):
    """Point pairs of list 1."""
    counts = np.asarray(trav.tree.box_target_counts_nonchild, dtype=np.int64)
    st = np.asarray(trav.neighbor_source_boxes_starts, dtype=np.int64)
    tgt = np.repeat(counts[np.asarray(trav.target_boxes)], np.diff(st))
    return int((tgt * counts[np.asarray(trav.neighbor_source_boxes_lists)]).sum())


def _tree_bytes(trav):
    t = trav.tree
    return (t.nboxes * (8 * t.dim + 1 + 8) + 4 * (2 * len(trav.target_boxes) + trav.nnz)
            + 8 * t.ntargets)


def work(case):
    kind = case["kind"]
    if kind == "table":
        # the tensor-product quadrature nodes of every (case, target point,
        # sub-simplex) of the stored entries, each with one kernel value and
        # its share of the q^dim modes' sums
        dim, q = case["dim"], case["q"]
        table = _table(case["kernel"], dim, q, 1.0)
        ids = table.get_reduced_table_data()[0]
        nq = q ** dim
        groups = len(np.unique(ids // (nq * nq) * nq + ids % nq))
        nodes = (2 ** dim * math.factorial(dim) * case.get("regular", 20) ** (dim - 1)
                 * (2 * case.get("radial", 61) + 1))
        cv = 1 if case["kernel"] == "laplace" else 2
        return {"bytes": 8 * cv * len(ids),
                "flops": nodes * (20.0 * groups + 2.0 * cv * len(ids))}
    if kind == "batch":
        total_b = total_f = 0
        for level, q, nrhs in _batch_problems(case):
            trav = _mesh(3, q, level, None, None)[0]
            total_b += _tree_bytes(trav) + 16 * nrhs * trav.tree.ntargets
            total_f += 2.0 * nrhs * _pairs(trav)
        return {"bytes": total_b, "flops": total_f}
    trav = _traversal(case)[0]
    n, pairs, nrhs = trav.tree.ntargets, _pairs(trav), case.get("nrhs", 1)
    if kind == "split":
        # distance, a logarithm or root, the series and the weighted sum
        return {"bytes": _tree_bytes(trav) + n * (8 * case["dim"] + 8 + 16),
                "flops": 50.0 * pairs}
    tc, cc = case["kernel"] != "laplace", case.get("complex_density", False)
    return {"bytes": _tree_bytes(trav) + nrhs * n * ((16 if cc else 8)
                                                     + (16 if tc or cc else 8)),
            "flops": 2.0 * pairs * nrhs * (2 if tc else 1) * (2 if cc else 1)}

# }}}


# {{{ the same results in plain torch, 64 bits

def _list1_geometry(trav):
    """Per list-1 pair: first target, first source (particle indices), the
    offset of the target centre in source box extents, the ratio of the
    extents and the source extent."""
    t = trav.tree
    st = np.asarray(trav.neighbor_source_boxes_starts, dtype=np.int64)
    tb = np.repeat(np.asarray(trav.target_boxes, dtype=np.int64), np.diff(st))
    sb = np.asarray(trav.neighbor_source_boxes_lists, dtype=np.int64)
    lev = np.asarray(t.box_levels, dtype=np.int64)
    ext = t.root_extent * 0.5 ** lev
    off = (np.asarray(t.box_centers)[:, tb] - np.asarray(t.box_centers)[:, sb]) / ext[sb]
    first = np.asarray(t.box_target_starts, dtype=np.int64)
    return first[tb], first[sb], off, ext[tb] / ext[sb], ext[sb]


def _list1_sum(trav, kernel, dim, q, extent, rhs):
    """sum over list 1 of the closed form's blocks times ``rhs`` [nrhs, N]."""
    nq = q ** dim
    first_t, first_s, off, ratio, ext = _list1_geometry(trav)
    key = np.concatenate([np.rint(off * 4.0), np.rint(ratio * 2.0)[None]]).astype(np.int64)
    cases, which = np.unique(key, axis=1, return_inverse=True)
    order = np.argsort(which.ravel(), kind="stable")
    bounds = np.concatenate([[0], np.cumsum(np.bincount(which.ravel()))])
    src, w = _nodes(dim, q)
    src_t = torch.from_numpy(src).cuda()
    w_t = torch.from_numpy(w).cuda()
    dtype = torch.complex128 if kernel != "laplace" or rhs.is_complex() else torch.float64
    # [box, rhs, point], boxes in particle order
    x = rhs.reshape(rhs.shape[0], -1, nq).permute(1, 0, 2).contiguous()
    out = torch.zeros(x.shape, dtype=dtype, device="cuda")
    for c in range(cases.shape[1]):
        sel = order[bounds[c]:bounds[c + 1]]
        centre = torch.from_numpy(cases[:dim, c] / 4.0 + 0.5).cuda()
        size = float(cases[dim, c]) / 2.0
        tgt = centre + size * (src_t - 0.5)
        block = _table_values(kernel, dim, q, extent, HELMHOLTZ_K, src_t[:, None, :],
                              w_t[:, None], tgt[None])           # [source, target]
        b_t = torch.from_numpy(first_t[sel] // nq).cuda()
        b_s = torch.from_numpy(first_s[sel] // nq).cuda()
        h = torch.from_numpy(np.ascontiguousarray(ext[sel])).cuda()
        xs = x[b_s]
        if kernel == "laplace":
            h2 = (h / extent) ** 2
            val = (xs * h2[:, None, None]) @ block.to(xs.dtype)
            if dim == 2:   # G(h r) = G(r) - log(h) / (2 pi)
                val = val + (xs @ (w_t * extent ** 2).to(xs.dtype))[:, :, None] * (
                    -h2 * torch.log(h / extent) / (2.0 * math.pi))[:, None, None]
        else:
            val = xs.to(dtype) @ block
        out.index_add_(0, b_t, val.to(dtype))
    return out.permute(1, 0, 2).reshape(rhs.shape)


def _split_exact(case, trav, weighted):
    """sum over list-1 points of weights x (G_k - G_0)(r), self limit added."""
    dim, nq, k = case["dim"], case["q"] ** case["dim"], case["k"]
    first_t, first_s, _, _, _ = _list1_geometry(trav)
    pts = _points(trav).reshape(dim, -1, nq)
    x = weighted.reshape(-1, nq)
    out = torch.zeros(x.shape, dtype=torch.complex128, device="cuda")
    gamma = 0.5772156649015329
    lk = math.log(0.5 * k) + gamma
    for lo in range(0, len(first_t), 8192):
        b_t = torch.from_numpy(first_t[lo:lo + 8192] // nq).cuda()
        b_s = torch.from_numpy(first_s[lo:lo + 8192] // nq).cuda()
        d2 = ((pts[:, b_t, None, :] - pts[:, b_s, :, None]) ** 2).sum(0)  # [pair, source, target]
        if dim == 3:
            kr = k * torch.sqrt(d2)
            half = 0.5 * kr
            # (exp(ikr) - 1) / (4 pi r) = exp(ikr/2) i sin(kr/2) / (2 pi r)
            sinc = torch.where(kr > 0, torch.sin(half) / torch.where(kr > 0, half, half + 1.0),
                               torch.ones_like(half))
            g = 1j * torch.polar(torch.ones_like(half), half) * sinc * (k / (4.0 * math.pi))
        else:
            log_r = 0.5 * torch.log(torch.where(d2 > 0, d2, torch.ones_like(d2)))
            re = torch.full_like(d2, -lk / (2.0 * math.pi))
            im = torch.full_like(d2, 0.25)
            term, harmonic = torch.ones_like(d2), 0.0
            for n in range(1, 40):
                term = term * d2 * (-0.25 * k * k / (n * n))
                harmonic += 1.0 / n
                re += term * ((harmonic - lk - log_r) / (2.0 * math.pi))
                im += 0.25 * term
            g = torch.complex(re, im)
        # at r = 0 the remainder takes its limit, the self term that is added back
        out.index_add_(0, b_t, torch.einsum("ps,pst->pt", x[b_s].to(g.dtype), g))
    return out.reshape(-1)


def _tanh_sinh(n):
    n = max(3, n)
    h = 1.0 / math.sqrt(n)
    t = h * np.arange(-n, n + 1)
    a = 0.5 * math.pi * np.sinh(t)
    x = 0.5 * (1.0 + np.tanh(a))
    w = 0.25 * math.pi * h * np.cosh(t) / np.cosh(np.minimum(np.abs(a), 300.0)) ** 2
    keep = (x > 0.0) & (x < 1.0)
    return x[keep], w[keep]


def _table_exact(case, extent, k):
    """The stored entries by the same Duffy quadrature: the box split at the
    target (clipped into it), each part into simplices mapped from the cube."""
    import itertools

    dim, q = case["dim"], case["q"]
    nq = q ** dim
    stored = _table(case["kernel"], dim, q, 1.0)
    ids = stored.get_reduced_table_data()[0]
    unit_targets = np.moveaxis(stored.get_case_target_points(), 0, -1)
    group, which = np.unique(ids // (nq * nq) * nq + ids % nq, return_inverse=True)
    rx, rw = _tanh_sinh(case.get("radial", 61))
    gx, gw = _gauss(case.get("regular", 20))
    axes = [torch.from_numpy(v).cuda() for v in [rx] + [gx] * (dim - 1)]
    waxes = [torch.from_numpy(v).cuda() for v in [rw] + [gw] * (dim - 1)]
    r = [g.ravel() for g in torch.meshgrid(*axes, indexing="ij")]
    wt = functools.reduce(torch.mul, [g.ravel() for g in torch.meshgrid(*waxes, indexing="ij")])
    for i in range(dim - 1):
        wt = wt * r[i] ** (dim - 1 - i)
    u = list(itertools.accumulate(r, torch.mul))
    nodes = torch.from_numpy(_gauss(q)[0] * extent).cuda()
    complex_valued = case["kernel"] != "laplace"
    vals = torch.zeros((len(group), nq), dtype=torch.complex128 if complex_valued
                       else torch.float64, device="cuda")

    def basis(y):
        cols = []
        for m in range(q):
            p = torch.ones_like(y)
            for j in range(q):
                if j != m:
                    p = p * ((y - nodes[j]) / (nodes[m] - nodes[j]))
            cols.append(p)
        return torch.stack(cols)                                   # [q, nodes]

    for gi, gid in enumerate(group):
        t = unit_targets[gid // nq, gid % nq] * extent
        c = np.clip(t, 0.0, extent)
        for signs in itertools.product((-1.0, 1.0), repeat=dim):
            length = [c[a] if signs[a] < 0 else extent - c[a] for a in range(dim)]
            if min(length) <= 0.0:
                continue
            for perm in itertools.permutations(range(dim)):
                y = [None] * dim
                for i, a in enumerate(perm):
                    y[a] = c[a] + signs[a] * length[a] * u[i]
                r2 = sum((t[a] - y[a]) ** 2 for a in range(dim))
                f = wt * float(np.prod(length))
                f = torch.where(r2 > 0, f, torch.zeros_like(f))
                rr = torch.sqrt(torch.where(r2 > 0, r2, torch.ones_like(r2)))
                if not complex_valued:
                    g = 1.0 / (4 * math.pi * rr) if dim == 3 else -torch.log(rr) / (2 * math.pi)
                elif dim == 3:
                    g = torch.polar(1.0 / (4 * math.pi * rr), k * rr)
                else:
                    g = 0.25 * torch.complex(-torch.special.bessel_y0(k * rr),
                                             torch.special.bessel_j0(k * rr))
                g = g * f
                b = [basis(v).to(g.dtype) for v in y]
                left = b[0] if dim == 2 else (b[0][:, None] * b[1][None]).reshape(q * q, -1)
                vals[gi] += ((left * g) @ b[-1].T).reshape(-1)
    modes = torch.from_numpy((ids % (nq * nq)) // nq).cuda()
    return vals[torch.from_numpy(which.ravel()).cuda(), modes].cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "table":
        if case["dim"] == 3 and case["q"] > 4:
            return None
        s = prepare(case, seed)
        return _table_exact(case, s["extent"], s["k"])
    if kind == "batch":
        out = []
        for i, (level, q, nrhs) in enumerate(_batch_problems(case)):
            trav = _mesh(3, q, level, None, None)[0]
            rhs = _densities(97 * seed + i, _points(trav), nrhs)
            out.append(_list1_sum(trav, "laplace", 3, q, 1.0, rhs).reshape(-1))
        return out
    trav = _traversal(case)[0]
    rhs = _densities(seed, _points(trav), case.get("nrhs", 1), case.get("complex_density", False))
    if kind == "split":
        weights = torch.from_numpy(np.ascontiguousarray(trav.tree.weights)).cuda()
        return _split_exact(case, trav, rhs[0] * weights)
    got = _list1_sum(trav, case["kernel"], case["dim"], case["q"], _table_extent(case), rhs)
    if kind == "many":
        return got
    if kind == "drive":
        return [got[0]]
    if kind == "remesh":
        return {"potential": got[0], "points": None, "lists": None}
    return got[0]

# }}}
