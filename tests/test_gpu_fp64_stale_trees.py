"""Tree arrays written in place behind torch's back (``.data``, a kernel of the
caller's, a graph replay): FP64 evaluations follow the arrays.

The tensor-core path walks a schedule made from the arrays; every call compares
them with the copy the schedule was made from.  The oracle is the per-box
kernel, which reads the arrays (``eval_fp64`` without ``keep``); tolerance 1e-12
relative l2, both being FP64 sums of at most a few thousand terms.

Each change below keeps every index in its range, so that the arrays stay valid
for both kernels."""

import numpy as np
import pytest

from helpers import plan_and_view, rel_l2
from volumential_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _swap(a, i, j):
    a[i], a[j] = a[j].copy(), a[i].copy()


def _interior(w, n=2):
    """Indices of target boxes with full, equally long lists, far apart."""
    st = w.traversal.neighbor_source_boxes_starts
    full = np.flatnonzero(np.diff(st) == np.diff(st).max())
    return [int(full[k]) for k in np.linspace(0, len(full) - 1, n).astype(int)]


def _targets_and_lists(w, a):
    """Two target boxes change places, with their lists."""
    i, j = _interior(w)
    _swap(a["target_boxes"], i, j)
    st = a["starts"]
    m = st[i + 1] - st[i]
    li, lj = a["lists"][st[i]:st[i] + m].copy(), a["lists"][st[j]:st[j] + m].copy()
    a["lists"][st[i]:st[i] + m], a["lists"][st[j]:st[j] + m] = lj, li


def _lists(w, a):
    """One list entry is replaced by its neighbour in the list: a source that
    counts twice is no schedule's, only the per-box kernel's."""
    i, _ = _interior(w)
    s = a["starts"][i]
    a["lists"][s] = a["lists"][s + 1]


def _starts(w, a):
    """One pair moves from a target box's list to the one before it: adjacent
    boxes that share the neighbour."""
    st, ls, tb, ctr = a["starts"], a["lists"], a["target_boxes"], a["centers"]
    ext = w.tree.root_extent * 0.5 ** int(a["levels"][tb[0]])
    for i in range(1, len(tb)):
        c = ctr[:, tb[i - 1]]
        near = [p for p in range(st[i], st[i + 1])
                if np.abs(ctr[:, ls[p]] - c).max() < 1.25 * ext]
        if near and st[i + 1] - st[i] > 1:
            p = near[0]
            ls[st[i]], ls[p] = ls[p], ls[st[i]]
            st[i] += 1
            return
    raise AssertionError


def _centers(w, a):
    """The boxes mirrored: every coordinate along axis 0 negated."""
    a["centers"][0] *= -1.0


def _source_ranges(w, a):
    """Two boxes' sources change places."""
    i, j = (int(a["target_boxes"][k]) for k in _interior(w))
    _swap(a["src_starts"], i, j)


def _source_counts(w, a):
    i = int(a["target_boxes"][_interior(w)[0]])
    a["src_counts"][i] -= 1


def _modes(w, a):
    """Two sources of a box in one mode: their densities add."""
    s = a["src_starts"][a["target_boxes"][_interior(w)[0]]]
    a["smode"][s] = a["smode"][s + 1]


CHANGES = [_targets_and_lists, _lists, _starts, _centers, _source_ranges, _source_counts, _modes]


@pytest.mark.parametrize("dim,level,q,nrhs,cplx", [(2, 6, 5, 1, False), (2, 6, 5, 2, True),
                                                   (3, 3, 4, 1, False)])
@pytest.mark.parametrize("change", CHANGES, ids=[c.__name__[1:] for c in CHANGES])
def test_arrays_changed_in_place(cuda, dim, level, q, nrhs, cplx, change):
    torch = cuda
    w = W.uniform_workload("stale", dim, level, q, seed=51, nrhs=nrhs)
    plan, view, keep = plan_and_view(w)
    # (densities of one size everywhere: every change is seen)
    c = torch.from_numpy(np.random.default_rng(5).standard_normal(w.coefs.shape)).cuda()
    c = c * (1.0 - 0.5j if cplx else 1.0)
    out, ref = torch.empty_like(c), torch.empty_like(c)

    def evaluate():
        out.fill_(7.0)
        plan.eval_fp64(view, c, out, stream=0, nrhs=nrhs, keep=keep)
        plan.raise_on_status(0)
        plan.eval_fp64(view, c, ref, stream=0, nrhs=nrhs)
        plan.raise_on_status(0)
        return out.cpu().numpy(), ref.cpu().numpy()

    rows = nrhs * (2 if cplx else 1)
    for _ in range(3):
        got, first = evaluate()
        assert rel_l2(got, first) <= 1e-12
    assert view.fp64_schedules[rows][1] is not None
    host = {k: v.cpu().numpy() for k, v in keep.items()}
    change(w, host)
    for k, v in keep.items():
        version = v._version
        v.data.copy_(torch.from_numpy(host[k]))
        assert v._version == version
    for _ in range(4):
        got, now = evaluate()
        assert rel_l2(got, now) <= 1e-12
    assert rel_l2(now, first) > 1e-6 or change in (_targets_and_lists,)


def test_graph_replay_rewrites_the_lists(cuda):
    """A captured copy into the list array between two evaluations."""
    torch = cuda
    w = W.uniform_workload("stale_g", 2, 6, 5, seed=52)
    plan, view, keep = plan_and_view(w)
    c = torch.from_numpy(w.coefs).cuda()
    out, ref = torch.empty_like(c), torch.empty_like(c)
    host = {k: v.cpu().numpy() for k, v in keep.items()}
    _targets_and_lists(w, host)
    src = {k: torch.from_numpy(host[k]).cuda() for k in ("target_boxes", "lists")}
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for k, v in src.items():
            keep[k].copy_(v)
    # (captured, not run: the versions moved, so the arrays' first schedule is
    # made now)
    for _ in range(3):
        plan.eval_fp64(view, c, out, stream=0, keep=keep)
    assert view.fp64_schedules[1][1] is not None
    g.replay()
    torch.cuda.synchronize()
    for _ in range(3):
        plan.eval_fp64(view, c, out, stream=0, keep=keep)
        plan.eval_fp64(view, c, ref, stream=0)
        plan.raise_on_status(0)
        assert rel_l2(out.cpu().numpy(), ref.cpu().numpy()) <= 1e-12


@pytest.mark.parametrize("offset", [1, 4])
def test_arrays_at_odd_addresses(cuda, offset):
    """Arrays that start inside a larger one (4-byte steps, and 16-byte ones),
    changed in their last entries."""
    from volumential_gb300 import plan as plan_module
    from volumential_gb300.plan import tree_view_from_arrays

    torch = cuda
    w = W.uniform_workload("stale_o", 2, 6, 5, seed=53)
    plan, view, keep = plan_and_view(w)
    k = {}
    for name, t in keep.items():
        big = torch.zeros(offset + t.numel(), dtype=t.dtype, device="cuda")
        k[name] = big[offset:].view(t.shape)
        k[name].copy_(t)
    args = dict(zip(plan_module._VIEW_ARGS, (k[n] for n in plan_module._VIEW_KEYS)))
    v, k = tree_view_from_arrays(root_extent=view.root_extent, **args)
    c = torch.from_numpy(np.random.default_rng(6).standard_normal(w.n_points)).cuda()
    out, ref = torch.empty_like(c), torch.empty_like(c)

    def evaluate():
        plan.eval_fp64(v, c, out, stream=0, keep=k)
        plan.eval_fp64(v, c, ref, stream=0)
        plan.raise_on_status(0)
        assert rel_l2(out.cpu().numpy(), ref.cpu().numpy()) <= 1e-12

    for _ in range(3):
        evaluate()
    assert v.fp64_schedules[1][1] is not None and not v.fp64_schedules[1][1].is_stale()
    box = int(k["lists"][-1])
    s = int(k["src_starts"][box]) + int(k["src_counts"][box]) - 1
    k["smode"].data[s] = int(k["smode"][s - 1])       # two sources in one mode
    for _ in range(3):
        evaluate()
    assert v.fp64_schedules[1][1] is None             # the per-box kernel again
