"""Trees whose particle order is the user's against the general reordering.

For ``ParticleTree`` the wrangler neither gathers through an identity
permutation nor uploads box-local ids; a subclass with its own (same or
permuted) order takes the general way.  Both must agree on every input form.
"""

import numpy as np
import pytest

from helpers import wrangler_for
from volumential_gb300 import workloads as W
from volumential_gb300.expansion_wrangler_fpnd import _compute_box_local_ids
from volumential_gb300.tree_build import ParticleTree

pytestmark = pytest.mark.gpu


class _OwnOrder(ParticleTree):
    """The same tree with orders of its own (identity unless set)."""

    order = None

    @property
    def sorted_target_ids(self):
        return np.arange(self.ntargets) if self.order is None else self.order

    @property
    def user_source_ids(self):
        return np.arange(self.ntargets) if self.order is None else np.argsort(self.order)


def _pair(dim=2, q=3):
    w = W.uniform_workload("io", dim, 3, q, seed=5)
    fast = wrangler_for(w)
    slow = wrangler_for(w)
    slow.tree = _OwnOrder(**{k: getattr(w.tree, k) for k in ParticleTree.__dataclass_fields__})
    return w, fast, slow


def _forms(torch, n):
    a = np.random.default_rng(1).standard_normal((2, n))
    dev = torch.from_numpy(a).cuda()
    return {
        "numpy": a[0], "numpy-2d": a, "cpu": torch.from_numpy(a[1]), "cuda": dev[0].clone(),
        "cuda-2d": dev, "strided": dev.t().contiguous().t()[1], "complex": dev[0] + 1j * dev[1],
        "longer": torch.cat([dev[0], dev[1][:5]]), "float32": dev[0].float(),
    }


def test_reordering_agrees_with_the_general_path(cuda):
    torch = cuda
    w, fast, slow = _pair()
    for name, x in _forms(torch, w.n_points).items():
        for f in ("reorder_sources", "reorder_targets"):
            a, b = getattr(fast, f)(x), getattr(slow, f)(x)
            assert a.dtype == b.dtype and torch.equal(a, b) and a.is_contiguous(), name
            if hasattr(x, "is_cuda") and x.is_cuda:
                assert a.untyped_storage().data_ptr() != x.untyped_storage().data_ptr(), name
        t = torch.as_tensor(x).cuda()
        a, b = fast.reorder_potentials([t])[0], slow.reorder_potentials([t])[0]
        assert torch.equal(a, b)
        assert a.untyped_storage().data_ptr() != t.untyped_storage().data_ptr()
    with pytest.raises(IndexError):
        fast.reorder_sources(torch.zeros(w.n_points - 1, dtype=torch.float64, device="cuda"))


@pytest.mark.parametrize("dim,q", [(2, 1), (2, 5), (3, 4)])
def test_local_ids_agree_with_the_general_path(cuda, dim, q):
    w, fast, slow = _pair(dim, q)
    nq = q ** dim
    want = _compute_box_local_ids(slow.tree, nq)
    assert np.array_equal(_compute_box_local_ids(fast.tree, nq), want)
    payload = {"table_data_shapes": {"n_q_points": nq}}
    ids = fast._device_local_ids(payload)
    assert ids.is_cuda and np.array_equal(ids.cpu().numpy(), want)
    assert np.array_equal(slow._device_local_ids(payload), want)
    # a permuted order is followed, and its ids are not taken from a memo
    slow.tree.order = np.random.default_rng(2).permutation(w.n_points)
    assert np.array_equal(slow._device_local_ids(payload), want[slow.tree.order])
    with pytest.raises(ValueError, match="not divisible"):
        fast._device_local_ids({"table_data_shapes": {"n_q_points": w.n_points + 1}})
    fast.tree.sources_are_targets = False
    with pytest.raises(ValueError, match="coincide"):
        fast._device_local_ids(payload)
