"""Error of the FP64 tensor-core path per target point, against sums in extended
precision (64 significant bits on x86, 113 on Arm): densities in all boxes, in
one box and in one point, at every phase of the digits, and tables whose blocks
lie many decades apart.

Bound.  A target row's scale is 2^(E + 2), E the largest exponent of
density row + block over its own pairs with a nonzero density, each rounded up to
a multiple of 8 (by at most 2^5 and 2^7, after the density's two extra leading
bits and the largest value of a row or block up to twice 2^(e - 1)): at most
2^16 M with M = max over those pairs of max|x'| max|T|.  Dropped are the seven
digit products of weight 2^-80 per pair of points (zero-mean, |digit| <= 128, 74
in the mean square: 2^-66.2 together in the mean square) and digits beyond 2^-64
of either operand (less).  Over K source points that is 2^-66.2 sqrt(K) 2^16 M in
the mean square; six times that, plus one rounding of the result and one of
the reference's products."""

import ctypes as C

import numpy as np
import pytest

from helpers import plan_and_view
from volumential_gb300 import _lib
from volumential_gb300 import workloads as W
from volumential_gb300.batched import MixedSchedule
from volumential_gb300.kernels import HelmholtzKernel

pytestmark = pytest.mark.gpu


class _Reference:
    """Blocks of the list-1 pairs; sums in extended precision and M per box."""

    def __init__(self, torch, plan, view, keep):
        rows, signs = plan.orbit_index_map()
        keys = torch.empty(keep["lists"].numel(), dtype=torch.int32, device="cuda")
        _lib.check(_lib.lib().vl1_classify_pairs(plan.handle, C.byref(view), keys.data_ptr(),
                                                 C.c_void_p(0)), "vl1_classify_pairs")
        torch.cuda.synchronize()
        rows, signs, self.keys = (t.cpu().numpy() for t in (rows, signs, keys))
        self.k = {n: t.cpu().numpy() for n, t in keep.items()}
        self.nq, d = plan.nq, plan.desc
        table = plan._host["table"]
        self.blocks = {}
        for key in np.unique(self.keys):
            lev, c = divmod(int(key), plan.n_cases)
            self.blocks[int(key)] = table[lev][rows[c]] * signs[c]
        ext = view.root_extent * 0.5 ** self.k["levels"].astype(float)
        p = d.scaling_exponent
        self.scale = ext ** p / d.table_root_extent ** p
        assert d.displacement_kind == 0

    def sums(self, x):
        """(sums, M, K) of densities x [N]: [targets, nq] and per target box."""
        k, nq = self.k, self.nq
        ld = np.clongdouble if any(np.iscomplexobj(b) for b in self.blocks.values()) \
            else np.longdouble
        n_tb = len(k["target_boxes"])
        y, m = np.zeros((n_tb, nq), dtype=ld), np.zeros(n_tb)
        n = np.zeros(n_tb)
        for i in range(n_tb):
            for q in range(k["starts"][i], k["starts"][i + 1]):
                sb = k["lists"][q]
                s0 = k["src_starts"][sb]
                v = self.scale[sb] * x[s0:s0 + nq]     # as the kernels round it
                top = np.abs(v).max()
                if top == 0.0:
                    continue
                b = self.blocks[int(self.keys[q])]
                y[i] += v.astype(np.longdouble) @ b.astype(ld)
                part = np.maximum(np.abs(b.real).max(), np.abs(b.imag).max())
                m[i] = max(m[i], top * part)
                n[i] += np.count_nonzero(v)
        return y, m, n


def _steep(tables, dim, q):
    """Blocks 2^-30 apart per unit of distance (a strongly damped kernel)."""
    nq = q ** dim
    for t in tables:
        ids = np.asarray(t._get_scalar_arithmetic_invariant_entry_info()["entry_ids"])
        vec = np.abs(np.asarray(t.interaction_case_vecs))[ids // (nq * nq)].sum(-1)
        t.data[:] *= 2.0 ** (-30.0 * vec / 4.0)


@pytest.mark.parametrize("dim,level,q,cplx", [(3, 2, 4, False), (3, 2, 3, False),
                                              (2, 3, 5, True), (3, 1, 5, False)])
@pytest.mark.parametrize("steep", [False, True])
def test_error_per_target(cuda, dim, level, q, cplx, steep):
    torch = cuda
    # (2D Laplace kernels add a displacement in FP64: the Helmholtz kernel here)
    kernel = dict(kernel=HelmholtzKernel(dim), complex_table=True) if cplx else {}
    w = W.uniform_workload("digits", dim, level, q, seed=71, **kernel)
    if steep:
        _steep(w.tables, dim, q)
    plan, view, keep = plan_and_view(w)
    ref = _Reference(torch, plan, view, keep)
    nq, n = q ** dim, w.n_points
    rng = np.random.default_rng(8)
    one_box, one_point = np.zeros(n), np.zeros(n)
    s = int(ref.k["src_starts"][ref.k["target_boxes"][len(ref.k["target_boxes"]) // 3]])
    one_box[s:s + nq] = rng.standard_normal(nq)
    one_point[s + nq // 2] = 1.7
    sched = MixedSchedule(plan, view, keep, 1, 0, int(_lib.lib().vl1_eval_fp64_item_keys(
        plan.handle)), workspace=False)
    out = torch.empty(n, dtype=torch.complex128 if cplx else torch.float64, device="cuda")
    tgt = np.concatenate([np.arange(nq) + ref.k["tgt_starts"][b] for b in ref.k["target_boxes"]])
    for x in (rng.standard_normal(n), one_box, one_point):
        for phase in range(8):
            v = x * 2.0 ** phase
            c = torch.from_numpy(v).cuda()
            _lib.check(_lib.lib().vl1_eval_fp64_tiles(
                plan.handle, C.byref(view), C.byref(sched.c_struct), c.data_ptr(),
                _lib.VL1_REAL64, 1, out.data_ptr(), C.c_void_p(0)), "vl1_eval_fp64_tiles")
            plan.raise_on_status(0)
            y, m, k = ref.sums(v)
            err = out.cpu().numpy()[tgt].reshape(y.shape) - y
            bound = 6.0 * 2.0 ** -50.2 * np.sqrt(k) * m
            for g, r in ((err.real, y.real), (err.imag, y.imag)):
                b = 2.0 ** -52 * np.abs(r) + bound[:, None]
                assert np.all(np.abs(g) <= b), (phase, float((np.abs(g)[b > 0] / b[b > 0]).max()))
