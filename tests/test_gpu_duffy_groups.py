"""The grouped Duffy build (all modes of a target together) against the
per-entry build: every instance of the kernel, radial rules of one and two
blocks of nodes, all radial kernels, a capped grid.

Tolerance: both sum the same quadrature; each product carries a few ulps and
the basis moments at most a factor of 2 (the Lebesgue constant of up to eight
Chebyshev points), so the entries agree within 1e-13 of the largest one."""

import ctypes as C

import numpy as np
import pytest

from volumential_gb300 import table_builder as TB
from volumential_gb300.kernels import (HelmholtzKernel, LaplaceKernel, RadialPowerKernel,
                                       RadialPowerLogKernel)
from volumential_gb300.nearfield_potential_table import NearFieldInteractionTable

pytestmark = pytest.mark.gpu


def _both(monkeypatch, dim, q, knl, reg, rad, max_ctas=0, extent=0.5):
    from volumential_gb300 import _lib

    cplx = knl.is_complex_valued
    t = NearFieldInteractionTable(q, dim=dim, sumpy_kernel=knl, source_box_extent=extent,
                                  dtype=np.complex128 if cplx else np.float64)
    ids = t._get_invariant_entry_info()["entry_ids"]
    pick = ids[np.unique(np.linspace(0, len(ids) - 1, 300).astype(int))]
    kw = dict(regular_quad_order=reg, radial_quad_order=rad, entry_ids=pick, store=False,
              max_ctas=max_ctas, **({"k": 5.0} if cplx else {}))
    _, grouped = TB.build_table_values(t, **kw)
    lib = _lib.lib()

    class PerEntry:
        def __getattr__(self, name):
            if name == "vl1_duffy_table_grouped":
                return lambda d, n, eg, ge, out, s: lib.vl1_duffy_table(d, out, s)
            return getattr(lib, name)

    with monkeypatch.context() as m:
        m.setattr(_lib, "lib", lambda: PerEntry())
        _, single = TB.build_table_values(t, **kw)
    return grouped, single


@pytest.mark.parametrize("dim,q", [(2, q) for q in (1, 2, 3, 4, 5, 6, 7, 8, 9)]
                         + [(3, q) for q in (1, 2, 3, 4, 5, 6, 7)])
@pytest.mark.parametrize("cplx", [False, True])
def test_instances(cuda, monkeypatch, dim, q, cplx):
    knl = (HelmholtzKernel if cplx else LaplaceKernel)(dim)
    a, b = _both(monkeypatch, dim, q, knl, 4, 11)
    assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b))


@pytest.mark.parametrize("dim,reg,rad,cap", [(2, 20, 61, 0), (3, 6, 64, 0), (2, 3, 200, 5),
                                             (3, 1, 63, 3), (2, 130, 11, 0)])
def test_rules_and_capped_grids(cuda, monkeypatch, dim, reg, rad, cap):
    a, b = _both(monkeypatch, dim, 3, HelmholtzKernel(dim), reg, rad, cap)
    assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b))
    full, _ = _both(monkeypatch, dim, 3, HelmholtzKernel(dim), reg, rad, 0)
    assert np.array_equal(a, full)     # the grid does not change the sums' order


@pytest.mark.parametrize("dim,knl", [(2, RadialPowerKernel(2, 2)), (2, RadialPowerLogKernel(2, 4)),
                                     (3, RadialPowerKernel(3, 3)), (3, RadialPowerKernel(3, 1))])
def test_power_kernels(cuda, monkeypatch, dim, knl):
    a, b = _both(monkeypatch, dim, 3, knl, 6, 21, extent=2.0)
    assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b))


def test_invalid_modes_and_descriptors(cuda):
    import torch

    from volumential_gb300 import _lib

    lib, d = _lib.lib(), _lib.DuffyDesc()
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    assert lib.vl1_duffy_table_grouped(None, 0, None, None, out.data_ptr(),
                                       C.c_void_p(0)) == _lib.VL1_E_ARG
    d.dim, d.q, d.n_entries = 4, 2, 1        # refused as by the per-entry build
    assert lib.vl1_duffy_table_grouped(C.byref(d), 1, out.data_ptr(), out.data_ptr(),
                                       out.data_ptr(), C.c_void_p(0)) == _lib.VL1_E_ARG
