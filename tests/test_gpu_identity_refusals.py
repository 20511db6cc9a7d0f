"""What the general reordering of potentials refuses, the identity order's does
too: tensors that are not on the device."""

import pytest

from test_gpu_identity_order import _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [0, 5])
def test_host_tensors(cuda, extra):
    w, fast, slow = _pair()
    x = cuda.zeros(w.n_points + extra, dtype=cuda.float64)
    for wr in (slow, fast):
        with pytest.raises(RuntimeError):
            wr.reorder_potentials([x])
    assert fast.reorder_sources(x).is_cuda and slow.reorder_sources(x).is_cuda
