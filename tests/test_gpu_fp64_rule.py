"""Which FP64 kernel a call takes, and that both agree there.

Trees of many small boxes on either side of the line between the per-box
kernel and the tensor-core path: the schedule that the rule keeps for the view
says which was taken from the second call on.  Both are FP64-accurate (a few
units of 2^-53 of the sums' magnitude), so they agree to 1e-13.
"""

import numpy as np
import pytest

from helpers import plan_and_view, rel_l2
from volumential_gb300 import workloads as W
from volumential_gb300.plan import as_device_tensor

pytestmark = pytest.mark.gpu

CASES = [  # dim, level, q, complex, tensor cores
    (2, 7, 3, False, True), (2, 6, 5, False, True), (2, 6, 3, False, False),
    (2, 7, 2, True, False), (3, 4, 2, False, False), (3, 3, 3, False, False),
    (2, 3, 3, False, False),
]


@pytest.mark.parametrize("dim,level,q,cplx,tiles", CASES)
def test_either_side_of_the_line(cuda, dim, level, q, cplx, tiles):
    torch = cuda
    w = W.uniform_workload("fr", dim, level, q, seed=17)
    plan, view, keep = plan_and_view(w)
    c = as_device_tensor(np.ascontiguousarray(w.coefs))[0]
    if cplx:
        c = c * (1.0 - 0.5j)
    stream = torch.cuda.current_stream().cuda_stream
    want = torch.empty_like(c)
    plan.eval_fp64(view, c, want, stream=stream)
    outs = []
    for _ in range(3):
        out = torch.full_like(c, float("nan"))
        plan.eval_fp64(view, c, out, stream=stream, keep=keep)
        outs.append(out)
    plan.raise_on_status(stream)
    assert (view.fp64_schedules[2 if cplx else 1][1] is not None) == tiles
    assert torch.equal(outs[1], outs[2])
    for out in outs:
        assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) <= 1e-13
