"""The launch shapes an untuned core takes: either side of the lines of the
rule (columns, levels, precision) the operator, the preconditioner and their
transposes give the bits of shape 0."""

import pytest
import torch

from suetes_b200.workloads import mountain_wave
from _cases import random_fields, shapes5, to_cuda

pytestmark = pytest.mark.gpu

SCALES = {"u": 1.0, "v": 1.0, "w": 0.5, "pi": 1e-3, "eta_dot": 1e-3}


# (5, 4, 156 / 157): the float64 column tile reaches 200 KB of shared memory
# between them; 141^2 and 142^2, 224^2: the matvec's and the march's lines
@pytest.mark.parametrize("dtype,shape", [
    (torch.float32, (33, 17, 9)), (torch.float32, (2, 2, 2)), (torch.float32, (5, 4, 320)),
    (torch.float32, (224, 223, 4)), (torch.float32, (247, 246, 3)), (torch.float32, (260, 260, 3)),
    (torch.float64, (5, 4, 156)), (torch.float64, (5, 4, 157)), (torch.float64, (141, 141, 4)),
    (torch.float64, (142, 142, 4)), (torch.float64, (174, 173, 3))])
def test_default_shapes_give_the_bits_of_shape_zero(dtype, shape):
    from suetes_b200.steppers import VerticalPreconditioner
    st, _, _ = mountain_wave(*shape, dtype=dtype, flat=True)
    ph, sol = st.physics, st.implicit_solver
    bg = ph.precompute_bg(ph.bg_state_ref())
    core = sol._core(dtype, bg)
    pre = VerticalPreconditioner(ph, st.dt, alpha=st.alpha)
    pre.precompute_banded(bg)
    x = to_cuda(random_fields(shapes5(*shape), 3, SCALES), dtype)
    calls = [lambda: sol.matvec_scaled(x, bg), lambda: pre(x), lambda: sol.matvec_scaled(x, bg, transpose=True),
             lambda: pre.transpose(x)]
    default = [f() for f in calls]
    chosen = core.tuning()
    core.set_tuning()
    for got, f in zip(default, calls):
        want = f()
        for k in got:
            assert torch.isfinite(want[k]).all() and torch.equal(got[k], want[k]), (k, chosen)
