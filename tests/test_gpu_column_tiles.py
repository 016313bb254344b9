"""The batched column tiles on either side of the line between one wide block
per tile and several small ones (148 tiles): the preconditioner and its
transpose give the bits of shape 0 at level counts below, at and past a round
of the wide block's loads (32 levels a row of threads, two rows in flight)."""

import pytest
import torch

from suetes_b200.workloads import mountain_wave
from _cases import random_fields, shapes5, to_cuda

pytestmark = pytest.mark.gpu

SCALES = {"u": 1.0, "v": 1.0, "w": 0.5, "pi": 1e-3, "eta_dot": 1e-3}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(32, 148, 3), (32, 149, 3), (33, 74, 2), (33, 75, 5), (5, 4, 31), (40, 3, 32),
                                   (7, 6, 33), (31, 5, 63), (32, 4, 64), (65, 2, 65), (9, 8, 129)])
def test_column_tiles_give_the_bits_of_shape_zero(shape, dtype):
    from suetes_b200.steppers import VerticalPreconditioner
    st, _, _ = mountain_wave(*shape, dtype=dtype, flat=True)
    ph, sol = st.physics, st.implicit_solver
    bg = ph.precompute_bg(ph.bg_state_ref())
    core = sol._core(dtype, bg)
    pre = VerticalPreconditioner(ph, st.dt, alpha=st.alpha)
    pre.precompute_banded(bg)
    x = to_cuda(random_fields(shapes5(*shape), 3, SCALES), dtype)
    core.set_tuning(precond_tile=4, precond_t_tile=4)
    default = [pre(x), pre.transpose(x)]
    core.set_tuning()
    for got, want in zip(default, [pre(x), pre.transpose(x)]):
        for k in got:
            assert torch.isfinite(want[k]).all() and torch.equal(got[k], want[k]), k
