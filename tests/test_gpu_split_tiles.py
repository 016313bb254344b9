"""One step of the split-explicit core against the float64 oracle at the sizes
where the tiled slow-forcing kernels can go wrong: grids shorter than the
upwind stencil and the Laplacian's rim (indices clamp or wrap onto one cell
several times, on every choice of periodic axes), tiles of 32 x 8 columns with
one column over, level counts around the chunks of 8 and 16 a block walks, and
a grid large enough for the longer chunk.

Bound: float64 rounding 1.1e-16 over a few thousand dependent operations of a
step; 1e-10 leaves two decades for the cancellation in w and eta_dot.
"""

import pytest
import torch

from _cases import rel_l2, to_cuda
from test_gpu_split_vjp_gather import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,periodic", [
    ((2, 2, 2), ()), ((2, 3, 3), (0, 1)), ((3, 2, 4), (0,)), ((5, 4, 8), (1,)), ((33, 9, 9), (0, 1)),
    ((32, 8, 16), ()), ((31, 17, 17), (0,)), ((65, 7, 33), (1,)), ((298, 235, 17), ())])
def test_step_is_the_oracles(shape, periodic):
    ost, pst, s0 = _case(shape, periodic)
    ref = ost.step(dict(s0), 0.0, None, lambda s, f: s)
    out = pst.step(to_cuda(s0), 0.0, None, lambda s, f: s)
    errs = {k: rel_l2(out[k], ref[k]) for k in ("u", "v", "w", "eta_dot", "pi", "th_v", "rho")}
    assert max(errs.values()) < 1e-10, errs


# past the shared memory of a tile of 32 columns (133 levels in float64), of 16 (266), and into the march
@pytest.mark.parametrize("nz", [133, 134, 266, 267])
def test_column_solve_at_many_levels(nz):
    test_step_is_the_oracles((17, 2, nz), ())
