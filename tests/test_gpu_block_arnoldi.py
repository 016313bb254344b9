"""The block Arnoldi cycle of the CUDA GMRES (several operator applications
per orthogonalisation) against the oracle's one-step Arnoldi, at the sizes
where its blocks and row tiles end: restarts below, at and past a multiple of
the block width and of the 8-row tiles, grids of a few blocks and of fewer
elements than one, Krylov spaces smaller than a cycle.
"""

import pytest
import torch

from _cases import build, mountain, random_fields, rel_l2, shapes5, to_cuda

pytestmark = pytest.mark.gpu

SCALES = {"u": 1.0, "v": 1.0, "w": 0.5, "pi": 1e-3, "eta_dot": 1e-3}


def _pair(shape, dt, restart, maxiter, method, tol):
    from oracle.steppers import SemiImplicitSolver3D as Oracle
    from suetes_b200 import SemiImplicitSolver3D
    h = mountain if shape[2] > 4 else None  # two levels leave no room for the mountain
    o = build("oracle", *shape, 2000.0, 2000.0, 500.0, h=h, dt=dt)
    p = build("cuda", *shape, 2000.0, 2000.0, 500.0, h=h, device="cuda", dt=dt)
    rhs = random_fields(shapes5(*shape), 7, SCALES)
    for k in ("w", "eta_dot"):
        rhs[k][:, :, 0] = 0.0
        rhs[k][:, :, -1] = 0.0
    kw = dict(solver_tol=tol, solver_maxiter=maxiter, solver_restart=restart, solve_method=method)
    return o[2], p[2], Oracle(o[2], dt, **kw), SemiImplicitSolver3D(p[2], dt, **kw), rhs


def _bg(ph):
    return ph.precompute_bg(ph.bg_state_ref())


# One cycle is the minimiser over a Krylov space that both forms span: their
# float64 iterates differ by the rounding of the basis, 2.2e-16 times the
# square root of the reduction length (under 1e3) times the conditioning of a
# block's vectors (at most 1 / sqrt(5e-4) = 45 at six columns): 1e-11.  The
# bound below leaves two decades for the least-squares problem's own
# conditioning.
@pytest.mark.parametrize("method", ["batched", "incremental"])
@pytest.mark.parametrize("restart", [1, 2, 3, 5, 6, 7, 8, 13, 30, 31])
def test_one_cycle_is_the_oracles(restart, method):
    oph, pph, osol, psol, rhs = _pair((11, 9, 7), 20.0, restart, 1, method, 1e-14)
    ref = osol.solve(rhs, _bg(oph))
    out = psol.solve(to_cuda(rhs), _bg(pph))
    assert psol.last_info["arnoldi_steps"] == osol.last_stats["forward"]["arnoldi_steps"]
    for k in ref:
        assert rel_l2(out[k], ref[k]) < 1e-9, (k, rel_l2(out[k], ref[k]))


# past the widest row-tile steps (100, 128 rows), and a grid shorter than the
# launch's blocks; two cycles, the second restarting from the first
@pytest.mark.parametrize("shape,restart", [((40, 36, 20), 12), ((9, 8, 6), 64), ((9, 8, 6), 100), ((9, 8, 6), 128)])
def test_two_cycles_are_the_oracles(shape, restart):
    oph, pph, osol, psol, rhs = _pair(shape, 60.0, restart, 2, "batched", 1e-13)
    ref = osol.solve(rhs, _bg(oph))
    out = psol.solve(to_cuda(rhs), _bg(pph))
    assert psol.last_info["cycles"] == osol.last_stats["forward"]["cycles"]
    for k in ref:
        assert rel_l2(out[k], ref[k]) < 1e-8, (k, rel_l2(out[k], ref[k]))


# 2x2x2 cells: the Krylov space is exhausted inside a cycle, in the middle of
# a block; the cycle ends there and the solve still converges
@pytest.mark.parametrize("method", ["batched", "incremental"])
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-11), (torch.float32, 1e-6)])
def test_exhausted_space_ends_the_block(method, dtype, tol):
    oph, pph, osol, psol, rhs = _pair((2, 2, 2), 60.0, 60, 20, method, tol)
    bg = _bg(pph)
    b = to_cuda(rhs, dtype)
    out = psol.solve(b, bg)
    assert psol.last_info["converged"], psol.last_info
    assert all(torch.isfinite(v).all() for v in out.values())
    # the stopping test bounds ||M r|| by tol ||b||; the true residual is ||M^-1|| times that, M^-1 of the
    # columns bounded by 1 + radius^2 (radius 16.6 here)
    assert float(psol.relative_residual(out, b, bg)) < 300.0 * tol


def test_zero_right_hand_side():
    _, pph, _, psol, rhs = _pair((9, 8, 6), 60.0, 30, 5, "batched", 1e-8)
    out = psol.solve({k: torch.zeros_like(v, device="cuda") for k, v in rhs.items()}, _bg(pph))
    assert psol.last_info["converged"]
    assert all(float(v.abs().max()) == 0.0 for v in out.values())


# acoustic radius 1.1 (one column per block) and 4.4 (six): both follow the oracle's cycles
@pytest.mark.parametrize("dt", [4.0, 16.0])
def test_either_side_of_the_block_rule(dt):
    oph, pph, osol, psol, rhs = _pair((16, 12, 8), dt, 20, 6, "batched", 1e-10)
    ref = osol.solve(rhs, _bg(oph))
    out = psol.solve(to_cuda(rhs), _bg(pph))
    assert psol.last_info["cycles"] == osol.last_stats["forward"]["cycles"]
    for k in ref:
        assert rel_l2(out[k], ref[k]) < 1e-8, (k, rel_l2(out[k], ref[k]))
