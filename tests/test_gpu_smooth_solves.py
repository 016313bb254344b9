"""Solves of smooth right-hand sides: one or two cosine modes excite only the
slow end of the operator's spectrum, and short Krylov spaces nearly hold the
solution.  The reference is the one-column Arnoldi process in plain torch on
the package's own operator and preconditioner, in the solve's precision
(smooth float32 vectors carry rounding noise that the operator amplifies, so
the float64 oracle's minimum is out of reach for any float32 form)."""

import math

import pytest
import torch

from _cases import build, mountain, random_fields, rel_l2, shapes5, to_cuda

pytestmark = pytest.mark.gpu

SHAPE, SPACING = (24, 20, 8), (500.0, 500.0, 1000.0)
KEYS = ("u", "v", "w", "pi", "eta_dot")
# Two forms of a cycle span the same space up to the rounding of their vectors, and the minimum is flat to second
# order; past 30 steps of a smooth float32 right-hand side the spaces hold noise, and the minima differ by a few per
# cent.  The floor, against ||M b||: eps times sqrt(30) steps of ||M A|| about 1 to 17.
RATIO = 1.05
FLOOR = {torch.float32: 1e-5, torch.float64: 1e-13}


def cosine(shape, waves):
    f = torch.ones((), dtype=torch.float64)
    for axis, (n, m) in enumerate(zip(shape, waves)):
        at = [1] * 3
        at[axis] = n
        f = f * torch.cos(math.pi * m * (torch.arange(n, dtype=torch.float64) + 0.5) / n).reshape(at)
    return f


def smooth_rhs(waves, shape=SHAPE):
    rhs = {k: torch.zeros(s, dtype=torch.float64) for k, s in shapes5(*shape).items()}
    rhs["pi"] = 1e-3 * cosine(shape, waves)
    return rhs


class Problem:
    """The package's solver from a zero guess, and the reference cycle on the same operator."""

    def __init__(self, dt, method, restart=30, maxiter=1, tol=1e-14, h=None, shape=SHAPE, transpose=False,
                 periodic=()):
        from suetes_b200 import SemiImplicitSolver3D
        from suetes_b200.steppers import VerticalPreconditioner
        p = build("cuda", *shape, *SPACING, h=h, periodic=periodic, device="cuda", dt=dt)
        self.bg = p[2].precompute_bg(p[2].bg_state_ref())
        self.shapes = shapes5(*shape)
        self.solver = SemiImplicitSolver3D(p[2], dt, solver_tol=tol, solver_maxiter=maxiter, solver_restart=restart,
                                           solve_method=method)
        self.transpose = transpose
        self.solver.adjoint_normalize = False  # residuals in the units of the right-hand side
        self.pre = VerticalPreconditioner(p[2], dt)
        self.pre.precompute_banded(self.bg)

    def solve(self, rhs, dtype):
        b = to_cuda(rhs, dtype)
        if self.transpose:
            return self.solver.solve_transpose(b, self.bg), self.solver.last_transpose_info
        out = self.solver.solve(b, self.bg, x0={k: torch.zeros_like(v) for k, v in b.items()})
        return out, self.solver.last_info

    def _flat(self, d):
        return torch.cat([d[k].reshape(-1) for k in KEYS])

    def _fields(self, x):
        parts = torch.split(x, [math.prod(self.shapes[k]) for k in KEYS])
        return {k: t.reshape(self.shapes[k]) for k, t in zip(KEYS, parts)}

    def _A(self, x):
        return self._flat(self.solver.matvec_scaled(self._fields(x), self.bg, transpose=self.transpose))

    def _M(self, x):
        f = self._fields(x)
        return self._flat(self.pre.transpose(f) if self.transpose else self.pre(f))

    def reference(self, rhs, dtype, steps):
        """(||M b||, ||M (b - A x)|| after a cycle of ``steps`` from zero), residuals formed in float64."""
        scale = 1e-3 if self.transpose else 1e3  # of pi, the only field the right-hand sides here have
        b = self._flat({k: v * (scale if k == "pi" else 1.0) for k, v in to_cuda(rhs).items()})
        v = self._M(b.to(dtype)).double()
        first = float(v.norm())
        H = torch.zeros(steps + 1, steps, dtype=torch.float64)
        V = [(v / first).to(dtype)]
        for j in range(steps):
            w = self._M(self._A(V[j]))
            for i in range(j + 1):  # projections of one vector, as classical Gram-Schmidt has them
                H[i, j] = torch.dot(V[i].double(), w.double()).cpu()
            for i in range(j + 1):
                w = w - H[i, j].to("cuda", dtype) * V[i]
            H[j + 1, j] = w.double().norm().cpu()
            V.append((w.double() / H[j + 1, j].cuda()).to(dtype))
        e = torch.zeros(steps + 1, 1, dtype=torch.float64)
        e[0] = first
        y = torch.linalg.lstsq(H, e).solution[:, 0].cuda()
        x = sum(y[j] * V[j].double() for j in range(steps))
        return first, float(self._M((b - self._A(x)).to(dtype)).double().norm())


# A cycle takes all its steps, and reaches what they can, whatever spectrum the right-hand side excites
@pytest.mark.parametrize("method", ["batched", "incremental"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("restart", [30, 17])
@pytest.mark.parametrize("dt", [1.0, 3.2, 8.0, 16.0])
@pytest.mark.parametrize("waves", [(0, 1, 1), (1, 1, 1), (2, 1, 0)])
def test_cycle_takes_all_its_steps(waves, dt, restart, dtype, method):
    p = Problem(dt, method, restart)
    rhs = smooth_rhs(waves)
    _, info = p.solve(rhs, dtype)
    first, least = p.reference(rhs, dtype, info["arnoldi_steps"])
    # an incremental cycle leaves when its estimate meets the tolerance (float64 at the smallest step) or nothing above
    # the rounding of its vectors is left to orthogonalise (float32 there: the residual is at 4 eps of the first)
    spent = info["converged"] or info["residual_norm"] <= 4 * torch.finfo(dtype).eps * first
    assert info["cycles"] == 1 and (info["arnoldi_steps"] == restart or spent), (info, first)
    assert info["residual_norm"] <= RATIO * least + FLOOR[dtype] * first, (info, least, first)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dt", [3.2, 8.0])
def test_transposed_cycle_takes_all_its_steps(dt, dtype):
    p = Problem(dt, "batched", 30, h=mountain, transpose=True)
    rhs = smooth_rhs((1, 1, 1))
    _, info = p.solve(rhs, dtype)
    assert info["cycles"] == 1 and info["arnoldi_steps"] == 30, info
    first, least = p.reference(rhs, dtype, 30)
    assert info["residual_norm"] <= RATIO * least + FLOOR[dtype] * first, (info, least, first)


# The blocks of a smooth right-hand side keep their columns: the cycle is not done over one column at a time, which
# would add four launches for each of its 30 steps to the 60 operator and preconditioner launches, at most 14 block
# launches and about 20 others of a solve.
@pytest.mark.parametrize("method", ["batched", "incremental"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dt", [0.2, 1.0, 3.2, 8.0, 16.0])
@pytest.mark.parametrize("waves", [(0, 1, 1), (1, 1, 1), (2, 1, 0)])
def test_smooth_blocks_keep_their_columns(waves, dt, dtype, method):
    from suetes_b200.core import kernel_launches
    p = Problem(dt, method, 30)
    rhs = smooth_rhs(waves)
    p.solve(rhs, dtype)
    before = kernel_launches()
    p.solve(rhs, dtype)
    assert kernel_launches() - before < 60 + 14 + 40


# Periodic axes, whose duplicate faces are unknowns of their own: a right-hand side that differs there too.  One
# float64 cycle of 13 against the oracle's; the bound is that of the one-cycle tests of test_gpu_block_arnoldi.
@pytest.mark.parametrize("periodic", [(0,), (1,), (0, 1)])
def test_periodic_cycle_is_the_oracles(periodic):
    from oracle.steppers import SemiImplicitSolver3D as Oracle
    from suetes_b200 import SemiImplicitSolver3D
    shape, dt = (11, 9, 7), 8.0
    rhs = random_fields(shapes5(*shape), 7, {"u": 1.0, "v": 1.0, "w": 0.5, "pi": 1e-3, "eta_dot": 1e-3})
    kw = dict(solver_tol=1e-14, solver_maxiter=1, solver_restart=13)
    o = build("oracle", *shape, *SPACING, h=mountain, periodic=periodic, dt=dt)[2]
    p = build("cuda", *shape, *SPACING, h=mountain, periodic=periodic, device="cuda", dt=dt)[2]
    ref = Oracle(o, dt, **kw).solve(rhs, o.precompute_bg(o.bg_state_ref()))
    out = SemiImplicitSolver3D(p, dt, **kw).solve(to_cuda(rhs), p.precompute_bg(p.bg_state_ref()))
    for k in ref:
        assert rel_l2(out[k], ref[k]) < 1e-9, (k, rel_l2(out[k], ref[k]))


@pytest.mark.parametrize("periodic", [(0,), (1,), (0, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_periodic_transposed_cycle(periodic, dtype):
    p = Problem(8.0, "batched", 13, h=mountain, transpose=True, periodic=periodic)
    rhs = random_fields(p.shapes, 7, {"u": 1.0, "v": 1.0, "w": 0.5, "pi": 1e3, "eta_dot": 0.0})
    _, info = p.solve(rhs, dtype)
    first, least = p.reference(rhs, dtype, 13)
    assert info["residual_norm"] <= RATIO * least + FLOOR[dtype] * first, (info, least, first)


# A cycle that is cut short is still the least residual of the steps it took
@pytest.mark.parametrize("dt,waves", [(8.0, (0, 1, 1)), (8.0, (1, 1, 1)), (3.2, (1, 1, 1)), (12.0, (2, 1, 0))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_cycle_is_the_least_residual_of_its_steps(dt, waves, dtype):
    p = Problem(dt, "batched")
    rhs = smooth_rhs(waves)
    _, info = p.solve(rhs, dtype)
    first, least = p.reference(rhs, dtype, info["arnoldi_steps"])
    assert info["residual_norm"] <= RATIO * least + FLOOR[dtype] * first, (info, least, first)


# Spaces that end inside a block: a right-hand side the coupling does not see
# (constant pi', one level of w), and grids of a few cells.  The solve
# converges as the one-column form does: within two cycles to the rounding.
@pytest.mark.parametrize("method", ["batched", "incremental"])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-6), (torch.float64, 1e-11)])
@pytest.mark.parametrize("what", ["pi", "w", "cells"])
def test_space_that_ends_inside_a_block(what, dtype, tol, method):
    shape = (3, 3, 3) if what == "cells" else SHAPE
    p = Problem(8.0, method, 100 if what == "cells" else 30, maxiter=2, tol=tol, shape=shape)
    rhs = smooth_rhs((1, 1, 1) if what == "cells" else (0, 0, 0), shape)
    if what == "w":
        rhs["w"][:, :, 3] = 1.0
        rhs["pi"].zero_()
    out, info = p.solve(rhs, dtype)
    assert info["converged"], info
    assert all(torch.isfinite(v).all() for v in out.values())


@pytest.mark.parametrize("dtype,tol,method", [(torch.float32, 1e-7, "batched"), (torch.float32, 1e-7, "incremental"),
                                              (torch.float64, 1e-11, "incremental")])
def test_shortened_blocks_in_graphs(dtype, tol, method):
    """A member whose Krylov space ends inside a block beside one whose does not: eager steps, branch graphs and
    grouped graphs give the same bits and statistics."""
    from suetes_b200 import DeviceState, PingPong
    from suetes_b200.workloads import rising_bubble
    members = []
    for n in ((3, 3, 3), (18, 12, 10)):
        st, state, _ = rising_bubble(*n, radius=150.0, center=(0.0, 0.0, 100.0), dtype=dtype, device="cuda",
                                     solver_tol=tol, solver_restart=100, solve_method=method, solver_maxiter=4)
        members.append((st, st.to_device_state(state, dtype), None))
    branch, grouped = PingPong(members), PingPong(members, grouped=True)
    for g in (branch, grouped):
        g.step()
        g.step()
    for m, (st, ds, _) in enumerate(members):
        a, b = ds, DeviceState(ds.core)
        for _ in range(branch.steps_done + 2):
            st.step_device(a, b)
            a, b = b, DeviceState(ds.core)
        for k in ("u", "v", "w", "eta_dot", "pi_p", "th_p", "rho"):
            assert torch.isfinite(a.t[k]).all()
            assert torch.equal(branch.current()[m].t[k], a.t[k]), (m, k)
            assert torch.equal(grouped.current()[m].t[k], a.t[k]), (m, k)
        assert branch.info(m)["solves"] == grouped.info(m)["solves"]
