"""The gathered transposes of the split-explicit core (acoustic sub-step and
upwind advection) against the float64 oracle's autograd, at the sizes where
they can go wrong: grids shorter than the four-point upwind stencil, whose
positions clamp or wrap onto one cell several times, on every choice of
periodic axes; level counts around the chunks a thread walks (4) and the
column tiles' last column (32 of them); the levels past which the column
solve marches instead of holding its tile in shared memory.

Bound: the sweep is linear, a few hundred operations deep, and sums in
float64 with one rounding per element, so float64 agrees with the autograd to
some thousand times 1.1e-16 of the largest cotangent; 1e-10 leaves three
decades.
"""

import pytest
import torch

from _cases import C, build, mountain, random_fields, rel_l2, shapes5
from test_gpu_split import DX, KW
from test_gpu_split_vjp import IN, NATIVE, _cotangents, _native_vjp, _oracle_vjp

pytestmark = pytest.mark.gpu


def _case(shape, periodic, ns=3, dt=2.0):
    from oracle.split_explicit import SplitExplicitStepper3D as OSp
    from suetes_b200 import SplitExplicitStepper3D as PSp
    h = mountain if shape[2] > 4 else None
    dz = min(500.0, 10000.0 / shape[2])
    o = build("oracle", *shape, DX, DX, dz, h=h, periodic=periodic, dt=dt, **KW)
    p = build("cuda", *shape, DX, DX, dz, h=h, periodic=periodic, device="cuda", dt=dt, **KW)
    ost, pst = OSp(o[2], dt, ns, alpha=0.5), PSp(p[2], dt, ns, alpha=0.5)
    s0 = random_fields(shapes5(*shape), 5, {"u": 4.0, "v": 4.0, "w": 0.1, "pi": 1e-4, "eta_dot": 0.0})
    s0["u"] += 1.0
    s0["pi"] += o[2].pi_bg
    s0["th_v"] = o[2].theta_bg + random_fields({"m": shape}, 6, {"m": 1.0})["m"]
    s0["rho"] = C["p0"] / (C["Rd"] * s0["th_v"]) * s0["pi"] ** (C["cvd"] / C["Rd"])
    s0["eta_dot"], s0["w"] = ost._diagnose_eta_dot(s0)
    return ost, pst, s0


@pytest.mark.parametrize("shape,periodic", [
    ((2, 2, 2), ()), ((2, 3, 3), (0, 1)), ((3, 2, 4), (0,)), ((4, 5, 5), (1,)), ((5, 4, 9), (0, 1)),
    ((31, 3, 8), ()), ((32, 2, 5), (1,)), ((33, 9, 7), (0,)), ((3, 3, 201), ())])
def test_gathered_sweep_is_the_oracles(shape, periodic):
    ost, pst, s0 = _case(shape, periodic)
    cot = _cotangents(s0, 11)
    ref = _oracle_vjp(ost, s0, cot)
    got = _native_vjp(pst, s0, cot, torch.float64)
    again = _native_vjp(pst, s0, cot, torch.float64)
    errs = {k: rel_l2(got[NATIVE[k]], ref[k]) for k in IN}
    assert max(errs.values()) < 1e-10, errs
    assert all(torch.equal(got[NATIVE[k]], again[NATIVE[k]]) for k in IN)
