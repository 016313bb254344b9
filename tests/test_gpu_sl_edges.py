"""Semi-Lagrangian gathers where their row addresses can go wrong: fields of
one to five columns along x (the shared address of a row needs four), points
on, between and past the edges, level counts around the four a thread forms
velocities for.

Bounds: the 64 weights of a point sum to at most 1.25^3 = 2 in magnitude, so
rounding is 64 * 2 * eps of the largest value, 1.5e-14 and 8e-6; the relative
norm over many points stays a decade below: 2e-14 and 2e-6 with the inputs
rounded to the field's type first.  Departure points: two gathers of eight
terms, displacements of up to 1.5 cells: 1e-13 and 2e-6 of a cell."""

import pytest
import torch

from _cases import build, max_abs, random_fields, rel_l2, shapes5, to_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limiter", [False, True])
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 2e-14), (torch.float32, 2e-6)])
@pytest.mark.parametrize("ex", [1, 2, 3, 4, 5, 33])
def test_tricubic_on_short_rows(ex, dtype, tol, limiter):
    from oracle.ops import tensor_product_interp_3d as ref_interp
    from suetes_b200 import tensor_product_interp_3d
    gen = torch.Generator().manual_seed(ex)
    f = torch.randn(ex, 4, 3, generator=gen, dtype=torch.float64).to(dtype).double()
    at = torch.tensor([-3.0, -0.25, 0.0, 0.5, 1.0, ex - 2.5, ex - 1.0, ex - 0.75, ex + 2.0], dtype=torch.float64)
    grid = torch.meshgrid(at, torch.tensor([-1.0, 0.0, 1.5, 2.75, 3.0, 5.0], dtype=torch.float64),
                          torch.tensor([-0.5, 0.25, 1.0, 2.0, 2.5], dtype=torch.float64), indexing="ij")
    coords = torch.stack(grid).to(dtype).double()
    ref = ref_interp(f, coords, use_limiter=limiter)
    out = tensor_product_interp_3d(f.to("cuda", dtype), coords.to("cuda", dtype), use_limiter=limiter)
    assert rel_l2(out, ref) < tol, rel_l2(out, ref)


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 2e-6)])
@pytest.mark.parametrize("shape", [(2, 3, 2), (3, 2, 3), (5, 4, 4), (33, 3, 5), (6, 5, 8)])
def test_departure_points_on_small_grids(shape, dtype, tol):
    from oracle.steppers import SemiLagrangianAdvector3D as OA
    from suetes_b200 import SemiLagrangianAdvector3D as PA
    o = build("oracle", *shape, 1000.0, 1000.0, 500.0, dt=100.0)
    p = build("cuda", *shape, 1000.0, 1000.0, 500.0, device="cuda", dt=100.0)
    s = random_fields({k: v for k, v in shapes5(*shape).items() if k in ("u", "v", "eta_dot")}, 3,
                      {"u": 15.0, "v": 15.0, "eta_dot": 0.01})
    s = {k: v.to(dtype).double() for k, v in s.items()}
    for loc in ("m", "u", "v", "w"):
        ref = OA(o[0], o[2], 100.0).compute_departure_indices(s, loc=loc)
        out = PA(p[0], p[2], 100.0).compute_departure_indices(to_cuda(s, dtype), loc=loc)
        bound = tol * (1.0 if dtype == torch.float64 else max(8.0, float(max(shape))))  # a coordinate's own rounding
        assert max_abs(out, ref) < bound, (loc, max_abs(out, ref))


# A diverged wind: the midpoints lie past the largest integer (or are not
# numbers) and the gathers take the nearest edge.  Uniform winds interpolate
# to themselves, so the points are known: index minus displacement, with the
# rounding of four float products.
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 2e-6)])
@pytest.mark.parametrize("wind", [1e12, -1e12, 3e30, -3e30, float("inf"), float("-inf"), float("nan")])
def test_departure_points_of_a_diverged_wind(wind, dtype, tol):
    from suetes_b200 import SemiLagrangianAdvector3D as PA
    shape = (8, 5, 4)
    p = build("cuda", *shape, 1000.0, 1000.0, 500.0, device="cuda", dt=100.0)
    adv = PA(p[0], p[2], 100.0)
    for axis in ("u", "v", "eta_dot"):
        s = {k: torch.zeros(v, dtype=dtype, device="cuda") for k, v in shapes5(*shape).items()
             if k in ("u", "v", "eta_dot")}
        s[axis] += wind
        for loc in ("m", "u", "v", "w"):
            out = adv.compute_departure_indices(s, loc=loc)
            if abs(wind) < float("inf"):
                assert torch.isfinite(out).all()
                if axis != "eta_dot":  # dt wind m / dx, the map factor 1 to 1e-6 on this grid
                    along = out[0 if axis == "u" else 1].double() / (-0.1 * wind)
                    assert float((along - 1.0).abs().max()) < tol + 1e-5
            else:
                assert not torch.isfinite(out).all()
