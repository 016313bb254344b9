"""The shared-memory flux-form sweep against the oracle where its tiles end:
lines shorter and longer than a warp, counts that are no multiple of a block's
32 lines or eight segments, and lines past the shared-memory bound (the
one-thread form), on open and periodic axes."""

import pytest
import torch

from _cases import build, random_fields, rel_l2, shapes5, to_cuda

pytestmark = pytest.mark.gpu

DT = 20.0


# float64: sums of N terms in another order, N 2^-53 on values of order one
# against results of order one: 1e-13 at 870.  float32: one rounding per sweep
# and two in the mass, 2^-24 each in the 2-norm: 3.6e-7.
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 1e-6)])
@pytest.mark.parametrize("periodic", [(), (0, 1)])
@pytest.mark.parametrize("shape", [(2, 3, 2), (7, 5, 9), (33, 31, 8), (64, 33, 40), (870, 3, 2), (3, 870, 2)])
def test_transport_matches_oracle(shape, periodic, dtype, tol):
    from oracle.steppers import FluxFormAdvector as Oracle
    from suetes_b200 import FluxFormAdvector
    nx, ny, nz = shape
    og, _, oph = build("oracle", *shape, 1000.0, 1000.0, 400.0, periodic=periodic, dt=DT)
    pg, _, pph = build("cuda", *shape, 1000.0, 1000.0, 400.0, periodic=periodic, device="cuda", dt=DT)
    # Courant numbers up to 2.4 along x and y, 0.8 along z
    st = random_fields(shapes5(*shape), 5, {"u": 120.0, "v": 120.0, "w": 1.0, "pi": 1e-3, "eta_dot": 0.04})
    st["eta_dot"][:, :, 0] = 0.0
    st["eta_dot"][:, :, -1] = 0.0
    gen = torch.Generator().manual_seed(6)
    rho = 0.5 + torch.rand(shape, generator=gen, dtype=torch.float64)
    st = {k: v.to(dtype).double() for k, v in st.items()}
    rho = rho.to(dtype).double()
    obg, pbg = (ph.precompute_bg(ph.bg_state_ref()) for ph in (oph, pph))
    ref = Oracle(og, DT, periodic_axes=periodic).advect_3d_split(rho, st, obg)
    out = FluxFormAdvector(pg, DT, periodic_axes=periodic, physics=pph).advect_3d_split(
        rho.to("cuda", dtype), to_cuda(st, dtype), pbg)
    assert out.shape == ref.shape
    assert rel_l2(out, ref) < tol, rel_l2(out, ref)
