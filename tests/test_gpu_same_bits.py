"""One rule for every solve: the same step gives the same bits whether its
solves are recorded or not, alone or grouped with members of any time step."""

import pytest
import torch

from suetes_b200.workloads import rising_bubble

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "eta_dot", "pi_p", "th_p", "rho")


def _member(n, dtype, dt, method, tol):
    st, state, bc = rising_bubble(*n, dx=50.0, radius=200.0, center=(0.0, 0.0, 200.0), dtype=dtype, dt=dt,
                                  solver_tol=tol, solver_restart=30, solver_maxiter=30, solve_method=method)
    return st, st.to_device_state(state), bc


@pytest.mark.parametrize("method", ["batched", "incremental"])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-7), (torch.float64, 1e-10)])
@pytest.mark.parametrize("dt", [0.1, 0.25, 1.0, 3.0])
def test_recorded_step_is_the_plain_step(dt, dtype, tol, method):
    from suetes_b200 import DeviceState, StepGraph
    from suetes_b200.adjoint import _taped_step
    st, ds, _ = _member((17, 14, 11), dtype, dt, method, tol)
    plain = DeviceState(ds.core)
    st.step_device(ds, plain)
    taped, rec = _taped_step(st, ds, None)
    flat = [t for solve in rec for t in solve]
    out = DeviceState(ds.core)
    graph = StepGraph([(st, ds, out, None)], tapes=[[torch.empty_strided(t.shape, t.stride(), dtype=t.dtype, device=t.device) for t in flat]])
    graph.launch()
    for k in FIELDS:
        assert torch.equal(taped.t[k], plain.t[k]), k
        assert torch.equal(out.t[k], plain.t[k]), k


@pytest.mark.parametrize("dtype,tol,method", [(torch.float32, 1e-7, "batched"), (torch.float32, 1e-7, "incremental"),
                                              (torch.float64, 1e-10, "batched")])
def test_grouped_members_of_unequal_steps(dtype, tol, method):
    """Acoustic radius 1.1, 11 and 27 in one grouped graph: each member's own eager bits and statistics."""
    from suetes_b200 import DeviceState, StepGraph
    members, refs, infos = [], [], []
    for n, dt in (((16, 12, 10), 0.1), ((20, 14, 12), 1.0), ((12, 18, 9), 2.5)):
        st, ds, _ = _member(n, dtype, dt, method, tol)
        ref = DeviceState(ds.core)
        infos.append(st.step_device(ds, ref))
        refs.append(ref)
        members.append((st, ds, DeviceState(ds.core), None))
    graph = StepGraph(members, grouped=True)
    graph.launch()
    for m, ref in enumerate(refs):
        for k in FIELDS:
            assert torch.equal(members[m][2].t[k], ref.t[k]), (m, k)
        got = graph.info(m)["solves"]
        for q in range(2):
            for key in ("cycles", "arnoldi_steps", "converged", "residual_norm"):
                assert got[q][key] == infos[m]["solves"][q][key], (m, q, key)
