"""The autotuner stays inside the workspace of a solve, down to a restart of
one (two basis vectors), and leaves the core's results as they were."""

import ctypes

import pytest
import torch

from suetes_b200 import _lib
from suetes_b200.workloads import rising_bubble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("restart", [1, 2, 30])
def test_autotune_stays_in_its_workspace(restart, dtype):
    st, state, _ = rising_bubble(17, 14, 11, dtype=dtype, device="cuda", solver_tol=1e-6, solver_restart=restart,
                                 solver_maxiter=40)
    core = st.core(dtype)
    n = int(core.lib.sisl_workspace_bytes(core.handle, _lib.WS_GMRES))
    past = 8 * 6 * 18 * 15 * 12 * 2  # two vectors and their padding
    buf = torch.full((n + past,), 0x5A, dtype=torch.uint8, device="cuda")
    t = _lib.SislTuning()
    _lib.check(core.lib.sisl_autotune(core.handle, buf.data_ptr(), n, core.stream, ctypes.byref(t)), "sisl_autotune")
    torch.cuda.synchronize()
    assert bool((buf[n:] == 0x5A).all())
    ds = st.to_device_state(state)
    tuned = type(ds)(core)
    st.step_device(ds, tuned)
    core.set_tuning()
    plain = type(ds)(core)
    st.step_device(ds, plain)
    for k in ("u", "v", "w", "eta_dot", "pi_p", "th_p"):
        assert torch.equal(tuned.t[k], plain.t[k]), k
