"""Bounded waits of the TMA-staged y-sweep that run out in the device-clocked loop.

As in test_tma_timeout.py the limit is set to 1 ns, so CTAs give up on boxes still
in flight and the call reports MHD_ERR_TIMEOUT.  The clock's status then changes
while the sweep runs; what the clock says afterwards has to be the step's own
dt and c_h (or no step at all, if CTA 0 came late enough to skip it), because the
workspace carries c_h on as the floor of every later CFL maximum."""
import pytest

import numpy as np

from mhd_gpu_acc_b200 import (
    F32,
    F64,
    GpuWorkspace,
    Grid2DGPU,
    compute_dt_gpu,
    get_n_case_config,
    init_gpu_workspace,
    initialise,
    set_gpu_physics_ch,
    set_gpu_physics_gamma,
)

pytestmark = pytest.mark.gpu
TIMEOUT = -8  # MHD_ERR_TIMEOUT


def _workspace(U, cfg):
    ws = GpuWorkspace()
    init_gpu_workspace(ws, U)
    set_gpu_physics_gamma(ws, cfg.gamma)
    set_gpu_physics_ch(ws, 0.0)
    ws.set_limiter(1)
    ws.set_sweep_shape(8, 0, 1)
    return ws


@pytest.mark.parametrize("dtype", [F64, F32])
def test_a_timed_out_step_leaves_a_defined_clock(dtype):
    n, t_end = 2048, 1.0
    cfg = get_n_case_config(4, 1)
    U0 = initialise(4, n, n, 2, cfg.extent)
    U, T = (Grid2DGPU(n, n, 2, *cfg.extent, dtype) for _ in range(2))
    bc = (0, 0, 0, 0)
    U.upload(U0)
    ws = _workspace(U, cfg)
    want = ws.run(U, T, cfg.cfl, t_end, 1, 2, bc)
    after = U.download()
    ws.destroy()

    U.upload(U0)
    ws = _workspace(U, cfg)
    dt = compute_dt_gpu(U, ws, cfg.cfl)  # sets c_h
    assert (dt, ws.ch) == (want.last_dt, want.ch)
    ws.set_tma_wait_limit(1)
    # step 1 times out, later ones are skipped
    info = ws.run(U, T, cfg.cfl, t_end, 4, 2, bc, raise_on_stop=False)
    assert info.status == TIMEOUT
    assert info.steps in (0, 1)
    assert info.ch == ws.ch == want.ch
    if info.steps:
        assert (info.t, info.last_dt) == (dt, dt)
    else:
        assert (info.t, info.last_dt) == (0.0, 0.0)

    # the workspace goes on as if the step had not been tried
    ws.set_tma_wait_limit(0)
    U.upload(U0)
    info = ws.run(U, T, cfg.cfl, t_end, 1, 2, bc)
    assert (info.steps, info.t, info.last_dt, info.ch) == (1, want.t, want.last_dt, want.ch)
    np.testing.assert_array_equal(U.download(), after)
    ws.destroy()
