"""Batch work lists with more ghost layers, and in FP32: every instance equals the
same problem advanced alone (FP64, bit for bit), and no launch shape, the lengths by
the size of the batch among them, changes a bit of any instance."""
import ctypes as C

import numpy as np
import pytest

from mhd_gpu_acc_b200 import F32, F64, GpuWorkspace, Grid2DGPU, init_gpu_workspace, load, set_gpu_physics_gamma
from mhd_gpu_acc_b200.batch import SQRT_4PI, Batch, instance

# the smallest grids, widths about a 28-cell segment and a 32-column strip, long and wide ones
SIZES = [(4, 4), (5, 33), (27, 9), (28, 8), (29, 7), (30, 64), (62, 63), (300, 301), (4, 300), (517, 61)]
BCS = [(0, 0, 0, 0), (1, 1, 2, 2), (2, 2, 0, 0)]


def _states(dtype, ng, tuning):
    descs = [instance(nx, ny, 5 / 3, 0.3, 5.0, bc=BCS[k % 3], ng=ng) for k, (nx, ny) in enumerate(SIZES)]
    batch = Batch(descs, dtype=dtype)
    if tuning:
        batch.set_tuning(*tuning)
    for i, d in enumerate(descs):
        batch.init_orszag_tang(i, 0.9 / SQRT_4PI, d.gamma)
    infos = batch.run(5)
    out = [batch.download(i) for i in range(len(descs))], [(i.steps, i.t, i.ch) for i in infos], descs
    batch.destroy()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("ng", [2, 3, 4])
def test_no_launch_shape_changes_a_bit(dtype, ng):
    states, infos, descs = _states(dtype, ng, None)
    for tuning in [(8, 64), (2, 7, 148, 296), (1, 4, 0, 0)]:
        other, other_infos, _ = _states(dtype, ng, tuning)
        assert other_infos == infos
        for i, (a, b) in enumerate(zip(states, other)):
            np.testing.assert_array_equal(a, b, err_msg=f"instance {i}, tuning {tuning}")
    if dtype != F64:
        return
    for i, d in enumerate(descs):
        U, T = (Grid2DGPU(d.nx, d.ny, ng, 0.0, 1.0, 0.0, 1.0, F64) for _ in range(2))
        assert load().mhd_initialise_orszag_tang(None, C.byref(U.g), 0.9 / SQRT_4PI, d.gamma, None) == 0
        ws = GpuWorkspace()
        init_gpu_workspace(ws, U)
        set_gpu_physics_gamma(ws, d.gamma)
        ws.set_limiter(1)
        info = ws.run(U, T, d.cfl, d.t_end, 5, 2, tuple(d.bc))
        assert infos[i] == (info.steps, info.t, info.ch), i
        np.testing.assert_array_equal(states[i], U.download(), err_msg=f"instance {i}")
