"""The work lists that a batch takes by its size: every instance equals the same
problem advanced alone, bit for bit (FP64), at the edges of the lists -- the
smallest grids, widths about one 28-cell segment and one 32-column strip, one wave
of equal tasks, several waves with shorter ones at the end, more units than
instances' clocks -- and under explicit tunings of the same batch."""
import ctypes as C

import numpy as np
import pytest

from mhd_gpu_acc_b200 import F64, GpuWorkspace, Grid2DGPU, init_gpu_workspace, load, set_gpu_physics_gamma
from mhd_gpu_acc_b200.batch import SQRT_4PI, Batch, instance

SMALL = [(4, 4), (5, 33), (27, 9), (28, 8), (29, 7), (30, 64), (31, 5), (62, 63), (300, 4), (4, 300)]
WAVES = [(300, 301)] * 6 + [(61, 517), (517, 61), (4, 4)]


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [SMALL, WAVES, SMALL[:1]], ids=["small", "waves", "one"])
@pytest.mark.parametrize("tuning", [None, (2, 7, 148, 296)])
def test_batch_work_lists(sizes, tuning):
    bcs = [(0, 0, 0, 0), (1, 1, 2, 2), (2, 2, 0, 0)]
    descs = [instance(nx, ny, 5 / 3, 0.3, 5.0, bc=bcs[k % 3]) for k, (nx, ny) in enumerate(sizes)]
    batch = Batch(descs, dtype=F64)
    if tuning:
        batch.set_tuning(*tuning)
    for i, d in enumerate(descs):
        batch.init_orszag_tang(i, 0.9 / SQRT_4PI, d.gamma)
    infos = batch.run(3) and batch.run(2)
    for i, d in enumerate(descs):
        # alone, c_h carried from the first three steps into the next two, as the batch carries it
        U, T = (Grid2DGPU(d.nx, d.ny, 2, 0.0, 1.0, 0.0, 1.0, F64) for _ in range(2))
        assert load().mhd_initialise_orszag_tang(None, C.byref(U.g), 0.9 / SQRT_4PI, d.gamma, None) == 0
        ws = GpuWorkspace()
        init_gpu_workspace(ws, U)
        set_gpu_physics_gamma(ws, d.gamma)
        ws.set_limiter(1)
        ws.run(U, T, d.cfl, d.t_end, 3, 2, tuple(d.bc))
        info = ws.run(U, T, d.cfl, d.t_end, 2, 2, tuple(d.bc))
        assert (infos[i].steps, infos[i].t, infos[i].ch) == (info.steps, info.t, info.ch), i
        np.testing.assert_array_equal(batch.download(i), U.download(), err_msg=f"instance {i}")
    batch.destroy()
