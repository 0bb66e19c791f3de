"""Adjoint gradients of grids that are not square, through the C ABI."""
import ctypes as C

import numpy as np
import pytest

from mhd_gpu_acc_b200 import F32, F64, load
from mhd_gpu_acc_b200.adjoint import amplitudes


class Adjoint:
    def __init__(self, nx, ny, nsteps, dtype=F64, limiter=1, solver=0):
        self.ptr = C.c_void_p()
        assert load().mhd_adjoint_create(nx, ny, dtype, limiter, 5.0 / 3.0, 0.4, 0.18, nsteps, 0, C.byref(self.ptr)) == 0
        if solver:
            assert load().mhd_adjoint_set_solver(self.ptr, solver) == 0

    def gradient(self, target, amp):
        target = np.ascontiguousarray(target, dtype=np.float64)
        assert load().mhd_adjoint_set_target(self.ptr, target.ctypes.data) == 0
        J, g = C.c_double(), np.zeros(16)
        assert load().mhd_adjoint_gradient(self.ptr, amp.ctypes.data, C.byref(J), g.ctypes.data) == 0
        return J.value, g

    def __del__(self):
        load().mhd_adjoint_destroy(self.ptr)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [F64, F32])
def test_gradient_of_a_very_tall_grid(dtype):
    """More rows than 65,535 blocks of 8 (524,276) or of 26 (1,703,906) cover.  One
    step of a column of square-ish cells has dt ~ dy, so rho moves by dt times
    a smooth function of y and the sums over the column, J / ny and the
    gradient, converge in 1 / ny: both grids have the same up to a few times
    2 pi 2 / 430000 = 3e-5 (FP64), and FP32 is within the other checks' 1e-2 of that."""
    got = []
    for ny in (430_000, 1_720_000):
        y = (np.arange(ny)[:, None] + 0.5) / ny
        target = 0.2 + 0.01 * np.sin(2 * np.pi * (y + np.array([[0.0, 0.25, 0.5, 0.75]])))
        J, g = Adjoint(4, ny, 1, dtype).gradient(target, amplitudes(0))
        got.append((J / ny, g))
    (J0, g0), (J1, g1) = got
    tol = 1e-3 if dtype == F64 else 1e-2
    assert np.linalg.norm(g0) > 0.0
    assert abs(J1 - J0) <= tol * J0
    assert np.linalg.norm(g1 - g0) <= tol * np.linalg.norm(g0), (g0, g1)
