"""Adjoint gradients of grids that are not square, through the C ABI."""
import ctypes as C
import importlib.util
import os

import numpy as np
import pytest

from mhd_gpu_acc_b200 import F32, F64, load
from mhd_gpu_acc_b200.adjoint import amplitudes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


def _cases():
    """perf/cases.py: its plain torch form of the scheme, differentiated by autograd in 64 bits."""
    spec = importlib.util.spec_from_file_location("mhd_cases", os.path.join(ROOT, "perf", "cases.py"))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def _objective(cases, nx, ny, solver, limiter, target, a):
    import torch

    amp = torch.tensor(a, dtype=torch.float64, device="cuda", requires_grad=True)
    U = cases._orszag_tang(nx, ny, 1.0 / np.sqrt(4.0 * np.pi), 5.0 / 3.0, amp)
    U, _, _, _ = cases._march(U, 10, 0.4, 1.0 / nx, 1.0 / ny, 5.0 / 3.0, solver, limiter, (0, 0, 0, 0))
    return 0.5 * ((U[0, 2:-2, 2:-2] - torch.as_tensor(target, device="cuda")) ** 2).sum(), amp


# both extents under, at and past the kernels' tiles of 26 (22 + 4 = 26, 48 + 4 = 52) and blocks of 8
@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["hll", "hlld"])
@pytest.mark.parametrize("limiter", ["minmod", "vanleer"])
@pytest.mark.parametrize("nx,ny", [(22, 48), (49, 23), (53, 74), (8, 5), (4, 100)])
def test_gradient_of_rectangles_equals_autograd(nx, ny, solver, limiter):
    """Ten steps.  FP64: both sides round to 1e-16 per operation, which ten steps of
    either grow to some 1e-13 (3e-14 measured at 256^2 x 16 steps); 1e-10 leaves
    room for a poorly conditioned amplitude.  FP32 within the other checks' 1e-2.

    HLLD's flux jumps with the sign of S_M where B_n has different signs on the two
    sides, and at 8 x 5 the symmetry of the flow puts a face at S_M = 0 to rounding
    (-1.2e-16): J has no gradient there, and each side's is that of the sign its
    rounding gave.  So a difference is let pass where the reference's own J jumps
    between a - 1e-7 and a + 1e-7, and nowhere else."""
    cases = _cases()
    a = amplitudes(0)
    y, x = (np.arange(ny)[:, None] + 0.5) / ny, (np.arange(nx)[None, :] + 0.5) / nx
    target = 0.22 + 0.01 * np.sin(2 * np.pi * (x + 2 * y))
    J, amp = _objective(cases, nx, ny, solver, limiter, target, a)
    J.backward()
    want = amp.grad.cpu().numpy()
    for dtype, tol in ((F64, 1e-10), (F32, 1e-2)):
        adj = Adjoint(nx, ny, 10, dtype, 0 if limiter == "minmod" else 1, 0 if solver == "hll" else 2)
        Jk, g = adj.gradient(target, a)
        if dtype == F64 and np.linalg.norm(g - want) > tol * np.linalg.norm(want):
            assert solver == "hlld", (g, want)
            jump = [_objective(cases, nx, ny, solver, limiter, target, a + h)[0].item()
                    - _objective(cases, nx, ny, solver, limiter, target, a - h)[0].item() for h in 1e-7 * np.eye(16)]
            assert np.linalg.norm(np.array(jump) / 2e-7 - want) > 10.0 * np.linalg.norm(want), (g, want)
            return
        assert abs(Jk - J.item()) <= tol * J.item()
        assert np.linalg.norm(g - want) <= tol * np.linalg.norm(want), (dtype, g, want)
