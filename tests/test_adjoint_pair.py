"""The paired adjoint functions (csrc/adj_pair.cuh) equal the general ones they
restate, to rounding (host build: needs nvcc, no GPU); on the GPU, gradients of
grids whose edges fall inside the kernels' tiles, and one segment of all steps
against many."""
import os
import subprocess

import numpy as np
import pytest

from mhd_gpu_acc_b200 import F32, F64
from mhd_gpu_acc_b200.adjoint import OTAdjoint, amplitudes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_paired_functions_equal_the_general_ones(tmp_path):
    exe = str(tmp_path / "adjpair")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-x", "cu", "-arch=sm_100a", "-I",
                    os.path.join(ROOT, "mhd_gpu_acc_b200", "csrc"),
                    os.path.join(ROOT, "tests", "adj_pair_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("limiter", [0, 1])
@pytest.mark.parametrize("n", [22, 23, 48, 53, 74])  # n + 4 under, at and past 26 and 52; ragged blocks of 8 columns
def test_gradient_at_tile_edges(n, limiter):
    """The FP64 gradient against central differences (h = 1e-6; the bound of the
    repository's other gradient checks), with one segment and with segments of 4."""
    grads = []
    for every in (0, 4):
        adj = OTAdjoint(n=n, nsteps=10, dtype=F64, limiter=limiter, checkpoint_every=every)
        _, target = adj.forward(amplitudes(1), want_rho=True)
        adj.set_target(target)
        a = amplitudes(0)
        grads.append(adj.gradient(a)[1])
    np.testing.assert_allclose(grads[0], grads[1], rtol=1e-10, atol=1e-14 * np.abs(grads[0]).max())
    fd = np.zeros(16)
    for k in range(16):
        e = np.zeros(16)
        e[k] = 1e-6
        fd[k] = (adj.forward(a + e) - adj.forward(a - e)) / 2e-6
    assert np.linalg.norm(grads[0] - fd) / np.linalg.norm(fd) <= 1e-4
    adj = OTAdjoint(n=n, nsteps=10, dtype=F32, limiter=limiter)
    adj.set_target(target)
    g32 = adj.gradient(a)[1]
    assert np.linalg.norm(g32 - grads[0]) / np.linalg.norm(grads[0]) <= 1e-2


@pytest.mark.gpu
def test_gradient_without_stored_x_swept_states():
    """A segment whose x-swept states exceed an eighth of the free memory (1024^2
    FP64, 160 steps: 12 GB more) recomputes them; the gradient is that of short
    segments, which keep them."""
    grads = []
    for every in (160, 8):
        adj = OTAdjoint(n=1024, nsteps=160, dtype=F64, checkpoint_every=every)
        adj.set_target(np.full((1024, 1024), 0.2))
        grads.append(adj.gradient(amplitudes(0))[1])
        adj.destroy()
    np.testing.assert_allclose(grads[0], grads[1], rtol=1e-10, atol=1e-14 * np.abs(grads[0]).max())
