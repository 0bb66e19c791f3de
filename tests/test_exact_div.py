"""Branch-free FP64 quotients and roots (csrc/exact_div.cuh) equal the operators
bit for bit, on the host and with the GPU's own seeds; the sweeps' FP64 physics
(csrc/phys_exact_sweep.cuh) equals the reference-ordered functions bit for bit
(host)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _build(tmp_path, name):
    exe = str(tmp_path / name)
    subprocess.run(["nvcc", "-std=c++17", "-O2", "--fmad=false", "-arch=sm_100a", "-Xcompiler", "-mfma", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(ROOT, "mhd_gpu_acc_b200", "csrc"),
                    os.path.join(ROOT, "tests", name + ".cu"), "-o", exe], check=True)
    return exe


def _passes(*cmd):
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_quotients_and_roots_on_the_host(tmp_path):
    _passes(_build(tmp_path, "exact_div_check"), "host")


def test_sweep_physics_equals_the_reference_order(tmp_path):
    _passes(_build(tmp_path, "exact_sweep_check"))


@pytest.mark.gpu
def test_quotients_and_roots_on_the_gpu(tmp_path):
    _passes(_build(tmp_path, "exact_div_check"), "device")
