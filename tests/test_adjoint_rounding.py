"""The adjoint sweeps' reciprocals and roots are correctly rounded: compiled with the
build's own flags for either precision, they equal the operators bit for bit."""
import os
import subprocess

import pytest

from mhd_gpu_acc_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("source", ["adj_f32.cu", "adj_f64.cu", "adjoint.cu"])
def test_no_approximate_arithmetic(source):
    assert not [f for f in build.CU_SOURCES[source] if "fast" in f or "prec" in f or "ftz" in f]


@pytest.mark.gpu
@pytest.mark.parametrize("source", ["adj_f32.cu", "adj_f64.cu"])
def test_reciprocals_and_roots_equal_the_operators(tmp_path, source):
    exe = str(tmp_path / "adj_round_check")
    subprocess.run(["nvcc", "-std=c++17", "-O3", "-arch=sm_100a", *build.CU_SOURCES[source], "-I",
                    os.path.join(ROOT, "mhd_gpu_acc_b200", "csrc"), os.path.join(ROOT, "tests", "adj_round_check.cu"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
