"""Branch-free FP64 quotients and roots (csrc/exact_div.cuh) equal the operators bit
for bit wherever their range tests let operands through."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("where", ["host", pytest.param("device", marks=pytest.mark.gpu)])
def test_quotients_and_roots_over_the_declared_ranges(tmp_path, where):
    exe = str(tmp_path / "exact_range_check")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "--fmad=false", "-arch=sm_100a", "-Xcompiler", "-mfma", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(ROOT, "mhd_gpu_acc_b200", "csrc"),
                    os.path.join(ROOT, "tests", "exact_range_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe, where], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
