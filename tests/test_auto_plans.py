"""The task plans that the sweeps take by the size of the launch cover every cell
exactly once (index arithmetic, compiled for the host: needs nvcc, no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# one cell; a segment of one chunk (28 cells) and its neighbours; the one-wave
# limits of x and y from both sides; ragged and large extents
SIZES = [(2, 2), (27, 3), (28, 4), (29, 5), (60, 61), (800, 4), (4, 3000), (515, 1031), (543, 557), (767, 769),
         (1100, 1090), (2048, 2048), (4096, 1500), (3001, 2999)]


@pytest.mark.skipif(shutil.which("nvcc") is None and not os.path.exists("/usr/local/cuda/bin/nvcc"),
                    reason="needs nvcc")
def test_auto_plans_cover_every_cell_once(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "auto_plan_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-x", "cu", "-Wno-deprecated-gpu-targets", "-I",
                    os.path.join(ROOT, "mhd_gpu_acc_b200", "csrc"), os.path.join(ROOT, "tests", "auto_plan_check.cu"),
                    "-o", exe], check=True)
    r = subprocess.run([exe, *[str(v) for s in SIZES for v in s]], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
