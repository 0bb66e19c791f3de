"""The workspace's device and page-locked scratch (host code of csrc/capi.cu on a
fake CUDA runtime: needs nvcc, no GPU)."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def build_on_fake_runtime(tmp_path, check, *sources):
    """tests/<check>.cu with the library's host sources, linked without the CUDA
    runtime; symbols that the check never calls stay unresolved."""
    exe, csrc, tests = str(tmp_path / check), os.path.join(ROOT, "mhd_gpu_acc_b200", "csrc"), os.path.join(ROOT, "tests")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    objs = []
    for src in [os.path.join(tests, check + ".cu"), os.path.join(tests, "fake_cuda.cpp"),
                *(os.path.join(csrc, s) for s in sources)]:
        objs.append(str(tmp_path / (os.path.basename(src) + ".o")))
        subprocess.run([nvcc, "-std=c++17", "-O1", "-arch=sm_100a", "-Xcompiler", "-fPIC", "-I", csrc, "-c", src, "-o",
                        objs[-1]], check=True)
    subprocess.run(["g++", *objs, "-o", exe, "-Wl,--unresolved-symbols=ignore-all", "-lpthread", "-ldl"], check=True)
    return exe


def test_workspace_scratch(tmp_path):
    r = subprocess.run([build_on_fake_runtime(tmp_path, "workspace_check", "capi.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
