"""The batched engine's work lists and error paths (host code of csrc/batch_api.cu on
a fake CUDA runtime: needs nvcc, no GPU)."""
import subprocess

from test_workspace import build_on_fake_runtime


def test_batch_lists(tmp_path):
    r = subprocess.run([build_on_fake_runtime(tmp_path, "batch_check", "batch_api.cu", "capi.cu")], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stdout + r.stderr
