"""split_layout_test.cu (host only, runs on the CPU): the tensor-core form's
word coordinates for k up to 2^31, where operands of the size would not fit a
test."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_split_layout(tmp_path):
    nvcc = shutil.which("nvcc") or os.path.join(
        os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    pkg = os.path.join(REPO, "jet_gb300")
    exe = str(tmp_path / "split_layout_test")
    cmd = [nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
           "-I" + os.path.join(REPO, "include"), "-I" + os.path.join(pkg, "csrc"),
           os.path.join(REPO, "tests", "cpp", "split_layout_test.cu"), "-L" + pkg, "-ljetgpu",
           "-Xlinker", "-rpath", "-Xlinker", pkg, "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-4000:]
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-2000:]
    assert res.stdout.startswith("ok ")
