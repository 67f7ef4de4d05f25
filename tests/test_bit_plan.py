"""bit_plan_test.cu (host only, runs on the CPU): the bit-permutation plan of
power-of-2 transposes replayed against the plain permutation; and, on the GPU,
transposes on both sides of the size where that kernel takes over from the
gather kernel, batched and with long runs, bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bit_plan(tmp_path):
    nvcc = shutil.which("nvcc") or os.path.join(
        os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    pkg = os.path.join(REPO, "jet_gb300")
    exe = str(tmp_path / "bit_plan_test")
    cmd = [nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
           "-I" + os.path.join(REPO, "include"), "-I" + os.path.join(pkg, "csrc"),
           os.path.join(REPO, "tests", "cpp", "bit_plan_test.cu"), "-L" + pkg, "-ljetgpu",
           "-Xlinker", "-rpath", "-Xlinker", pkg, "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-4000:]
    res = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-2000:]
    assert res.stdout.startswith("ok ")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n,batch", [(12, 1), (15, 1), (16, 1), (17, 1), (18, 1), (21, 1), (12, 32),
                                     (12, 33), (14, 7)])
def test_transposes_around_the_threshold(cuda, n, batch, dtype):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(n + batch)
    x = (rng.standard_normal((batch,) + (2,) * n)
         + 1j * rng.standard_normal((batch,) + (2,) * n)).astype(dtype)
    xd = torch.from_numpy(x.ravel()).to(cuda)
    for perm in (list(rng.permutation(n)), list(range(n // 3, n)) + list(range(n // 3)),
                 list(range(n))[::-1]):
        perm = [int(v) for v in perm]
        got = capi.permute(xd, [2] * n, perm, batch=batch).cpu().numpy()
        want = x.transpose([0] + [v + 1 for v in perm]).ravel()
        assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
