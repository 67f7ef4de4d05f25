"""Small outputs over a long k read in place: closing_plan_test.cu replays the
kernel's plan on the CPU; on the GPU, every tile, both operands' orders and the
workspace's least size against complex128.

An output of k terms is off by at most 2 k + 4 roundings of sums of |a| |b|
(|z| as |re| + |im|), whatever their order; the reference is complex128, so
complex128 gets twice that."""
import os
import shutil
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_closing_plan(tmp_path):
    nvcc = shutil.which("nvcc") or os.path.join(
        os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    pkg = os.path.join(REPO, "jet_gb300")
    exe = str(tmp_path / "closing_plan_test")
    cmd = [nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
           "-I" + os.path.join(REPO, "include"), "-I" + os.path.join(pkg, "csrc"),
           os.path.join(REPO, "tests", "cpp", "closing_plan_test.cu"), "-L" + pkg, "-ljetgpu",
           "-Xlinker", "-rpath", "-Xlinker", pkg, "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-4000:]
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout[-2000:] + res.stderr[-2000:]
    assert res.stdout.startswith("ok ")


OUTPUTS = [(1, 1), (1, 5), (2, 3), (3, 4), (4, 1), (4, 4), (3, 5), (4, 5), (5, 1), (5, 4)]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("m,n", OUTPUTS)
@pytest.mark.parametrize("k,order", [(11, "free last"), (11, "mixed"), (14, "A in order"),
                                     (15, "mixed"), (17, "free first")])
def test_orders(cuda, m, n, k, order, dtype):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m + 10 * n + 100 * k)
    # Places in memory of the permuted operands' axes.
    a_perm, b_perm = list(range(m + k)), list(range(k + n))
    if order == "free last":
        a_perm = a_perm[k:] + a_perm[:k]
    elif order == "free first":
        b_perm = b_perm[n:] + b_perm[:n]
    else:
        b_perm = [int(x) for x in rng.permutation(k + n)]
        if order == "mixed":
            a_perm = [int(x) for x in rng.permutation(m + k)]
    M, N, K = 2 ** m, 2 ** n, 2 ** k
    a = (rng.standard_normal(M * K) + 1j * rng.standard_normal(M * K)).astype(dtype)
    b = (rng.standard_normal(K * N) + 1j * rng.standard_normal(K * N)).astype(dtype)
    ad, bd = (torch.from_numpy(x).to(cuda) for x in (a, b))
    got = capi.contract(ad, [2] * (m + k), a_perm, bd, [2] * (k + n), b_perm, M, N, K)
    am = a.reshape([2] * (m + k)).transpose(a_perm).reshape(M, K)
    bm = b.reshape([2] * (k + n)).transpose(b_perm).reshape(K, N)
    want = am.astype(np.complex128) @ bm.astype(np.complex128)
    size = (np.abs(am.real) + np.abs(am.imag)).astype(float) @ (np.abs(bm.real) + np.abs(bm.imag))
    eps = (2 * K + 4) * (2.0 ** -24 if dtype == "complex64" else 2.0 ** -52)
    assert np.all(np.abs(got.cpu().numpy().reshape(M, N) - want) <= eps * size)
