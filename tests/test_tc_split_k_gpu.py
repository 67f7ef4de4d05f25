"""Tensor-core products whose k is cut into ranges (few tiles, long k): ragged
ranges and tiles, each word format, the 3M product, and what happens when the
workspace holds only what an uncut product needs.

Bounds, elementwise against sum |a| |b| (|z| as |re| + |im|): a product term is
off by 3 * 2^-18 (BF16: two pieces of 8 bits, lo lo dropped) or 3 * 2^-21
(TF32, FP16: pieces of 11 bits); tensor-core sums of a chunk, folds and the
sum of the ranges add at most as much again. 3M's products are of re + im:
three times that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(128, 128, 1024), (129, 200, 1000), (300, 127, 4097), (512, 640, 777), (256, 64, 8192),
          (1000, 1000, 260)]


@pytest.mark.parametrize("algo", [0, 1])
@pytest.mark.parametrize("form", ["tf32x3", "bf16x3", "fp16x3"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_ranges(cuda, m, n, k, form, algo):
    import torch

    from jet_gb300 import capi

    prec = {"tf32x3": capi.PREC_TF32X3, "bf16x3": capi.PREC_BF16X3,
            "fp16x3": capi.PREC_FP16X3}[form]
    rng = np.random.default_rng(m + n + k)
    a = (rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))).astype(np.complex64)
    b = (rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))).astype(np.complex64)
    ad = torch.from_numpy(a.T.copy().ravel()).to(cuda)
    bd = torch.from_numpy(b.ravel()).to(cuda)
    got = capi.contract(ad, [k, m], [1, 0], bd, [k, n], [0, 1], m, n, k, precision=prec,
                        algo=algo).cpu().numpy().reshape(m, n)
    want = a.astype(np.complex128) @ b.astype(np.complex128)
    size = (np.abs(a.real) + np.abs(a.imag)).astype(float) @ (np.abs(b.real) + np.abs(b.imag))
    eps = 6 * 2.0 ** (-18 if form == "bf16x3" else -21) * (3 if algo else 1)
    assert np.all(np.abs(got - want) <= eps * size)


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_uncut_with_the_smaller_workspace(cuda, m, n, k):
    """A workspace of what a batch of one needs is enough, gives the batched
    executors' bits, and the allocation-free entry point takes the product."""
    import torch

    from jet_gb300 import capi

    gen = torch.Generator(device=cuda).manual_seed(k)
    a = torch.randn(m * k, generator=gen, device=cuda, dtype=torch.complex64)
    b = torch.randn(k * n, generator=gen, device=cuda, dtype=torch.complex64)
    args = ([m, k], [0, 1], b, [k, n], [0, 1], m, n, k)
    need = int(capi.lib.jetgpu_contract_batched_workspace_size(
        1, 2, capi.u64([m, k]), capi.i32([0, 1]), 0, 2, capi.u64([k, n]), capi.i32([0, 1]), 0, m,
        n, k, capi.C64, capi.PREC_FP16X3))
    ws = torch.empty(need, dtype=torch.uint8, device=cuda)
    one = capi.contract_batched(1, a, [m, k], [0, 1], 0, b, [k, n], [0, 1], 0, m, n, k,
                                precision=capi.PREC_FP16X3)
    out = torch.empty_like(one)
    capi.check(capi.lib.jetgpu_contract(
        a.data_ptr(), 2, capi.u64([m, k]), capi.i32([0, 1]), b.data_ptr(), 2, capi.u64([k, n]),
        capi.i32([0, 1]), out.data_ptr(), m, n, k, capi.C64, capi.PREC_FP16X3, 0, 0, 0,
        ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out, one)
    cut = capi.contract(a, *args, precision=capi.PREC_FP16X3)
    assert torch.linalg.vector_norm(cut - one) <= 2e-6 * torch.linalg.vector_norm(one)
    if need <= capi.lib.jetgpu_contract_noalloc_max_scratch():
        capi.check(capi.lib.jetgpu_contract_noalloc(
            capi._vp(a.data_ptr()), 2, capi.u64([m, k]), capi.i32([0, 1]), capi._vp(b.data_ptr()),
            2, capi.u64([k, n]), capi.i32([0, 1]), capi._vp(out.data_ptr()), capi.ctypes.c_uint64(m),
            capi.ctypes.c_uint64(n), capi.ctypes.c_uint64(k), capi.C64, capi.PREC_FP16X3, 0, 0, 0,
            capi._vp(torch.cuda.current_stream().cuda_stream)))
        assert torch.linalg.vector_norm(out - one) <= 2e-6 * torch.linalg.vector_norm(one)
