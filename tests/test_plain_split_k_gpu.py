"""Plain products of few tiles whose k jetgpu_contract cuts into ranges: ragged
and empty last ranges, both element types, tile edges; the uncut result where
the workspace holds no more than a batched contraction asks for; and no cut of
k <= 64, which grouped and skinny launches add in one order.

An output of k terms is off by at most 2 k + 4 roundings of sums of |a| |b|
(|z| as |re| + |im|); the reference is complex128, so complex128 gets twice
that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(17, 17, 256), (33, 40, 257), (64, 65, 1000), (32, 512, 512), (256, 64, 1024),
          (100, 100, 4099), (20, 300, 2047), (700, 600, 300)]


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_ranges(cuda, m, n, k, dtype):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m + n + k)
    a = (rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))).astype(dtype)
    b = (rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))).astype(dtype)
    ad = torch.from_numpy(a.T.copy().ravel()).to(cuda)
    bd = torch.from_numpy(b.ravel()).to(cuda)
    args = ([k, m], [1, 0], bd, [k, n], [0, 1], m, n, k)
    want = a.astype(np.complex128) @ b.astype(np.complex128)
    size = (np.abs(a.real) + np.abs(a.imag)).astype(float) @ (np.abs(b.real) + np.abs(b.imag))
    eps = (2 * k + 4) * (2.0 ** -24 if dtype == "complex64" else 2.0 ** -52)
    got = capi.contract(ad, *args)
    assert np.all(np.abs(got.cpu().numpy().reshape(m, n) - want) <= eps * size)
    # The workspace of a batch of one: its result, bit for bit.
    need = int(capi.lib.jetgpu_contract_batched_workspace_size(
        1, 2, capi.u64([k, m]), capi.i32([1, 0]), 0, 2, capi.u64([k, n]), capi.i32([0, 1]), 0, m,
        n, k, capi.dtype_code(ad.dtype), capi.PREC_FP32))
    one = capi.contract_batched(1, ad, [k, m], [1, 0], 0, bd, [k, n], [0, 1], 0, m, n, k)
    out = torch.empty_like(one)
    ws = torch.empty(max(need, 1), dtype=torch.uint8, device=cuda)
    capi.check(capi.lib.jetgpu_contract(
        ad.data_ptr(), 2, capi.u64([k, m]), capi.i32([1, 0]), bd.data_ptr(), 2, capi.u64([k, n]),
        capi.i32([0, 1]), out.data_ptr(), m, n, k, capi.dtype_code(ad.dtype), capi.PREC_FP32, 0, 0,
        0, ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream))
    small = int(capi.contract_workspace_size([k, m], [1, 0], [k, n], [0, 1], m, n, k,
                                             capi.dtype_code(ad.dtype), capi.PREC_FP32)) == need
    assert small or torch.equal(torch.view_as_real(out), torch.view_as_real(one))


def test_short_k_is_not_cut(cuda):
    import torch

    from jet_gb300 import capi

    gen = torch.Generator(device=cuda).manual_seed(2)
    for m, n, k in ((40, 50, 64), (64, 64, 255)):
        a = torch.randn(m * k, generator=gen, device=cuda, dtype=torch.complex64)
        b = torch.randn(k * n, generator=gen, device=cuda, dtype=torch.complex64)
        one = capi.multiply(a, b, m, n, k)
        got = capi.contract(a, [m, k], [0, 1], b, [k, n], [0, 1], m, n, k)
        assert torch.equal(torch.view_as_real(got), torch.view_as_real(one))
