"""jetgpu_contract_noalloc where jetgpu_contract cuts k into ranges: the same
bits where the size that jetgpu_contract asks for fits the library's scratch, operands in
order (which an uncut product needs no scratch for) among them; and the uncut
product's where only that fits."""
import pytest

pytestmark = pytest.mark.gpu


def _both(cuda, m, n, k, dtype, precision):
    import torch

    from jet_gb300 import capi

    gen = torch.Generator(device=cuda).manual_seed(m + n + k)
    a = torch.randn(m * k, generator=gen, device=cuda, dtype=getattr(torch, dtype))
    b = torch.randn(k * n, generator=gen, device=cuda, dtype=getattr(torch, dtype))
    code = capi.dtype_code(a.dtype)
    views = ([m, k], [0, 1], [k, n], [0, 1])
    asked = capi.contract_workspace_size(*views, m, n, k, code, precision)
    least = int(capi.lib.jetgpu_contract_batched_workspace_size(
        1, 2, capi.u64([m, k]), capi.i32([0, 1]), 0, 2, capi.u64([k, n]), capi.i32([0, 1]), 0, m, n,
        k, code, precision))
    out = torch.empty(m * n, dtype=a.dtype, device=cuda)
    capi.check(capi.lib.jetgpu_contract_noalloc(
        capi._vp(a.data_ptr()), 2, capi.u64([m, k]), capi.i32([0, 1]), capi._vp(b.data_ptr()), 2,
        capi.u64([k, n]), capi.i32([0, 1]), capi._vp(out.data_ptr()), capi.ctypes.c_uint64(m),
        capi.ctypes.c_uint64(n), capi.ctypes.c_uint64(k), code, precision, 0, 0, 0,
        capi._vp(torch.cuda.current_stream().cuda_stream)))
    cut = capi.contract(a, [m, k], [0, 1], b, [k, n], [0, 1], m, n, k, precision=precision)
    one = capi.contract_batched(1, a, [m, k], [0, 1], 0, b, [k, n], [0, 1], 0, m, n, k,
                                precision=precision)
    return asked, least, *(torch.view_as_real(x) for x in (out, cut, one))


@pytest.mark.parametrize("dtype,precision,m,n,k", [
    ("complex64", 0, 64, 64, 300), ("complex64", 0, 40, 50, 500), ("complex128", 0, 64, 64, 300),
    ("complex64", 0, 64, 64, 4096), ("complex128", 0, 33, 65, 1000), ("complex64", 1, 128, 100, 1024)])
def test_same_bits_within_the_scratch(cuda, dtype, precision, m, n, k):
    import torch

    from jet_gb300 import capi

    asked, least, out, cut, one = _both(cuda, m, n, k, dtype, precision)
    assert least < asked <= capi.lib.jetgpu_contract_noalloc_max_scratch()
    assert torch.equal(out, cut)


@pytest.mark.parametrize("m,n,k", [(1024, 1024, 512), (1000, 1000, 560)])
def test_uncut_beyond_the_scratch(cuda, m, n, k):
    import torch

    from jet_gb300 import capi

    asked, least, out, cut, one = _both(cuda, m, n, k, "complex64", capi.PREC_TF32X3)
    assert least <= capi.lib.jetgpu_contract_noalloc_max_scratch() < asked
    assert torch.equal(out, one)
    assert torch.linalg.vector_norm(out - cut) <= 2e-6 * torch.linalg.vector_norm(cut)
