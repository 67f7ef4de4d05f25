"""Plain products across the tiles that jetgpu_contract picks by shape: edges
of 32- and 64-wide tiles, k around the staged slices (8 and 16) and batches,
aligned and unaligned outputs.

A complex product of k terms in FP32 (FP64) FMAs is off by at most 2 k + 2
roundings of its partial sums, each at most the sum of |a| |b| (|z| as |re| +
|im|); the reference is complex128, so complex128 products get twice that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 100), (31, 33, 7), (32, 32, 65), (33, 31, 129), (64, 64, 72), (65, 127, 80),
          (100, 20, 300), (20, 100, 300), (640, 640, 17), (129, 1023, 66), (1031, 517, 70),
          (2048, 2048, 9), (700, 700, 81)]


def _check(a, b, got, eps):
    want = a.astype(np.complex128) @ b.astype(np.complex128)
    size = (np.abs(a.real) + np.abs(a.imag)).astype(float) @ (np.abs(b.real) + np.abs(b.imag))
    k = a.shape[1]
    assert np.all(np.abs(got - want) <= (2 * k + 2) * eps * size)


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_shapes(cuda, m, n, k, dtype):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m + 3 * n + 7 * k)
    a = (rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))).astype(dtype)
    b = (rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))).astype(dtype)
    eps = 2.0 ** -24 if dtype == "complex64" else 2.0 ** -52
    ad, bd = torch.from_numpy(a).to(cuda).ravel(), torch.from_numpy(b).to(cuda).ravel()
    for off in (0, 1):  # C on and off a 16-byte boundary
        out = torch.zeros(m * n + 2, dtype=ad.dtype, device=cuda)
        capi.multiply(ad, bd, m, n, k, out=out[off: off + m * n])
        got = out.cpu().numpy()
        _check(a, b, got[off: off + m * n].reshape(m, n), eps)
        assert not got[:off].any() and not got[off + m * n:].any()


@pytest.mark.parametrize("batch,m,n,k", [(3, 33, 65, 70), (9, 81, 27, 243), (40, 64, 64, 66)])
def test_batches_equal_single_products(cuda, batch, m, n, k):
    """Every tile adds the same k sequence: a batch has the bits of its products."""
    import torch

    from jet_gb300 import capi

    gen = torch.Generator(device=cuda).manual_seed(batch)
    a = torch.randn(batch * m * k, generator=gen, device=cuda, dtype=torch.complex64)
    b = torch.randn(batch * k * n, generator=gen, device=cuda, dtype=torch.complex64)
    got = capi.contract_batched(batch, a, [m, k], [0, 1], 1, b, [k, n], [0, 1], 1, m, n, k)
    for i in range(batch):
        one = capi.multiply(a[i * m * k:(i + 1) * m * k], b[i * k * n:(i + 1) * k * n], m, n, k)
        assert torch.equal(got[i * m * n:(i + 1) * m * n], one)
