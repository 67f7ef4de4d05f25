"""Small outputs over a long k: every tile of the kernel and its edges, k around
its slices (32 and 16) and ranges, batches.

An output of k terms is off by at most 2 k + 4 roundings of sums of |a| |b|
(|z| as |re| + |im|); the reference is complex128, so complex128 gets twice
that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OUTPUTS = [(2, 2), (4, 8), (5, 8), (4, 9), (8, 16), (9, 16), (2, 16), (8, 17), (16, 16), (3, 31),
           (16, 32), (17, 2), (32, 16), (25, 9)]


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("m,n", OUTPUTS)
@pytest.mark.parametrize("k,batch", [(2048, 1), (2049, 3), (4111, 1), (20011, 2)])
def test_tiles(cuda, m, n, k, batch, dtype):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m + 100 * n + k)
    a = (rng.standard_normal((batch, m, k)) + 1j * rng.standard_normal((batch, m, k)))
    b = (rng.standard_normal((batch, k, n)) + 1j * rng.standard_normal((batch, k, n)))
    a, b = a.astype(dtype), b.astype(dtype)
    ad, bd = (torch.from_numpy(x.ravel()).to(cuda) for x in (a, b))
    if batch > 1:
        got = capi.contract_batched(batch, ad, [m, k], [0, 1], 1, bd, [k, n], [0, 1], 1, m, n, k)
    else:
        got = capi.contract(ad, [m, k], [0, 1], bd, [k, n], [0, 1], m, n, k)
    want = a.astype(np.complex128) @ b.astype(np.complex128)
    size = (np.abs(a.real) + np.abs(a.imag)).astype(float) @ (np.abs(b.real) + np.abs(b.imag))
    eps = (2 * k + 4) * (2.0 ** -24 if dtype == "complex64" else 2.0 ** -52)
    assert np.all(np.abs(got.cpu().numpy().reshape(want.shape) - want) <= eps * size)
