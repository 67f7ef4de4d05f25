"""Vector products (one row or column, and dot products) around the groups of
loads their threads keep in flight, and reductions over k ranges in eights.

Each thread's compensated sums of four-product groups are off by a few FP32
roundings of sum |a| |b| (|z| as |re| + |im|): 16 allowed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("m,n", [(1, 1), (1, 9), (7, 1), (1, 300), (64, 1)])
@pytest.mark.parametrize("k", [1, 63, 255, 257, 1023, 4097, 8191, 65537])
def test_lengths(cuda, m, n, k, dtype):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m + n + k)
    a = (rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))).astype(dtype)
    b = (rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))).astype(dtype)
    got = capi.contract(torch.from_numpy(a.ravel()).to(cuda), [m, k], [0, 1],
                        torch.from_numpy(b.ravel()).to(cuda), [k, n], [0, 1], m, n, k)
    want = a.astype(np.complex128) @ b.astype(np.complex128)
    size = (np.abs(a.real) + np.abs(a.imag)).astype(float) @ (np.abs(b.real) + np.abs(b.imag))
    eps = 2.0 ** -24 if dtype == "complex64" else (8 + np.log2(k + 1)) * 2.0 ** -53
    assert np.all(np.abs(got.cpu().numpy().reshape(m, n) - want) <= 16 * eps * size)


@pytest.mark.parametrize("n_values", [1, 3, 5])
def test_slice_gather_widths(cuda, n_values):
    """Slice values on both sides of 2^32 (the sliced axes repeat far beyond
    their extents there): 32- and 64-bit index arithmetic agree with numpy."""
    import torch

    from jet_gb300 import capi

    shape, axes = [3, 4, 5, 2], [1, 2]
    x = np.arange(120, dtype=np.complex64).reshape(shape)
    xd = torch.from_numpy(x.ravel()).to(cuda)
    for strides in ([5, 1], [1 << 33, 1]):
        for first in (0, 7, (1 << 32) - 2, (1 << 32) + 11, 3 << 40):
            got = capi.slice_gather(xd, shape, axes, strides, first, n_values).cpu().numpy()
            want = []
            for v in range(first, first + n_values):
                i, j = (v // strides[0]) % 4, (v // strides[1]) % 5
                want.append(x[:, i, j, :].ravel())
            assert np.array_equal(got, np.concatenate(want))
