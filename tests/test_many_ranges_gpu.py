"""Plain complex64 products of few outputs whose long k is cut into many ranges:
the kernels that add the ranges (a warp or a thread per output, on both sides
of the line between them) on operands of small integers, whose sums are exact
in any order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(17, 17, 16384), (17, 17, 65537), (2, 40, 262147), (33, 3, 262144), (20, 40, 100003),
          (32, 64, 65536), (33, 62, 65599), (64, 64, 65536), (64, 64, 262143), (64, 65, 131072),
          (90, 91, 70001), (2, 65, 1000000)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_exact(cuda, m, n, k):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m + n + k)

    def draw(*shape):  # |re|, |im| <= 2: sums of k <= 2^20 products stay below 2^24
        return rng.integers(-2, 3, shape) + 1j * rng.integers(-2, 3, shape)

    a, b = draw(m, k), draw(k, n)
    ad = torch.from_numpy(a.astype(np.complex64).ravel()).to(cuda)
    bd = torch.from_numpy(b.astype(np.complex64).ravel()).to(cuda)
    got = capi.contract(ad, [m, k], [0, 1], bd, [k, n], [0, 1], m, n, k).cpu().numpy()
    assert np.array_equal(got.reshape(m, n), a @ b)


@pytest.mark.parametrize("m,n,k", [(79, 2248, 3356), (300, 300, 2816), (128, 700, 4000),
                                   (200, 1000, 1536), (33, 2000, 5000)])
def test_no_further_off_than_a_batch_of_one(cuda, m, n, k):
    """jetgpu_contract cuts k at least as often as the batched rule does, so its
    sums are no further from complex128 (10 % for the sample)."""
    import torch

    from jet_gb300 import capi

    gen = torch.Generator(device=cuda).manual_seed(m + n + k)
    a = torch.randn(m * k, generator=gen, device=cuda, dtype=torch.complex64)
    b = torch.randn(k * n, generator=gen, device=cuda, dtype=torch.complex64)
    want = (a.reshape(m, k).to(torch.complex128) @ b.reshape(k, n).to(torch.complex128)).ravel()
    got = capi.contract(a, [m, k], [0, 1], b, [k, n], [0, 1], m, n, k)
    one = capi.contract_batched(1, a, [m, k], [0, 1], 0, b, [k, n], [0, 1], 0, m, n, k)
    off = torch.linalg.vector_norm(got - want)
    assert off <= 1.1 * torch.linalg.vector_norm(one - want)
