"""Plain complex64 products of a short k and many outputs, on both sides of the
lines where they get tiles of their own: k around 8, 16 and 32, ragged edges,
batches, outputs off a 16-byte boundary. Every tile adds the same k sequence,
so blocks of the output equal the products of the blocks alone (few tiles, the
other kernels) bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


def _operands(cuda, *sizes):
    import torch

    gen = torch.Generator(device=cuda).manual_seed(sum(sizes))
    return [torch.randn(n, generator=gen, device=cuda, dtype=torch.complex64) for n in sizes]


@pytest.mark.parametrize("k", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33])
@pytest.mark.parametrize("m,n", [(17, 9800), (20, 30001), (32, 4864), (32, 4896), (65, 9728),
                                 (33, 5000), (65537, 33), (4001, 260)])
def test_blocks(cuda, m, n, k):
    import torch

    from jet_gb300 import capi

    a, b = _operands(cuda, m * k, k * n)
    a2, b2 = a.reshape(m, k), b.reshape(k, n)
    for off in (0, 1):
        out = torch.zeros(m * n + 2, dtype=a.dtype, device=cuda)
        capi.multiply(a, b, m, n, k, out=out[off: off + m * n])
        got = out[off: off + m * n].reshape(m, n)
        for r in {0, m // 2, max(0, m - 40)}:
            for c in {0, n // 2, max(0, n - 70)}:
                h, w = min(40, m - r), min(70, n - c)
                one = capi.multiply(a2[r: r + h].contiguous().ravel(),
                                    b2[:, c: c + w].contiguous().ravel(), h, w, k)
                assert torch.equal(got[r: r + h, c: c + w], one.reshape(h, w))
        assert not out[:off].any() and not out[off + m * n:].any()


@pytest.mark.parametrize("k", [3, 8, 27, 32])
@pytest.mark.parametrize("batch,m,n", [(64, 27, 81), (200, 20, 100), (9, 27, 2187), (30, 32, 65)])
def test_batches(cuda, batch, m, n, k):
    import torch

    from jet_gb300 import capi

    a, b = _operands(cuda, batch * m * k, batch * k * n)
    got = capi.contract_batched(batch, a, [m, k], [0, 1], 1, b, [k, n], [0, 1], 1, m, n, k)
    for i in range(batch):
        one = capi.multiply(a[i * m * k:(i + 1) * m * k].clone(), b[i * k * n:(i + 1) * k * n].clone(),
                            m, n, k)
        assert torch.equal(got[i * m * n:(i + 1) * m * n], one)
