"""Closing steps (small outputs over a long k) on operands of small integers,
whose sums are exact in any order: a k that is left out, read twice or read
from a neighbour's place shows in any output, at every k. Interleaved operands
read in place, with the workspace that jetgpu_contract asks for and with the
least that it takes; and packed operands with ragged k, whose last tiles are
part full.

Sums of k <= 2^17 products of at most 8 stay below 2^24."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OUTPUTS = [(1, 1), (1, 5), (2, 3), (3, 4), (4, 1), (4, 4), (3, 5), (4, 5), (5, 1), (5, 4)]
PACKED = [(2, 2), (4, 8), (5, 8), (4, 9), (8, 16), (9, 16), (2, 16), (8, 17), (16, 16), (3, 31),
          (16, 32), (17, 2), (32, 16), (25, 9)]


def _draw(rng, *shape):
    return rng.integers(-2, 3, shape) + 1j * rng.integers(-2, 3, shape)


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("m,n", OUTPUTS)
@pytest.mark.parametrize("k,order", [(11, "mixed"), (12, "free first"), (14, "A in order"),
                                     (15, "free last"), (17, "mixed")])
def test_in_place(cuda, m, n, k, order, dtype):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m + 10 * n + 100 * k)
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
    a, b = _draw(rng, M * K), _draw(rng, K * N)
    want = (a.reshape([2] * (m + k)).transpose(a_perm).reshape(M, K)
            @ b.reshape([2] * (k + n)).transpose(b_perm).reshape(K, N))
    ad, bd = (torch.from_numpy(x.astype(dtype)).to(cuda) for x in (a, b))
    views = ([2] * (m + k), a_perm, bd, [2] * (k + n), b_perm, M, N, K)
    got = capi.contract(ad, *views).cpu().numpy().reshape(M, N)
    assert np.array_equal(got, want)
    least = int(capi.lib.jetgpu_contract_batched_workspace_size(
        1, m + k, capi.u64(views[0]), capi.i32(a_perm), 0, k + n, capi.u64(views[3]),
        capi.i32(b_perm), 0, M, N, K, capi.dtype_code(ad.dtype), capi.PREC_FP32))
    ws = torch.empty(max(least, 1), dtype=torch.uint8, device=cuda)
    got = capi.contract(ad, *views, workspace=ws).cpu().numpy().reshape(M, N)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("m,n", PACKED)
@pytest.mark.parametrize("k,batch", [(2048, 1), (2049, 3), (4111, 1), (20011, 2), (100003, 1)])
def test_packed(cuda, m, n, k, batch, dtype):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m + 100 * n + k)
    a, b = _draw(rng, batch, m, k), _draw(rng, batch, k, n)
    ad, bd = (torch.from_numpy(x.astype(dtype).ravel()).to(cuda) for x in (a, b))
    if batch > 1:
        got = capi.contract_batched(batch, ad, [m, k], [0, 1], 1, bd, [k, n], [0, 1], 1, m, n, k)
    else:
        got = capi.contract(ad, [m, k], [0, 1], bd, [k, n], [0, 1], m, n, k)
    assert np.array_equal(got.cpu().numpy().reshape(batch, m, n), a @ b)
