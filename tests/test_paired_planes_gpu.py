"""Tensor-core contractions on paired planes (hi and lo words of a block in one
128-byte row, where k is whole blocks of 32 words, 16 of TF32) and, around
them, on planar ones: k at the edges of a block, rows at the edges of a tile,
the three kernels that write the planes (bit permutation, tiles, gather), and
batches.

The products add the terms of every accumulator in the same order on both, so
the results must equal the two-stage entry points' (jetgpu_split_planes and
jetgpu_gemm_split, planar) bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # (A shape, A order, B shape, B order, free axes of A, free axes of B)
    ([40, 33], [0, 1], [33, 50], [0, 1], 1, 1),
    ([31, 130], [1, 0], [31, 7], [0, 1], 1, 1),
    ([32, 129], [1, 0], [200, 32], [1, 0], 1, 1),
    ([63, 128], [1, 0], [63, 65], [0, 1], 1, 1),
    ([17, 300], [1, 0], [140, 17], [1, 0], 1, 1),
    ([3] * 11, [4, 1, 9, 0, 7, 10, 2, 8, 3, 6, 5], [3] * 10, [1, 7, 4, 0, 9, 2, 3, 8, 5, 6], 6, 5),
    ([3] * 12, [0, 2, 4, 6, 8, 10, 1, 3, 5, 7, 9, 11], [3] * 12,
     [11, 9, 7, 5, 3, 1, 0, 2, 4, 6, 8, 10], 6, 6),
    ([2] * 18, list(range(17, -1, -1)), [2] * 17, [3, 1, 16, 0, 5, 2, 4, 6, 15, 8, 7, 9, 10, 11,
                                                  12, 13, 14], 8, 7),
    ([2] * 12, [11, 0, 10, 1, 9, 2, 8, 3, 7, 4, 6, 5], [2] * 11, list(range(11)), 7, 6),
]


@pytest.mark.parametrize("fmt", ["tf32x3", "bf16x3", "fp16x3"])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_equals_planar_stages(cuda, case, fmt):
    import torch

    from jet_gb300 import capi

    a_shape, a_perm, b_shape, b_perm, fa, fb = CASES[case]
    m = int(np.prod([a_shape[i] for i in a_perm[:fa]]))
    k = int(np.prod([a_shape[i] for i in a_perm[fa:]]))
    n = int(np.prod([b_shape[i] for i in b_perm[len(b_perm) - fb:]]))
    gen = torch.Generator(device=cuda).manual_seed(case)
    a = torch.randn(m * k, generator=gen, device=cuda, dtype=torch.complex64)
    b = torch.randn(k * n, generator=gen, device=cuda, dtype=torch.complex64)
    prec, word, code = {"tf32x3": (capi.PREC_TF32X3, torch.float32, capi.FMT_TF32),
                        "bf16x3": (capi.PREC_BF16X3, torch.int16, capi.FMT_BF16),
                        "fp16x3": (capi.PREC_FP16X3, torch.int16, capi.FMT_FP16)}[fmt]
    # The workspace is all ones (NaN, or the largest finite words): a padding
    # word that is not written shows.
    ws = torch.full((1 << 26,), 255, dtype=torch.uint8, device=cuda)
    got = capi.contract(a, a_shape, a_perm, b, b_shape, b_perm, m, n, k, precision=prec,
                        workspace=ws)
    al = 4 if code == capi.FMT_TF32 else 8
    kp = (k + al - 1) // al * al
    e = torch.empty(2, dtype=torch.int32, device=cuda)
    capi.max_exponent(a, out=e[0:1])
    capi.max_exponent(b, out=e[1:2])
    pa = torch.empty(4 * m * kp, dtype=word, device=cuda)
    pb = torch.empty(4 * n * kp, dtype=word, device=cuda)
    bt = b_perm[len(b_perm) - fb:] + b_perm[:len(b_perm) - fb]
    fp16 = code == capi.FMT_FP16
    capi.split_planes(a, a_shape, a_perm, m, k, kp, pa, code, e_max=e[0:1] if fp16 else None)
    capi.split_planes(b, b_shape, bt, n, k, kp, pb, code, e_max=e[1:2] if fp16 else None)
    want = torch.empty(m * n, dtype=torch.complex64, device=cuda)
    capi.gemm_split(pa, pb, m, n, k, kp, want, code, e_max2=e if fp16 else None)
    if k >= 512:  # contract may cut k
        assert torch.linalg.vector_norm(got - want) <= 1e-5 * torch.linalg.vector_norm(want)
    else:
        assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("batch,m,n,k", [(3, 130, 70, 45), (5, 128, 128, 64), (2, 33, 257, 100)])
def test_batches_equal_single_products(cuda, batch, m, n, k, mode):
    import torch

    from jet_gb300 import capi

    gen = torch.Generator(device=cuda).manual_seed(batch * 10 + mode)
    a = torch.randn(batch * m * k, generator=gen, device=cuda, dtype=torch.complex64)
    b = torch.randn(batch * k * n, generator=gen, device=cuda, dtype=torch.complex64)
    if mode == 1:
        args = ([m, k], [0, 1], 1, b, [k, n], [0, 1], 1)
    else:  # one tensor whose order leads with the batch axis
        args = ([batch, m, k], [0, 1, 2], 2, b, [batch, k, n], [0, 1, 2], 2)
    got = capi.contract_batched(batch, a, *args, m, n, k, precision=capi.PREC_TF32X3)
    for i in range(batch):
        one = capi.contract(a[i * m * k:(i + 1) * m * k], [m, k], [0, 1],
                            b[i * k * n:(i + 1) * k * n], [k, n], [0, 1], m, n, k,
                            precision=capi.PREC_TF32X3)
        assert torch.equal(torch.view_as_real(got[i * m * n:(i + 1) * m * n]),
                           torch.view_as_real(one))
