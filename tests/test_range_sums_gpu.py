"""Sums of the k ranges of one complex64 product (a contraction whose k is cut):
partial sums near the largest float that cancel, sums that overflow, and
cancellation among partial sums of very different size. Every partial sum here
is one operand value times 1, so the results are known exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BIG = float(np.float32(1.75 * 2.0 ** 127))  # also a TF32 and BF16 number
ROWS = [  # values at four k, one in each quarter; their exact sum rounded to a float
    ([BIG, BIG, -BIG, -1.5 * 2.0 ** 127], 2.0 ** 125),
    ([-BIG, -BIG, BIG, 1.5 * 2.0 ** 127], -(2.0 ** 125)),
    ([BIG, BIG, -BIG, -BIG], 0.0),
    ([BIG, BIG, 0.0, 0.0], np.inf),
    ([-BIG, -BIG, 0.0, -1.0], -np.inf),
    ([2.0 ** 40, 1.0, -(2.0 ** 40), 0.5], 1.5),
    ([2.0 ** 30, 1.0, 2.0 ** -20, -(2.0 ** 30)], 1.0 + 2.0 ** -20),
    ([1.0, 2.0, 3.0, 4.0], 10.0),
]


@pytest.mark.parametrize("form", ["fp32", "tf32x3", "bf16x3"])
def test_sums(cuda, form):
    import torch

    from jet_gb300 import capi

    prec = {"fp32": capi.PREC_FP32, "tf32x3": capi.PREC_TF32X3,
            "bf16x3": capi.PREC_BF16X3}[form]
    m, n, k = (64, 64, 1024) if form == "fp32" else (128, 128, 1024)
    size = [int(f(*a)) for f, a in (
        (capi.contract_workspace_size, ([m, k], [0, 1], [k, n], [0, 1], m, n, k, capi.C64, prec)),
        (capi.lib.jetgpu_contract_batched_workspace_size,
         (1, 2, capi.u64([m, k]), capi.i32([0, 1]), 0, 2, capi.u64([k, n]), capi.i32([0, 1]), 0, m,
          n, k, capi.C64, prec)))]
    assert size[0] > size[1], "k is not cut: nothing to test"
    a = np.zeros((m, k), dtype=np.complex64)
    want = np.zeros((m, n), dtype=np.complex64)
    for i in range(m):
        re, re_sum = ROWS[i % len(ROWS)]
        im, im_sum = ROWS[(i // len(ROWS)) % len(ROWS)]
        for q in range(4):
            a.real[i, q * k // 4 + 5] = re[q]
            a.imag[i, q * k // 4 + 5] = im[q]
        want.real[i], want.imag[i] = re_sum, im_sum
    b = torch.ones(k * n, dtype=torch.complex64, device=cuda)
    got = capi.contract(torch.from_numpy(a.ravel()).to(cuda), [m, k], [0, 1], b, [k, n], [0, 1], m,
                        n, k, precision=prec).cpu().numpy().reshape(m, n)
    assert np.array_equal(got.real, want.real)
    assert np.array_equal(got.imag, want.imag)
