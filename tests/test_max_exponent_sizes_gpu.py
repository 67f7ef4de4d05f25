"""Max-exponent pass (jetgpu_max_exponent): sizes around its 16-byte packs and
its per-CTA share, operands that start off a 16-byte boundary, and the largest
element at either end. The exponents are exact integers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 7, 8, 255, 2047, 2048, 2049, 4099, 1245183, 1245185, 5000001]


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("offset", [0, 1])
def test_sizes_and_alignment(cuda, n, dtype, offset):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(n)
    x = (rng.uniform(0.5, 1, n) + 1j * rng.uniform(-1, -0.5, n)).astype(dtype)
    full = torch.zeros(n + offset, dtype=getattr(torch, dtype), device=cuda)
    full[offset:] = torch.from_numpy(x).to(cuda)
    if offset:
        full[0] = 2.0 ** 60  # not part of the operand
    v = full[offset:]
    # -1, or 0 where a value just under 1 has rounded up to it
    top = max(np.abs(x.real).max(), np.abs(x.imag).max())
    assert capi.max_exponent(v) == int(np.frexp(top)[1]) - 1
    for at in (0, n // 2, n - 1):
        w = full.clone()[offset:]
        w[at] = 1j * 2.0 ** 37
        assert capi.max_exponent(w) == 37
    w = full.clone()[offset:]
    w.zero_()
    assert capi.max_exponent(w) == -1000
