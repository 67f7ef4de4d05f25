"""BF16x3 products whose Ar B and Ai B terms are summed apart: sizes around a
tile, a stage (32 k) and a chunk (128 k), in both layouts of the stages.

Bound, elementwise against sum |a| |b| (with |z| as |re| + |im|): the split
x = hi + lo + d has |d| <= 2^-18 |x|, and lo lo <= 2^-18 |a| |b| is dropped, so
a product is off by at most 3 * 2^-18; the 24 tensor-core sums of a chunk and
the FP32 folds add at most 2^-18 more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 2])
@pytest.mark.parametrize("m,n,k", [(2, 2, 1), (128, 128, 31), (129, 127, 32), (130, 64, 33),
                                   (127, 257, 127), (256, 128, 128), (65, 129, 129),
                                   (384, 200, 257), (1000, 500, 1031)])
def test_tile_stage_and_chunk_edges(cuda, m, n, k, variant):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m * 7 + n * 3 + k)
    a = (rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))).astype(np.complex64)
    b = (rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))).astype(np.complex64)
    capi.set_tc_variant(variant)
    try:
        got = capi.contract(torch.from_numpy(a.T.copy().ravel()).to(cuda), [k, m], [1, 0],
                            torch.from_numpy(b.ravel()).to(cuda), [k, n], [0, 1], m, n, k,
                            precision=capi.PREC_BF16X3).cpu().numpy().reshape(m, n)
    finally:
        capi.set_tc_variant(0)
    want = a.astype(np.complex128) @ b.astype(np.complex128)
    size = (np.abs(a.real) + np.abs(a.imag)).astype(float) @ (np.abs(b.real) + np.abs(b.imag))
    assert np.all(np.abs(got - want) <= 4 * 2.0 ** -18 * size)
