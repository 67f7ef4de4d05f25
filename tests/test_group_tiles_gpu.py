"""Grouped launches where the kernel's two ways through a tile meet: the work
limit of a tile read straight through the tables, k at the edges of eight and
of its longest k, partial and full 32 x 32 tiles, tasks without outputs, and
256 tasks in one launch.

An output of k terms is off by at most 2 k + 2 FP32 roundings of sums of |a|
|b| (|z| as |re| + |im|)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(cuda, shapes, seed):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(seed)
    tasks, host = [], []
    for batch, m, n, k in shapes:
        a = (rng.standard_normal((k, batch, m)) + 1j * rng.standard_normal((k, batch, m)))
        b = (rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k)))
        a, b = a.astype(np.complex64), b.astype(np.complex64)
        tab = lambda shape, axes: torch.from_numpy(capi.view_offsets(shape, axes)).to(cuda)  # noqa: E731
        tasks.append(dict(
            A=torch.from_numpy(a.ravel()).to(cuda), B=torch.from_numpy(b.ravel()).to(cuda),
            C=torch.full((batch * m * n + 1,), 7.0, dtype=torch.complex64, device=cuda),
            batch=batch, m=m, n=n, k=k, a_bat=tab(a.shape, [1]), a_row=tab(a.shape, [2]),
            a_col=tab(a.shape, [0]), b_bat=torch.zeros(batch, dtype=torch.int64, device=cuda),
            b_row=tab(b.shape, [1]), b_col=tab(b.shape, [0])))
        host.append((a.transpose(1, 2, 0), b.T))
    keep = capi.contract_group(tasks)
    torch.cuda.synchronize()
    for t, (a, b) in zip(tasks, host):
        got = t["C"].cpu().numpy()
        assert got[-1] == 7
        want = a.astype(np.complex128) @ b.astype(np.complex128)
        size = (np.abs(a.real) + np.abs(a.imag)).astype(float) @ (np.abs(b.real) + np.abs(b.imag))
        got = got[:-1].reshape(want.shape)
        assert np.all(np.abs(got - want) <= (2 * t["k"] + 2) * 2.0 ** -24 * size)
    del keep


@pytest.mark.parametrize("k", [1, 7, 8, 9, 16, 17, 63, 64, 65, 100])
def test_tiles(cuda, k):
    _run(cuda, [(1, 32, 32, k), (1, 33, 31, k), (2, 64, 4, k), (3, 1, 1, k), (1, 2, 100, k),
                (5, 8, 16, k), (1, 16, 32, k)], k)


def test_256_tasks_with_empty_ones(cuda):
    shapes = [(1 + i % 3, 1 + i % 5, 1 + i % 7, 1 + i % 11) for i in range(256)]
    for i in (0, 1, 100, 254):
        shapes[i] = (1, 0, 4, 2)
    _run(cuda, shapes, 1)
