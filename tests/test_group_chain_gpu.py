"""Chains of grouped launches whose tables were uploaded beforehand
(jetgpu_contract_group_uploaded): every level reads the one before, direct and
staged tiles and tasks of no k among them, back to back and replayed from a
graph, bit for bit against one synchronised launch per level."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEVELS = 24


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("m,n", [(2, 2), (16, 16), (33, 31), (128, 64)])
def test_chain(cuda, m, n, dtype):
    import torch

    from jet_gb300 import capi

    rng = np.random.default_rng(m)
    dt = getattr(torch, dtype)
    # Level l: x[l + 1] (m x n) = x[l] (m x n) w[l] (n x n), and a task of no k
    # that clears the level's second output.
    x = torch.zeros((LEVELS + 1, m, n), dtype=dt, device=cuda)
    clear = torch.ones((LEVELS, m, n), dtype=dt, device=cuda)
    w = torch.from_numpy(((rng.standard_normal((LEVELS, n, n))
                           + 1j * rng.standard_normal((LEVELS, n, n))) / n).astype(dtype)).to(cuda)
    first = torch.from_numpy((rng.standard_normal((m, n)) + 0j).astype(dtype)).to(cuda)
    table = np.concatenate([[0], np.arange(m) * n, np.arange(n) * n, np.arange(n)]).astype(np.int64)
    tab = torch.from_numpy(table).to(cuda)
    base = tab.data_ptr()
    arr = (capi.GroupTask * (2 * LEVELS))()
    for lv in range(LEVELS):
        for q, k, c in ((arr[2 * lv], n, x[lv + 1]), (arr[2 * lv + 1], 0, clear[lv])):
            q.A, q.B, q.C = x[lv].data_ptr(), w[lv].data_ptr(), c.data_ptr()
            q.batch, q.m, q.n, q.k = 1, m, n, k
            q.a_bat = q.b_bat = base
            q.a_row, q.a_col = base + 8, base + 8 * (1 + m + n)
            q.b_row, q.b_col = base + 8 * (1 + m), base + 8 * (1 + m + n)
    raw = torch.frombuffer(bytearray(bytes(arr)), dtype=torch.uint8).to(cuda)
    size = 2 * ctypes.sizeof(capi.GroupTask)
    tiles = 2 * int(capi.lib.jetgpu_group_tiles(1, m, n))
    code = capi.dtype_code(dt)

    def chain(launch):
        x.zero_()
        x[0].copy_(first)
        clear.fill_(1)
        for lv in range(LEVELS):
            launch(raw.data_ptr() + size * lv, 2, tiles, code)

    def one_by_one(*args):
        capi.contract_group_at(*args)
        torch.cuda.synchronize()

    chain(one_by_one)
    want = x.clone()
    assert not clear.any() and want[-1].abs().max() > 0
    for _ in range(5):
        chain(capi.contract_group_uploaded)
        assert torch.equal(x, want) and not clear.any()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(capi.contract_group_uploaded)
    for _ in range(5):
        x.zero_()
        graph.replay()
        assert torch.equal(x, want) and not clear.any()
