"""The allocation-free sort with crowded cells (needs a GPU): cells on both
sides of the edges between comparisons, a block and several to a cell (1,024 and 16,384
particles), bitmaps of one word to a thread and of the most (32), everything in one
cell, and cells whose indices lie together or apart; against the oracle's stable sort.  Integers: no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [[1024], [1025], [1, 5, 15, 16, 17, 18, 33, 64, 511, 1023, 1024, 1025, 5000, 16384, 16385, 40000],
                                    [1100] * 400, [32768], [32769], [1 << 20], [3, (1 << 20) - 3]])
@pytest.mark.parametrize("sort", [False, True])
def test_crowded_cells(pbf_mod, oracle_mod, cuda_device, counts, sort):
    import torch
    dev = torch.device("cuda", cuda_device)
    params = pbf_mod.load_scenario("dam_break_32k")
    n, grid = sum(counts), 1 << 17
    params.particleCount, params.gridBufSize = n, grid
    rng = np.random.default_rng(len(counts))
    cell = np.repeat(np.arange(len(counts)), counts)
    if not sort:
        cell = rng.permutation(cell)
    pred = np.zeros((n, 4), np.float32)
    pred[:, :3] = (np.stack([cell % 8, cell // 8 % 8, cell // 64], axis=1) + rng.uniform(0.2, 0.8, (n, 3))) * params.h
    keys, perm, cells = oracle_mod.sort(params, pred)
    d_pred = torch.from_numpy(pred).to(dev)
    d_keys, d_perm, d_cells = (torch.full((k,), -7, dtype=torch.int32, device=dev) for k in (n, n, 2 * grid))
    for table in (d_cells.data_ptr(), None):
        pbf_mod.sort_state_noalloc(params, d_pred.data_ptr(), d_keys.data_ptr(), d_perm.data_ptr(), table,
                                   torch.cuda.current_stream(dev).cuda_stream)
        torch.cuda.synchronize(dev)
        assert np.array_equal(d_keys.cpu().numpy().view(np.uint32), keys[:n])
        assert np.array_equal(d_perm.cpu().numpy().view(np.uint32), perm[:n])
        d_keys.fill_(-7)
        d_perm.fill_(-7)
    assert np.array_equal(d_cells.cpu().numpy().view(np.uint32), cells)
