"""The allocation-free sort at the edges of how a cell is ordered (needs a GPU):
128 and 129 particles (compared, or sorted by a block), 4,096 and 4,097 (by a block,
or tile by tile), bitmaps and networks of every size, the most large cells there
can be, tiles with a remainder, few cells for many particles (65,536 and one more),
more than 32 particles to a key, and as many cells as there are keys; against the
oracle's stable sort.  Integers: no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {"compared": ([128], 1 << 10), "block": ([129], 1 << 10), "both": ([127, 128, 129, 130, 255, 256, 257, 1, 2], 1 << 10),
         "block_most": ([4096], 1 << 10), "large_least": ([4097], 1 << 10), "remainder": ([4097, 4095, 4096, 8191], 1 << 12),
         "apart": ([300, 513, 1025, 2049, 4096, 4097, 150000], 1 << 14), "most_large": ([4097] * 255, 1 << 17),
         "even": ([256] * 256, 1 << 12), "contended": ([256] * 256 + [1], 1 << 12), "radix": ([33] * 1986, 2048),
         "every_key": ([129] * 63 + [4200], 64), "few_keys": ([900, 5000, 1], 1023)}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("sort", [False, True])
def test_edges(pbf_mod, oracle_mod, cuda_device, name, sort):
    import torch
    dev = torch.device("cuda", cuda_device)
    counts, grid = CASES[name]
    params = pbf_mod.load_scenario("dam_break_32k")
    n = sum(counts)
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
    for _ in range(2):
        pbf_mod.sort_state_noalloc(params, d_pred.data_ptr(), d_keys.data_ptr(), d_perm.data_ptr(), d_cells.data_ptr(),
                                   torch.cuda.current_stream(dev).cuda_stream)
        torch.cuda.synchronize(dev)
        assert np.array_equal(d_keys.cpu().numpy().view(np.uint32), keys[:n])
        assert np.array_equal(d_perm.cpu().numpy().view(np.uint32), perm[:n])
        assert np.array_equal(d_cells.cpu().numpy().view(np.uint32), cells)
        d_keys.fill_(-7)
        d_perm.fill_(-7)
