"""A substep's sort by counting and by radix passes (needs a GPU): the sorted
keys, the permutation and the cell table equal the oracle's at the edges of the
rule that chooses between them (key ranges of at most 2^20, or 16 keys a
particle, and of at least one key to 64 particles are counted), of the scan's 1,024-key chunks, and of the blocks of 256
particles; also with every particle in one cell.  Integers: no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


EDGES = [
    (1, 1), (255, 1023), (256, 1024), (257, 1025), (700, 3), (3001, 4095), (3001, 4096),
    (3001, (1 << 20) - 1), (3001, 1 << 20), (3001, (1 << 20) + 1), (70001, 16 * 70001), (70001, 16 * 70001 + 1),
    (640, 10), (641, 10),  # 64 particles a key are counted, more are not
]


@pytest.mark.parametrize("n,grid", EDGES)
def test_sort_of_a_substep(pbf_mod, oracle_mod, cuda_device, n, grid):
    params = pbf_mod.load_scenario("dam_break_32k")
    params.particleCount, params.gridBufSize = n, grid
    side = int(np.ceil(n ** (1 / 3)))
    pos = pbf_mod.scene_block(side, side, side, 0.05, (0.025,) * 3, 0.02, 3)[:n].copy()
    vel = np.zeros_like(pos)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(2)
        keys, perm, cells = sim.read_sort()
        got = sim.read_state()
    *want, debug = oracle_mod.step(params, pos, vel, 2, debug=True)
    assert np.array_equal(keys, debug["keys"]) and np.array_equal(perm, debug["perm"])
    assert np.array_equal(cells, debug["cells"])
    for g, o in zip(got, want):
        assert np.array_equal(g.view(np.uint32), o.view(np.uint32))


@pytest.mark.parametrize("n,grid", EDGES + [(1 << 20, 524288), (1 << 20, 600000)])
def test_allocation_free_sort(pbf_mod, oracle_mod, cuda_device, n, grid):
    """The same edges, and the largest key range that fits its array at 2^20 particles with one that does not;
    each case twice, with and without the cell table, over what the other calls left in the array."""
    import torch
    dev = torch.device("cuda", cuda_device)
    params = pbf_mod.load_scenario("dam_break_32k")
    params.particleCount, params.gridBufSize = n, grid
    side = int(np.ceil(n ** (1 / 3)))
    pred = pbf_mod.scene_block(side, side, side, 0.05, (0.025,) * 3, 0.05, 3)[:n].copy()
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


def test_all_particles_in_one_cell(pbf_mod, oracle_mod, cuda_device):
    params = pbf_mod.load_scenario("dam_break_32k")
    params.particleCount, params.h, params.h_2 = 1500, 100.0, 1.0e4
    rng = np.random.default_rng(5)
    pos = np.zeros((1500, 4), np.float32)
    pos[:, :3] = rng.uniform(10.0, 90.0, (1500, 3))
    vel = np.zeros_like(pos)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(1)
        keys, perm, _ = sim.read_sort()
    assert np.array_equal(perm[:1500], np.arange(1500)) and len(set(keys[:1500])) == 1
