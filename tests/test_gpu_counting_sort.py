"""A substep's sort by counting and by radix passes (needs a GPU): the sorted
keys, the permutation and the cell table equal the oracle's at the edges of the
rule that chooses between them (key ranges of at most 2^20, or 16 keys a
particle, are counted), of the scan's 1,024-key chunks, and of the blocks of 256
particles; also with every particle in one cell.  Integers: no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,grid", [
    (1, 1), (255, 1023), (256, 1024), (257, 1025), (700, 3), (3001, 4095), (3001, 4096),
    (3001, (1 << 20) - 1), (3001, 1 << 20), (3001, (1 << 20) + 1), (70001, 16 * 70001), (70001, 16 * 70001 + 1),
])
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
