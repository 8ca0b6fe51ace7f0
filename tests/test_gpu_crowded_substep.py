"""Substeps whose cells hold more particles than are ranked one by one (needs a
GPU): 256 and 257 to a cell, in input order (whole warps of one cell) and in any
order; the sort and the state are the oracle's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    a = np.array(a, np.float32, copy=True)
    a.view(np.uint32)[np.isnan(a)] = 0x7FC00000
    return a.view(np.uint32)


@pytest.mark.parametrize("counts", [[256, 257], [1000], [31, 700, 288, 1, 33, 320], [5, 2500], [3300]])
@pytest.mark.parametrize("sort", [True, False])
def test_crowded_cells_of_a_substep(pbf_mod, oracle_mod, cuda_device, counts, sort):
    params = pbf_mod.load_scenario("dam_break_32k")
    n = params.particleCount = sum(counts)
    rng = np.random.default_rng(n)
    cell = np.repeat(np.arange(len(counts)), counts)
    if not sort:
        cell = rng.permutation(cell)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = (np.stack([2 + 3 * cell, np.full(n, 4), np.full(n, 5)], axis=1) + rng.uniform(0.1, 0.9, (n, 3))) * params.h
    vel = np.zeros_like(pos)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        for substep in (1, 2):
            sim.Step(1)
            keys, perm, cells = sim.read_sort()
            got = sim.read_state()
            *want, debug = oracle_mod.step(params, pos, vel, substep, debug=True)
            assert np.array_equal(keys, debug["keys"]) and np.array_equal(perm, debug["perm"])
            assert np.array_equal(cells, debug["cells"])
            for g, o in zip(got, want):
                assert np.array_equal(_bits(g), _bits(o))


@pytest.mark.parametrize("grid", [16, 64, 150])
@pytest.mark.parametrize("per_cell", [8, 40])
def test_keys_that_many_cells_share(pbf_mod, oracle_mod, cuda_device, grid, per_cell):
    """Runs whose candidates are many and mostly another cell's, beside runs of truly crowded cells."""
    params = pbf_mod.load_scenario("dam_break_32k")
    n = params.particleCount = 6000
    params.gridBufSize, params.boxClamp = grid, 0
    rng = np.random.default_rng(grid + per_cell)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = 0.3 + rng.random((n, 3)) * (n / per_cell) ** (1.0 / 3.0) * params.h
    vel = np.zeros_like(pos)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(2)
        got = sim.read_state()
    for g, o in zip(got, oracle_mod.step(params, pos, vel, 2)):
        assert np.array_equal(_bits(g), _bits(o))
