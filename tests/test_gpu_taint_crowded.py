"""Irregular positions that the position pass makes among crowded cells (needs a
GPU): the box's low wall at 1e-20, so that every particle it stops has a coordinate
below 2^-27 and all around it divide the IEEE way, with cells of a few particles and
of many more than one lane marks alone; bit for bit the oracle's substeps."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2500, 6000, 30000])
@pytest.mark.parametrize("per_cell", [6, 31, 33, 400])
def test_wall_of_irregular_positions(pbf_mod, oracle_mod, cuda_device, n, per_cell):
    params = pbf_mod.load_scenario("dam_break_32k")
    params.particleCount, params.simIterations = n, 2
    params.xMin = params.yMin = params.zMin = np.float32(1.0e-20)
    params.boxClamp = 1
    rng = np.random.default_rng(n + per_cell)
    pos = np.zeros((n, 4), np.float32)
    side = min((n / per_cell) ** (1.0 / 3.0), 10.0)
    pos[:, :3] = rng.random((n, 3)) * side * params.h
    vel = np.zeros_like(pos)
    vel[:, :3] = rng.normal(-1.0, 1.0, (n, 3))  # towards the low walls
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(2)
        got = sim.read_state()
    want = oracle_mod.step(params, pos, vel, 2)
    assert (np.abs(want[0][:, :3]) == np.float32(1.0e-20)).any()
    for g, o in zip(got, want):
        assert np.array_equal(g.view(np.uint32), o.view(np.uint32))
