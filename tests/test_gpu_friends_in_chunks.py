"""Friends builds of cells so full that a run's candidates pass through shared
memory in chunks of 384 (needs a GPU), with 1, 4, 8 and 16 particles to a warp:
bit for bit the oracle's substeps, with circles below, at and beyond their
limits, every friend kept or only the inner circles, and lists of one chunk and
of many."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2500, 9000, 20000, 50001])
@pytest.mark.parametrize("per_cell,fields", [(18, {}), (40, {}), (40, {"completeNeighbours": 1}),
                                             (100, {"friendsCircles": 2, "particlesPerCircle": 64}), (60, {"particlesPerCircle": 7})])
def test_crowded_cells(pbf_mod, oracle_mod, cuda_device, n, per_cell, fields):
    params = pbf_mod.load_scenario("dam_break_32k")
    params.particleCount = n
    for name, value in fields.items():
        setattr(params, name, value)
    rng = np.random.default_rng(n + per_cell)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = 0.3 + rng.random((n, 3)) * (n / per_cell) ** (1.0 / 3.0) * params.h
    vel = np.zeros_like(pos)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(1)
        got = sim.read_state()
    for g, o in zip(got, oracle_mod.step(params, pos, vel, 1)):
        assert np.array_equal(g.view(np.uint32), o.view(np.uint32))


def test_clusters(pbf_mod, oracle_mod, cuda_device):
    params = pbf_mod.load_scenario("dam_break_32k")
    n = params.particleCount = 6000
    rng = np.random.default_rng(2)
    pos = np.zeros((n, 4), np.float32)
    centre = 0.4 + rng.random((4, 3)) * 0.8
    pos[:, :3] = centre[rng.integers(0, 4, n)] + rng.normal(0.0, 0.01, (n, 3))
    vel = np.zeros_like(pos)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(1)
        got = sim.read_state()
    for g, o in zip(got, oracle_mod.step(params, pos, vel, 1)):
        assert np.array_equal(g.view(np.uint32), o.view(np.uint32))
