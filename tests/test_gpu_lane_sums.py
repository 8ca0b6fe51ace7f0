"""Four and eight lanes to a particle in the solver passes (up to 24,576 and
4,096 particles; needs a GPU): bit for bit the oracle's substeps on both sides
of the edges, with lists from none to full, with every rule that changes what a
sum starts from or takes, and with positions that are not finite."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(pbf, n, **fields):
    params, pos, vel = pbf.make_double_dam_break(n, 2, 7)
    for name, value in fields.items():
        setattr(params, name, value)
    rng = np.random.default_rng(n)
    vel[:, :3] = rng.normal(0.0, 0.3, (n, 3))
    return params, pos, vel


def _bits(a):
    a = np.array(a, np.float32, copy=True)
    a.view(np.uint32)[np.isnan(a)] = 0x7FC00000
    return a.view(np.uint32)


@pytest.mark.parametrize("n", [2, 33, 4096, 4097, 24576, 24577])
def test_edges_of_the_lane_rules(pbf_mod, oracle_mod, cuda_device, n):
    params, pos, vel = _scene(pbf_mod, n)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(2)
        got = sim.read_state()
    for g, o in zip(got, oracle_mod.step(params, pos, vel, 2)):
        assert np.array_equal(g.view(np.uint32), o.view(np.uint32))


@pytest.mark.parametrize("n", [2500, 6000])
@pytest.mark.parametrize("fields", [{"completeNeighbours": 1}, {"zeroDistanceGuard": 0}, {"particlesPerCircle": 1},
                                    {"friendsCircles": 1, "particlesPerCircle": 3}, {"particlesPerCircle": 25}])
def test_lane_sums_match_oracle(pbf_mod, oracle_mod, cuda_device, n, fields):
    params, pos, vel = _scene(pbf_mod, n, **fields)
    pos[17, 0] = np.float32(1.0e-20)  # its neighbours divide the IEEE way
    pos[n - 9, 1] = np.float32("inf")
    pos[n // 2, 2] = np.float32("nan")
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(3)
        got = sim.read_state()
    for g, o in zip(got, oracle_mod.step(params, pos, vel, 3)):
        assert np.array_equal(_bits(g), _bits(o))
