"""Small scenes, where four lanes share a particle in the solver passes (up to
16,384 particles) and the friends build takes 4, 8, 16 or 32 particles to a warp
(up to 16,384, 49,152, 196,608 and above; needs a GPU): bit for bit the oracle's
substeps on both sides of each edge, and the same with the balanced thread map
and persistent grids, which keep one lane to a particle."""
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


@pytest.mark.parametrize("n", [5, 4096, 16384, 16385, 49152, 49153, 196608, 196609])
def test_edges_of_the_small_scene_rules(pbf_mod, oracle_mod, cuda_device, n):
    params, pos, vel = _scene(pbf_mod, n)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(2)
        got = sim.read_state()
    for g, o in zip(got, oracle_mod.step(params, pos, vel, 2)):
        assert np.array_equal(g.view(np.uint32), o.view(np.uint32))


@pytest.mark.parametrize("fields", [{}, {"relaxedMath": 1}, {"completeNeighbours": 1}, {"zeroDistanceGuard": 0}])
def test_four_lanes_and_one_agree(pbf_mod, cuda_device, fields):
    params, pos, vel = _scene(pbf_mod, 6000, **fields)
    pos[17, 0] = np.float32(1.0e-20)  # a coordinate below 2^-27: its neighbours divide the IEEE way
    states = []
    for tail in ([0, 0, 0], [0, 1, 0], [0, 0, 1]):
        with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
            sim.set_launch_shape(sim.launch_shape()[:5] + tail)
            sim.Step(3)
            states.append(sim.read_state())
    for other in states[1:]:
        for a, b in zip(states[0], other):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
