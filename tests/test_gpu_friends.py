"""The friends build where its shared memory, its limits and its warps end (needs
a GPU): the builds by warps (friends algorithms 0 and 2) and by one thread per
particle (1) must give the oracle's substep bit for bit, and the same lists.

The configurations cover ragged particle counts, candidate sequences longer than
the shared buffer (split runs and chunks), more accepted candidates than the
list holds (a second walk), circles over their limit, one to eight circles, hash
collisions under a modulo that is no power of two, and cells with few particles.
Integer decisions and the exact contract: no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# name: dims, h, spacing, circles, per circle, gridBufSize
CASES = {
    "one_particle": ((1, 1, 1), 0.1, 0.05, 5, 50, 4096),
    "ragged_33": ((3, 11, 1), 0.1, 0.05, 5, 50, 4096),
    "ragged_1331": ((11, 11, 11), 0.1, 0.05, 5, 50, 4096),
    "many_candidates": ((15, 13, 14), 0.15, 0.05, 5, 50, 4096),
    "more_than_the_list": ((12, 12, 12), 0.2, 0.05, 5, 63, 4096),
    "eight_circles": ((12, 13, 11), 0.15, 0.05, 8, 64, 4096),
    "one_circle": ((12, 11, 10), 0.1, 0.05, 1, 20, 4096),
    "circles_over_their_limit": ((12, 11, 10), 0.15, 0.05, 5, 3, 4096),
    "hash_collisions": ((10, 9, 11), 0.1, 0.05, 5, 50, 61),
    "one_key": ((6, 5, 7), 0.1, 0.05, 5, 50, 1),
    "few_to_a_cell": ((14, 12, 13), 0.1, 0.09, 5, 50, 8192),
}


@pytest.mark.parametrize("name", list(CASES))
def test_builds_agree_with_the_oracle(pbf_mod, oracle_mod, cuda_device, name):
    dims, h, spacing, circles, per_circle, grid = CASES[name]
    params = pbf_mod.load_scenario("dam_break_32k")
    params.h, params.h_2 = h, np.float32(h) * np.float32(h)
    params.friendsCircles, params.particlesPerCircle, params.gridBufSize = circles, per_circle, grid
    pos = pbf_mod.scene_block(*dims, spacing, (0.02, 0.03, 0.025), 0.3 * spacing, 17)
    params.particleCount = len(pos)
    vel = np.zeros_like(pos)
    want = oracle_mod.step(params, pos, vel, 1)[:3]
    lists = []
    for algorithm in (0, 1, 2):
        with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
            sim.set_launch_shape(sim.launch_shape()[:5] + [algorithm])
            sim.Step(1)
            got = sim.read_state()
            lists.append(sim.read_friends())
        for g, o in zip(got, want):
            assert np.array_equal(g.view(np.uint32), o.view(np.uint32)), f"algorithm {algorithm}"
    for counts, rows in lists[1:]:
        assert np.array_equal(counts, lists[0][0]) and np.array_equal(rows, lists[0][1])


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.0e38])
def test_coordinates_that_are_not_finite(pbf_mod, cuda_device, value):
    params = pbf_mod.load_scenario("dam_break_32k")
    pos = pbf_mod.scene_block(9, 8, 10, 0.05, (0.02, 0.03, 0.025), 0.01, 5)
    params.particleCount = len(pos)
    pos[100, 0] = value
    pos[333, 2] = value
    lists = []
    for algorithm in (0, 1):
        with pbf_mod.Simulation.create(params, pos, np.zeros_like(pos), device=cuda_device) as sim:
            sim.set_launch_shape(sim.launch_shape()[:5] + [algorithm])
            sim.Step(1)
            lists.append(sim.read_friends())
    assert np.array_equal(lists[0][0], lists[1][0]) and np.array_equal(lists[0][1], lists[1][1])
