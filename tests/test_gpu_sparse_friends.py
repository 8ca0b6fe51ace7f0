"""Scenes of 600,000 particles and more, whose friends are left to one
thread per particle where most runs are short (needs a GPU): sparse, dense, mixed,
one particle fewer, and a last warp of a few; the state of two substeps is
the oracle's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spray(rng, n, per_cell, low, h):
    return low + rng.random((n, 3)) * (n / per_cell) ** (1.0 / 3.0) * h


@pytest.mark.parametrize("parts", [[(600_003, 0.5)], [(600_000, 6.0)], [(250_000, 0.3), (300_000, 8.0), (50_001, 2.2)],
                                   [(599_999, 1.0)]])
@pytest.mark.parametrize("grid", [1 << 19, 300_007, 1 << 14])
def test_sparse_warps(pbf_mod, oracle_mod, cuda_device, parts, grid):
    params = pbf_mod.load_scenario("dam_break_32k")
    n = params.particleCount = sum(count for count, _ in parts)
    params.gridBufSize, params.boxClamp, params.simIterations = grid, 0, 1
    rng = np.random.default_rng(n + grid)
    pos = np.zeros((n, 4), np.float32)
    at, low = 0, 0.3
    for count, per_cell in parts:
        x = _spray(rng, count, per_cell, low, params.h)
        pos[at:at + count, :3] = x
        at, low = at + count, float(x.max()) + 0.3
    pos[n // 3, 0] = np.float32(1.0e-20)  # its neighbours divide the IEEE way
    vel = np.zeros_like(pos)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.Step(2)
        got = sim.read_state()
    for g, o in zip(got, oracle_mod.step(params, pos, vel, 2)):
        assert np.array_equal(g.view(np.uint32), o.view(np.uint32))
