"""Sprites of every width class on both sides of the particle count from which their
fragments are tested early (needs a GPU): tiny, small, as wide as a tile, and wider,
many over one another; the images equal the oracle's bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _canon(a):
    a = np.array(a, np.float32, copy=True)
    a.view(np.uint32)[np.isnan(a)] = 0x7FC00000
    return a.view(np.uint32)


@pytest.mark.parametrize("n", [99999, 100000])
@pytest.mark.parametrize("size", [0.5, 1.5, 3.0, 5.0, 8.0])
def test_frames_match_the_oracle(pbf_mod, oracle_mod, cuda_device, n, size):
    params = pbf_mod.load_scenario("dam_break_32k")
    params.particleCount, params.h, params.h_2 = n, 2.0, 4.0
    pos = pbf_mod.scene_block(47, 47, 47, 0.55, (0.3, 0.3, 0.3), 0.05, 3)[:n].copy()
    pos[:, 3] = np.linspace(0.0, 40.0, n, dtype=np.float32)
    side = 0.55 * 47
    cam = pbf_mod.render_camera((0.5 * side, 0.9 * side, 2.2 * side), (0.5 * side, 0.45 * side, 0.5 * side), (0.0, 1.0, 0.0),
                                45.0, 150, 110, size)
    with pbf_mod.Simulation.create(params, pos, np.zeros_like(pos), device=cuda_device) as sim:
        for mode in (1, 0):
            sim.render_frame(cam, mode)
            want = oracle_mod.render(cam, mode, params, pos)
            assert np.array_equal(_canon(sim.render_read(cam, 1)), _canon(want[0])), f"splat, mode {mode}"
            assert np.array_equal(_canon(sim.render_read(cam, 0)), _canon(want[2])), f"frame, mode {mode}"
