"""Launches that a rendered frame counts (needs a GPU): those it makes, under a plain
perspective projection and under others."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,kernels", [(0, 11), (1, 4), (2, 4)])
@pytest.mark.parametrize("plain", [True, False])
def test_launches_of_a_frame(pbf_mod, cuda_device, mode, kernels, plain):
    params = pbf_mod.load_scenario("dam_break_32k")
    params.h, params.h_2 = 2.0, 4.0
    pos = pbf_mod.scene_block(8, 8, 8, 0.55, (0.3, 0.3, 0.3), 0.05, 11)
    params.particleCount = len(pos)
    cam = pbf_mod.render_camera((4.4, 8.0, 30.0), (4.4, 4.0, 4.4), (0.0, 1.0, 0.0), 45.0, 64, 48, 1.0)
    if not plain:
        cam.projection[2] = 0.01
    with pbf_mod.Simulation.create(params, pos, np.zeros_like(pos), device=cuda_device) as sim:
        before = sim.launch_count()
        sim.render_frame(cam, mode)
        assert sim.launch_count() - before == kernels
