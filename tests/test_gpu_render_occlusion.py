"""The splat with occlusion bounds (needs a GPU): the images equal the oracle's bit
for bit where sprites hide one another many times over, at odd image sizes, with
sprites from one pixel to wider than the image, from inside the volume, and under
projections that are no plain perspective, which take no bounds.  Frames of
another size and mode in between leave nothing behind."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _canon(a):
    a = np.array(a, np.float32, copy=True)
    a.view(np.uint32)[np.isnan(a)] = 0x7FC00000
    return a.view(np.uint32)


# name: eye, width, height, point size, entries set in the projection
CASES = {
    "deep": ((4.4, 8.0, 30.0), 160, 120, 1.0, {}),
    "odd_size": ((4.4, 8.0, 30.0), 131, 77, 1.3, {}),
    "one_tile": ((4.4, 8.0, 30.0), 8, 8, 1.0, {}),
    "one_pixel": ((4.4, 8.0, 30.0), 1, 1, 1.0, {}),
    "small_sprites": ((4.4, 8.0, 60.0), 96, 64, 0.05, {}),
    "wide_sprites": ((4.4, 5.0, 12.0), 100, 90, 6.0, {}),
    "inside": ((4.1, 4.2, 4.3), 90, 70, 0.7, {}),
    "skewed": ((4.4, 8.0, 30.0), 120, 90, 1.0, {2: 0.01}),
    "scaled_w": ((4.4, 8.0, 30.0), 120, 90, 1.0, {11: -1.25}),
}


@pytest.mark.parametrize("name", list(CASES))
def test_frames_match_the_oracle(pbf_mod, oracle_mod, cuda_device, name):
    eye, width, height, size, entries = CASES[name]
    params = pbf_mod.load_scenario("dam_break_32k")
    params.h, params.h_2 = 2.0, 4.0
    pos = pbf_mod.scene_block(14, 15, 16, 0.55, (0.3, 0.3, 0.3), 0.05, 11)
    params.particleCount = len(pos)
    pos[:, 3] = np.linspace(0.0, 40.0, len(pos), dtype=np.float32)
    cam = pbf_mod.render_camera(eye, (4.4, 4.0, 4.4), (0.0, 1.0, 0.0), 45.0, width, height, size)
    for k, value in entries.items():
        cam.projection[k] = value
    other = pbf_mod.render_camera((9.0, 9.0, 9.0), (4.4, 4.0, 4.4), (0.0, 1.0, 0.0), 60.0, 64, 48, 0.9)
    with pbf_mod.Simulation.create(params, pos, np.zeros_like(pos), device=cuda_device) as sim:
        for mode in (0, 2, 0):
            sim.render_frame(cam, mode)
            want = oracle_mod.render(cam, mode, params, pos)
            assert np.array_equal(_canon(sim.render_read(cam, 1)), _canon(want[0])), f"splat, mode {mode}"
            assert np.array_equal(_canon(sim.render_read(cam, 0)), _canon(want[2])), f"frame, mode {mode}"
            sim.render_frame(other, 1)
