"""The launch shape that the autotuner reports (needs a GPU): the friends block size
stays the caller's where the build by warps is chosen, which has its own, instead of
the size that the fastest of equal trials happened to name."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [96, 416])
def test_friends_block_of_the_build_by_warps(pbf_mod, cuda_device, block):
    params, pos, vel = pbf_mod.make_double_dam_break(65536, 2, 3)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        shape = sim.launch_shape()
        shape[0] = block
        sim.set_launch_shape(shape)
        sim.Step(2)
        for _ in range(3):
            tuned = sim.autotune(trial_substeps=1)
            assert tuned == sim.launch_shape()
            assert tuned[5] == 1 and tuned[0] in (64, 128, 256, 512) or tuned[5] == 0 and tuned[0] == block
            sim.set_launch_shape(shape)
