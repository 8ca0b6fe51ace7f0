"""Each route of a substep against the oracle, named for what runs now (needs a GPU):
the friends build by warps and by threads, with the plain and the balanced thread map
and with complete neighbour sets; the shape value 2, which acts as 0; batches small
enough for one particle to a friends warp; and relaxed passes on both sides of the
edge of their shared lanes."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


def _run(pbf, params, pos, vel, substeps, device, tail):
    with pbf.Simulation.create(params, pos, vel, device=device) as sim:
        sim.set_launch_shape(sim.launch_shape()[:5] + tail)
        sim.Step(substeps)
        return sim.read_state()


@pytest.mark.parametrize("algorithm", [0, 1], ids=["warps", "threads"])
@pytest.mark.parametrize("balance", [0, 1], ids=["plain", "balanced"])
@pytest.mark.parametrize("complete", [0, 1], ids=["cut", "complete"])
def test_friends_builds(pbf_mod, oracle_mod, cuda_device, algorithm, balance, complete):
    params, pos, vel = pbf_mod.make_double_dam_break(13824, 3, 7)
    params.completeNeighbours = complete
    pos[17, 0] = np.float32(1.0e-20)  # its neighbours divide the IEEE way
    got = _run(pbf_mod, params, pos, vel, 3, cuda_device, [algorithm, balance, 0])
    assert _same(got, oracle_mod.step(params, pos, vel, 3))


def test_shape_value_2_acts_as_0(pbf_mod, cuda_device):
    params, pos, vel = pbf_mod.make_double_dam_break(5000, 2, 7)
    assert _same(_run(pbf_mod, params, pos, vel, 2, cuda_device, [2, 0, 0]),
                 _run(pbf_mod, params, pos, vel, 2, cuda_device, [0, 0, 0]))


@pytest.mark.parametrize("counts", [[1, 700, 33], [2048, 2048], [2048, 2049]])
def test_small_batches(pbf_mod, oracle_mod, cuda_device, counts):
    scenes, positions = pbf_mod.make_batch_scenes(first=len(counts))
    for p, n in zip(scenes, counts):
        p.particleCount = n
    positions = [x[:n].copy() for x, n in zip(positions, counts)]
    pos = np.concatenate(positions)
    with pbf_mod.Simulation.create(scenes, pos, np.zeros_like(pos), device=cuda_device) as sim:
        offs = sim.scene_offsets()
        sim.Step(2)
        bp, bv, _ = sim.read_state()
    for s, (p, x) in enumerate(zip(scenes, positions)):
        part = slice(int(offs[s]), int(offs[s + 1]))
        assert _same((bp[part], bv[part]), oracle_mod.step(p, x, np.zeros_like(x), 2)[:2])


@pytest.mark.parametrize("n", [4096, 4097, 16384, 16385])
def test_relaxed_lanes_keep_the_sums(pbf_mod, cuda_device, n):
    params, pos, vel = pbf_mod.make_double_dam_break(n, 2, 7)
    params.relaxedMath = 1
    vel[:, :3] = np.random.default_rng(n).normal(0.0, 0.3, (n, 3))
    shared = _run(pbf_mod, params, pos, vel, 3, cuda_device, [0, 0, 0])
    assert _same(shared, _run(pbf_mod, params, pos, vel, 3, cuda_device, [0, 0, 1]))  # persistent: one lane
