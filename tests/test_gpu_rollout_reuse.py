"""What a rollout leaves behind for the next one (needs a GPU): checkpoints that a
later forward pass takes up again, fewer or more of them, accumulators that the
reverse pass leaves at zero, and frames replayed from a graph in between.  Every
gradient is compared with that of a fresh context; the adjoint's sums are unordered,
so within the tolerance of the rollout's other tests, which a value left from another
pass exceeds by far.  Positions are the plain substeps', bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRAD_TOL = 1e-3


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / max(np.linalg.norm(np.ravel(b)), 1e-30))


def _scene(pbf, **fields):
    params, pos, vel = pbf.make_rollout_scene(16, 16, 16)
    for name, value in fields.items():
        setattr(params, name, value)
    vel[:, :3] = np.random.default_rng(11).normal(0.0, 0.05, (params.particleCount, 3)).astype(np.float32)
    return params, pos, vel


def _dldx(n, seed):
    g = np.zeros((n, 4), np.float32)
    g[:, :3] = np.random.default_rng(seed).normal(0.0, 1.0, (n, 3))
    return g


def _gradient(pbf, params, pos, vel, device, substeps, every, dldx):
    with pbf.Simulation.create(params, pos, vel, device=device) as sim:
        sim.rollout_forward(substeps, every)
        return sim.rollout_backward(dldx)


def _close(got, want):
    return _rel(got[0][:, :3], want[0][:, :3]) < GRAD_TOL and abs(got[1] - want[1]) < GRAD_TOL * abs(want[1]) \
        and _rel(got[2], want[2]) < GRAD_TOL


def test_rollouts_after_one_another(pbf_mod, cuda_device):
    params, pos, vel = _scene(pbf_mod)
    n = params.particleCount
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        for k, (substeps, every) in enumerate([(6, 2), (6, 6), (7, 3), (4, 1), (6, 2)]):
            sim.write_state(pos, vel)
            dldx = _dldx(n, k)
            sim.rollout_forward(substeps, every)
            first, second = sim.rollout_backward(dldx), sim.rollout_backward(dldx)
            want = _gradient(pbf_mod, params, pos, vel, cuda_device, substeps, every, dldx)
            assert _close(first, want) and _close(second, want), (substeps, every)
            sim.step_async(3)  # frames from a graph between two rollouts
            sim.synchronize()


def test_positions_are_the_substeps_of_a_graph(pbf_mod, cuda_device):
    params, pos, vel = _scene(pbf_mod)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as a, \
         pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as b:
        b.use_graph(True)
        for substeps, every in ((5, 2), (3, 3)):
            a.rollout_forward(substeps, every)
            after = a.read_state()
            a.rollout_backward(_dldx(params.particleCount, substeps))
            b.step_async(substeps)
            b.synchronize()
            want = b.read_state()
            for x, y in zip(after, want):
                assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
            # the reverse pass recomputes segments; positions, velocities and ids are put back to the rollout's end
            for x, y in zip(a.read_state()[:2], want[:2]):
                assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
            assert np.array_equal(a.read_ids(), b.read_ids())


@pytest.mark.parametrize("fields", [{"particlesPerCircle": 7}, {"friendsCircles": 2, "particlesPerCircle": 64},
                                    {"friendsCircles": 8, "particlesPerCircle": 3}])
def test_other_row_lengths_on_the_tape(pbf_mod, oracle_mod, cuda_device, fields):
    params, pos, vel = _scene(pbf_mod, **fields)
    target_params = pbf_mod.rollout_target_params(params)
    R = oracle_mod.Rollout(params, pos, vel, 4)
    target = oracle_mod.Rollout(target_params, pos, vel, 4).final_by_id32().astype(np.float64)
    _, dv64, dc64, dg64 = R.grad(target)
    _, x64 = R.replay()
    dldx = np.zeros((R.n, 4), np.float64)
    dldx[:, :3] = 2.0 * (x64[:, :3] - target[:, :3]) / (3.0 * R.n)
    _, dv32, dc32, dg32 = R.grad_f32(target, dldx)
    got = _gradient(pbf_mod, params, pos, vel, cuda_device, 4, 2, dldx.astype(np.float32))
    for g, f32, f64 in ((got[0][:, :3], dv32[:, :3], dv64[:, :3]), (got[1], dc32, dc64), (got[2], dg32, dg64)):
        assert _rel(g, f64) < max(2.0 * _rel(f32, f64), 1e-5)
