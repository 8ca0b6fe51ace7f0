"""The direction of vorticity confinement in the reverse pass (needs a GPU).

In the interior of a lattice that turns as a rigid body eta = -G sum |omega_j| k
nearly cancels: its direction is that of the rounding errors of its sum, and its
derivative scales with 1/|eta|.  The reverse pass sums eta in FP32 over the friends
in list order with fused multiply-adds; the oracle takes the same eta and does all
else in FP64 over the same FP32 values.  Evaluated in FP32 on the
CPU, that reverse pass is 4e-7 to 9e-7 off in these scenes, and with the eta that
the forward pass sums, 1e-3 to 5e-2.  The tolerance, ten times the former, is a
hundredth of the latter.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize("substeps", [2, 4])
@pytest.mark.parametrize("dims", [(12, 11, 13), (9, 9, 9), (16, 16, 16)])
def test_reverse_pass_sums_eta_in_list_order(pbf_mod, oracle_mod, cuda_device, dims, substeps):
    params, _, vel = pbf_mod.make_rollout_scene(*dims)
    pos = pbf_mod.scene_block(*dims, 0.05, (0.025, 0.025, 0.025), 0.0, 1)
    arm = pos[:, :3] - pos[:, :3].mean(0)
    vel[:, :3] = np.cross(np.array([1.0, 0.5, 0.25]), arm).astype(np.float32)
    dldx = np.zeros((len(pos), 4), np.float32)
    dldx[:, :3] = np.random.default_rng(3).normal(0.0, 1.0, (len(pos), 3))
    want, _ = oracle_mod.rollout_grad_at(params, pos, vel, substeps, dldx)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.rollout_forward(substeps, substeps)
        got, _, _ = sim.rollout_backward(dldx)
    rel = float(np.linalg.norm(got[:, :3] - want) / np.linalg.norm(want))
    print(f"{dims}, {substeps} substeps: dv0 {rel:.2e} off")
    assert rel < TOL
