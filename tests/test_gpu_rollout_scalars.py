"""dL/d viscosityFactor over many particles (needs a GPU).

Every block of every substep but the last adds its part to one total.  Rounded to
FP32 at each of them, the total of the 16,384 additions here drifts by some 1e-6; in
64 bits it keeps the accuracy of its terms, whose factors (POLY6, the XSPH factor, the
result itself) are each rounded to FP32 once: 6e-8 apiece.  The adjoint of the
velocities is along the velocities themselves, so that the terms have one sign.  The
tolerance is eight roundings of 6e-8.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 5e-7


@pytest.mark.parametrize("dims, substeps", [((64, 64, 64), 3), ((64, 32, 32), 9)])
def test_viscosity_gradient_of_many_blocks(pbf_mod, oracle_mod, cuda_device, dims, substeps):
    params, pos, vel = pbf_mod.make_rollout_scene(*dims)
    vel[:, :3] = np.random.default_rng(5).normal(0.0, 0.05, (len(pos), 3)).astype(np.float32)
    dldx = vel.copy()
    _, want = oracle_mod.rollout_grad_at(params, pos, vel, substeps, dldx)
    with pbf_mod.Simulation.create(params, pos, vel, device=cuda_device) as sim:
        sim.rollout_forward(substeps, substeps)
        got = [sim.rollout_backward(dldx)[1] for _ in range(3)]
    rel = [abs(g - want) / abs(want) for g in got]
    print(f"{dims}, {substeps} substeps: dL/d viscosityFactor {want:.6e}, off by {rel}")
    assert max(rel) < TOL
