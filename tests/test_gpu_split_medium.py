"""Batches of medium size run in a few parts once a solve has enough steps (split_parts in
csrc/fsm_api.cu): the same results as one launch sequence, bit for bit, whatever the steps between
the waits of the parts, and frames from every part."""

import numpy as np
import pytest
import torch

from test_gpu_split import _unsplit
from torchfsm_gb300 import initial, pde

pytestmark = pytest.mark.gpu


# two parts (as many as samples), three parts with an uneven last one, three channels in 3D
@pytest.mark.parametrize("build,shape,batch,channels", [
    (lambda: pde.NavierStokesVorticity(500), (512, 512), 3, 1),
    (lambda: pde.Burgers(0.02), (256, 256), 13, 2),
    (lambda: pde.NavierStokes(200), (256, 256), 14, 2),
    (lambda: pde.Burgers(0.05), (64, 64, 64), 3, 3),
    (lambda: pde.Burgers(0.05), (128, 64, 64), 2, 3)], ids=["512", "convection", "leray", "cube", "two"])
@pytest.mark.parametrize("steps", [16, 19])
def test_medium_batch_in_parts(build, shape, batch, channels, steps):
    u = torch.tensor(initial.band_limited(shape, batch, channels, 5, 3, 0.3), dtype=torch.float32, device="cuda")
    op = build()
    op.integrate(u_0=u, mesh=[(0, 2 * np.pi, n) for n in shape], dt=1e-3, step=1)
    integ = op._state_dict["integrator"]
    plan = integ.plan
    assert plan.launch_count(steps, batch) == min(3, batch) * plan.launch_count(steps, 0)
    assert plan.launch_count(15, batch) == plan.launch_count(15, 0)  # few steps: one sequence
    st0 = integ.spectral.to_half(u).contiguous()
    a, b = st0.clone(), st0.clone()
    slots = [-1] * steps + [0]
    traj = torch.empty((batch, 1) + tuple(st0.shape[1:]), dtype=torch.complex64, device="cuda")
    plan.integrate_half(a, steps, slots=slots, traj=traj)
    _unsplit(plan, b, steps)
    assert torch.equal(a, b) and torch.equal(traj[:, 0], b)
