"""Where a 2D solve leaves the resident kernel for the passes in parts (resident_config in
csrc/fsm_resident.cu): the choice on either side of the line, and the same results bit for bit."""

import pytest
import torch

from test_gpu_resident import BURG, NSVEL, VORT, _passes, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build,channels,shape,batch,steps,resident", [
    (VORT, 1, (128, 128), 80, 16, True), (VORT, 1, (128, 128), 200, 12, False), (VORT, 1, (128, 128), 128, 16, False),
    (VORT, 1, (128, 128), 128, 12, True),  # too few steps for parts
    (BURG, 2, (128, 128), 64, 16, True), (BURG, 2, (128, 128), 100, 16, False), (NSVEL, 2, (128, 128), 100, 16, True),
    (BURG, 2, (128, 256), 24, 16, True), (BURG, 2, (128, 256), 32, 16, False), (NSVEL, 2, (128, 256), 32, 16, True)])
def test_line_between_resident_kernel_and_parts(build, channels, shape, batch, steps, resident):
    plan, sp, u, _ = _setup(build, shape, batch, channels, 1e-3)
    assert (plan.launch_count(steps, batch) == 1) == resident
    a = sp.to_half(u).contiguous()
    b = a.clone()
    plan.integrate_half(a, steps)
    _passes(plan, b, steps)
    assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))


@pytest.mark.parametrize("batch,launches", [(8, 1), (2000, 2)])
def test_a_full_device_returns_sooner(batch, launches):
    """A batch that fills the device advances at most 256 steps a launch, others 2048; frames on either side of
    the boundary."""
    plan, sp, u, _ = _setup(VORT, (32, 32), batch, 1, 1e-3)
    assert plan.launch_count(256, batch) == 1 and plan.launch_count(258, batch) == launches
    a = sp.to_half(u).contiguous()
    b, frame = a.clone(), a.clone()
    traj = torch.empty((batch, 3) + tuple(a.shape[1:]), dtype=a.dtype, device=a.device)
    plan.integrate_half(a, 258, slots=[-1] * 255 + [0, 1, -1, 2], traj=traj)
    _passes(plan, b, 258)
    assert torch.equal(a, b) and torch.equal(traj[:, 2], a)
    for i, steps in enumerate((255, 256)):
        c = frame.clone()
        _passes(plan, c, steps)
        assert torch.equal(traj[:, i], c)
