"""Where a 2D solve leaves the resident kernel for the passes in parts (resident_config in
csrc/fsm_resident.cu): the choice on either side of the line, and the same results bit for bit."""

import pytest
import torch

from test_gpu_resident import BURG, NSVEL, VORT, _passes, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build,channels,batch,steps,resident", [
    (VORT, 1, 80, 16, True), (VORT, 1, 200, 12, False), (VORT, 1, 128, 16, False),
    (VORT, 1, 128, 12, True),  # too few steps for parts
    (BURG, 2, 64, 16, True), (BURG, 2, 100, 16, False), (NSVEL, 2, 100, 16, True)])
def test_line_between_resident_kernel_and_parts(build, channels, batch, steps, resident):
    plan, sp, u, _ = _setup(build, (128, 128), batch, channels, 2e-3)
    assert (plan.launch_count(steps, batch) == 1) == resident
    a = sp.to_half(u).contiguous()
    b = a.clone()
    plan.integrate_half(a, steps)
    _passes(plan, b, steps)
    assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))
