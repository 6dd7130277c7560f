"""A value that is not finite in a mode that the dealias mask drops: the passes do not read such modes
for the nonlinear term (they skip the zero columns of mask times spectrum), so it stays in its mode, and
every physical value of the result is not finite, as with the mask multiplied."""

import math

import pytest
import torch

from torchfsm_gb300 import initial, pde

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,mode", [((16, 32, 64), (1, 2, 30)), ((16, 32, 64), (1, 14, 2)), ((16, 32, 64), (7, 2, 2)),
                                        ((16, 64, 128), (1, 2, 60)), ((16, 64, 128), (1, 30, 2)), ((32, 64), (2, 30)),
                                        ((32, 64), (14, 2)), ((256, 512), (2, 250))])
def test_infinite_dropped_mode_reaches_every_physical_value(shape, mode):
    nd = len(shape)
    u = torch.tensor(initial.band_limited(shape, 2, nd, 4, 3, 0.3), dtype=torch.float32, device="cuda")
    op = pde.Burgers(0.02)
    op.integrate(u_0=u, mesh=[(0, 2 * math.pi, n) for n in shape], dt=1e-3, step=1)
    it = op._state_dict["integrator"]
    clean = it.spectral.to_half(u).contiguous()
    half = clean.clone()
    half[(0, 0) + mode] = complex(math.inf, 0.0)
    it.plan.integrate_half(half, 3)
    it.plan.integrate_half(clean, 3)
    assert not torch.isfinite(it.spectral.to_physical(half)[0, 0]).any()
    assert torch.equal(half[1], clean[1])  # the other sample is untouched
