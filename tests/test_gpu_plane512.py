"""The 512-point register transforms of the 2D passes (16 x 2 x 16 over a full warp) in either axis,
with every nonlinear term, against the FP64 oracle; and the transforms themselves against numpy."""

import math

import numpy as np
import pytest
import torch

from oracle import spectral as S
from torchfsm_gb300 import initial, pde

pytestmark = pytest.mark.gpu

TWO_PI = 2 * math.pi
TERMS = {
    "vorticity": (lambda: pde.NavierStokesVorticity(200), 1, [(1 / 200, ("laplacian",))], [(-1.0, "vorticity_convection")]),
    "convection": (lambda: pde.Burgers(0.02), 2, [(0.02, ("laplacian",))], [(-1.0, "convection")]),
    "leray": (lambda: pde.NavierStokes(100), 2, [(0.01, ("laplacian",))], [(1.0, "ns_pressure_convection")]),
    "ks": (lambda: pde.KuramotoSivashinskyHighDim(), 1, [(-1.0, ("laplacian",)), (-1.0, ("biharmonic",))],
           [(-1.0, "ks_convection")]),
}


@pytest.mark.parametrize("term", sorted(TERMS))
@pytest.mark.parametrize("shape", [(512, 16), (16, 512), (512, 64), (64, 512)])
def test_every_term_with_a_512_point_axis(term, shape):
    build, channels, lin, nl = TERMS[term]
    length = 10 * math.pi if term == "ks" else TWO_PI
    mesh = [(0, length, n) for n in shape]
    u0 = initial.band_limited(shape, 2, channels, 4, 7, 0.3).astype(np.float32)
    dt, steps = 2e-4, 5
    got = build().integrate(u_0=torch.tensor(u0, device="cuda"), mesh=mesh, dt=dt, step=steps)
    ref, _ = S.integrate(u0.astype(np.float64), mesh, lin, nl, dt, steps)
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5  # the parity tests' bound


def test_transforms_of_512_points():
    shape = (512, 512)
    u = torch.randn((3, 1) + shape, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    op = pde.NavierStokesVorticity(100)
    op.integrate(u_0=u, mesh=[(0, TWO_PI, n) for n in shape], dt=1e-3, step=1)
    sp = op._state_dict["integrator"].spectral
    half = sp.to_half(u)
    ref = np.fft.rfftn(u.cpu().numpy().astype(np.float64), axes=(-2, -1))
    # FP32 transforms: log2(512^2) = 18 butterfly levels of 2^-24 each, rms: 18 x 6e-8
    assert S.rel_l2(torch.view_as_real(half).cpu().numpy(), np.stack([ref.real, ref.imag], -1)) < 1.1e-6
    assert S.rel_l2(sp.to_physical(half).cpu().numpy(), u.cpu().numpy()) < 2.2e-6
