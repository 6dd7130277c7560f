"""The 2D and 3D passes with an axis of 128 to 512 points, whose transforms take 16 points a lane, at both
dealias rates that have kernels of their own (the 2/3 rule's columns, every column) and for every
nonlinear term, against the FP64 oracle. These kernels run at the 128-register cap, several with spills; nvcc
13.0.88 was seen to compile packed sums wrong in a loop at that cap, and a wrong product shows here."""

import math

import numpy as np
import pytest
import torch

from oracle import spectral as S
from test_gpu_plane512 import TERMS
from test_gpu_resident import _passes
from torchfsm_gb300 import initial, pde
from torchfsm_gb300.integrator import SETDRKIntegrator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate", [2 / 3, 1.0])
@pytest.mark.parametrize("shape", [(16, 128), (16, 256), (16, 512), (128, 16), (256, 16), (512, 16)])
@pytest.mark.parametrize("term", sorted(TERMS))
def test_2d_passes(term, shape, rate):
    build, channels, lin, nl = TERMS[term]
    length = 10 * math.pi if term == "ks" else 2 * math.pi
    mesh = [(0, length, n) for n in shape]
    u0 = initial.band_limited(shape, 2, channels, 4, 7, 0.3).astype(np.float32)
    u = torch.tensor(u0, device="cuda")
    dt, steps = 1e-3, 4
    op = build()
    op.set_de_aliasing_rate(rate)
    op.integrate(u_0=u, mesh=mesh, dt=dt, step=1)
    it = op._state_dict["integrator"]
    half = it.spectral.to_half(u).contiguous()
    _passes(it.plan, half, steps)
    ref, _ = S.integrate(u0.astype(np.float64), mesh, lin, nl, dt, steps, de_aliasing_rate=rate)
    assert S.rel_l2(it.spectral.to_physical(half).cpu().numpy(), ref) < 1e-5  # the parity tests' bound
    op = build()  # a scheme dispatched at run time
    op.set_de_aliasing_rate(rate)
    op.set_integrator(SETDRKIntegrator.SETDRK3)
    got = op.integrate(u_0=u, mesh=mesh, dt=dt, step=steps)
    ref, _ = S.integrate(u0.astype(np.float64), mesh, lin, nl, dt, steps, integrator="setdrk3", de_aliasing_rate=rate)
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5


@pytest.mark.parametrize("rate", [2 / 3, 1.0])
@pytest.mark.parametrize("shape", [(128, 16, 16), (256, 16, 16), (16, 128, 64), (16, 256, 16), (16, 64, 128),
                                   (16, 16, 256), (16, 32, 256)])
@pytest.mark.parametrize("term", ["convection", "leray", "ks"])
def test_3d_passes(term, shape, rate):
    length = 10 * math.pi if term == "ks" else 2 * math.pi
    lin = [(-1.0, ("laplacian",)), (-1.0, ("biharmonic",))] if term == "ks" else [(0.05, ("laplacian",))]
    nl = {"convection": [(-1.0, "convection")], "leray": [(1.0, "ns_pressure_convection")], "ks": [(-1.0, "ks_convection")]}[term]
    op = {"convection": lambda: pde.Burgers(0.05), "leray": lambda: pde.NavierStokes(20), "ks": pde.KuramotoSivashinskyHighDim}[term]()
    op.set_de_aliasing_rate(rate)
    mesh = [(0, length, n) for n in shape]
    u0 = initial.band_limited(shape, 1, 1 if term == "ks" else 3, 3, 6, 0.3).astype(np.float32)
    got = op.integrate(u_0=torch.tensor(u0, device="cuda"), mesh=mesh, dt=1e-3, step=3)
    ref, _ = S.integrate(u0.astype(np.float64), mesh, lin, nl, 1e-3, 3, de_aliasing_rate=rate)
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5
