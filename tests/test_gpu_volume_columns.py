"""The 3D passes exchange only the columns that the dealias mask keeps: the 2/3 rule's prefix, other
rates (every column), and no dealiasing, on unequal axes, against the FP64 oracle."""

import math

import pytest
import torch

from oracle import spectral as S
from torchfsm_gb300 import initial, pde

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate", [2 / 3, 0.5, 0.9, 1.0])
@pytest.mark.parametrize("term", ["convection", "leray", "ks"])
@pytest.mark.parametrize("shape", [(16, 32, 64), (64, 16, 16), (32, 128, 16)])
def test_rates_on_unequal_axes(rate, term, shape):
    length = 10 * math.pi if term == "ks" else 2 * math.pi
    channels = 1 if term == "ks" else 3
    op = {"convection": lambda: pde.Burgers(0.05), "leray": lambda: pde.NavierStokes(20),
          "ks": pde.KuramotoSivashinskyHighDim}[term]()
    lin = {"convection": [(0.05, ("laplacian",))], "leray": [(0.05, ("laplacian",))],
           "ks": [(-1.0, ("laplacian",)), (-1.0, ("biharmonic",))]}[term]
    nl = {"convection": [(-1.0, "convection")], "leray": [(1.0, "ns_pressure_convection")],
          "ks": [(-1.0, "ks_convection")]}[term]
    op.set_de_aliasing_rate(rate)
    mesh = [(0, length, n) for n in shape]
    u0 = initial.band_limited(shape, 2, channels, 3, 5, 0.3).astype("float32")
    got = op.integrate(u_0=torch.tensor(u0, device="cuda"), mesh=mesh, dt=2e-3, step=4)
    ref, _ = S.integrate(u0.astype("float64"), mesh, lin, nl, 2e-3, 4, de_aliasing_rate=rate)
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5  # the parity tests' bound


# the plane kernel at the largest plane of each y length, and the first sizes beyond it
@pytest.mark.parametrize("shape", [(16, 16, 256), (16, 32, 128), (16, 64, 64), (16, 128, 32), (16, 256, 16), (16, 64, 128),
                                   (16, 32, 32)])
@pytest.mark.parametrize("term", ["convection", "leray"])
def test_plane_kernel_sizes(term, shape):
    op = pde.Burgers(0.05) if term == "convection" else pde.NavierStokes(20)
    nl = [(-1.0, "convection")] if term == "convection" else [(1.0, "ns_pressure_convection")]
    mesh = [(0, 2 * math.pi, n) for n in shape]
    u0 = initial.band_limited(shape, 2, 3, 3, 6, 0.3).astype("float32")
    got = op.integrate(u_0=torch.tensor(u0, device="cuda"), mesh=mesh, dt=1e-3, step=3)
    ref, _ = S.integrate(u0.astype("float64"), mesh, [(0.05, ("laplacian",))], nl, 1e-3, 3)
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5  # the parity tests' bound
