"""The 1D line kernel (csrc/fsm_line.cu) at every length it has, against the FP64 oracle: the passes
and exchanges of a transform differ with the length, and SETDRK4 keeps its state in registers up to
2048 points and in shared memory otherwise (as the other schemes do at every length)."""

import math

import numpy as np
import pytest
import torch

from oracle import spectral as S
from torchfsm_gb300 import initial, pde
from torchfsm_gb300.integrator import RKIntegrator, SETDRKIntegrator

pytestmark = pytest.mark.gpu

LENGTHS = [16, 32, 64, 128, 256, 512, 1024, 2048, 4096]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("scheme", ["setdrk4", "setdrk3", "RK4"])
def test_burgers_every_length(n, scheme):
    steps, dt, batch = 12, 0.2 / n, 3
    u0 = initial.band_limited((n,), batch, 1, 4, n, 0.5).astype(np.float32)
    op = pde.Burgers(0.01)
    if scheme == "setdrk3":
        op.set_integrator(SETDRKIntegrator.SETDRK3)
    elif scheme == "RK4":
        op.set_integrator(RKIntegrator.RK4)
        dt = min(dt, 0.5 / (0.01 * (math.pi * n) ** 2))  # inside the explicit stability limit
    got = op.integrate(u_0=torch.tensor(u0, device="cuda"), mesh=[(0, 1, n)], dt=dt, step=steps)
    ref, _ = S.integrate(u0.astype(np.float64), [(0, 1, n)], [(0.01, ("laplacian",))], [(-1.0, "convection")], dt,
                         steps, integrator=scheme)
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5  # the parity tests' bound


@pytest.mark.parametrize("n", LENGTHS)
def test_ks_batch_mean_and_dispersion_every_length(n):
    L, steps = 8 * math.pi, 8
    mesh = [(0, L, n)]
    u0 = initial.band_limited((n,), 2, 1, 4, n + 1, 0.5).astype(np.float32)
    u = torch.tensor(u0, device="cuda")
    dt = 0.02 if n <= 256 else 0.002
    got = pde.KuramotoSivashinskyHighDim().integrate(u_0=u, mesh=mesh, dt=dt, step=steps)
    ref, _ = S.integrate(u0.astype(np.float64), mesh, [(-1.0, ("laplacian",)), (-1.0, ("biharmonic",))],
                         [(-1.0, "ks_convection")], dt, steps)
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5
    # KdV: odd symbol, complex Nyquist mode
    got = pde.KortewegDeVries().integrate(u_0=u, mesh=mesh, dt=1e-4, step=steps)
    ref, _ = S.integrate(u0.astype(np.float64), mesh, [(-1.0, ("spatial_derivative", 0, 3))], [(6.0, "convection")],
                         1e-4, steps)
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5
