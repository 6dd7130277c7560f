"""Short 1D lines (16 to 64 points) with the schemes dispatched at run time, whose update spreads the modes
over the warp (csrc/fsm_line.cu): per-sample symbols, a source per sample, recorded frames and the KS batch
mean, against the FP64 oracle."""

import numpy as np
import pytest
import torch

from oracle import spectral as S
from torchfsm_gb300 import initial, pde
from torchfsm_gb300.integrator import ETDRKIntegrator, RKIntegrator, SETDRKIntegrator
from torchfsm_gb300.operator import Convection, Laplacian
from torchfsm_gb300.traj_recorder import AutoRecorder, IntervalController

pytestmark = pytest.mark.gpu

SCHEMES = {"etdrk2": ETDRKIntegrator.ETDRK2, "setdrk1": SETDRKIntegrator.SETDRK1, "setdrk3": SETDRKIntegrator.SETDRK3,
           "RK4": RKIntegrator.RK4, "Dorpi45": RKIntegrator.Dorpi45}


@pytest.mark.parametrize("n", [16, 32, 64])
@pytest.mark.parametrize("scheme", sorted(SCHEMES))
def test_symbols_sources_and_frames_per_sample(n, scheme):
    batch, steps, dt = 5, 9, 2e-3
    mesh = [(0.0, 1.0, n)]
    u0 = initial.band_limited((n,), batch, 1, 4, n, 0.5).astype(np.float32)
    src = initial.band_limited((n,), batch, 1, 3, n + 1, 0.5).astype(np.float32)
    nu = np.linspace(0.001, 0.01, batch).reshape(batch, 1, 1)
    op = (torch.tensor(nu, device="cuda") * Laplacian() - Convection()) + torch.tensor(src, device="cuda")
    op.set_integrator(SCHEMES[scheme])
    rec = AutoRecorder(control_func=IntervalController(interval=3))
    got = op.integrate(u_0=torch.tensor(u0, device="cuda"), mesh=mesh, dt=dt, step=steps, trajectory_recorder=rec)
    src_hat = S.OMesh(mesh).fft(src.astype(np.float64))
    _, ref = S.integrate(u0.astype(np.float64), mesh, [(nu, ("laplacian",))],
                         [(-1.0, "convection"), (1.0, ("source", src_hat))], dt, steps, integrator=scheme,
                         record=lambda k: k % 3 == 0)
    assert got.shape == ref.shape
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5  # the parity tests' bound


@pytest.mark.parametrize("n", [16, 32, 64])
def test_ks_batch_mean(n):
    mesh = [(0.0, 30.0, n)]
    u0 = initial.band_limited((n,), 3, 1, 4, n, 0.5).astype(np.float32)
    op = pde.KuramotoSivashinskyHighDim()
    op.set_integrator(SETDRKIntegrator.SETDRK3)
    got = op.integrate(u_0=torch.tensor(u0, device="cuda"), mesh=mesh, dt=0.01, step=8)
    ref, _ = S.integrate(u0.astype(np.float64), mesh, [(-1.0, ("laplacian",)), (-1.0, ("biharmonic",))],
                         [(-1.0, "ks_convection")], 0.01, 8, integrator="setdrk3")
    assert S.rel_l2(got.cpu().numpy(), ref) < 1e-5
