"""Linear symbols that differ between the channels of a velocity (a viscosity per channel): a table
set of its own per channel in every kernel that reads them. (Channels with equal symbols share one set.)"""

import math

import numpy as np
import pytest
import torch

from oracle import spectral as S
from test_gpu_adjoint import _torch_step_adjoint
from test_gpu_resident import _passes
from torchfsm_gb300 import adjoint, initial
from torchfsm_gb300.integrator import RKIntegrator, SETDRKIntegrator
from torchfsm_gb300.operator import Convection, Laplacian, NSPressureConvection

pytestmark = pytest.mark.gpu

TWO_PI = 2 * math.pi
NU = (0.05, 0.01, 0.02)


def _case(term, shape, batch, scheme=None, seed=3):
    nd = len(shape)
    nu = torch.tensor(NU[:nd], dtype=torch.float64, device="cuda").reshape((1, nd) + (1,) * nd)
    op = nu * Laplacian() + (NSPressureConvection() if term == "leray" else -Convection())
    if scheme is not None:
        op.set_integrator(scheme)
    u0 = initial.band_limited(shape, batch, nd, 4, seed, 0.3).astype(np.float32)
    return op, u0, [(0, TWO_PI, n) for n in shape]


def _exact(term, u0, mesh, dt, steps, scheme="setdrk4"):
    nd = len(mesh)
    nu = np.array(NU[:nd]).reshape((1, nd) + (1,) * nd)
    nl = [(1.0, "ns_pressure_convection")] if term == "leray" else [(-1.0, "convection")]
    return S.integrate(u0.astype(np.float64), mesh, [(nu, ("laplacian",))], nl, dt, steps, integrator=scheme)[0]


# batches that fill a cluster's shared memory with every table, and ones that leave tables in global memory
@pytest.mark.parametrize("term", ["convection", "leray"])
@pytest.mark.parametrize("shape,batch", [((32, 32), 2), ((64, 32), 5), ((128, 128), 9), ((128, 128), 60), ((64, 256), 40)])
def test_resident_kernel(term, shape, batch):
    op, u0, mesh = _case(term, shape, batch)
    dt, steps = 2e-3, 6
    got = op.integrate(u_0=torch.tensor(u0, device="cuda"), mesh=mesh, dt=dt, step=steps)
    it = op._state_dict["integrator"]
    assert it.plan.launch_count(steps, batch) == 1
    assert it.plan.tables().shape[1] == 2 * shape[0] * (shape[1] // 2 + 1)
    half = it.spectral.to_half(torch.tensor(u0, device="cuda")).contiguous()
    _passes(it.plan, half, steps)
    assert torch.equal(got, it.spectral.to_physical(half))
    ref = _exact(term, u0[:2], mesh, dt, steps)
    assert S.rel_l2(got[:2].cpu().numpy(), ref) < 1e-5  # the parity tests' bound


@pytest.mark.parametrize("term", ["convection", "leray"])
@pytest.mark.parametrize("scheme,name", [(SETDRKIntegrator.SETDRK4, "setdrk4"), (SETDRKIntegrator.SETDRK3, "setdrk3"),
                                         (RKIntegrator.RK4, "RK4")], ids=["setdrk4", "setdrk3", "rk4"])
@pytest.mark.parametrize("shape", [(512, 16), (64, 512), (16, 32, 32), (32, 16, 64), (16, 64, 128)])
def test_passes(term, scheme, name, shape):
    op, u0, mesh = _case(term, shape, 2, scheme)
    dt, steps = 2e-4, 4
    got = op.integrate(u_0=torch.tensor(u0, device="cuda"), mesh=mesh, dt=dt, step=steps)
    assert S.rel_l2(got.cpu().numpy(), _exact(term, u0, mesh, dt, steps, name)) < 1e-5


@pytest.mark.parametrize("shape", [(32, 64), (16, 16, 32)])
def test_step_adjoint(shape):
    nd, dt = len(shape), 1e-3
    op, u0, mesh = _case("convection", shape, 2)
    u0 = torch.tensor(u0, device="cuda")
    with torch.no_grad():
        op.integrate(u_0=u0, mesh=mesh, dt=dt, step=1)
    plan = op._state_dict["integrator"].plan
    h = shape[-1] // 2 + 1
    L64 = op._linear_coef64(u0.device)
    L64 = L64.expand(L64.shape[:2] + shape)[..., :h]
    adj = adjoint.ConvectionAdjoint(plan, plan.program, L64, dt)
    u = adj.sp.to_half(u0).contiguous()
    ub = (adj.sp.to_half(torch.tensor(initial.band_limited(shape, 2, nd, 7, 4, 1.0), dtype=torch.float32,
                                      device="cuda")) / adj.ntot).contiguous()
    tb = torch.zeros((6,) + tuple(u.shape), dtype=torch.float64, device="cuda")
    tb_ref = torch.zeros_like(tb)
    out, ref = adj.step_adjoint(u, ub, tb), _torch_step_adjoint(adj, u, ub, tb_ref)

    def rel(a, b):
        return float((a - b).abs().pow(2).sum().sqrt() / b.abs().pow(2).sum().sqrt())

    assert rel(out, ref) <= 1e-5  # the bound of the same comparison for one symbol
    for t in range(6):
        assert rel(tb[t], tb_ref[t]) <= 1e-5, t
