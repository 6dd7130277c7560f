"""Hand-written adjoint against the reference's autograd gradients (FP64 golden vectors)."""

import os

import numpy as np
import pytest
import torch

import cases as C
from torchfsm_gb300.operator import Convection, Laplacian

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", sorted(C.GRAD_CASES))
@pytest.mark.parametrize("checkpoint", [7, 50])
def test_adjoint_matches_reference_autograd(name, checkpoint):
    from torchfsm_gb300 import adjoint

    c = C.GRAD_CASES[name]
    g = np.load(os.path.join(GOLDEN, f"{name}.npz"))
    dev = torch.device("cuda", 0)
    u0 = torch.tensor(g["u0"], dtype=torch.float32, device=dev, requires_grad=True)
    target = torch.tensor(g["target"], dtype=torch.float32, device=dev)
    nu = torch.tensor(c["nu"], dtype=torch.float32, device=dev, requires_grad=True)
    op = nu * Laplacian() - Convection()
    with torch.no_grad():
        op.integrate(u_0=u0.detach(), mesh=c["mesh"], dt=c["dt"], step=1)
    out = adjoint.integrate_with_grad(op, u0, c["dt"], c["step"], checkpoint=checkpoint)
    loss = ((out - target) ** 2).mean()
    loss.backward()
    assert abs(loss.item() - float(g["loss"])) <= 1e-4 * float(g["loss"])
    gu = u0.grad.double().cpu().numpy()
    err_u = np.linalg.norm(gu - g["grad_u0"]) / np.linalg.norm(g["grad_u0"])
    err_nu = abs(nu.grad.item() - float(g["grad_nu"])) / abs(float(g["grad_nu"]))
    print(f"{name} checkpoint {checkpoint}: grad_u0 rel {err_u:.2e}, grad_nu rel {err_nu:.2e}")
    assert err_u <= 1e-4 and err_nu <= 1e-4


def test_integrate_autograd_entry():
    """op.integrate itself routes to the adjoint when the input or nu requires grad."""
    c = C.GRAD_CASES["grad_burgers1d_n64"]
    g = np.load(os.path.join(GOLDEN, "grad_burgers1d_n64.npz"))
    dev = torch.device("cuda", 0)
    u0 = torch.tensor(g["u0"], dtype=torch.float32, device=dev, requires_grad=True)
    nu = torch.tensor(c["nu"], dtype=torch.float32, device=dev, requires_grad=True)
    op = nu * Laplacian() - Convection()
    out = op.integrate(u_0=u0, mesh=c["mesh"], dt=c["dt"], step=c["step"])
    loss = ((out - torch.tensor(g["target"], dtype=torch.float32, device=dev)) ** 2).mean()
    loss.backward()
    err_nu = abs(nu.grad.item() - float(g["grad_nu"])) / abs(float(g["grad_nu"]))
    assert err_nu <= 1e-4


def _torch_step_adjoint(adj, u, ub, tbar):
    """One SETDRK4 adjoint step as tensor arithmetic (tables from the FP64 contour formulas, the
    nonlinear term and its vector-Jacobian product from ConvectionAdjoint)."""
    E, E2, c1, c4, c5, c6 = adj.tabs
    fl = []
    n0 = adj.nonlinear(u, fl)
    a1 = E2 * u + c1 * n0
    n1 = adj.nonlinear(a1, fl)
    a2 = E2 * u + c1 * n1
    n2 = adj.nonlinear(a2, fl)
    a3 = E2 * a1 + c1 * (2 * n2 - n0)
    n3 = adj.nonlinear(a3, fl)

    def acc(t, x, y):
        tbar[t] += (x.conj() * y).real.double()

    u_bar = E * ub
    acc(0, ub, u)
    n0b = c4 * ub
    acc(3, ub, n0)
    n1b = 2 * c5 * ub
    n2b = 2 * c5 * ub
    acc(4, ub, 2 * (n1 + n2))
    n3b = c6 * ub
    acc(5, ub, n3)
    a3b = adj.nonlinear_vjp(a3, n3b, fl[3])
    a1b = E2 * a3b
    acc(1, a3b, a1)
    n2b = n2b + 2 * c1 * a3b
    n0b = n0b - c1 * a3b
    acc(2, a3b, 2 * n2 - n0)
    a2b = adj.nonlinear_vjp(a2, n2b, fl[2])
    u_bar = u_bar + E2 * a2b
    acc(1, a2b, u)
    n1b = n1b + c1 * a2b
    acc(2, a2b, n1)
    a1b = a1b + adj.nonlinear_vjp(a1, n1b, fl[1])
    u_bar = u_bar + E2 * a1b
    acc(1, a1b, u)
    n0b = n0b + c1 * a1b
    acc(2, a1b, n0)
    return u_bar + adj.nonlinear_vjp(u, n0b, fl[0])


@pytest.mark.parametrize("name", sorted(C.GRAD_CASES))
def test_native_step_adjoint_matches_tensor_formulation(name):
    """fsm_step_adjoint (fused kernels, the plan's tables) against the same step written as
    FP32 tensor arithmetic: the state cotangent and the six table cotangents."""
    from torchfsm_gb300 import adjoint

    c = C.GRAD_CASES[name]
    g = np.load(os.path.join(GOLDEN, f"{name}.npz"))
    dev = torch.device("cuda", 0)
    op = c["nu"] * Laplacian() - Convection()
    u0 = torch.tensor(g["u0"], dtype=torch.float32, device=dev)
    with torch.no_grad():
        op.integrate(u_0=u0, mesh=c["mesh"], dt=c["dt"], step=1)
    plan = op._state_dict["integrator"].plan
    h = plan.shape[-1] // 2 + 1
    L64 = op._linear_coef64(dev)
    L64 = L64.expand(L64.shape[:2] + tuple(plan.shape))[..., :h]
    adj = adjoint.ConvectionAdjoint(plan, plan.program, L64, c["dt"])
    u = adj.sp.to_half(u0).contiguous()
    gen = torch.Generator().manual_seed(5)
    ub = (adj.sp.to_half(torch.randn(tuple(u0.shape), generator=gen).to(dev)) / adj.ntot).contiguous()
    tb_native = torch.zeros((6,) + tuple(u.shape), dtype=torch.float64, device=dev)
    tb_torch = torch.zeros_like(tb_native)
    out_native = adj.step_adjoint(u, ub, tb_native)
    out_torch = _torch_step_adjoint(adj, u, ub, tb_torch)
    torch.cuda.synchronize()

    def rel(a, b):
        return float((a - b).abs().pow(2).sum().sqrt() / b.abs().pow(2).sum().sqrt())

    assert rel(out_native, out_torch) <= 1e-5
    for t in range(6):
        assert rel(tb_native[t], tb_torch[t]) <= 1e-5, t
    # without table cotangents the state cotangent is the same
    out2 = adj.step_adjoint(u, ub, None)
    assert torch.equal(out2, out_native)


@pytest.mark.parametrize("name", sorted(C.GENERIC_GRAD_CASES))
def test_recomputed_segments_match_reference_autograd(name):
    """Programs outside the hand-written Convection adjoint (vorticity NS, high-dimensional KS, KdV):
    the fused forward with checkpoints, segments recomputed in torch arithmetic and differentiated by
    autograd, against the reference's float64 autograd."""
    case = C.GENERIC_GRAD_CASES[name]
    g = np.load(os.path.join(GOLDEN, f"{name}.npz"))
    dev = torch.device("cuda", 0)
    M = C.namespace("torchfsm_gb300")
    coef = torch.tensor(case["coef"], dtype=torch.float32, device=dev, requires_grad=True)
    op = C.build_generic_grad_op(name, M, coef)
    u0 = torch.tensor(g["u0"], dtype=torch.float32, device=dev, requires_grad=True)
    target = torch.tensor(g["target"], dtype=torch.float32, device=dev)
    out = op.integrate(u_0=u0, mesh=case["mesh"], dt=case["dt"], step=case["step"])
    loss = ((out - target) ** 2).mean()
    loss.backward()
    ref_u = g["grad_u0"]
    err_u = float(np.linalg.norm(u0.grad.cpu().numpy() - ref_u) / np.linalg.norm(ref_u))
    err_c = abs(coef.grad.item() - float(g["grad_coef"])) / abs(float(g["grad_coef"]))
    # 1e-4, or twice the reference's own float32 autograd error where that floor is higher (KdV: the
    # i k^3 symbol amplifies every step's rounding; the reference's FP32 gradient is 1.9e-4 off)
    tol_u = max(1e-4, 2 * float(g["fp32_grad_u0_rel_l2"]))
    tol_c = max(1e-4, 2 * float(np.nan_to_num(g["fp32_grad_coef_rel"])))  # NaN: the float32 autograd is NaN
    print(f"{name}: grad u0 rel-L2 {err_u:.2e} (bound {tol_u:.1e}), grad coef rel {err_c:.2e} (bound {tol_c:.1e})")
    assert err_u <= tol_u and err_c <= tol_c


def test_table_derivatives_of_the_library_match_the_contour_formulas():
    """fsm_adj_table_derivs over both of its branches (series for |dt L| < 0.5, closed forms above)
    and the switch between them, against the contour means in float64."""
    from torchfsm_gb300 import _lib, adjoint

    dt = 0.01
    z = torch.cat([torch.tensor([0.0, -1e-9, 1e-6, -0.4999999, -0.5, 0.5, 0.4999999, 3.0]),
                   -torch.logspace(-6, 3, 400)]).double().cuda()
    L = (z / dt).contiguous()
    out = torch.empty((6, L.numel()), dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().fsm_adj_table_derivs(L.numel(), L.data_ptr(), dt, out.data_ptr(),
                                                torch.cuda.current_stream().cuda_stream))
    ref = adjoint._table_derivatives(L.to(torch.complex128), dt, 32, 2.0)
    for t in range(6):
        # at |z| = 0.5 the closed forms lose 4/z^4 x 2^-53 x ~10 = 7e-14 of values of order 0.1
        scale = ref[t].abs().max()
        assert float((out[t] - ref[t]).abs().max() / scale) < 1e-11, t


@pytest.mark.parametrize("shape,batch", [((16, 16), 1), ((32, 64), 3), ((64, 32), 2), ((16, 128), 5), ((128, 256), 1),
                                         ((16, 512), 2), ((512, 16), 1)])
def test_2d_step_adjoint_every_row_length(shape, batch):
    """The fused row kernel of the 2D adjoint step at every last-axis length, batches of one and odd
    ones, against the step written as FP32 tensor arithmetic."""
    from torchfsm_gb300 import adjoint, initial

    dev = torch.device("cuda", 0)
    dt = 1e-3
    mesh = [(0.0, 2 * np.pi, n) for n in shape]
    op = 0.02 * Laplacian() - Convection()
    u0 = torch.tensor(initial.band_limited(shape, batch, 2, 5, 3, 0.5), dtype=torch.float32, device=dev)
    with torch.no_grad():
        op.integrate(u_0=u0, mesh=mesh, dt=dt, step=1)
    plan = op._state_dict["integrator"].plan
    h = shape[-1] // 2 + 1
    L64 = op._linear_coef64(dev)
    L64 = L64.expand(L64.shape[:2] + tuple(shape))[..., :h]
    adj = adjoint.ConvectionAdjoint(plan, plan.program, L64, dt)
    u = adj.sp.to_half(u0).contiguous()
    ub = (adj.sp.to_half(torch.tensor(initial.band_limited(shape, batch, 2, 7, 4, 1.0), dtype=torch.float32,
                                      device=dev)) / adj.ntot).contiguous()
    tb = torch.zeros((6,) + tuple(u.shape), dtype=torch.float64, device=dev)
    tb_ref = torch.zeros_like(tb)
    out, ref = adj.step_adjoint(u, ub, tb), _torch_step_adjoint(adj, u, ub, tb_ref)
    torch.cuda.synchronize()

    def rel(a, b):
        return float((a - b).abs().pow(2).sum().sqrt() / b.abs().pow(2).sum().sqrt())

    assert rel(out, ref) <= 1e-5  # the bound of the same comparison above
    for t in range(6):
        assert rel(tb[t], tb_ref[t]) <= 1e-5, t
