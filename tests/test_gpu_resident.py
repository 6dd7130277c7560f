"""The resident 2D kernel (csrc/fsm_resident.cuh) against the column and row passes: one cluster per
sample or two launches per stage, the same arithmetic, so the results are equal bit for bit. The
passes are reached through the profiled integrate, which never takes the resident kernel."""

import ctypes
import math

import numpy as np
import pytest
import torch

from oracle import spectral as S
from torchfsm_gb300 import _lib, initial, operator, pde

pytestmark = pytest.mark.gpu

TWO_PI = 2 * math.pi


def _passes(plan, state, steps):
    ws = torch.empty(plan.workspace_bytes(state.shape[0], steps), dtype=torch.uint8, device=state.device)
    ms, cnt = (ctypes.c_double * 4)(), (ctypes.c_int64 * 4)()
    _lib.check(_lib.load().fsm_integrate_profiled(
        plan.handle, state.shape[0], ctypes.c_void_p(state.data_ptr()), steps, ctypes.c_void_p(ws.data_ptr()),
        ctypes.c_size_t(ws.numel()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ms, cnt))
    torch.cuda.synchronize()


def _setup(build, shape, batch, channels, dt, seed=3):
    u0 = initial.band_limited(shape, batch, channels, 5, seed, 0.3)
    u = torch.tensor(u0, dtype=torch.float32, device="cuda")
    op = build()
    op.integrate(u_0=u, mesh=[(0, TWO_PI, n) for n in shape], dt=dt, step=1)
    integ = op._state_dict["integrator"]
    return integ.plan, integ.spectral, u, u0


VORT = lambda: pde.NavierStokesVorticity(200)  # noqa: E731
BURG = lambda: pde.Burgers(0.02)  # noqa: E731
NSVEL = lambda: pde.NavierStokes(100)  # noqa: E731


# smallest and largest axes, both orders of a rectangle, batches at one cluster, several sizes of
# cluster and more than one wave
@pytest.mark.parametrize("build,channels", [(VORT, 1), (BURG, 2), (NSVEL, 2)], ids=["vorticity", "convection", "leray"])
@pytest.mark.parametrize("shape,batch", [((32, 32), 1), ((32, 32), 161), ((64, 64), 5), ((64, 64), 33), ((32, 256), 3),
                                         ((256, 32), 17), ((128, 128), 9), ((128, 64), 2), ((64, 256), 7)])
def test_resident_equals_passes(build, channels, shape, batch):
    plan, sp, u, _ = _setup(build, shape, batch, channels, 2e-3)
    assert plan.launch_count(6, batch) == 1  # the resident kernel takes it
    a = sp.to_half(u).contiguous()
    b = a.clone()
    plan.integrate_half(a, 6)
    _passes(plan, b, 6)
    assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))


def test_resident_largest_vorticity_grid():
    plan, sp, u, _ = _setup(VORT, (256, 256), 8, 1, 1e-3)
    assert plan.launch_count(3, 8) == 1
    a = sp.to_half(u).contiguous()
    b = a.clone()
    plan.integrate_half(a, 3)
    _passes(plan, b, 3)
    assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))


def test_resident_batched_symbol_source_and_complex_symbol():
    B = 6
    nu = torch.linspace(0.01, 0.05, B, dtype=torch.float64, device="cuda").reshape(B, 1, 1, 1)
    src = torch.tensor(initial.band_limited((64, 32), B, 1, 3, 8, 0.5), dtype=torch.float32, device="cuda")
    build = lambda: nu * operator.Laplacian() + 0.7 * operator.SpatialDerivative(0, 1) - operator.VorticityConvection() + src  # noqa: E731,E501
    plan, sp, u, _ = _setup(build, (64, 32), B, 1, 2e-3)
    assert plan.launch_count(6, B) == 1
    a = sp.to_half(u).contiguous()
    b = a.clone()
    plan.integrate_half(a, 6)
    _passes(plan, b, 6)
    assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))


def test_resident_frames_equal_shorter_runs():
    plan, sp, u, _ = _setup(BURG, (64, 64), 3, 2, 2e-3)
    st0 = sp.to_half(u).contiguous()
    rec = st0.clone()
    traj = torch.empty((3, 3) + tuple(st0.shape[1:]), dtype=torch.complex64, device="cuda")
    plan.integrate_half(rec, 5, slots=[0, -1, 1, -1, -1, 2], traj=traj)
    for frame, k in enumerate((0, 2, 5)):
        ref = st0.clone()
        if k:
            _passes(plan, ref, k)
        assert torch.equal(traj[:, frame], ref)


def test_resident_long_run_of_several_launches():
    """More steps than one launch takes: the state passes from launch to launch."""
    plan, sp, u, _ = _setup(VORT, (32, 32), 2, 1, 1e-3)
    steps = 2048 + 3
    assert plan.launch_count(steps, 2) == 2
    a = sp.to_half(u).contiguous()
    b = a.clone()
    plan.integrate_half(a, steps)
    _passes(plan, b, steps)
    assert torch.equal(torch.view_as_real(a), torch.view_as_real(b))


@pytest.mark.parametrize("build,channels", [(VORT, 1), (BURG, 2)], ids=["vorticity", "convection"])
def test_resident_captured_and_without_steps(build, channels):
    """A captured call replays on the data it then finds; no steps leave the state as it was, recorded as frame 0."""
    plan, sp, u, _ = _setup(build, (64, 32), 3, channels, 2e-3)
    st0 = sp.to_half(u).contiguous()
    ref = st0.clone()
    plan.integrate_half(ref, 4)
    static = torch.zeros_like(st0)
    ws = torch.empty(plan.workspace_bytes(3, 4), dtype=torch.uint8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.integrate_half(static, 4, workspace=ws)
    for _ in range(2):
        static.copy_(st0)
        graph.replay()
        assert torch.equal(static, ref)
    still = st0.clone()
    traj = torch.zeros((3, 1) + tuple(st0.shape[1:]), dtype=torch.complex64, device="cuda")
    plan.integrate_half(still, 0, slots=[0], traj=traj)
    assert torch.equal(still, st0) and torch.equal(traj[:, 0], st0)


def test_resident_matches_the_fp64_oracle():
    shape, steps, dt = (64, 32), 20, 5e-3
    plan, sp, u, u0 = _setup(NSVEL, shape, 3, 2, dt)
    a = sp.to_half(u).contiguous()
    plan.integrate_half(a, steps)
    ref, _ = S.integrate(u0.astype(np.float32).astype(np.float64), [(0, TWO_PI, n) for n in shape],
                         [(0.01, ("laplacian",))], [(1.0, "ns_pressure_convection")], dt, steps)
    assert S.rel_l2(sp.to_physical(a).cpu().numpy(), ref) < 1e-5  # the parity tests' bound
