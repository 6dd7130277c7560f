"""The workloads this framework is timed on, through its public entry points.

A case names a program (``torchfsm_gb300.pde``), a periodic mesh, a batch, a time step and a
call: ``integrate`` (the final field), ``record`` (a recorded trajectory), ``grad`` (a loss and
its gradients) or ``apply`` (one evaluation of the right-hand side). Meshes have power-of-two
axes (what the library takes); batches are odd as well as even. Inputs are seeded random fields
with the spectra of this repository's own workloads. ``exact`` computes the same outputs in
float64 with plain torch on full complex spectra.
"""

from __future__ import annotations

import math

import torch

TWO_PI = 2.0 * math.pi


def _case(name, program, n, batch, steps, dt, call="integrate", every=1, length=TWO_PI):
    n = tuple(n) + (0,) * (3 - len(n))
    return {"name": name, "program": program, "n0": n[0], "n1": n[1], "n2": n[2], "batch": batch, "steps": steps,
            "dt": dt, "call": call, "every": every, "length": length}


def listed():
    return [
        # the README's first example: one small 1D solve, every frame kept (latency of one call)
        _case("burgers1d_128_b1_traj", "burgers", (128,), 1, 200, 0.01, "record", 1, 1.0),
        # a few medium 1D Kuramoto-Sivashinsky solves, as served one request at a time (odd batch)
        _case("ks1d_1024_b7", "ks", (1024,), 7, 200, 0.05, length=32 * math.pi),
        # the largest 1D request of the serving stream
        _case("ks1d_4096_b32", "ks", (4096,), 32, 100, 0.01, length=32 * math.pi),
        # the smallest 2D request of the serving stream: launches and latency
        _case("burgers2d_64_b1", "burgers", (64, 64), 1, 100, 0.005),
        # generating training trajectories: small vorticity fields, every tenth frame kept
        _case("ns2d_64_b4_traj", "vorticity", (64, 64), 4, 100, 0.005, "record", 10),
        # forced velocity Navier-Stokes (Leray projection) on a rectangular mesh, odd batch
        _case("nsvel2d_128x256_b9", "ns", (128, 256), 9, 40, 0.002),
        # this repository's headline benchmark workload, 50 of its steps
        _case("ns2d_256_b64", "vorticity", (256, 256), 64, 50, 0.001),
        # the largest 2D mesh the library takes, a few samples
        _case("ns2d_512_b5", "vorticity", (512, 512), 5, 40, 0.0005),
        # a right-hand side evaluation of a batch of fields (residuals, physics losses)
        _case("apply_ns2d_256_b16", "vorticity", (256, 256), 16, 1, 0.001, "apply"),
        # fitting initial fields and viscosities: one iteration, operator, forward, loss and backward
        _case("burgers2d_grad_128_b16", "burgers", (128, 128), 16, 50, 0.005, "grad"),
        # 3D velocity fields at a size for datasets (odd batch)
        _case("burgers3d_64_b3", "burgers", (64, 64, 64), 3, 20, 0.005),
        # the 3D benchmark workload, 4 of its steps
        _case("burgers3d_256_b1", "burgers", (256, 256, 256), 1, 4, 0.001),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["line", "line", "plane", "plane", "plane", "plane", "grad", "apply", "volume"])
    if kind == "line":
        program = rng.choice(["burgers", "ks"])
        n, batch = rng.choice([128, 256, 512, 1024, 2048, 4096]), _log_int(rng, 1, 48)
        steps = _log_int(rng, 50, 200)
        if program == "burgers":
            return _unnamed("burgers", (n,), batch, steps, min(0.01, 0.4 / n), rng, 1.0)
        return _unnamed("ks", (n,), batch, steps, 0.05 if n <= 1024 else 0.01, rng, 32 * math.pi)
    if kind == "volume":
        n = [rng.choice([32, 64, 128]) for _ in range(3)]
        batch = max(1, _log_int(rng, 1, 4))
        return _unnamed("burgers", n, batch, _log_int(rng, 4, 20), 0.2 / max(n), rng, TWO_PI)
    n = [rng.choice([32, 64, 128, 256, 512]) for _ in range(2)]
    batch = _log_int(rng, 1, max(2, min(64, 64 * 65536 // (n[0] * n[1]))))
    dt = min(0.005, 0.25 / max(n))
    program = rng.choice(["burgers", "vorticity", "vorticity", "ns"])
    if kind == "apply":
        c = _unnamed(program, n, batch, 1, dt, rng, TWO_PI)
        return dict(c, call="apply", every=1)
    if kind == "grad":
        n = [min(v, 128) for v in n]
        batch = min(batch, 16)
        return dict(_unnamed("burgers", n, batch, _log_int(rng, 10, 50), dt, rng, TWO_PI), call="grad", every=1)
    return _unnamed(program, n, batch, _log_int(rng, 10, 50), dt, rng, TWO_PI)


def _unnamed(program, n, batch, steps, dt, rng, length):
    c = _case("", program, n, batch, steps, dt, length=length)
    del c["name"]
    if rng.random() < 0.3:
        c.update(call="record", every=max(1, steps // rng.randint(2, 8)))
    return c


def _shape(case):
    return tuple(n for n in (case["n0"], case["n1"], case["n2"]) if n)


def _channels(case):
    return len(_shape(case)) if case["program"] in ("burgers", "ns") else 1


def _viscosity(case):
    """Burgers: nu; the Navier-Stokes programs: 1 / Re."""
    if case["program"] == "burgers":
        return 0.005 if len(_shape(case)) == 3 else 0.01
    return 0.001 if case["program"] == "vorticity" else 0.01


def _random_field(shape, batch, channels, spectrum, generator):
    """Gaussian random fields [batch, channels, *shape] (float64, unit RMS) whose Fourier amplitudes
    at integer wavenumber |k| are ``spectrum(|k|)``."""
    dims = tuple(range(-len(shape), 0))
    noise = torch.randn((batch, channels) + shape, dtype=torch.float64, device="cuda", generator=generator)
    k2 = 0.0
    for i, n in enumerate(shape):
        k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
        k2 = k2 + k.reshape([-1 if j == i else 1 for j in range(len(shape))]) ** 2
    u = torch.fft.ifftn(torch.fft.fftn(noise, dim=dims) * spectrum(k2.sqrt()), dim=dims).real
    return u / u.square().mean(dim=dims, keepdim=True).sqrt()


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    shape, batch, channels = _shape(case), case["batch"], _channels(case)
    if case["program"] == "vorticity":
        # shell spectrum k^4 exp(-(k/4)^2)
        amp = lambda k: torch.where(k > 0, k ** 1.5 * torch.exp(-((k / 4.0) ** 2) / 2), 0.0)  # noqa: E731
        u = _random_field(shape, batch, channels, amp, g)
    elif len(shape) == 3:
        # shell spectrum k^2 exp(-(k/3)^2)
        amp = lambda k: torch.where(k > 0, torch.exp(-((k / 3.0) ** 2) / 2), 0.0)  # noqa: E731
        u = _random_field(shape, batch, channels, amp, g)
    else:
        # band-limited Fourier series with a mean
        kmax = 8.0 if case["program"] == "ks" else 6.0
        u = _random_field(shape, batch, channels, lambda k: (k <= kmax).double(), g)
        if len(shape) == 2 or case["program"] == "burgers":
            u = 0.25 * u
        if len(shape) == 1 and case["program"] == "burgers":
            u = u + 0.5
    out = {"u0": u.float()}
    if case["call"] == "grad":
        out["nu"] = (0.01 + 0.01 * torch.rand((batch,) + (1,) * (len(shape) + 1), dtype=torch.float64, device="cuda",
                                              generator=g)).float()
        out["target"] = (0.25 * _random_field(shape, batch, channels, lambda k: (k <= 6.0).double(), g)).float()
    if case["program"] == "ns":
        # a steady body force, as a source term of the velocity equation
        f = 0.5 * _random_field(shape, 1, channels, lambda k: ((k > 2) & (k <= 4)).double(), g)
        out["force"] = f.float()
    return out


def _operator(case, data):
    from torchfsm_gb300 import operator, pde

    if case["call"] == "grad":
        return data["nu"] * operator.Laplacian() - operator.Convection()
    if case["program"] == "burgers":
        return pde.Burgers(_viscosity(case))
    if case["program"] == "ks":
        return pde.KuramotoSivashinsky()
    if case["program"] == "vorticity":
        return pde.NavierStokesVorticity(1.0 / _viscosity(case))
    return pde.NavierStokes(1.0 / _viscosity(case)) + data["force"]


def prepare(case, seed):
    from torchfsm_gb300.mesh import MeshGrid

    data = _inputs(case, seed)
    if case["call"] == "grad":
        data["u0"].requires_grad_(True)
        data["nu"].requires_grad_(True)
    mesh = MeshGrid([(0.0, case["length"], n) for n in _shape(case)], device="cuda")
    if case["call"] == "grad":  # the operator belongs to one set of viscosities: built for each iteration of a fit
        return {"case": case, "mesh": mesh, **data}
    op = _operator(case, data)
    with torch.no_grad():  # registers the mesh and builds the plan, as the first call of a program does
        if case["call"] == "apply":
            op(u=data["u0"], mesh=mesh)
        else:
            op.integrate(data["u0"], dt=case["dt"], step=1, mesh=mesh)
    return {"case": case, "op": op, **data}


def run(state):
    case, u0 = state["case"], state["u0"]
    if case["call"] == "grad":
        op = _operator(case, state)
        out = op.integrate(u0, dt=case["dt"], step=case["steps"], mesh=state["mesh"])
        loss = ((out - state["target"]) ** 2).mean()
        grad_u0, grad_nu = torch.autograd.grad(loss, (u0, state["nu"]))
        return {"field": out.detach(), "grad_u0": grad_u0, "grad_nu": grad_nu}
    op = state["op"]
    if case["call"] == "apply":
        return {"rhs": op(u=u0)}
    if case["call"] == "record":
        from torchfsm_gb300.traj_recorder import AutoRecorder, IntervalController

        recorder = AutoRecorder(control_func=IntervalController(interval=case["every"]))
        return {"trajectory": op.integrate(u0, dt=case["dt"], step=case["steps"], trajectory_recorder=recorder)}
    return {"field": op.integrate(u0, dt=case["dt"], step=case["steps"])}


def work(case):
    """Fields read and written once; the real transforms of every stage (2.5 N log2 N operations
    each) and about 40 operations per spectral point and channel for the stage's update."""
    shape, batch, c = _shape(case), case["batch"], _channels(case)
    nd, points = len(shape), math.prod(shape)
    field = 4.0 * batch * c * points
    transforms = {"vorticity": 5, "ks": 3}.get(case["program"], c * (nd + 2))
    if nd == 1:
        transforms = 3
    transform = 2.5 * points * math.log2(points)
    stages = 1 if case["call"] == "apply" else 4 * case["steps"]
    forward = batch * stages * (transforms * transform + 20.0 * c * points)
    if case["call"] == "record":
        frames = case["steps"] // case["every"] + 1
        return {"bytes": field * (1 + frames), "flops": forward + batch * c * frames * transform}
    if case["call"] == "grad":
        # the forward, its stages again, and each stage's vector-Jacobian product
        vjp = batch * stages * (c * (nd + 2) * transform + 40.0 * c * points)
        return {"bytes": 4 * field, "flops": 2 * forward + vjp}
    return {"bytes": 2 * field, "flops": forward}


# ---- float64, plain torch ------------------------------------------------------------------


class _Exact:
    """The programs on full complex spectra in float64."""

    def __init__(self, case, data):
        self.case, self.shape = case, _shape(case)
        nd = len(self.shape)
        self.dims = tuple(range(-nd, 0))
        self.k, self.mask = [], 1.0
        for i, n in enumerate(self.shape):
            view = [1, 1] + [-1 if j == i else 1 for j in range(nd)]
            f = torch.fft.fftfreq(n, case["length"] / n, dtype=torch.float64, device="cuda")
            self.k.append((2.0 * math.pi * f).reshape(view))
            keep = f.abs() <= f.abs().max() * (2.0 / 3.0)
            self.mask = self.mask * keep.double().reshape(view)
        self.lap = -sum(k * k for k in self.k)
        self.inv_lap = torch.where(self.lap == 0, 1.0, 1.0 / torch.where(self.lap == 0, 1.0, self.lap))
        self.source = self.fft(data["force"].double()) if "force" in data else None

    def fft(self, u):
        return torch.fft.fftn(u, dim=self.dims)

    def phys(self, u):
        return torch.fft.ifftn(u, dim=self.dims).real

    def symbol(self, nu):
        if self.case["program"] == "ks":
            return -self.lap - self.lap * self.lap
        return nu * self.lap

    def nonlinear(self, full):
        a = full * self.mask
        if self.case["program"] == "vorticity":
            psi = -a * self.inv_lap
            kx, ky = self.k
            return -self.fft(self.phys(1j * ky * psi) * self.phys(1j * kx * a)
                             - self.phys(1j * kx * psi) * self.phys(1j * ky * a))
        u = self.phys(a)
        conv = self.fft(sum(u[:, i:i + 1] * self.phys(1j * k * a) for i, k in enumerate(self.k)))
        if self.case["program"] != "ns":
            return -conv
        p = self.inv_lap * sum(1j * k * conv[:, i:i + 1] for i, k in enumerate(self.k))
        return torch.cat([1j * k * p for k in self.k], dim=1) - conv + self.source

    def tables(self, lin, m=16):
        """The SETDRK4 coefficients: means over m points of the unit circle around dt L."""
        dt = self.case["dt"]
        c = [0.0] * 4
        for j in range(1, m + 1):
            z = lin * dt + complex(math.cos(2 * math.pi * (j - 0.5) / m), math.sin(2 * math.pi * (j - 0.5) / m))
            e = torch.exp(z)
            terms = ((torch.exp(z / 2) - 1) / z, (-4 - z + e * (4 - 3 * z + z ** 2)) / z ** 3,
                     (2 + z + e * (z - 2)) / z ** 3, (-4 - 3 * z - z ** 2 + e * (4 - z)) / z ** 3)
            c = [a + dt * t.real / m for a, t in zip(c, terms)]
        return [torch.exp(dt * lin), torch.exp(0.5 * dt * lin)] + c

    def step(self, u, tab):
        e, e2, c1, c4, c5, c6 = tab
        n0 = self.nonlinear(u)
        a1 = e2 * u + c1 * n0
        n1 = self.nonlinear(a1)
        n2 = self.nonlinear(e2 * u + c1 * n1)
        n3 = self.nonlinear(e2 * a1 + c1 * (2 * n2 - n0))
        return e * u + c4 * n0 + 2 * c5 * (n1 + n2) + c6 * n3


def exact(case, seed):
    data = _inputs(case, seed)
    ex = _Exact(case, data)
    if case["call"] == "grad":
        return _exact_grad(case, data, ex)
    with torch.no_grad():
        u = ex.fft(data["u0"].double())
        lin = ex.symbol(_viscosity(case))
        if case["call"] == "apply":
            return {"rhs": ex.phys(lin * u + ex.nonlinear(u))}
        tab = ex.tables(lin)
        frames = []
        for i in range(case["steps"]):
            if case["call"] == "record" and i % case["every"] == 0:
                frames.append(ex.phys(u))
            u = ex.step(u, tab)
        if case["call"] == "record":
            if case["steps"] % case["every"] == 0:
                frames.append(ex.phys(u))
            return {"trajectory": torch.stack(frames, dim=1)}
        return {"field": ex.phys(u)}


def _exact_grad(case, data, ex):
    from torch.utils.checkpoint import checkpoint

    u0 = data["u0"].double().requires_grad_(True)
    nu = data["nu"].double().requires_grad_(True)
    tab = ex.tables(ex.symbol(nu))
    u = ex.fft(u0)
    for _ in range(case["steps"]):
        u = checkpoint(ex.step, u, tab, use_reentrant=False)
    out = ex.phys(u)
    loss = ((out - data["target"].double()) ** 2).mean()
    grad_u0, grad_nu = torch.autograd.grad(loss, (u0, nu))
    return {"field": out.detach(), "grad_u0": grad_u0, "grad_nu": grad_nu}
