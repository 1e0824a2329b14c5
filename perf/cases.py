"""The workloads by which the speed of this package is judged.

Each case is one call (or the short loop of calls) that a program built on the
package makes through its public entry points: the single-instance driver
loops of the reference, batched solves of thousands of instances in both
precisions, solves with boundaries and with the global Lax-Friedrichs flux,
the learned reconstruction, the discrete adjoint, the inverse problem and the
host-resident batch. Sizes are those of the package's own configurations and
tests, and odd sizes between them.

Initial states follow the batched configuration: a mean, an 8-mode Fourier
series with amplitudes N(0, 1)/k^2 and up to three jumps, as exact cell
averages; every second instance is a developed state instead (sawtooth fronts
with linear ramps between them, as Burgers' equation leaves them after
shocks have formed).

Work counts: bytes are one read and one write of the state per fused step (plus
the cotangent's in the reverse sweep); flops are those of the WENO-JS5 +
Rusanov + SSPRK33 step as the package's kernels count them (237 per cell and
step).
"""

from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

EPS = 1.0e-6
FLOP_STEP = 237  # per cell and SSPRK33 step
FLOP_REVERSE = 700  # per cell and reverse step (backward of the three stages)


# {{{ the cases


def listed():
    return [
        # the reference's driver loop (`for event in step(stepper, u0)`) on its
        # default grid: one small instance, a dt read back per step
        {"name": "driver_n256", "path": "driver", "n": 256, "nsteps": 20, "flux": "rusanov"},
        # the reference's adjoint driver: Lax-Friedrichs with the constant
        # reconstruction, checkpoints in memory, then adjoint_step
        {"name": "driver_adjoint_n256", "path": "driver_adjoint", "n": 256, "nsteps": 12},
        # a small parameter study: few instances, each of a few hundred cells
        {"name": "forward_f64_small", "path": "forward", "batch": 24, "nmin": 100, "nmax": 1000,
         "odd": True, "nsteps": 50, "dtype": "float64", "bc": "periodic", "flux": "rusanov",
         "layout": 1},
        # an uneven batch with sizes that divide into nothing
        {"name": "forward_f64_ragged", "path": "forward", "batch": 300, "nmin": 500, "nmax": 9000,
         "odd": True, "nsteps": 10, "dtype": "float64", "bc": "periodic", "flux": "rusanov",
         "layout": 2},
        # the batched configuration at its full size
        {"name": "forward_f64_large", "path": "forward", "batch": 4096, "nmin": 1024, "nmax": 16384,
         "odd": False, "nsteps": 2, "dtype": "float64", "bc": "periodic", "flux": "rusanov",
         "layout": 3},
        # the same batch with float32 states
        {"name": "forward_f32_large", "path": "forward", "batch": 4096, "nmin": 1024, "nmax": 16384,
         "odd": False, "nsteps": 10, "dtype": "float32", "bc": "periodic", "flux": "rusanov",
         "layout": 3},
        # inflow on the left, outflow on the right
        {"name": "forward_f64_boundary", "path": "forward", "batch": 256, "nmin": 300, "nmax": 5000,
         "odd": True, "nsteps": 10, "dtype": "float64", "bc": "dirichlet-neumann", "flux": "rusanov",
         "layout": 4},
        # the reference's default scheme (global Lax-Friedrichs), batched
        {"name": "forward_f64_lf", "path": "forward", "batch": 512, "nmin": 1024, "nmax": 4096,
         "odd": False, "nsteps": 5, "dtype": "float64", "bc": "periodic", "flux": "lf",
         "layout": 5},
        # the learned reconstruction on float64 states
        {"name": "learned_f64", "path": "learned", "batch": 768, "nmin": 1024, "nmax": 8192,
         "odd": False, "nsteps": 5, "dtype": "float64", "layout": 6},
        # gradients of a batched solve: checkpointed forward run and reverse sweep
        {"name": "adjoint_f64", "path": "adjoint", "batch": 96, "nmin": 1024, "nmax": 8192,
         "odd": False, "nsteps": 25, "dtype": "float64", "layout": 7},
        # one iteration of the LWR inverse problem with the learned scheme
        {"name": "inverse_learned_f32", "path": "inverse", "batch": 48, "nmin": 4096, "nmax": 16384,
         "odd": False, "nsteps": 49, "dtype": "float32", "layout": 8},
        # a batch that lives in host memory: copy in, steps, copy out
        {"name": "host_f64", "path": "host", "batch": 1024, "nmin": 1024, "nmax": 8192,
         "odd": False, "nsteps": 1, "dtype": "float64", "layout": 9},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["driver", "driver_adjoint", "forward", "forward", "forward", "forward",
                       "learned", "adjoint", "inverse", "host"])
    if path == "driver":
        return {"path": path, "n": _log_int(rng, 64, 65536), "nsteps": rng.randint(2, 30),
                "flux": rng.choice(["rusanov", "rusanov", "lf"])}
    if path == "driver_adjoint":
        return {"path": path, "n": _log_int(rng, 48, 2048), "nsteps": rng.randint(2, 20)}
    case = {"path": path, "nmin": _log_int(rng, 600, 2500), "odd": rng.random() < 0.5,
            "dtype": "float64", "layout": rng.randint(100, 10**6)}
    if path == "forward":
        kind = rng.choice(["f64", "f64", "f32", "bc", "lf"])
        case["nmin"] = _log_int(rng, 100, 2500)
        case["nmax"] = min(16384, _log_int(rng, case["nmin"] + 1, 12 * case["nmin"]))
        case["batch"] = _log_int(rng, 8, 1500)
        case["nsteps"] = rng.randint(2, 12)
        case["dtype"] = "float32" if kind == "f32" else "float64"
        case["bc"] = rng.choice(["dirichlet-neumann", "neumann", "dirichlet"]) if kind == "bc" else "periodic"
        case["flux"] = "lf" if kind == "lf" else "rusanov"
        return case
    case["nmax"] = min(16384, _log_int(rng, case["nmin"] + 1, 8 * case["nmin"]))
    if path == "learned":
        case.update(batch=_log_int(rng, 16, 700), nsteps=rng.randint(2, 6),
                    dtype=rng.choice(["float64", "float32"]))
    elif path == "adjoint":
        case.update(batch=_log_int(rng, 8, 80), nsteps=rng.randint(4, 25),
                    dtype=rng.choice(["float64", "float64", "float32"]))
    elif path == "inverse":
        case.update(batch=_log_int(rng, 8, 48), nsteps=rng.randint(4, 49), dtype="float32")
    else:
        case.update(batch=_log_int(rng, 64, 900), nsteps=rng.randint(1, 3))
    return case


# }}}


# {{{ inputs


def _sizes(case):
    """Cells of every instance (a plan is laid out for them once)."""
    rng = np.random.default_rng(1000 + case["layout"])
    lo, hi = case["nmin"], case["nmax"]
    if case["odd"]:
        return np.round(np.exp(rng.uniform(np.log(lo), np.log(hi), case["batch"]))).astype(np.int64)
    steps = []
    n = lo
    while n <= hi:
        steps.append(n)
        n *= 2
    return rng.choice(np.array(steps, dtype=np.int64), case["batch"])


def _coordinates(sizes, device):
    inst = torch.repeat_interleave(torch.arange(len(sizes), device=device),
                                   torch.tensor(sizes, device=device))
    off = torch.tensor(np.concatenate([[0], np.cumsum(sizes)[:-1]]), device=device)
    local = torch.arange(int(np.sum(sizes)), device=device) - off[inst]
    h = 2.0 / torch.tensor(sizes, dtype=torch.float64, device=device)[inst]
    return inst, -1.0 + local.double() * h, -1.0 + (local + 1).double() * h, h


def _fourier(rng, inst, fl, fr, h, B, scale=1.0):
    device = fl.device
    k = np.arange(1, 9)
    amp = torch.tensor(scale * rng.normal(0.0, 1.0, (B, 8)) / k**2, device=device)
    phi = torch.tensor(rng.uniform(0.0, 2.0 * np.pi, (B, 8)), device=device)
    u = torch.zeros_like(fl)
    for i in range(8):
        kp = (i + 1) * math.pi
        u += amp[inst, i] * (torch.cos(kp * fl + phi[inst, i]) - torch.cos(kp * fr + phi[inst, i])) / (kp * h)
    return u


def _burgers_state(sizes, seed, device="cuda"):
    """Packed exact cell averages of the initial states (float64)."""
    rng = np.random.default_rng(seed)
    B = len(sizes)
    inst, fl, fr, h = _coordinates(sizes, device)
    m = torch.tensor(rng.uniform(-0.5, 0.5, B), device=device)
    early = _fourier(rng, inst, fl, fr, h, B)
    nj = rng.integers(0, 4, B)
    hj = rng.uniform(-1.0, 1.0, (B, 3)) * (np.arange(3)[None, :] < nj[:, None])
    xj = torch.tensor(rng.uniform(-1.0, 1.0, (B, 3)), device=device)
    hj = torch.tensor(hj, device=device)
    for j in range(3):
        early += hj[inst, j] * torch.clamp((fr - xj[inst, j]) / h, 0.0, 1.0)
    # developed state: q fronts per period, ramps of slope 1/t between them
    q = torch.tensor(rng.integers(1, 4, B), device=device, dtype=torch.float64)[inst]
    a = torch.tensor(rng.uniform(0.2, 1.0, B), device=device)[inst]
    x0 = torch.tensor(rng.uniform(0.0, 1.0, B), device=device)[inst]

    def ramp(x):  # antiderivative of frac(q (x + 1) / 2 + x0) - 1/2, times q / 2
        s = q * (x + 1.0) / 2.0 + x0
        f = s - torch.floor(s)
        return 0.5 * f * (f - 1.0)

    late = a * (ramp(fr) - ramp(fl)) / (q * h / 2.0) + _fourier(rng, inst, fl, fr, h, B, 0.05)
    return m[inst] + torch.where(inst % 2 == 0, early, late)


def _lwr_state(sizes, seed, device="cuda"):
    """Packed densities in [0, 1]: a Fourier profile with two jam plateaus."""
    rng = np.random.default_rng(seed)
    B = len(sizes)
    inst, fl, fr, h = _coordinates(sizes, device)
    rho = 0.5 + 0.3 * _fourier(rng, inst, fl, fr, h, B)
    for _ in range(2):
        c = torch.tensor(rng.uniform(-0.8, 0.8, B), device=device)[inst]
        w = torch.tensor(rng.uniform(0.05, 0.2, B), device=device)[inst]
        part = torch.clamp((torch.minimum(fr, c + w / 2) - torch.maximum(fl, c - w / 2)) / h, 0.0, 1.0)
        rho = (1 - part) * rho + part * 0.95
    return torch.clamp(rho, 0.0, 1.0)


def _boundary_data(case, sizes, u0, seed):
    """set_boundary's arguments: inflow values near the instance's first and
    last cells, small outflow gradients."""
    if case["bc"] == "periodic":
        return None
    B = len(sizes)
    rng = np.random.default_rng(seed + 7)
    off = np.concatenate([[0], np.cumsum(sizes)])
    first = u0[torch.tensor(off[:-1], device=u0.device)]
    last = u0[torch.tensor(off[1:] - 1, device=u0.device)]
    ends = torch.stack([first, last], dim=1)[:, :, None].expand(B, 2, 3)
    dirichlet = (ends + torch.tensor(rng.normal(0.0, 0.01, (B, 2, 3)), device=u0.device)).contiguous()
    neumann = torch.tensor(rng.normal(0.0, 0.05, (B, 2)), device=u0.device)
    left, _, right = case["bc"].partition("-")
    return {"left": left, "right": right or left, "dirichlet": dirichlet, "neumann": neumann}


def _driver_state(n, seed, a=-1.0, b=1.0):
    rng = np.random.default_rng(seed)
    f = torch.linspace(a, b, n + 1, dtype=torch.float64, device="cuda")
    fl, fr, h = f[:-1], f[1:], (b - a) / n
    ph = rng.uniform(0.0, 2.0 * math.pi, 2)
    A = rng.uniform(0.3, 0.6, 2)
    k = 2.0 * math.pi / (b - a)
    u = torch.full_like(fl, 0.5)
    for i in range(2):
        kp = (i + 1) * k
        u += A[i] / (i + 1) * (torch.cos(kp * fl + ph[i]) - torch.cos(kp * fr + ph[i])) / (kp * h)
    return u


# }}}


# {{{ prepare and run


def _scheme(flux, equation="burgers", learned=False):
    from pyshocks_gb300 import burgers, reconstruction
    from pyshocks_gb300 import learned as ln

    if learned:
        rec = ln.LearnedWENO(params=ln.load_default_params())
    else:
        rec = reconstruction.make_reconstruction_from_name("wenojs53", eps=EPS)
    if equation == "lwr":
        return burgers.LWRRusanov(rec=rec)
    return burgers.make_scheme_from_name(flux, rec=rec)


def prepare(case, seed):
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import burgers, reconstruction, scalar
    from pyshocks_gb300.adjoint import CheckpointedSolve
    from pyshocks_gb300.batched import BatchedSolver, HostStepper
    from pyshocks_gb300.inverse import InverseProblem

    path = case["path"]
    s = {"case": case, "path": path}
    if path == "driver":
        n = case["n"]
        scheme = _scheme(case["flux"])
        grid = gb.make_uniform_cell_grid(a=-1.0, b=1.0, n=n, nghosts=3)
        u = _driver_state(n, seed)
        s["u0"] = torch.cat([u[-3:], u, u[:3]])
        bc = scalar.PeriodicBoundary()
        s["stepper"] = gb.timestepping.make_time_stepper(gb.bind(scheme, grid, bc), grid, bc, theta=1.0)
        return s
    if path == "driver_adjoint":
        n = case["n"]
        rec = reconstruction.make_reconstruction_from_name("default")
        scheme = burgers.make_scheme_from_name("lf", rec=rec, alpha=0.995)
        grid = gb.make_uniform_cell_grid(a=-1.5, b=1.5, n=n, nghosts=scheme.stencil_width)
        u = _driver_state(n, seed, -1.5, 1.5)
        s["u0"] = torch.cat([u[:1], u, u[-1:]])
        left, right = float(u[0]), float(u[-1])
        bc = scalar.make_dirichlet_boundary(ga=lambda t, x: torch.full_like(x, left),
                                            gb=lambda t, x: torch.full_like(x, right))
        s.update(scheme=gb.bind(scheme, grid, bc), grid=grid, bc=bc,
                 nbc=scalar.make_neumann_boundary(lambda t: 0.0))
        return s
    sizes = _sizes(case)
    dx = 2.0 / sizes.astype(np.float64)
    dtype = getattr(torch, case["dtype"])
    if path == "forward":
        s["solver"] = BatchedSolver(_scheme(case["flux"]), sizes, dx, dtype=dtype)
        s["u0"] = _burgers_state(sizes, seed)
        bc = _boundary_data(case, sizes, s["u0"], seed)
        if bc is not None:
            s["solver"].set_boundary(**bc)
        s["u0"] = s["u0"].to(dtype)
    elif path == "learned":
        s["solver"] = BatchedSolver(_scheme("rusanov", learned=True), sizes, dx, dtype=dtype)
        s["u0"] = _burgers_state(sizes, seed).to(dtype)
    elif path == "adjoint":
        solver = BatchedSolver(_scheme("rusanov"), sizes, dx, dtype=dtype, max_steps=case["nsteps"])
        s["checkpointed"] = CheckpointedSolve(solver, case["nsteps"])
        s["u0"] = _burgers_state(sizes, seed).to(dtype)
        inst, fl, fr, h = _coordinates(sizes, "cuda")
        s["target"] = s["u0"] + _fourier(np.random.default_rng(seed + 5), inst, fl, fr, h, len(sizes),
                                         0.05).to(dtype)
    elif path == "inverse":
        problem = InverseProblem(_scheme("rusanov", "lwr", learned=True), sizes, dx, case["nsteps"],
                                 dtype=dtype, lr=0.5)
        truth = _lwr_state(sizes, seed)
        problem.observe(truth)
        inst = problem.inst
        mean = torch.zeros(len(sizes), dtype=torch.float64, device="cuda").index_add_(0, inst, truth)
        s["guess"] = (mean / torch.tensor(sizes, device="cuda"))[inst]
        s["problem"] = problem
        problem.run(s["guess"], 1)  # the iteration's graph is captured once
    else:
        s["stepper"] = HostStepper(_scheme("rusanov"), sizes, dx, dtype=dtype)
        s["u_in"] = _burgers_state(sizes, seed).cpu().pin_memory()
        s["u_out"] = torch.empty_like(s["u_in"]).pin_memory()
    return s


def run(s):
    from pyshocks_gb300 import adjoint, apply_boundary, timestepping

    case, path = s["case"], s["path"]
    if path == "driver":
        for event in timestepping.step(s["stepper"], s["u0"], maxit=case["nsteps"]):
            pass
        return {"u": event.u, "t": event.t}
    if path == "driver_adjoint":
        from pyshocks_gb300.checkpointing import InMemoryCheckpoint

        grid, nbc = s["grid"], s["nbc"]
        stepper = timestepping.make_time_stepper(s["scheme"], grid, s["bc"], theta=1.0,
                                                 checkpoint=InMemoryCheckpoint("Iteration"))
        for event in timestepping.step(stepper, s["u0"], maxit=case["nsteps"]):
            pass
        for back in timestepping.adjoint_step(stepper, event.u, maxit=case["nsteps"],
                                              apply_boundary=lambda t, u, p: apply_boundary(nbc, grid, t, p)):
            pass
        return {"u": event.u, "p": back.p}
    if path in ("forward", "learned"):
        solver = s["solver"]
        solver.reset(s["u0"])
        u = solver.step(case["nsteps"])
        return {"u": u, "t": solver.time()}
    if path == "adjoint":
        u0 = s["u0"].detach().requires_grad_()
        u = adjoint.solve(u0, s["checkpointed"])
        misfit = 0.5 * ((u - s["target"]) ** 2).sum()
        misfit.backward()
        return {"u": u.detach(), "gradient": u0.grad}
    if path == "inverse":
        misfit = s["problem"].run(s["guess"], 1)
        return {"u0": s["problem"].u0, "misfit": misfit[0]}
    s["stepper"].advance(s["u_in"], s["u_out"], case["nsteps"])
    torch.cuda.current_stream().synchronize()
    return {"u": s["u_out"]}


def work(case):
    path = case["path"]
    if path == "driver":
        return {"bytes": 16 * case["n"] * case["nsteps"], "flops": FLOP_STEP * case["n"] * case["nsteps"]}
    if path == "driver_adjoint":
        # forward step and its transpose, constant reconstruction
        return {"bytes": 40 * case["n"] * case["nsteps"], "flops": 90 * case["n"] * case["nsteps"]}
    cells = int(_sizes(case).sum())
    width = 4 if case["dtype"] == "float32" else 8
    cs = cells * case["nsteps"]
    if path in ("adjoint", "inverse"):
        # forward, replay and reverse sweep: two, one and three accesses of a state
        return {"bytes": 6 * width * cs, "flops": (2 * FLOP_STEP + FLOP_REVERSE) * cs}
    return {"bytes": 2 * width * (cells if path == "host" else cs), "flops": FLOP_STEP * cs}


# }}}


# {{{ exact: the same results in 64 bits with plain torch


def _weno5(v, eps):
    """(left, right) face values of the cells with stencil v[0..4]."""

    def side(a, b, c, d, e):
        b0 = 13.0 / 12.0 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
        b1 = 13.0 / 12.0 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
        b2 = 13.0 / 12.0 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
        w0, w1, w2 = 0.1 / (eps + b0) ** 2, 0.6 / (eps + b1) ** 2, 0.3 / (eps + b2) ** 2
        f0 = (2 * a - 7 * b + 11 * c) / 6
        f1 = (-b + 5 * c + 2 * d) / 6
        f2 = (2 * c + 5 * d - e) / 6
        return (w0 * f0 + w1 * f1 + w2 * f2) / (w0 + w1 + w2)

    return side(*v[::-1]), side(*v)


def _flux(left, right, speed):
    """Numerical flux of Burgers' equation from the values of the two sides of a
    face (left: of the cell on its right)."""
    return 0.5 * (0.5 * left**2 + 0.5 * right**2) - 0.5 * speed * (left - right)


class _Packed:
    """Neighbours and per-instance maxima of a packed batch, by index tables."""

    def __init__(self, sizes, flux, bc=None):
        self.inst, _, _, self.h = _coordinates(sizes, "cuda")
        self.B, self.flux, self.bc = len(sizes), flux, bc
        n = torch.tensor(sizes, device="cuda")
        self.off = torch.cumsum(n, 0) - n
        self.n = n
        self.dx = 2.0 / n.double()
        lo, nn = self.off[self.inst], n[self.inst]
        local = torch.arange(self.inst.numel(), device="cuda") - lo
        self.at = {k: lo + (local + k) % nn for k in range(-3, 4) if k}
        self.local = local

    def shift(self, v, k, stage=0):
        """v_{i+k}; beyond a non-periodic instance's ends its ghost value."""
        if k == 0:
            return v
        w = v[self.at[k]]
        if self.bc is None:
            return w
        n = self.n[self.inst]
        pos = self.local + k
        for side, out, kind in ((0, pos < 0, self.bc["left"]), (1, pos >= n, self.bc["right"])):
            j = torch.nonzero(out).reshape(-1)
            b = self.inst[j]
            ghost = (-1 - pos[j]) if side == 0 else (pos[j] - n[j])
            if kind == "dirichlet":
                val = self.bc["dirichlet"][b, side, ghost]
            else:
                mirror = self.off[b] + (ghost if side == 0 else self.n[b] - 1 - ghost)
                val = v[mirror] - (2 * ghost + 1) * self.dx[b] * self.bc["neumann"][b, side]
            w = w.index_put((j,), val)
        return w

    def top(self, v):
        return torch.zeros(self.B, dtype=v.dtype, device=v.device).scatter_reduce(
            0, self.inst, v.detach().abs(), "amax")

    def rate(self, v):
        """dx times the operator: F_{i-1/2} - F_{i+1/2}."""
        w = [self.shift(v, k) for k in range(-3, 4)]
        _, r0 = _weno5(w[0:5], EPS)      # cell i - 1
        l1, r1 = _weno5(w[1:6], EPS)     # cell i
        l2, _ = _weno5(w[2:7], EPS)      # cell i + 1
        if self.flux == "lf":
            a = self.top(v)[self.inst]
            am = ap = a
        else:
            am = torch.maximum(w[2].abs(), w[3].abs())
            ap = torch.maximum(w[3].abs(), w[4].abs())
        return _flux(l1, r0, am) - _flux(l2, r1, ap)

    def step(self, u, dt):
        c = (dt / self.dx)[self.inst]
        k1 = u + c * self.rate(u)
        k2 = 0.75 * u + 0.25 * (k1 + c * self.rate(k1))
        return u / 3 + 2.0 / 3.0 * (k2 + c * self.rate(k2))

    def solve(self, u, nsteps):
        t = torch.zeros(self.B, dtype=torch.float64, device="cuda")
        for _ in range(nsteps):
            dt = 0.5 * self.dx / self.top(u) + 1.0e-15
            # (reverse mode recomputes each step: the whole tape would not fit)
            u = checkpoint(self.step, u, dt, use_reentrant=False) if u.requires_grad else self.step(u, dt)
            t = t + dt
        return u, t


def _exact_driver_adjoint(case, seed):
    n, nsteps = case["n"], case["nsteps"]
    dx = 3.0 / n
    nu, cfl = dx ** (0.995 - 1.0), 0.5 * dx ** (2 - 0.995)
    u = _driver_state(n, seed, -1.5, 1.5)
    left, right = u[:1].clone(), u[-1:].clone()

    def rate(v):
        v = torch.cat([left, v[1:-1], right])
        a = nu * v.abs().max()
        f = _flux(v[1:], v[:-1], a)
        zero = torch.zeros_like(f[:1])
        f = torch.cat([zero, f, zero])
        return (f[:-1] - f[1:]) / dx

    def advance(v, dt):
        k1 = v + dt * rate(v)
        k2 = 0.75 * v + 0.25 * (k1 + dt * rate(k1))
        return v / 3 + 2.0 / 3.0 * (k2 + dt * rate(k2))

    v = torch.cat([u[:1], u, u[-1:]])
    states, steps, t = [v], [], 0.0
    for _ in range(nsteps):
        dt = cfl / float(v[1:-1].abs().max()) + 1.0e-15
        v = advance(v, dt)
        steps.append((t + dt) - t)
        t = t + dt
        states.append(v)

    def ends(p):
        return torch.cat([p[1:2], p[1:-1], p[-2:-1]])

    p = ends(v)
    for m in range(nsteps - 1, -1, -1):
        w = states[m].detach().requires_grad_()
        (p,) = torch.autograd.grad(advance(w, steps[m]), w, p)
        p = ends(p)
    return {"u": v, "p": p}


def exact(case, seed):
    path = case["path"]
    if path in ("learned", "inverse"):
        return None  # the trust band switches on roundings of the network
    if path == "driver_adjoint":
        return _exact_driver_adjoint(case, seed)
    if path == "driver":
        n = case["n"]
        packed = _Packed(np.array([n]), case["flux"])
        u, t = packed.solve(_driver_state(n, seed), case["nsteps"])
        return {"u": torch.cat([u[-3:], u, u[:3]]), "t": float(t[0])}
    sizes = _sizes(case)
    if path == "forward":
        u = _burgers_state(sizes, seed)
        packed = _Packed(sizes, case["flux"], _boundary_data(case, sizes, u, seed))
        u, t = packed.solve(u.to(getattr(torch, case["dtype"])).double(), case["nsteps"])
        return {"u": u, "t": t}
    packed = _Packed(sizes, "rusanov")
    if path == "host":
        u = _burgers_state(sizes, seed)
        return {"u": packed.solve(u, case["nsteps"])[0]}
    u0 = _burgers_state(sizes, seed).to(getattr(torch, case["dtype"]))
    inst, fl, fr, h = _coordinates(sizes, "cuda")
    target = u0 + _fourier(np.random.default_rng(seed + 5), inst, fl, fr, h, len(sizes), 0.05).to(u0.dtype)
    u0 = u0.double().requires_grad_()
    u, _ = packed.solve(u0, case["nsteps"])
    (0.5 * ((u - target.double()) ** 2).sum()).backward()
    return {"u": u.detach(), "gradient": u0.grad}


# }}}
