"""The calls whose time counts: what users of the solver run, through its public
entry points, over the grid sizes, step counts, schemes and options they use.

``listed()`` names the fixed cases and ``draw(rng)`` gives further ones of the
same ranges; ``prepare`` makes what a program holds before the call (inputs on
the GPU, a solver or an ensemble handle), ``run`` is one pass, ``work`` the
bytes and operations a pass cannot do without, and ``exact`` the same outputs
from plain torch in float64.

Launch shapes are the library's defaults: a program that does not call the
autotuner gets them.  Time steps keep every run well conditioned (see
``_stable_dt``), so outputs of different rounding can be compared.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ns_solver_jax_differential_distributed_gb300 as nsgb
from ns_solver_jax_differential_distributed_gb300 import ensemble as ens

TWO_PI = 2.0 * math.pi
DEV = "cuda"


def _f32(x: float) -> float:
    return float(np.float32(x))


def _stable_dt(N: int, nu: float, scheme: str) -> float:
    """A time step at which rounding noise does not grow: states have rms speed
    1 (maximum about 3) on [0, 2 pi]^2.  Upwind: a tenth of the grid spacing,
    half the diffusive limit.  Central with forward Euler also needs
    (u dt / dx)^2 / 2 near the diffusion number."""
    dx = TWO_PI / N
    return _f32(min(0.1 * dx, dx * dx / (8.0 * nu), 1e-3 if scheme == "central" else 5e-3))


# ------------------------------------------------------------------- cases
def listed():
    return [
        # one solver step of the smallest grids: a caller that steps by itself
        # (its own forcing schedule, a coupled model); launches and host time
        {"name": "step_n64", "kind": "step", "N": 64, "scheme": "central", "theta_len": 2},
        # ChorinProjector.step with an explicit force field, the strategy-object
        # API, at an ordinary size
        {"name": "projector_n512", "kind": "projector", "N": 512, "scheme": "upwind"},
        # the single operators of PeriodicDifferentialOps and the advection
        # schemes, one after another, as custom projectors compose them
        {"name": "operators_n2048", "kind": "operators", "N": 2048, "scheme": "central"},
        # the spectral pressure solve alone, at the largest supported grid
        {"name": "poisson_n8192", "kind": "poisson", "N": 8192},
        # the reference's default grid: CLI runs, studies and parity checks
        {"name": "rollout_n128", "kind": "rollout", "N": 128, "scheme": "central", "steps": 100, "theta_len": 3},
        # an ordinary production rollout (sample configuration's N = 1024)
        {"name": "rollout_n1024", "kind": "rollout", "N": 1024, "scheme": "central", "steps": 101, "theta_len": 3},
        # the headline grid, fewer steps than the benchmark's 200
        {"name": "rollout_n4096", "kind": "rollout", "N": 4096, "scheme": "upwind", "steps": 48, "theta_len": 3},
        # jit_gradient from the zero state as the reference's gradient
        # benchmark and its optimiser study call it (N = 128, 328 steps)
        {"name": "jit_gradient_n128", "kind": "jit_gradient", "N": 128, "scheme": "central", "steps": 328,
         "every": 0, "theta_len": 2},
        # a differentiable rollout inside a torch program: J.backward() to theta
        # and u0, with checkpoints (a served gradient's interval of 50)
        {"name": "autograd_n256", "kind": "autograd", "N": 256, "scheme": "upwind", "steps": 150, "every": 50,
         "theta_len": 3},
        # the differentiation benchmark's grid and scheme, every state kept
        {"name": "gradient_n1024", "kind": "gradient", "N": 1024, "scheme": "upwind", "steps": 100, "every": 0,
         "theta_len": 3},
        # an ensemble of uneven solves, sizes drawn as in the ensemble benchmark
        {"name": "ensemble_60", "kind": "ensemble", "members": 60, "scheme": "central", "steps": 100, "n_max": 512},
        # gradient requests of mixed size and length advanced in lock-step, as
        # the serving loop batches them (checkpoints every 50 steps)
        {"name": "grad_batch_12", "kind": "grad_batch", "members": 12, "scheme": "upwind", "steps_min": 40,
         "steps_max": 140, "every": 50, "n_max": 512},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2(rng, lo: int, hi: int) -> int:
    return 1 << rng.randint(lo.bit_length() - 1, hi.bit_length() - 1)


def draw(rng):
    kind = rng.choice(["step", "projector", "operators", "poisson", "rollout", "rollout", "rollout",
                       "jit_gradient", "gradient", "gradient", "autograd", "ensemble", "grad_batch"])
    scheme = rng.choice(["central", "upwind"])
    tl = rng.choice([2, 3])
    if kind == "step":
        return {"kind": kind, "N": _pow2(rng, 16, 4096), "scheme": scheme, "theta_len": tl}
    if kind == "projector":
        return {"kind": kind, "N": _pow2(rng, 16, 4096), "scheme": scheme}
    if kind == "operators":
        return {"kind": kind, "N": _pow2(rng, 16, 4096), "scheme": scheme}
    if kind == "poisson":
        return {"kind": kind, "N": _pow2(rng, 16, 8192)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(8, 60), "scheme": scheme, "steps": _log_int(rng, 17, 120),
                "n_max": rng.choice([256, 512])}
    if kind == "grad_batch":
        lo = _log_int(rng, 20, 60)
        return {"kind": kind, "members": rng.randint(3, 12), "scheme": scheme, "steps_min": lo,
                "steps_max": lo + rng.randint(10, 60), "every": rng.choice([1, 7, 50]),
                "n_max": rng.choice([256, 512])}
    if kind == "rollout":
        N = _pow2(rng, 16, 4096)
        return {"kind": kind, "N": N, "scheme": scheme, "steps": _log_int(rng, 1, 300 if N <= 1024 else 48),
                "theta_len": tl}
    # gradients: every = 0 leaves the checkpoint policy to the solver
    N = _pow2(rng, 16, 1024)
    return {"kind": kind, "N": N, "scheme": scheme, "steps": _log_int(rng, 9, 200 if N <= 512 else 100),
            "every": rng.choice([0, 1, 7, 50]), "theta_len": tl}


# ------------------------------------------------------------------ inputs
def _u0(N: int, seed: int) -> torch.Tensor:
    """Divergence-free velocity of rms speed 1 from a random streamfunction of
    the modes 1 <= |k| <= min(32, N/4), amplitude |k|^-3 (the workloads'
    initial states, formed on the GPU)."""
    K = min(32, N // 4)
    g = torch.Generator().manual_seed(seed)
    c = torch.randn(2 * K + 1, K + 1, 2, generator=g, dtype=torch.float64)
    kx = torch.arange(-K, K + 1, dtype=torch.float64)[:, None]
    ky = torch.arange(0, K + 1, dtype=torch.float64)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    amp = torch.where((k >= 1) & (k <= K), k.clamp(min=1.0) ** -3.0, torch.zeros_like(k))
    psi = torch.view_as_complex(c) * amp
    out = []
    for h in (1j * ky * psi, -1j * kx * psi):
        full = torch.zeros(N, N // 2 + 1, dtype=torch.complex128, device=DEV)
        h = h.to(DEV)
        full[: K + 1, : K + 1] = h[K:]
        full[N - K:, : K + 1] = h[:K]
        out.append(torch.fft.irfft2(full, s=(N, N)))
    u = torch.stack(out)
    return (u / torch.sqrt((u[0] ** 2 + u[1] ** 2).mean())).to(torch.float32).contiguous()


def _theta(nu: float, n: int, rng) -> np.ndarray:
    th = np.array([1.0, 0.5, nu]) * (1.0 + 0.2 * rng.uniform(-1.0, 1.0, 3))
    return th[:n].astype(np.float32)


def _nu(scheme: str) -> float:
    return 1e-3 if scheme == "central" else 5e-4


def _solver(case, nu: float):
    N = case["N"]
    every = case.get("every", 0)
    return nsgb.SingleCoreNSSolver(
        nsgb.make_grid(N, TWO_PI), nsgb.Phys(nu=nu, mu0=0.5, sigma0=0.1, C=1.0),
        nsgb.Time(dt=_stable_dt(N, nu, case["scheme"]), steps=case.get("steps", 1)), case["scheme"],
        checkpoint_every=every or None)


def _members(case, seed: int):
    """(N, nu, theta, steps, u0 seed) of an ensemble's or a batch's members."""
    rng = np.random.default_rng(seed)
    # sizes are a draw of their own, the same for every seed: the work of a
    # case does not change with its inputs
    sizes = np.random.default_rng(case["members"])
    out = []
    for i in range(case["members"]):
        if case["kind"] == "ensemble":
            N = int(sizes.choice([64, 128, 256, 512], p=[0.4, 0.3, 0.2, 0.1]))
            steps = case["steps"]
            nu = float(np.exp(rng.uniform(math.log(1e-3), math.log(1e-2))))
        else:
            N = int(sizes.choice([128, 256, 512]))
            steps = int(sizes.integers(case["steps_min"], case["steps_max"] + 1))
            nu = _nu(case["scheme"])
        th = _theta(nu, 3, rng)
        out.append((min(N, case["n_max"]), nu, th, steps, seed * 1009 + i))
    return out


def _inputs(case, seed: int):
    """The tensors (and member lists) that ``run`` and ``exact`` share."""
    kind = case["kind"]
    if kind in ("ensemble", "grad_batch"):
        return {"members": [(N, nu, th, steps, _u0(N, s)) for (N, nu, th, steps, s) in _members(case, seed)]}
    rng = np.random.default_rng(seed)
    N = case["N"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    if kind == "poisson":
        rhs = torch.randn(N, N, generator=g, device=DEV)
        return {"rhs": rhs - rhs.mean()}
    nu = _nu(case["scheme"])
    out = {"nu": nu}
    if kind != "jit_gradient":
        out["u0"] = _u0(N, seed)
    if kind == "projector":
        out["f"] = torch.randn(2, N, N, generator=g, device=DEV)
    if kind in ("projector", "operators"):
        return out
    out["theta"] = torch.from_numpy(_theta(nu, case["theta_len"], rng)).to(DEV)
    out["t"] = _f32(rng.uniform(0.0, 1.0))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = dict(_inputs(case, seed), kind=kind)
    if kind == "poisson":
        s["poisson"] = nsgb.SpectralPoissonSolver(case["N"], case["N"], TWO_PI / case["N"])
    elif kind == "ensemble":
        dt = 1e-3
        specs = [ens.SolveSpec(N=N, u0=u0.cpu().numpy(), theta=th, nu=nu, dt=dt, scheme=case["scheme"])
                 for (N, nu, th, _, u0) in s["members"]]
        s["ensemble"] = ens.Ensemble(specs, steps=case["steps"])
    elif kind == "grad_batch":
        s["batch"] = ens.GradientBatch()
        s["members"] = [(u0, torch.from_numpy(th).to(DEV), steps, nu, _stable_dt(N, nu, case["scheme"]))
                        for (N, nu, th, steps, u0) in s["members"]]
        s["scheme"], s["every"] = case["scheme"], case["every"]
    else:
        s["solver"] = _solver(case, s["nu"])
    return s


# --------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind == "poisson":
        return state["poisson"](state["rhs"])
    if kind == "ensemble":
        J, us = state["ensemble"].run()
        return [J] + list(us)
    if kind == "grad_batch":
        gb = state["batch"]
        ids = [gb.add(u0, th, steps, state["every"], TWO_PI, nu, dt, state["scheme"], want_du0=True)
               for (u0, th, steps, nu, dt) in state["members"]]
        gb.run()
        out = [[*gb.result(k), gb.du0(k)] for k in ids]
        for k in ids:
            gb.release(k)
        return out
    solver = state["solver"]
    if kind == "step":
        return solver.step(state["u0"], state["theta"], state["t"])
    if kind == "projector":
        return solver.projector.step(state["u0"], state["f"])
    if kind == "operators":
        ops, adv = solver.projector.ops, solver.projector.advection
        u = state["u0"]
        gx, gy = ops.grad(u[0])
        return [gx, gy, ops.divergence(u), ops.laplacian(u[0]), ops.laplacian(u[1]),
                adv.advect(u[0], u[0], u[1], ops), adv.advect(u[1], u[0], u[1], ops)]
    if kind == "rollout":
        return list(solver.rollout(state["u0"], state["theta"]))
    if kind == "jit_gradient":
        return solver.jit_gradient(state["theta"])
    if kind == "gradient":
        return list(solver.gradient(state["u0"], state["theta"], want_u0_grad=True))
    if kind == "autograd":
        th = state["theta"].detach().requires_grad_()
        u0 = state["u0"].detach().requires_grad_()
        J, u = solver.rollout(u0, th)
        J.backward()
        return [J.detach(), u, th.grad, u0.grad]
    raise ValueError(kind)


# -------------------------------------------------------------------- work
def _step_flops(N: int) -> float:
    """Per cell: the stencils (about 60) and two real 2-D transforms of
    2.5 log2(N^2) each."""
    return 60.0 + 10.0 * math.log2(N)


def work(case):
    """Bytes: 32 per cell and solver step (the state in and out, two transpose
    passes of the spectrum), 112 per cell and step with its gradient; single
    calls count their inputs and outputs."""
    kind = case["kind"]
    if kind == "ensemble":
        cells = float(sum(N * N * st for (N, _, _, st, _) in _members(case, 0)))
        return {"bytes": 32.0 * cells, "flops": 140.0 * cells}
    if kind == "grad_batch":
        cells = float(sum(N * N * st for (N, _, _, st, _) in _members(case, 0)))
        return {"bytes": 112.0 * cells, "flops": 400.0 * cells}
    N = case["N"]
    NN = float(N * N)
    if kind == "poisson":
        return {"bytes": 8.0 * NN, "flops": 10.0 * math.log2(N) * NN}
    if kind == "operators":
        # each call reads its inputs and writes its outputs once:
        # grad 4+8, divergence 8+4, two laplacians 8, two advections 8+4 each
        return {"bytes": (12 + 12 + 16 + 24) * NN, "flops": 50.0 * NN}
    if kind == "step":
        return {"bytes": 16.0 * NN + 16.0 * NN, "flops": _step_flops(N) * NN}
    if kind == "projector":
        return {"bytes": 24.0 * NN + 16.0 * NN, "flops": _step_flops(N) * NN}
    cells = NN * case["steps"]
    if kind == "rollout":
        return {"bytes": 32.0 * cells, "flops": _step_flops(N) * cells}
    return {"bytes": 112.0 * cells, "flops": 3.0 * _step_flops(N) * cells}


# ------------------------------------------------------------------- exact
def _roll(f, s, d):
    return torch.roll(f, s, d)


def _grad64(f, dx):
    return (_roll(f, -1, -2) - _roll(f, 1, -2)) / (2 * dx), (_roll(f, -1, -1) - _roll(f, 1, -1)) / (2 * dx)


def _lap64(f, dx):
    return (_roll(f, 1, -2) + _roll(f, -1, -2) + _roll(f, -1, -1) + _roll(f, 1, -1) - 4 * f) / (dx * dx)


def _adv64(f, ux, uy, dx, scheme):
    if scheme == "central":
        fx, fy = _grad64(f, dx)
        return -(ux * fx + uy * fy)
    dfx = torch.where(ux >= 0, f - _roll(f, 1, -2), _roll(f, -1, -2) - f) / dx
    dfy = torch.where(uy >= 0, f - _roll(f, 1, -1), _roll(f, -1, -1) - f) / dx
    return -(ux * dfx + uy * dfy)


def _poisson64(rhs, L):
    N = rhs.shape[-1]
    kx = torch.fft.fftfreq(N, L / N, dtype=torch.float64, device=rhs.device) * TWO_PI
    ky = torch.fft.rfftfreq(N, L / N, dtype=torch.float64, device=rhs.device) * TWO_PI
    k2 = kx[:, None] ** 2 + ky[None, :] ** 2
    k2[0, 0] = math.inf
    return torch.fft.irfft2(-torch.fft.rfft2(rhs) / k2, s=(N, N))


def _project64(us, L, dt):
    N = us.shape[-1]
    dx = L / N
    gx, gy = _grad64(us[0], dx)[0], _grad64(us[1], dx)[1]
    px, py = _grad64(_poisson64((gx + gy) / dt, L), dx)
    return torch.stack([us[0] - dt * px, us[1] - dt * py])


def _step64(u, fx, fy, nu, dt, scheme):
    N = u.shape[-1]
    dx = TWO_PI / N
    ux = u[0] + dt * (nu * _lap64(u[0], dx) + _adv64(u[0], u[0], u[1], dx, scheme) + fx)
    uy = u[1] + dt * (nu * _lap64(u[1], dx) + _adv64(u[1], u[0], u[1], dx, scheme) + fy)
    return _project64(torch.stack([ux, uy]), TWO_PI, dt)


def _forcing64(theta, t, N):
    x = TWO_PI * (torch.arange(N, dtype=torch.float64, device=theta.device) / N)
    mu = 0.5 + torch.sin(TWO_PI * theta[0] * t)
    sig = 0.1 + torch.cos(TWO_PI * theta[1] * t) ** 2
    r = x - mu
    d = r - torch.round(r)
    return torch.exp(-(d * d) / (2 * sig * sig))[:, None]


def _rollout64(u0, theta, nu, dt, steps, scheme):
    N = u0.shape[-1]
    dx2 = (TWO_PI / N) ** 2
    nu = theta[2] if theta.numel() == 3 else nu
    J, u = torch.zeros((), dtype=torch.float64, device=u0.device), u0
    for i in range(steps):
        fx = _forcing64(theta, i * dt, N)
        J = J + dt * dx2 * (u[0] * fx).sum()
        u = _step64(u, fx, 0.0, nu, dt, scheme)
    return J, u


def _gradient64(u0, theta, nu, dt, steps, scheme):
    """(J, u_final, dJ/dtheta, dJ/du0) by reverse-mode autograd, step by step
    (only the states are kept, each step's graph is rebuilt in turn)."""
    N = u0.shape[-1]
    dx2 = (TWO_PI / N) ** 2
    states, u = [], u0.double()
    th = theta.double()
    J = torch.zeros((), dtype=torch.float64, device=u0.device)
    nu_of = (lambda t: t[2]) if theta.numel() == 3 else (lambda t: nu)
    with torch.no_grad():
        for i in range(steps):
            states.append(u)
            fx = _forcing64(th, i * dt, N)
            J = J + dt * dx2 * (u[0] * fx).sum()
            u = _step64(u, fx, 0.0, nu_of(th), dt, scheme)
    lam, gth = torch.zeros_like(u), torch.zeros_like(th)
    for i in reversed(range(steps)):
        t = th.detach().requires_grad_()
        v = states.pop().requires_grad_()
        fx = _forcing64(t, i * dt, N)
        J_i = dt * dx2 * (v[0] * fx).sum()
        w = _step64(v, fx, 0.0, nu_of(t), dt, scheme)
        a, b = torch.autograd.grad(J_i + (w * lam).sum(), (t, v))
        gth, lam = gth + a, b
    return J, u, gth, lam


def exact(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    if kind == "poisson":
        return _poisson64(x["rhs"].double(), TWO_PI)
    if kind == "ensemble":
        got = [_rollout64(u0.double(), torch.from_numpy(th).to(DEV).double(), nu, 1e-3, steps, case["scheme"])
               for (N, nu, th, steps, u0) in x["members"]]
        return [torch.stack([J for J, _ in got])] + [u for _, u in got]
    if kind == "grad_batch":
        out = []
        for (N, nu, th, steps, u0) in x["members"]:
            J, _, g, du0 = _gradient64(u0, torch.from_numpy(th).to(DEV), nu, _stable_dt(N, nu, case["scheme"]),
                                       steps, case["scheme"])
            out.append([J, g, du0])
        return out
    N, scheme, nu = case["N"], case["scheme"], x["nu"]
    dt = _stable_dt(N, nu, scheme)
    dx = TWO_PI / N
    if kind == "operators":
        u = x["u0"].double()
        gx, gy = _grad64(u[0], dx)
        div = _grad64(u[0], dx)[0] + _grad64(u[1], dx)[1]
        return [gx, gy, div, _lap64(u[0], dx), _lap64(u[1], dx), _adv64(u[0], u[0], u[1], dx, scheme),
                _adv64(u[1], u[0], u[1], dx, scheme)]
    if kind == "projector":
        f = x["f"].double()
        return _step64(x["u0"].double(), f[0], f[1], nu, dt, scheme)
    th = x["theta"].double()
    if kind == "step":
        return _step64(x["u0"].double(), _forcing64(th, x["t"], N), 0.0, th[2] if th.numel() == 3 else nu, dt, scheme)
    if kind == "rollout":
        return list(_rollout64(x["u0"].double(), th, nu, dt, case["steps"], scheme))
    u0 = torch.zeros(2, N, N, device=DEV) if kind == "jit_gradient" else x["u0"]
    J, u, g, du0 = _gradient64(u0, th, nu, dt, case["steps"], scheme)
    if kind == "jit_gradient":
        return g
    return [J, g, du0] if kind == "gradient" else [J, u, g, du0]
