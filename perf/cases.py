"""The work that a user of this framework has it do, as cases that can be timed
and compared: time loops of 1D and 2D Euler solvers, batches of problems,
stage pipelines over patches, and rollouts with their gradients, each through
the public entry points and over the sizes that the configurations, tests and
benchmark use.

A case is a dict of plain values; ``kind`` names the entry point:

  dropin1d    nest's own 1D solver interface on host arrays (Euler1DGPU)
  solver1d    one 1D domain (Solver), FP64 or FP32 form
  adjoint1d   1D rollout and the gradient of a density misfit (Adjoint)
  solver2d    one 2D domain (Solver), FP64 or FP32 form
  batch2d     many periodic 2D problems of uneven sizes (Batch), host arrays
  adjoint2d   2D rollout and its gradient, with handles kept (Adjoint) or
              under torch autograd (rollout_2d)
  pipeline1d  nest's sod1d step as device stages over patches (sod1d_pipeline)

``exact`` restates the scheme in plain torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import nest_b200 as nb
from nest_b200 import adjoint as nba

GAMMA = 1.4
CFL = 0.4
BC = {"periodic": nb.BC_PERIODIC, "outflow": nb.BC_OUTFLOW}
LIMITER = {"minmod": 0, "mc": nb.FLAG_LIMITER_MC, "none": nb.FLAG_LIMITER_NONE}


def listed():
    return [
        # nest's CPU-vs-GPU test run: a program written against nest's interface, host arrays in and out
        {"name": "dropin1d_sod_100", "kind": "dropin1d", "n": 100, "t_final": 0.1, "cfl": 0.3},
        # the Sod shock tube run to its usual end: one resident time loop
        {"name": "solver1d_sod_1024_f64", "kind": "solver1d", "n": 1024, "precision": "f64", "bc": "outflow",
         "limiter": "minmod", "init": "sod", "t_final": 0.2},
        # a fine 1D domain in the FP32 form, an odd size: one launch per step
        {"name": "solver1d_50021_f32", "kind": "solver1d", "n": 50021, "precision": "f32", "bc": "periodic",
         "limiter": "minmod", "init": "fourier", "steps": 256},
        # sensitivity of a 1D flow to its initial state: forward sweep, checkpoints, reverse sweep
        {"name": "adjoint1d_65536_f64", "kind": "adjoint1d", "n": 65536, "precision": "f64", "steps": 256,
         "every": 64},
        # the 2D Riemann problem at scale, plain form
        {"name": "solver2d_4096_f64", "kind": "solver2d", "nx": 4096, "ny": 4096, "precision": "f64",
         "bc": "outflow", "limiter": "minmod", "init": "riemann", "steps": 20, "totals": False, "repair": False},
        # the same in the FP32 form with FP64 totals and positivity repair
        {"name": "solver2d_4096_f32", "kind": "solver2d", "nx": 4096, "ny": 4096, "precision": "f32",
         "bc": "outflow", "limiter": "minmod", "init": "riemann", "steps": 20, "totals": True, "repair": True},
        # an ordinary 2D run on a ragged, oblong domain
        {"name": "solver2d_517x1003_f64", "kind": "solver2d", "nx": 517, "ny": 1003, "precision": "f64",
         "bc": "periodic", "limiter": "minmod", "init": "kh", "steps": 48, "totals": False, "repair": False},
        # a small 2D run, where launches and latency count
        {"name": "solver2d_256x192_f32", "kind": "solver2d", "nx": 256, "ny": 192, "precision": "f32",
         "bc": "periodic", "limiter": "minmod", "init": "kh", "steps": 200, "totals": False, "repair": False},
        # a batch of independent Kelvin-Helmholtz problems of uneven sizes, states from and to the host
        {"name": "batch2d_48_f32", "kind": "batch2d", "count": 48, "lo": 64, "hi": 256, "unit": 64,
         "precision": "f32", "steps": 500, "totals": True, "repair": True},
        # gradient of a 2D flow with respect to its initial state, FP32 form, binomial checkpoints,
        # in a loop that keeps its solver and checkpoints
        {"name": "adjoint2d_512_f32", "kind": "adjoint2d", "nx": 512, "ny": 512, "precision": "f32", "steps": 48,
         "policy": "binomial", "param": 12, "init": "kh", "autograd": False},
        # the same as an autograd function, plain form on a ragged domain, uniform checkpoints
        {"name": "adjoint2d_250x333_f64", "kind": "adjoint2d", "nx": 250, "ny": 333, "precision": "f64",
         "steps": 32, "policy": "uniform", "param": 8, "init": "fourier", "autograd": True},
        # nest's sod1d example as stages over its four patches, run to its end
        {"name": "pipeline1d_sod_400x4", "kind": "pipeline1d", "n": 400, "patches": 4, "limiter": "minmod",
         "t_final": 0.2},
    ]


def draw(rng):
    def size(lo, hi):  # spread over the logarithm, odd sizes among them
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["dropin1d", "solver1d", "adjoint1d", "solver2d", "solver2d", "solver2d", "batch2d",
                       "adjoint2d", "pipeline1d"])
    precision = rng.choice(["f64", "f32"])
    if kind == "dropin1d":
        n = size(64, 4096)
        return {"kind": kind, "n": n, "t_final": round(min(0.1, 30.0 / n), 6), "cfl": rng.choice([0.3, 0.4])}
    if kind == "solver1d":
        return {"kind": kind, "n": size(128, 200000), "precision": precision,
                "bc": rng.choice(["outflow", "periodic"]), "limiter": rng.choice(["minmod", "minmod", "mc"]),
                "init": rng.choice(["sod", "fourier"]), "steps": size(32, 400)}
    if kind == "adjoint1d":
        return {"kind": kind, "n": size(1000, 65536), "precision": precision, "steps": size(32, 256),
                "every": rng.choice([16, 32, 64])}
    if kind == "solver2d":
        nx, ny = size(48, 4096), size(48, 4096)
        fp32 = precision == "f32"
        return {"kind": kind, "nx": nx, "ny": ny, "precision": precision,
                "bc": rng.choice(["outflow", "periodic"]),
                "limiter": "minmod" if fp32 else rng.choice(["minmod", "minmod", "mc"]),
                "init": rng.choice(["kh", "riemann"]),
                "steps": max(12, min(200, size(3, 8) * 2 ** 21 // (nx * ny))),
                "totals": rng.random() < 0.3, "repair": fp32 and rng.random() < 0.5}
    if kind == "batch2d":
        return {"kind": kind, "count": size(4, 64), "lo": 48, "hi": rng.choice([128, 200, 320]),
                "unit": rng.choice([1, 16, 64]), "precision": precision, "steps": size(48, 300),
                "totals": rng.random() < 0.5, "repair": precision == "f32" and rng.random() < 0.5}
    if kind == "adjoint2d":
        return {"kind": kind, "nx": size(64, 512), "ny": size(64, 512), "precision": precision,
                "steps": size(8, 48), "policy": rng.choice(["binomial", "uniform"]), "param": size(3, 12),
                "init": rng.choice(["kh", "fourier"]), "autograd": rng.random() < 0.5}
    patches = size(2, 24)
    n = max(size(200, 4000), 16 * patches)
    return {"kind": kind, "n": n, "patches": patches, "limiter": rng.choice(["minmod", "mc"]),
            "t_final": round(min(0.2, 80.0 / n), 6)}


# -- inputs -------------------------------------------------------------------


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _cons(rho, vel, p):
    """Conserved state from density, velocity components and pressure."""
    ke = 0.0
    for w in vel:
        ke = ke + 0.5 * rho * w * w
    return torch.stack([rho, *[rho * w for w in vel], p / (GAMMA - 1.0) + ke])


def _sod(n, seed, device):
    """A Sod tube whose jump and states move a little with the seed."""
    r = np.random.default_rng(seed)
    at, hi, lo = 0.5 + 0.04 * r.uniform(-1, 1), r.uniform(0.9, 1.1), r.uniform(0.11, 0.14)
    x = (torch.arange(n, dtype=torch.float64, device=device) + 0.5) / n
    left = (x < at).double()
    return _cons(lo + (hi - lo) * left, [torch.zeros_like(x)], 0.8 * lo + (hi - 0.8 * lo) * left)


def _fourier(shape, seed, device, modes):
    """Smooth periodic fields in every variable (a sum of random modes)."""
    r = np.random.default_rng(seed)
    axes = [(torch.arange(m, dtype=torch.float64, device=device) + 0.5) / m for m in shape]
    out = []
    for _ in range(len(shape) + 2):
        f = torch.zeros(shape, dtype=torch.float64, device=device)
        if len(shape) == 1:
            for k in range(1, modes + 1):
                a, ph = r.standard_normal(), r.uniform(0, 2 * np.pi)
                f += a * torch.cos(2 * np.pi * k * axes[0] + ph)
        else:
            for kx in range(modes + 1):
                for ky in range(modes + 1):
                    if kx or ky:
                        a, ph = r.standard_normal(), r.uniform(0, 2 * np.pi)
                        f += a * torch.cos(2 * np.pi * (kx * axes[0][:, None] + ky * axes[1][None, :]) + ph)
        out.append(f / f.abs().max())
    return _cons(1.0 + 0.4 * out[0], [0.3 * f for f in out[1:-1]], 1.0 + 0.4 * out[-1])


def _riemann(nx, ny, seed, device):
    """The diagonal 2D Riemann problem; the line and the states move with the seed."""
    r = np.random.default_rng(seed)
    at, hi, lo = 1.0 + 0.04 * r.uniform(-1, 1), r.uniform(0.9, 1.1), r.uniform(0.11, 0.14)
    x = (torch.arange(nx, dtype=torch.float64, device=device) + 0.5) / nx
    y = (torch.arange(ny, dtype=torch.float64, device=device) + 0.5) / ny
    left = ((x[:, None] + y[None, :]) < at).double()
    rho = lo + (hi - lo) * left
    z = torch.zeros_like(rho)
    return _cons(rho, [z, z], 0.8 * lo + (hi - 0.8 * lo) * left)


def _kh(nx, ny, seed, device):
    """A periodic Kelvin-Helmholtz layer with seeded noise on the transverse velocity."""
    r = np.random.default_rng(seed)
    x = (torch.arange(nx, dtype=torch.float64, device=device) + 0.5) / nx
    y = (torch.arange(ny, dtype=torch.float64, device=device) + 0.5) / ny
    band = ((y - 0.5).abs() < 0.25)[None, :].expand(nx, ny)
    rho, u = 1.0 + band.double(), band.double() - 0.5
    noise = torch.from_numpy(r.uniform(-1e-3, 1e-3, size=(nx, ny))).to(device)
    v = 0.01 * torch.sin(4 * np.pi * x)[:, None] + noise
    return _cons(rho, [u, v], torch.full_like(rho, 2.5))


def _initial(case, seed, device):
    """The case's initial state in the precision that the solver takes, [vars][cells...]."""
    kind = case["kind"]
    if kind in ("dropin1d", "pipeline1d"):
        return _sod(case["n"], seed, device)
    init = case.get("init", "fourier")
    if kind in ("solver1d", "adjoint1d"):
        U = _sod(case["n"], seed, device) if init == "sod" else _fourier((case["n"],), seed, device, 16)
    elif init == "riemann":
        U = _riemann(case["nx"], case["ny"], seed, device)
    elif init == "kh":
        U = _kh(case["nx"], case["ny"], seed, device)
    else:
        U = _fourier((case["nx"], case["ny"]), seed, device, 3)
    return U if case["precision"] == "f64" else U.float()


def _batch(case, seed):
    """Sizes (the same for every seed) and initial states of a batch, on the host."""
    r = np.random.default_rng(1000 * case["count"] + case["hi"])
    sides = np.arange(case["lo"], case["hi"] + 1, case["unit"])
    nx, ny = r.choice(sides, size=case["count"]), r.choice(sides, size=case["count"])
    dtype = np.float64 if case["precision"] == "f64" else np.float32
    states = [_kh(int(a), int(b), seed * 1009 + k, "cpu").numpy().astype(dtype)
              for k, (a, b) in enumerate(zip(nx, ny))]
    return [int(a) for a in nx], [int(b) for b in ny], states


def prepare(case, seed):
    kind, dev = case["kind"], "cuda"
    s = {"case": case}
    if kind == "dropin1d":
        n = case["n"]
        s["solver"] = nb.Euler1DGPU(n, 2, 1.0 / n, GAMMA)
        U = np.zeros((3, n + 4))
        U[:, 2:-2] = _initial(case, seed, "cpu").numpy()
        s["U"] = U
        return s
    if kind == "batch2d":
        nx, ny, s["states"] = _batch(case, seed)
        flags = (nb.FLAG_TOTALS if case["totals"] else 0) | (nb.FLAG_REPAIR if case["repair"] else 0)
        s["batch"] = nb.Batch(nx, ny, gamma=GAMMA, bc=nb.BC_PERIODIC,
                              precision=nb.F64 if case["precision"] == "f64" else nb.F32, flags=flags)
        return s
    U = _initial(case, seed, dev).contiguous()
    if kind == "pipeline1d":
        s["pipe"] = nb.sod1d_pipeline(case["n"], case["patches"], cfl=CFL, gamma=GAMMA,
                                      limiter=("minmod", "mc", "none").index(case["limiter"]))
        s["U"] = torch.from_numpy(s["pipe"].scatter(U.cpu().numpy())).to(dev)
        return s
    s["U"] = U
    if case.get("autograd"):
        return s
    prec = nb.F64 if case["precision"] == "f64" else nb.F32
    if kind == "adjoint1d":
        s["solver"] = nb.Solver(1, case["n"], bc=nb.BC_PERIODIC, gamma=GAMMA, precision=prec,
                                flags=nb.FLAG_NO_RESIDENT)
        s["adjoint"] = nba.Adjoint(s["solver"], case["steps"], nba.UNIFORM, case["every"])
        s["target"] = _initial(case, seed + 500009, dev)[0].contiguous()
        return s
    if kind == "adjoint2d":
        s["solver"] = nb.Solver(2, case["nx"], case["ny"], bc=nb.BC_PERIODIC, gamma=GAMMA, precision=prec)
        policy = nba.BINOMIAL if case["policy"] == "binomial" else nba.UNIFORM
        s["adjoint"] = nba.Adjoint(s["solver"], case["steps"], policy, case["param"])
        return s
    flags = LIMITER[case["limiter"]]
    if kind == "solver2d":
        flags |= (nb.FLAG_TOTALS if case["totals"] else 0) | (nb.FLAG_REPAIR if case["repair"] else 0)
        s["solver"] = nb.Solver(2, case["nx"], case["ny"], bc=BC[case["bc"]], gamma=GAMMA, precision=prec, flags=flags)
    else:
        s["solver"] = nb.Solver(1, case["n"], bc=BC[case["bc"]], gamma=GAMMA, precision=prec, flags=flags)
    return s


# -- one pass -----------------------------------------------------------------


def _advance(solver, case, U):
    solver.reset_time()
    solver.upload_device(U.data_ptr(), nb.LAYOUT_INTERIOR)
    if "t_final" in case:
        solver.run_to(case["t_final"], CFL)
    else:
        solver.step(case["steps"], CFL)
    out = torch.empty_like(U)
    solver.download_device(out.data_ptr(), nb.LAYOUT_INTERIOR)
    time, steps = solver.time()
    return {"U": out, "time": time, "steps": steps}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dropin1d":
        s = state["solver"]
        s.upload(state["U"])
        steps = s.run(case["t_final"], case["cfl"])
        return {"U": s.download()[:, 2:-2], "steps": steps}
    if kind in ("solver1d", "solver2d"):
        out = _advance(state["solver"], case, state["U"])
        if case.get("totals"):
            out["totals"] = state["solver"].totals()
        return out
    if kind == "batch2d":
        b = state["batch"]
        b.reset()
        for p, U in enumerate(state["states"]):
            b.upload(p, U, nb.LAYOUT_INTERIOR)
        b.step(case["steps"], CFL)
        times, steps = b.times()
        U = np.concatenate([b.download(p, nb.LAYOUT_INTERIOR).ravel() for p in range(b.count)])
        out = {"U": U, "times": times, "steps": steps}
        if case["totals"]:
            out["totals"] = b.totals()
        return out
    if case.get("autograd"):
        U0 = state["U"].clone().requires_grad_(True)
        policy = nba.BINOMIAL if case["policy"] == "binomial" else nba.UNIFORM
        UT = nba.rollout_2d(U0, case["steps"], CFL, policy, case["param"])
        loss = (0.5 * UT[2] * UT[2] / UT[0]).mean()
        loss.backward()
        return {"U": UT.detach(), "loss": loss.detach(), "grad": U0.grad}
    if kind.startswith("adjoint"):
        s, adj, U = state["solver"], state["adjoint"], state["U"]
        s.upload_device(U.data_ptr(), nb.LAYOUT_INTERIOR)
        adj.forward(CFL)
        UT = torch.empty_like(U)
        s.download_device(UT.data_ptr(), nb.LAYOUT_INTERIOR)
        # the adjoint of the final state, in the solver's device layout
        if kind == "adjoint1d":
            lam = torch.zeros((3, case["n"] + 4), dtype=U.dtype, device=U.device)
            inner = lambda a: a[:, 2:-2]  # noqa: E731
            inner(lam)[0] = UT[0] - state["target"]
        else:
            _, pitch, plane = s.state_ptr()
            nx, ny = case["nx"], case["ny"]
            lam = torch.zeros((4, plane), dtype=U.dtype, device=U.device)
            inner = lambda a: a[:, :(nx + 4) * pitch].view(4, nx + 4, pitch)[:, 2:-2, 2:ny + 2]  # noqa: E731
            V = UT.clone().requires_grad_(True)
            loss = (0.5 * V[2] * V[2] / V[0]).mean()
            inner(lam).copy_(torch.autograd.grad(loss, V)[0])
        lam0 = torch.empty_like(lam)
        torch.cuda.current_stream().synchronize()  # the reverse sweep runs on the solver's own stream
        adj.backward_device(lam.data_ptr(), lam0.data_ptr())
        return {"U": UT, "grad": inner(lam0).contiguous()}
    pipe = state["pipe"]
    pipe.set_clock()
    U = state["U"].clone()
    torch.cuda.current_stream().synchronize()  # the stages run on the pipeline's own stream
    steps = pipe.run(U.data_ptr(), case["t_final"])
    return {"U": torch.from_numpy(pipe.gather(U.cpu().numpy())), "time": pipe.clock()[0], "steps": steps}


def work(case):
    """Per step the state is read once and written once; about 110 operations a cell, stage and
    axis. The reverse of a step reads the state and two adjoints and writes one, at about three times
    a step's operations, and a checkpointed sweep repeats the forward steps once."""
    kind = case["kind"]
    size = 4 if case.get("precision") == "f32" else 8
    if kind == "batch2d":
        r = np.random.default_rng(1000 * case["count"] + case["hi"])
        sides = np.arange(case["lo"], case["hi"] + 1, case["unit"])
        nx, ny = r.choice(sides, size=case["count"]), r.choice(sides, size=case["count"])
        cells, axes = int((nx.astype(np.int64) * ny).sum()), 2
    elif kind in ("solver2d", "adjoint2d"):
        cells, axes = case["nx"] * case["ny"], 2
    else:
        cells, axes = case["n"], 1
    # the fastest signal of these tubes moves at about 2.2 cell widths per unit time and cell
    steps = case["steps"] if "steps" in case else int(2.2 * case["t_final"] * case["n"] / case.get("cfl", CFL)) + 1
    step_bytes, step_flops = 2 * (axes + 2) * size * cells, 220 * axes * cells
    if kind.startswith("adjoint"):
        return {"bytes": float(steps * 4 * step_bytes), "flops": float(steps * 5 * step_flops)}
    return {"bytes": float(steps * step_bytes), "flops": float(steps * step_flops)}


# -- the scheme in plain torch, 64 bits ---------------------------------------


def _limit(a, b, kind):
    def mm(x, y):
        return torch.where(x * y <= 0, torch.zeros_like(x), torch.where(x.abs() < y.abs(), x, y))

    if kind == "minmod":
        return mm(a, b)
    if kind == "mc":
        return mm(2 * a, mm(0.5 * (a + b), 2 * b))
    return 0.5 * (a + b)


def _prims(U):
    rho = U[0]
    vel = [U[k] / rho for k in range(1, len(U) - 1)]
    p = (GAMMA - 1) * (U[-1] - sum(0.5 * rho * w * w for w in vel))
    return torch.stack([rho, *vel, torch.where(p < 0, torch.zeros_like(p), p)])


def _flux(L, R, axis):
    """HLLE flux with Davis speeds along velocity component `axis`."""
    def side(W):
        rho, vel, p = W[0], W[1:-1], W[-1]
        n, c = vel[axis], torch.sqrt(GAMMA * p / rho)
        E = p / (GAMMA - 1) + sum(0.5 * rho * w * w for w in vel)
        U = torch.stack([rho, *[rho * w for w in vel], E])
        F = U * n
        F = torch.cat([F[:1 + axis], (F[1 + axis] + p)[None], F[2 + axis:-1], ((E + p) * n)[None]])
        return U, F, n - c, n + c

    UL, FL, aL, bL = side(L)
    UR, FR, aR, bR = side(R)
    SL, SR = torch.where(aR < aL, aR, aL), torch.where(bL < bR, bR, bL)
    mid = (SR * FL - SL * FR + SL * SR * (UR - UL)) / (SR - SL)
    return torch.where(SL >= 0, FL, torch.where(SR <= 0, FR, mid))


def _rate(U, axes, limiter):
    """Sum over the axes of (flux out - flux in) / spacing for every cell; `axes` holds, for each
    axis, the spacing and the cells at offsets -2, -1, 1 and 2."""
    W = _prims(U)
    out = 0.0
    for axis, (h, a2, a1, b1, b2) in enumerate(axes):
        Wa2, Wa, Wb, Wb2 = (W[:, k] for k in (a2, a1, b1, b2))
        sa, s, sb = _limit(Wa - Wa2, W - Wa, limiter), _limit(W - Wa, Wb - W, limiter), _limit(Wb - W, Wb2 - Wb, limiter)
        out = out + (_flux(W + 0.5 * s, Wb - 0.5 * sb, axis) - _flux(Wa + 0.5 * sa, W - 0.5 * s, axis)) / h
    return out


def _step(U, dt, axes, limiter):
    V = U - dt * _rate(U, axes, limiter)
    return 0.5 * (U + V - dt * _rate(V, axes, limiter))


def _axes(shape, bc, device):
    cell = torch.arange(math.prod(shape), device=device).reshape(shape)
    out = []
    for d, n in enumerate(shape):
        def at(k, d=d, n=n):
            i = torch.arange(n, device=device) + k
            i = i % n if bc == "periodic" else i.clamp(0, n - 1)
            return cell.index_select(d, i).reshape(-1)
        out.append((1.0 / n, at(-2), at(-1), at(1), at(2)))
    return out


def _speeds(U, floor):
    W = _prims(U)
    rho, p = (W[0].clamp(min=1e-10), W[-1].clamp(min=1e-10)) if floor else (W[0], W[-1])
    c = torch.sqrt(GAMMA * p / rho)
    return [w.abs() + c for w in W[1:-1]]


def _dt(U, axes, cfl):
    return cfl * min(float(h / s.max()) for (h, *_), s in zip(axes, _speeds(U, len(axes) > 1)))


def _march(U, axes, case, keep=None):
    """The time loop: (state, time, steps); `keep` receives (state, dt) of every step."""
    limiter, cfl = case.get("limiter", "minmod"), case.get("cfl", CFL)
    t, steps, end = 0.0, 0, case.get("t_final", math.inf)
    while t < end and steps < case.get("steps", 1 << 30):
        dt = min(_dt(U, axes, cfl), end - t)
        if keep is not None:
            keep.append((U, dt))
        U = _step(U, dt, axes, limiter)
        t, steps = t + dt, steps + 1
    return U, t, steps


def _exact_batch(case, seed, device):
    nx, ny, states = _batch(case, seed)
    if sum(a * b for a, b in zip(nx, ny)) * case["steps"] > 1.5e9:
        return None
    first, parts, base = [], [], 0
    for a, b in zip(nx, ny):
        first.append([(h, *[k + base for k in rest]) for h, *rest in _axes((a, b), "periodic", device)])
        base += a * b
    axes = []
    for d in range(2):
        h = torch.cat([torch.full((a * b,), first[p][d][0], dtype=torch.float64, device=device)
                       for p, (a, b) in enumerate(zip(nx, ny))])
        axes.append((h, *[torch.cat([f[d][k] for f in first]) for k in range(1, 5)]))
    owner = torch.cat([torch.full((a * b,), p, dtype=torch.int64, device=device) for p, (a, b) in enumerate(zip(nx, ny))])
    U = torch.cat([torch.from_numpy(u).to(device).double().reshape(4, -1) for u in states], dim=1)
    t = torch.zeros(len(nx), dtype=torch.float64, device=device)
    for _ in range(case["steps"]):
        rate = [torch.zeros_like(t).scatter_reduce_(0, owner, s / h, "amax") for (h, *_), s in zip(axes, _speeds(U, True))]
        dt = CFL / torch.maximum(*rate)
        U = _step(U, dt[owner], axes, "minmod")
        t = t + dt
    at = 0
    for a, b in zip(nx, ny):
        parts.append(U[:, at:at + a * b].reshape(-1))
        at += a * b
    out = {"U": torch.cat(parts), "times": t, "steps": None}
    if case["totals"]:
        sums = torch.zeros(4, len(nx), dtype=torch.float64, device=device).index_add_(1, owner, U)
        out["totals"] = (sums / torch.tensor([a * b for a, b in zip(nx, ny)], device=device)).T.contiguous()
    return out


def exact(case, seed):
    kind, device = case["kind"], _device()
    if kind == "batch2d":
        return _exact_batch(case, seed, device)
    U0 = _initial(case, seed, device).double()
    shape = tuple(U0.shape[1:])
    bc = case.get("bc", "periodic")
    axes = _axes(shape, bc, device)
    U = U0.reshape(len(U0), -1)
    if kind == "pipeline1d":
        # every patch reconstructs its first and last cell from the one neighbour it has there
        n, m = case["n"], case["patches"]
        h, a2, a1, b1, b2 = axes[0]
        per, extra = divmod(n, m)
        starts = torch.tensor([k * per + min(k, extra) for k in range(m)], device=device)
        lasts = torch.cat([starts[1:], torch.tensor([n], device=device)]) - 1
        a2, b2 = a2.clone(), b2.clone()
        a2[starts], b2[lasts] = a1[starts], b1[lasts]
        axes = [(h, a2, a1, b1, b2)]
    if not kind.startswith("adjoint"):
        U, t, steps = _march(U, axes, case)
        out = {"U": U.reshape(U0.shape), "steps": steps}
        if kind != "dropin1d":
            out["time"] = t
        if case.get("totals"):
            out["totals"] = U.sum(dim=1) / U.shape[1]
        return out
    kept = []
    UT, _, _ = _march(U, axes, case, kept)
    if kind == "adjoint1d":
        lam = torch.zeros_like(UT)
        lam[0] = UT[0] - _initial(case, seed + 500009, device)[0].double()
        out = {}
    else:
        V = UT.clone().requires_grad_(True)
        loss = (0.5 * V[2] * V[2] / V[0]).mean()
        lam, = torch.autograd.grad(loss, V)
        out = {"loss": loss.detach()}
    for V, dt in reversed(kept):
        V = V.detach().requires_grad_(True)
        lam, = torch.autograd.grad(_step(V, dt, axes, "minmod"), V, lam)
    out["U"], out["grad"] = UT.reshape(U0.shape), lam.reshape(U0.shape)
    return out
