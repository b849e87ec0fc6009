"""The FP64 plain form outside the range of its branch-free division and square
root (nest_b200/csrc/f64div.cuh): states whose scales, or single cells of
which, leave the range run with the IEEE operations instead.  Every case equals
the oracle bit for bit, whichever of the two a row, face or cell takes."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import BC_OUTFLOW, BC_PERIODIC

pytestmark = pytest.mark.gpu

# density and pressure scales (in range; SI units; below 2^-128; above 2^128;
# a sound speed of 1e38), gamma (one with gamma - 1 under the kernels' bound)
SCALES = [(1.0, 1.0, 1.4), (1.2, 1e5, 1.4), (1e-45, 1e-44, 1.4), (1e45, 1e47, 1.4), (1e-36, 1e38, 1.4),
          (1.0, 1.0, 1.0 + 2.0 ** -22)]


def smooth(shape, rng):
    """A random smooth periodic field in [-1, 1]."""
    axes = np.meshgrid(*[2 * np.pi * (np.arange(m) + 0.5) / m for m in shape], indexing="ij")
    f = sum(rng.standard_normal() * np.cos(sum(k * a for k, a in zip(ks, axes)) + rng.uniform(0, 6.28))
            for ks in np.ndindex(*(3,) * len(shape)) if any(ks))
    return f / np.abs(f).max()


def state(shape, rs, ps, gamma, cells, seed):
    """Conserved state with ghosts; `cells` plants what leaves the range."""
    rng = np.random.default_rng(seed)
    rho = rs * (1 + 0.4 * smooth(shape, rng))
    p = ps * (1 + 0.4 * smooth(shape, rng))
    vel = [0.3 * np.sqrt(ps / rs) * smooth(shape, rng) for _ in shape]
    if cells == "tiny":
        # velocities from the smallest subnormal up, of either sign, zeros
        # among them, next to ordinary ones
        for v in vel:
            m = rng.random(shape) < 0.5
            t = np.ldexp(rng.uniform(1, 2, shape), rng.integers(-1074, -100, shape)) * rng.choice([-1.0, 1.0], shape)
            v[m] = np.where(rng.random(shape) < 0.3, rng.choice([0.0, -0.0, 5e-324], shape), t)[m]
    elif cells == "light":
        # a few cells lighter than the range, at rest (stationary contacts)
        rho[rng.random(shape) < 0.02] = rs * 1e-41
        p[...] = ps
        vel = [0 * v for v in vel]
    U = np.zeros((len(shape) + 2,) + tuple(m + 4 for m in shape))
    inner = (slice(None),) + (slice(2, -2),) * len(shape)
    U[inner] = np.stack([rho, *[rho * v for v in vel], p / (gamma - 1) + sum(0.5 * rho * v * v for v in vel)])
    return U


def time_step(U, dxs, gamma):
    """A stable step (the 2D solver's own rule has floors that these scales pass)."""
    V = U[(slice(None),) + (slice(2, -2),) * len(dxs)]
    vel = [V[k] / V[0] for k in range(1, len(V) - 1)]
    p = (gamma - 1) * (V[-1] - sum(0.5 * V[0] * v * v for v in vel))
    c = np.sqrt(gamma * p / V[0])
    return 0.2 * min(dx / (np.abs(v) + c).max() for dx, v in zip(dxs, vel))


CASES = [(s, "plain") for s in SCALES] + [(SCALES[0], "tiny"), (SCALES[1], "tiny"), (SCALES[0], "light")]


@pytest.mark.parametrize("scale,cells", CASES)
@pytest.mark.parametrize("limiter", [0, 1])
def test_2d_matches_oracle(gpu, oracle, scale, cells, limiter):
    nx, ny, (rs, ps, gamma) = 53, 61, scale
    U = state((nx, ny), rs, ps, gamma, cells, 5)
    want = U.copy()
    oracle.set_limiter(limiter)
    try:
        dt = time_step(U, (1 / nx, 1 / ny), gamma)
        _, t, _ = oracle.run2d(want, nx, ny, 2, 1 / nx, 1 / ny, gamma, 0.4, nsteps=7, bc=BC_PERIODIC,
                               dts_in=np.full(7, dt))
    finally:
        oracle.set_limiter(0)
    s = gpu.Solver(2, nx, ny, bc=BC_PERIODIC, gamma=gamma, flags=gpu.FLAG_LIMITER_MC if limiter else 0)
    s.upload(U)
    s.step_dt(7, dt)
    got = s.download()
    assert s.time()[0] == t and np.isfinite(want).all()
    assert np.array_equal(got[:, 2:-2, 2:-2].view(np.int64), want[:, 2:-2, 2:-2].view(np.int64))


@pytest.mark.parametrize("scale,cells", CASES)
@pytest.mark.parametrize("n,tiled", [(100, False), (613, False), (613, True)])
@pytest.mark.parametrize("limiter", [0, 1])
def test_1d_matches_oracle(gpu, oracle, scale, cells, n, tiled, limiter):
    rs, ps, gamma = scale
    U = state((n,), rs, ps, gamma, cells, 9)
    want = U.copy()
    oracle.set_limiter(limiter)
    try:
        _, t, _ = oracle.run1d(want, n, 2, 1 / n, gamma, 0.4, nsteps=7, bc=BC_OUTFLOW)
    finally:
        oracle.set_limiter(0)
    s = gpu.Solver(1, n, bc=BC_OUTFLOW, gamma=gamma,
                   flags=(gpu.FLAG_LIMITER_MC if limiter else 0) | (gpu.FLAG_NO_RESIDENT if tiled else 0))
    s.upload(U)
    s.step(7, 0.4)
    got = s.download()
    assert s.time()[0] == t and np.isfinite(want).all()
    assert np.array_equal(got[:, 2:-2].view(np.int64), want[:, 2:-2].view(np.int64))
