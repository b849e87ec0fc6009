"""The resident 1D time loop at the sizes where its form or its chunks change: one
CTA or a cluster, chunks of equal and of unequal size, full and nearly empty
last warps, both boundary conditions.  State, time and step count equal the
oracle's bit for bit, and so does a run cut into launches of one step."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import BC_OUTFLOW, BC_PERIODIC

pytestmark = pytest.mark.gpu
G = 1.4


def initial(n):
    rng = np.random.default_rng(n)
    x = (np.arange(n) + 0.5) / n
    rho = np.where(x < 0.45, 1.0, 0.125) * (1 + 0.02 * rng.random(n))
    u = 0.1 * np.sin(2 * np.pi * x)
    u[rng.random(n) < 0.1] = 0.0
    p = np.where(x < 0.45, 1.0, 0.1) * (1 + 0.02 * rng.random(n))
    U = np.zeros((3, n + 4))
    U[:, 2:-2] = np.stack([rho, rho * u, p / (G - 1) + 0.5 * rho * u * u])
    return U


@pytest.mark.parametrize("n", [31, 62, 63, 248, 255, 256, 257, 271, 272, 303, 432, 433, 1025, 1424, 1425, 4079, 4080])
@pytest.mark.parametrize("bc", [BC_OUTFLOW, BC_PERIODIC])
def test_matches_oracle(gpu, oracle, n, bc):
    U = initial(n)
    want = U.copy()
    _, t, _ = oracle.run1d(want, n, 2, 1 / n, G, 0.4, nsteps=11, bc=bc)
    for pieces in ([11], [1, 1, 2, 7]):
        s = gpu.Solver(1, n, bc=bc, gamma=G)
        s.upload(U)
        for k in pieces:
            s.step(k, 0.4)
        got = s.download()
        assert s.time()[0] == t and s.time()[1] == 11
        assert np.array_equal(got[:, 2:-2].view(np.int64), want[:, 2:-2].view(np.int64))
