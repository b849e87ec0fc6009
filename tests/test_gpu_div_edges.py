"""The branch-free division (nest_b200/csrc/f64div.cuh) by the divisor whose
reciprocal comes nearest to a midpoint of two doubles, (2 - ulp) 2^k: quotients of
powers of two and of their neighbours, alone and in the solvers, against IEEE."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import BC_PERIODIC
from test_gpu_div import check

pytestmark = pytest.mark.gpu
G = 1.4
EDGE = 2.0 - 2.0 ** -52


def test_powers_of_two_over_edge_divisors(gpu):
    from nest_b200 import _capi as A
    j, k = np.meshgrid(np.arange(-400, 400), np.arange(-400, 400, 7), indexing="ij")
    a, b = 2.0 ** j.ravel().astype(float), EDGE * 2.0 ** k.ravel().astype(float)
    assert check(A.lib, a, b).all()
    assert check(A.lib, -a, b).all()


def test_neighbours(gpu):
    """Numerators around 1 and 2, divisors of the last 256 significands below 2 and
    the first 256 above 1."""
    from nest_b200 import _capi as A
    i = np.arange(1, 257) * 2.0 ** -52
    b = np.concatenate([2.0 - i, [1.0], 1.0 + i])
    a = np.concatenate([1.0 - 0.5 * i, [1.0], 1.0 + i, 2.0 - i, 2.0 + 2.0 * i])
    a, b = (v.ravel() for v in np.meshgrid(a, b, indexing="ij"))
    assert check(A.lib, a, b).all()
    assert check(A.lib, a * 2.0 ** -300, b * 2.0 ** 55).all()


def edge_state(shape, seed):
    """Density 2 - ulp, momenta powers of two, smooth pressure."""
    rng = np.random.default_rng(seed)
    mom = [rng.choice([-1.0, 1.0], shape) * 2.0 ** -rng.integers(1, 6, shape).astype(float) for _ in shape]
    p = 1.0 + 0.2 * rng.random(shape)
    U = np.zeros((len(shape) + 2,) + tuple(m + 4 for m in shape))
    U[(slice(None),) + (slice(2, -2),) * len(shape)] = np.stack(
        [np.full(shape, EDGE), *mom, p / (G - 1) + sum(0.5 * m * m / EDGE for m in mom)])
    return U


@pytest.mark.parametrize("n,resident", [(100, True), (1000, True), (1000, False)])
def test_1d_matches_oracle(gpu, oracle, n, resident):
    U = edge_state((n,), n)
    want = U.copy()
    oracle.run1d(want, n, 2, 1 / n, G, 0.4, nsteps=2, bc=BC_PERIODIC)
    s = gpu.Solver(1, n, bc=BC_PERIODIC, gamma=G, flags=0 if resident else gpu.FLAG_NO_RESIDENT)
    s.upload(U)
    s.step(2, 0.4)
    assert np.array_equal(s.download()[:, 2:-2].view(np.int64), want[:, 2:-2].view(np.int64))


def test_2d_matches_oracle(gpu, oracle):
    nx, ny = 61, 67
    U = edge_state((nx, ny), 3)
    want = U.copy()
    oracle.run2d(want, nx, ny, 2, 1 / nx, 1 / ny, G, 0.4, nsteps=2, bc=BC_PERIODIC)
    s = gpu.Solver(2, nx, ny, bc=BC_PERIODIC, gamma=G)
    s.upload(U)
    s.step(2, 0.4)
    assert np.array_equal(s.download()[:, 2:-2, 2:-2].view(np.int64), want[:, 2:-2, 2:-2].view(np.int64))
