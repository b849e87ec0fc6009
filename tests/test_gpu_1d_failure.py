"""A failing step of the tiled 1D form on grids of several waves of blocks: the
step in which a cell fails completes on every cell, and nothing runs after it."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import BC_OUTFLOW, BC_PERIODIC

pytestmark = pytest.mark.gpu
G = 1.4


def failing(n, halo=2):
    """Noise, so that a step changes every cell, and a uniform stretch with p < 0 near
    one end, whose blocks are among the first."""
    rng = np.random.default_rng(n)
    U = np.zeros((3, n + 2 * halo))
    rho = 1 + 0.2 * rng.random(n)
    u = 0.2 * rng.standard_normal(n)
    p = 1 + 0.2 * rng.random(n)
    V = np.stack([rho, rho * u, p / (G - 1) + 0.5 * rho * u * u])
    V[:, 20:60] = np.array([1.0, 1.0, 0.4])[:, None]
    U[:, halo:-halo] = V
    return U


@pytest.mark.parametrize("n", [5003, 1_000_003, 3_000_017])
@pytest.mark.parametrize("bc", [BC_OUTFLOW, BC_PERIODIC])
def test_failing_step_completes(gpu, oracle, n, bc):
    U = failing(n)
    want = U.copy()
    oracle.run1d(want, n, 2, 1 / n, G, 0.4, nsteps=1, bc=bc)
    s = gpu.Solver(1, n, bc=bc, gamma=G, flags=gpu.FLAG_NO_RESIDENT)
    for steps in (2, 4, 19):
        s.upload(U)
        s.reset_time()
        for _ in range(2):
            with pytest.raises(gpu.NestError) as e:
                s.step(steps, 0.4)
                s.sync()
            assert "at step 1 " in str(e.value)
            got = s.download()
            assert np.array_equal(got[:, 2:-2].view(np.int64), want[:, 2:-2].view(np.int64))


@pytest.mark.parametrize("n", [5003, 1_000_003])
def test_failing_step_completes_f32(gpu, n):
    """FP32 against the two stage launches of one step, which run to their end."""
    U = failing(n).astype(np.float32)
    ends = []
    for steps in (1, 2, 18):
        s = gpu.Solver(1, n, bc=BC_PERIODIC, gamma=G, precision=gpu.F32, flags=gpu.FLAG_NO_RESIDENT)
        s.upload(U)
        with pytest.raises(gpu.NestError):
            s.step(steps, 0.4)
            s.sync()
        ends.append(s.download()[:, 2:-2])
        s.close()
    moved = np.abs(ends[0] - U[:, 2:-2]).max(axis=0)
    assert (moved > 1e-3).mean() > 0.9
    for e in ends[1:]:
        assert np.abs(e - ends[0]).max() < 1e-4


def test_stays_failed_across_forms(gpu):
    """A failure in a one-launch step stops later stage launches and the other way
    round, also behind a new clock; an upload clears it."""
    n = 70001
    U = failing(n)
    good = U.copy()
    good[:, 2:-2] = np.array([1.0, 0.1, 2.5])[:, None]
    s = gpu.Solver(1, n, bc=BC_PERIODIC, gamma=G, flags=gpu.FLAG_NO_RESIDENT)

    def fails(f):
        with pytest.raises(gpu.NestError):
            f()
            s.sync()

    for first in (1, 2):
        s.upload(U)
        fails(lambda: s.step(first, 0.4))
        at = s.download()
        for again in (1, 2, 3, 16):
            fails(lambda: s.step(again, 0.4))
            s.set_time(0.0, 0)
            fails(lambda: s.step(again, 0.4))
        assert np.array_equal(s.download()[:, 2:-2].view(np.int64), at[:, 2:-2].view(np.int64))
        s.upload(good)
        s.reset_time()
        s.step(5, 0.4)
        s.sync()
        assert s.time()[1] == 5
