"""The waits between the CTAs of the resident 1D loop run into their limit: the
launch ends by itself with an error, the process goes on, and a solver with the
usual limit is not affected."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import BC_OUTFLOW, BC_PERIODIC, sod_ic_1d

pytestmark = pytest.mark.gpu
G = 1.4


@pytest.mark.parametrize("n", [256, 1024, 4080])
@pytest.mark.parametrize("bc", [BC_OUTFLOW, BC_PERIODIC])
def test_no_wait_allowed(gpu, oracle, monkeypatch, n, bc):
    U = sod_ic_1d(n)
    monkeypatch.setenv("NEST_1D_WAIT_POLLS", "0")
    s = gpu.Solver(1, n, bc=bc, gamma=G)
    monkeypatch.delenv("NEST_1D_WAIT_POLLS")
    s.upload(U)
    for _ in range(2):
        with pytest.raises(gpu.NestError, match="ran into its limit"):
            s.step(5, 0.4)
            s.sync()
        assert np.array_equal(s.download()[:, 2:-2], U[:, 2:-2])
    want = U.copy()
    oracle.run1d(want, n, 2, 1 / n, G, 0.4, nsteps=5, bc=bc)
    s = gpu.Solver(1, n, bc=bc, gamma=G)
    s.upload(U)
    s.step(5, 0.4)
    assert np.array_equal(s.download()[:, 2:-2].view(np.int64), want[:, 2:-2].view(np.int64))


@pytest.mark.parametrize("polls", [1, 5, 20, 80])
def test_short_waits_fail_or_give_the_answer(gpu, oracle, monkeypatch, polls):
    n = 1024
    U = sod_ic_1d(n)
    want = U.copy()
    oracle.run1d(want, n, 2, 1 / n, G, 0.4, nsteps=50, bc=BC_OUTFLOW)
    monkeypatch.setenv("NEST_1D_WAIT_POLLS", str(polls))
    for _ in range(5):
        s = gpu.Solver(1, n, bc=BC_OUTFLOW, gamma=G)
        s.upload(U)
        try:
            s.step(50, 0.4)
            s.sync()
        except gpu.NestError as e:
            assert "ran into its limit" in str(e)
        else:
            assert np.array_equal(s.download()[:, 2:-2].view(np.int64), want[:, 2:-2].view(np.int64))
        s.close()
