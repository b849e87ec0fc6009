"""dt sequences that change on a live solver and a live adjoint: every sweep uses the
sequence that it was given last, as fresh objects do, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
G = 1.4


def state(n, seed):
    x = (np.arange(n + 4) - 2 + 0.5) / n
    rho = 1 + 0.2 * np.sin(2 * np.pi * x + seed)
    u = 0.3 * np.cos(2 * np.pi * x)
    return np.stack([rho, rho * u, (1 + 0.1 * np.cos(2 * np.pi * x)) / (G - 1) + 0.5 * rho * u * u])


def sequences(n, steps):
    rng = np.random.default_rng(n)
    return [0.2 / n * (1 + rng.random(steps)) for _ in range(4)]


@pytest.mark.parametrize("policy,param", [(0, 16), (0, 5), (1, 6)])
def test_adjoint_follows_its_last_sequence(gpu, policy, param):
    from nest_b200.adjoint import Adjoint
    n, steps = 1500, 48
    lam = np.zeros((3, n + 4))
    lam[:, 2:-2] = np.random.default_rng(1).standard_normal((3, n))
    lam[:, :2], lam[:, -2:] = lam[:, -4:-2], lam[:, 2:4]

    def sweep(s, a, dts, seed):
        s.upload(state(n, seed))
        a.forward(0.4, dts)
        return a.backward(lam)

    def make():
        s = gpu.Solver(1, n, bc=gpu.BC_PERIODIC, gamma=G, flags=gpu.FLAG_NO_RESIDENT)
        return s, Adjoint(s, steps, policy, param)
    live = make()
    for seed, dts in enumerate(sequences(n, steps) + [None]):
        got, want = sweep(*live, dts, seed), sweep(*make(), dts, seed)
        assert np.array_equal(got.view(np.int64), want.view(np.int64))


@pytest.mark.parametrize("n,resident", [(300, True), (1500, False)])
def test_solver_follows_its_last_sequence(gpu, n, resident):
    steps = 40

    def make():
        return gpu.Solver(1, n, bc=gpu.BC_PERIODIC, gamma=G, flags=0 if resident else gpu.FLAG_NO_RESIDENT)

    def run(s, dts):
        s.upload(state(n, 0))
        s.reset_time()
        s.freeze_dts(dts)
        s.step(len(dts), 0.4)
        return s.download()
    live = make()
    seqs = sequences(n, steps)
    for dts in seqs + [seqs[0][:17], np.concatenate(seqs), seqs[1]]:
        got, want = run(live, dts), run(make(), dts)
        assert np.array_equal(got.view(np.int64), want.view(np.int64))
