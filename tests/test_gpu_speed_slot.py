"""The wave-speed word of nest_solver_speed_slot in 1D: what a caller writes there
(a maximum over several domains) sets the next step's dt, also when it asks for the
address again, and whatever kind of step came before."""
from __future__ import annotations

import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
G = 1.4


def state(n):
    x = (np.arange(n + 4) - 2 + 0.5) / n
    rho = 1 + 0.2 * np.sin(2 * np.pi * x)
    u = 0.3 * np.cos(2 * np.pi * x)
    return np.stack([rho, rho * u, np.ones_like(x) / (G - 1) + 0.5 * rho * u * u])


def word(ptr):
    import torch
    o = types.SimpleNamespace(__cuda_array_interface__={
        "shape": (1,), "typestr": "<f8", "data": (ptr, False), "version": 3})
    return torch.as_tensor(o, device="cuda")


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("before", [0, 1, 2, 3, 4, 18, 35])
def test_written_speed_sets_dt(gpu, prec, before):
    import torch
    n, cfl = 5000, 0.4
    precision = gpu.F64 if prec == "f64" else gpu.F32
    s = gpu.Solver(1, n, bc=gpu.BC_PERIODIC, gamma=G, flags=gpu.FLAG_NO_RESIDENT, precision=precision)
    s.upload(state(n).astype(np.float64 if prec == "f64" else np.float32))
    if before:
        s.step(before, cfl)
    s.sync()
    t0 = s.time()[0]
    for k in range(4):
        v = word(s.speed_slot_ptr())
        s.sync()
        speed = float(v.item())
        # dt of the next step, from the value as the steps left it
        assert 1.0 < speed < 2.0
        v.fill_(2.0 * speed)
        torch.cuda.synchronize()
        again = word(s.speed_slot_ptr())
        s.sync()
        assert again.data_ptr() == v.data_ptr() and again.item() == 2.0 * speed
        s.stage(1, cfl)
        s.stage(2, cfl)
        s.sync()
        t1 = s.time()[0]
        assert t1 == t0 + cfl * (1.0 / n) / (2.0 * speed)
        t0 = t1


def test_value_is_the_steps_own(gpu):
    """The word holds the maximum that the last step reduced: no second pass over the
    state replaces it, and a one-launch step reads it from there."""
    import torch
    n, cfl = 5000, 0.4
    a, b = (gpu.Solver(1, n, bc=gpu.BC_PERIODIC, gamma=G, flags=gpu.FLAG_NO_RESIDENT) for _ in range(2))
    for s in (a, b):
        s.upload(state(n))
    for k in (2, 1, 4, 3, 16, 2):
        a.step(k, cfl)
        b.step(k, cfl)
        v = word(a.speed_slot_ptr())
        a.sync()
        torch.cuda.synchronize()
        assert v.item() > 1.0
    assert a.time() == b.time()
    assert np.array_equal(a.download().view(np.int64), b.download().view(np.int64))
