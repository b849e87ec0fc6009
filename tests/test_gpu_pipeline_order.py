"""Stage orders that nest_pipeline_add accepts and sod1d does not use, in the
one-launch form of 1D pipelines against a launch per stage (the same list padded
beyond what the one-launch form takes): the same state, work arrays and errors, bit for bit."""
from __future__ import annotations

import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
G = 1.4


def initial(n, seed=0):
    rng = np.random.default_rng(seed + n)
    x = (np.arange(n) + 0.5) / n
    rho = np.where(x < 0.5, 1.0, 0.125) * (1 + 0.05 * rng.random(n))
    u = 0.2 * np.sin(2 * np.pi * x)
    p = np.where(x < 0.5, 1.0, 0.1) * (1 + 0.02 * rng.random(n))
    return np.stack([rho, rho * u, p / (G - 1) + 0.5 * rho * u * u])


def bits(a):
    return np.where(np.isnan(a), np.nan, a).view(np.int64)


def forms(n, patches, stages, nwork=3):
    """The list in its one-launch form and with a launch per stage."""
    from nest_b200 import pipeline as P
    for pad in (0, 33):
        p = P.Pipeline(1, n, patches, nwork=nwork)
        for kind, kw in stages(P):
            p.add(kind, **kw)
        for _ in range(pad):
            p.add(P.COPY, src=nwork, dst=nwork)
        yield p


def work_view(p, index):
    import torch
    from nest_b200 import _capi as A
    ptr = A.C.c_void_p()
    A.check(A.lib.nest_pipeline_buffer(p._h, index, A.C.byref(ptr)), "nest_pipeline_buffer")
    o = types.SimpleNamespace(__cuda_array_interface__={
        "shape": (p.size,), "typestr": "<f8", "data": (ptr.value, False), "version": 3})
    return torch.as_tensor(o, device="cuda")


@pytest.mark.parametrize("n,patches", [(40, 2), (400, 4), (640, 7), (900, 6), (16000, 9)])
@pytest.mark.parametrize("every", [1, 3])
def test_check_right_behind_cfl(gpu, n, patches, every):
    """A CHECK with no barrier between it and the CFL stage before it: the step in
    which it fails completes everywhere, and nothing runs after it."""
    import torch

    def stages(P):
        return [(P.EXCHANGE, dict(src=0)), (P.CFL_DT, dict(src=0, param=0.3)), (P.CHECK, dict(src=0, param=every)),
                (P.EULER_RHS, dict(src=0, dst=2)), (P.COPY, dict(src=2, dst=0)), (P.CLOCK, {})]
    U = initial(n)
    if every == 1:
        U[2, n // 3] = 0.4 * 0.5 * U[1, n // 3] ** 2 / U[0, n // 3]  # one cell with p < 0
    else:  # uniform with p < 0, wider than two steps reach from both sides
        U[:, n // 4:n // 2] = np.array([1.0, 1.0, 0.4])[:, None]
    for _ in range(3):
        ends = []
        for p in forms(n, patches, stages):
            d = torch.from_numpy(p.scatter(U)).cuda()
            torch.cuda.synchronize()
            with pytest.raises(gpu.NestError) as e:
                p.run(d.data_ptr(), 1e9, max_steps=24)
            torch.cuda.synchronize()
            ends.append((str(e.value), d.cpu().numpy(), work_view(p, 2).cpu().numpy()))
            p.close()
        assert f"at step {every} " in ends[0][0] and f"at step {every} " in ends[1][0]
        if every == 1:  # a single failing cell: one record
            assert ends[0][0] == ends[1][0]
        assert np.array_equal(bits(ends[0][1]), bits(ends[1][1]))
        assert np.array_equal(bits(ends[0][2]), bits(ends[1][2]))


@pytest.mark.parametrize("n,patches", [(60, 2), (300, 3), (640, 7), (900, 6), (8193, 24), (16000, 9)])
def test_work_array_as_the_state(gpu, n, patches):
    """The state is work array 1, which the list uses under both names: what one
    index's stage reads from neighbours is what the other's stage overwrites."""
    import torch

    def stages(P):
        return [(P.CFL_DT, dict(src=0, param=0.3)), (P.EXCHANGE, dict(src=0)), (P.EULER_RHS, dict(src=0, dst=2)),
                (P.COPY, dict(src=2, dst=1)), (P.EXCHANGE, dict(src=1)), (P.EULER_RHS, dict(src=0, dst=3)),
                (P.AVERAGE, dict(src=2, aux=3, dst=1)), (P.CHECK, dict(src=1, param=4)), (P.CLOCK, {})]
    for _ in range(3):
        ends = []
        for p in forms(n, patches, stages, nwork=4):
            d = work_view(p, 1)
            d.copy_(torch.from_numpy(p.scatter(initial(n))))
            torch.cuda.synchronize()
            steps = p.run(d.data_ptr(), 1e9, max_steps=16)
            p.execute(d.data_ptr())
            ends.append((steps, p.clock(), [work_view(p, w).cpu().numpy() for w in (1, 2, 3)]))
            p.close()
        assert ends[0][:2] == ends[1][:2] and ends[0][0] == 16
        for a, b in zip(ends[0][2], ends[1][2]):
            assert np.isfinite(a).all() and np.array_equal(bits(a), bits(b))


@pytest.mark.parametrize("n,patches", [(40, 2), (640, 7), (900, 6), (16000, 9)])
@pytest.mark.parametrize("steps", [3, 8])
def test_cfl_stage_last(gpu, n, patches, steps):
    """The stage that ends a run comes last: the executions that a launch per stage
    still enqueues refresh the halos, unless the run ends with a batch of eight."""
    import torch

    def stages(P):
        return [(P.EXCHANGE, dict(src=0)), (P.EULER_RHS, dict(src=0, dst=2)), (P.COPY, dict(src=2, dst=0)),
                (P.EXCHANGE, dict(src=2)), (P.CLOCK, {}), (P.CFL_DT, dict(src=0, param=0.3))]
    ends = []
    for p in forms(n, patches, stages):
        d = torch.from_numpy(p.scatter(initial(n))).cuda()
        torch.cuda.synchronize()
        p.set_clock(0.0, 0.1 / n, 0)
        for _ in range(steps - 1):
            p.execute(d.data_ptr())
        t, dt, done = p.clock()
        assert done == steps - 1
        p.set_clock(0.0, 0.1 / n, 0)
        d.copy_(torch.from_numpy(p.scatter(initial(n))))
        torch.cuda.synchronize()
        count = p.run(d.data_ptr(), t + 0.5 * dt)  # ends in step `steps`
        ends.append((count, p.clock(), d.cpu().numpy(), work_view(p, 2).cpu().numpy()))
        p.close()
    assert ends[0][:2] == ends[1][:2] and ends[0][0] == steps
    for a, b in zip(ends[0][2:], ends[1][2:]):
        assert np.array_equal(bits(a), bits(b))
