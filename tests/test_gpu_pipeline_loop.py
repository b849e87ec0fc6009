"""The one-launch form of 1D pipelines (one CTA, or one thread-block cluster)
against a launch per stage: a stage list longer than the one-launch form takes is
run stage by stage, so the same pipeline padded with copies of a buffer onto
itself must give the same state (halos included), clock and errors, bit for bit, at the sizes where the form changes."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
G = 1.4


def initial(n, seed, scale=1.0):
    rng = np.random.default_rng(seed)
    x = (np.arange(n) + 0.5) / n
    rho = scale * (np.where(x < 0.5, 1.0, 0.125) * (1 + 0.05 * np.sin(6 * np.pi * x)) + 0.01 * rng.random(n))
    u = 0.2 * np.sin(2 * np.pi * x)
    u[rng.random(n) < 0.2] = 0.0
    p = scale * np.where(x < 0.5, 1.0, 0.1) * (1 + 0.02 * rng.random(n))
    return np.stack([rho, rho * u, p / (G - 1) + 0.5 * rho * u * u])


def pair(n, patches, limiter=0, halo=2, order="sod1d"):
    """The pipeline in its one-launch form and, padded, with a launch per stage."""
    from nest_b200 import pipeline as P
    out = []
    for pad in (0, 30):
        if order == "sod1d":
            p = P.sod1d_pipeline(n, patches, halo=halo, limiter=limiter)
        else:  # the exchange and a check first, forward Euler, two clocks' worth of stages last
            p = P.Pipeline(1, n, patches, halo=halo, limiter=limiter, nwork=3)
            p.add(P.EXCHANGE, src=P.STATE).add(P.CHECK, src=P.STATE, param=3).add(P.CFL_DT, src=P.STATE, param=0.3)
            p.add(P.EULER_RHS, src=P.STATE, dst=2).add(P.AVERAGE, src=2, aux=2, dst=3).add(P.COPY, src=3, dst=P.STATE)
            p.add(P.EXCHANGE, src=3).add(P.CLOCK)
        for _ in range(pad):
            p.add(P.COPY, src=1, dst=1)
        out.append(p)
    return out


@pytest.mark.parametrize("n,patches,limiter,halo,order", [
    (33, 3, 0, 2, "sod1d"), (400, 4, 1, 3, "sod1d"), (640, 7, 0, 2, "other"), (641, 7, 0, 2, "sod1d"),
    (1000, 5, 2, 2, "other"), (8192, 16, 0, 2, "sod1d"), (8193, 24, 1, 2, "other"), (16384, 9, 0, 2, "sod1d"),
    (16385, 9, 0, 2, "sod1d")])
def test_matches_a_launch_per_stage(gpu, n, patches, limiter, halo, order):
    import torch
    ends = []
    for p in pair(n, patches, limiter, halo, order):
        smooth = limiter == 2
        U = initial(n, n)
        if smooth:  # the unlimited reconstruction needs a smooth state
            x = (np.arange(n) + 0.5) / n
            U = np.stack([1 + 0.1 * np.sin(2 * np.pi * x), 0.1 * np.cos(2 * np.pi * x), 2.5 + 0 * x])
        d = torch.from_numpy(p.scatter(U)).cuda()
        steps = [p.run(d.data_ptr(), 1e9, max_steps=13)]  # whole batches of 8
        p.execute(d.data_ptr())
        clocks = [p.clock()]
        steps.append(p.run(d.data_ptr(), clocks[0][0] + 20.5 * clocks[0][1]))  # clips the last step
        clocks.append(p.clock())
        ends.append((steps, clocks, d.cpu().numpy()))
        p.close()
    assert ends[0][0] == ends[1][0] and ends[0][0][0] == 16
    assert ends[0][1] == ends[1][1]
    assert np.isfinite(ends[0][2]).all()
    assert np.array_equal(ends[0][2].view(np.int64), ends[1][2].view(np.int64))


@pytest.mark.parametrize("n,patches", [(400, 4), (900, 6)])
def test_failures_and_scales(gpu, n, patches):
    """A positivity failure stops both forms at the same step, cell and state;
    states outside the branch-free arithmetic's range agree too."""
    import torch
    for scale, break_it in ((1.0, True), (1e-45, False)):
        ends = []
        for p in pair(n, patches):
            U = initial(n, 3, scale)
            if break_it:
                U[1, n // 4:n // 2], U[2, n // 4:n // 2] = 2.0 * U[0, n // 4:n // 2], 0.4
            d = torch.from_numpy(p.scatter(U)).cuda()
            msg = ""
            try:
                p.run(d.data_ptr(), 1e9, max_steps=24)
            except gpu.NestError as e:
                msg = str(e)
            torch.cuda.synchronize()
            ends.append((msg, d.cpu().numpy()))
            p.close()
        assert ("at step 10 " in ends[0][0]) == break_it
        if not break_it:
            assert ends[0][0] == ends[1][0] == ""
            assert np.array_equal(ends[0][1].view(np.int64), ends[1][1].view(np.int64))


@pytest.mark.parametrize("n,patches,nwork,alias", [
    (28, 1, 3, False), (29, 1, 3, False), (84, 3, 3, False), (87, 3, 3, False), (300, 20, 3, False),
    (301, 10, 3, True), (630, 2, 16, False), (1300, 13, 3, False), (1400, 100, 3, False), (15000, 2, 3, False)])
def test_shared_faces_and_buffers(gpu, n, patches, nwork, alias):
    """Patches around the cells of a warp that shares faces (28) and too short
    for it; buffers too large for shared memory, and a work array passed as
    the state: state and work arrays equal a launch per stage, bit for bit."""
    import torch
    from nest_b200 import _capi as A
    from nest_b200 import pipeline as P
    ends = []
    for pad in (0, 30):
        p = P.Pipeline(1, n, patches, nwork=nwork)
        p.add(P.CFL_DT, src=P.STATE, param=0.4).add(P.EXCHANGE, src=P.STATE).add(P.COPY, src=P.STATE, dst=1)
        p.add(P.EULER_RHS, src=P.STATE, dst=2).add(P.COPY, src=2, dst=P.STATE).add(P.EXCHANGE, src=P.STATE)
        p.add(P.EULER_RHS, src=P.STATE, dst=2).add(P.AVERAGE, src=1, aux=2, dst=P.STATE).add(P.CLOCK)
        for _ in range(pad):
            p.add(P.COPY, src=1, dst=1)
        U = torch.from_numpy(p.scatter(initial(n, n))).cuda()
        work = []
        for w in range(1, nwork + 1):
            ptr = A.C.c_void_p()
            A.check(A.lib.nest_pipeline_buffer(p._h, w, A.C.byref(ptr)), "nest_pipeline_buffer")
            work.append(ptr.value)

        def view(ptr):
            import types
            o = types.SimpleNamespace(__cuda_array_interface__={
                "shape": (p.size,), "typestr": "<f8", "data": (ptr, False), "version": 3})
            return torch.as_tensor(o, device="cuda")
        state = view(work[2]) if alias else U
        state.copy_(U)
        torch.cuda.synchronize()
        steps = p.run(state.data_ptr(), 1e9, max_steps=8)
        p.execute(state.data_ptr())
        clock = p.clock()
        ends.append((steps, clock, state.cpu().numpy(), [view(w).cpu().numpy() for w in work]))
        p.close()
    assert ends[0][:2] == ends[1][:2] and ends[0][1][2] == 9
    assert np.isfinite(ends[0][2]).all()
    assert np.array_equal(ends[0][2].view(np.int64), ends[1][2].view(np.int64))
    for a, b in zip(ends[0][3], ends[1][3]):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))
