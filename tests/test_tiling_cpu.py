"""Default launch shapes, worked out on the host, and the tuner's use of its cache."""
from __future__ import annotations

import ctypes as C
import json

import numpy as np
import pytest


def test_default_shapes():
    from nest_b200.tuning import default_tiling
    for form in ("f32", "f64"):
        rows = [default_tiling(form, n, n)[0] for n in (8, 64, 256, 512, 1024, 4096)]
        assert rows[0] == 1 and rows == sorted(rows) and rows[-1] in (16, 24)


def test_bad_descriptions_are_refused():
    from nest_b200 import _capi as A
    r, w = C.c_int(), C.c_int()
    for kw in (dict(dim=1, nx=64, ny=64), dict(dim=2, nx=3, ny=64), dict(dim=2, nx=64, ny=2)):
        d = A.SolverDesc(halo=2, gamma=1.4, precision=A.F64, **kw)
        assert A.lib.nest_solver_default_tiling(C.byref(d), C.byref(r), C.byref(w)) == 1
    assert A.lib.nest_solver_default_tiling(None, C.byref(r), C.byref(w)) == 1


def test_cached_sweep_without_the_default_is_not_used(tmp_path, monkeypatch):
    """A cached sweep of tall tiles only does not answer for a small domain."""
    from nest_b200 import tuning
    monkeypatch.setattr(tuning, "CACHE", tmp_path / "cache.json")
    monkeypatch.setattr(tuning, "_device_key", lambda: "gpu")
    old = {"rows_per_tile": 16, "warps_per_block": 1, "ms_per_step": 1.0, "candidates": {"16x1": 1.0, "32x4": 2.0}}
    tuning.CACHE.write_text(json.dumps({"gpu|f32|256x192": old, "gpu|f32|4096x4096": old}))
    assert tuning.best_tiling("f32", 4096, 4096, tune_if_missing=False) == (16, 1)
    default = tuning.default_tiling("f32", 256, 192)
    assert default[0] < 8
    assert tuning.best_tiling("f32", 256, 192, tune_if_missing=False) == default


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_default_can_be_set_back(gpu, prec):
    from nest_b200.tuning import default_tiling, sweep
    nx, ny = 256, 192
    rows, warps = default_tiling(prec, nx, ny)
    flags = gpu.FLAG_TOTALS
    s = gpu.Solver(2, nx, ny, precision=gpu.F32 if prec == "f32" else gpu.F64, flags=flags)
    U = np.ones((4, nx + 4, ny + 4)) * np.array([1.0, 0.1, -0.2, 2.5])[:, None, None]
    U[0] += 0.1 * np.random.default_rng(1).random(U[0].shape)
    ends = []
    for shape in (None, (16, 4), (rows, warps), (8, 1)):
        if shape:
            s.set_tiling(*shape)
        s.upload(U.astype(s.dtype))
        s.step(4, 0.4)
        ends.append((s.download()[:, 2:-2, 2:-2], s.totals()))
    for e in ends[1:]:
        assert np.array_equal(e[0], ends[0][0])
        np.testing.assert_allclose(e[1], ends[0][1], rtol=1e-12, atol=1e-12)
    assert np.array_equal(ends[2][1], ends[0][1])
    for bad in (0, rows - 1, 4097):
        with pytest.raises(gpu.NestError):
            s.set_tiling(bad, 1)
    times = sweep(prec, nx, ny, steps=2, rows=(16,), warps=(1,))
    assert set(times) == {(rows, warps), (16, 1)}


@pytest.mark.gpu
def test_batch_default_can_be_set_back(gpu):
    nx, ny = [64, 96, 48], [64, 70, 33]
    b = gpu.Batch(nx, ny)
    rows, warps = b.default_tiling()
    items = b.info()[1:]
    b.set_tiling(16, 1, 4)
    assert b.info()[1:] != items
    b.set_tiling(rows, warps)
    assert b.info()[1:] == items
    with pytest.raises(gpu.NestError):
        b.set_tiling(rows - 1, warps)
