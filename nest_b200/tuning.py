"""Launch-shape autotuner for the 2D stage kernels.

The tunables are the rows each warp marches per tile and the warps per block
(nest_solver_set_tiling).  A sweep times every candidate with profiled steps
(CUDA events between the stage kernels) on a scratch solver of the requested
size and keeps the fastest.  The shape that a solver or batch of that size starts
with, whose tiles are short on small domains, is always among the candidates.
Results are cached in JSON keyed by (device name, SM count, form, nx, ny); the cache
ships with the package (tuning_cache.json) and is extended at run time.  An entry
whose sweep has not timed the present default is swept again.
"""
from __future__ import annotations

import json
import os
from pathlib import Path

import numpy as np

CACHE = Path(os.environ.get("NEST_B200_TUNING", Path(__file__).resolve().parent / "tuning_cache.json"))
ROWS = (16, 24, 32, 64, 128)
WARPS = (1, 2, 4, 8)


def default_tiling(form: str, nx: int, ny: int):
    """(rows per tile, warps per block) that a solver of this form and size starts with."""
    import ctypes as C

    from . import _capi as A
    d = A.SolverDesc(dim=2, nx=nx, ny=ny, halo=2, dx=1.0 / nx, dy=1.0 / ny, gamma=1.4, bc_x=A.BC_OUTFLOW,
                     bc_y=A.BC_OUTFLOW, precision=A.F32 if form == "f32" else A.F64)
    r, w = C.c_int(), C.c_int()
    A.check(A.lib.nest_solver_default_tiling(C.byref(d), C.byref(r), C.byref(w)), "nest_solver_default_tiling")
    return r.value, w.value


def _device_key():
    import torch
    p = torch.cuda.get_device_properties(torch.cuda.current_device())
    return f"{p.name}|{p.multi_processor_count}"


def _load():
    if CACHE.exists():
        try:
            return json.loads(CACHE.read_text())
        except (OSError, json.JSONDecodeError):
            return {}
    return {}


def _key(form, nx, ny):
    return f"{_device_key()}|{form}|{nx}x{ny}"


def sweep(form: str, nx: int, ny: int, steps: int = 6, rows=ROWS, warps=WARPS):
    """Time every (rows, warps) candidate and the default shape; returns
    {(rows, warps): ms per step}."""
    import nest_b200 as nb
    from nest_b200.problems import riemann_2d
    prec = nb.F32 if form == "f32" else nb.F64
    U = riemann_2d(nx, ny)
    if form == "f32":
        U = U.astype(np.float32)
    s = nb.Solver(2, nx, ny, bc=nb.BC_OUTFLOW, precision=prec)
    times = {}
    for r, w in dict.fromkeys([default_tiling(form, nx, ny)] + [(r, w) for r in rows for w in warps]):
        s.set_tiling(r, w)
        s.upload(U)
        s.step_profiled(2, 0.4)  # warm
        _, _, tot = s.step_profiled(steps, 0.4)
        times[(r, w)] = tot / steps
    s.close()
    return times


def autotune(form: str, nx: int, ny: int, steps: int = 6, save: bool = True):
    times = sweep(form, nx, ny, steps)
    best = min(times, key=times.get)
    if save:
        cache = _load()
        cache[_key(form, nx, ny)] = {"rows_per_tile": best[0], "warps_per_block": best[1],
                                      "ms_per_step": times[best],
                                      "candidates": {f"{r}x{w}": t for (r, w), t in sorted(times.items())}}
        try:
            CACHE.write_text(json.dumps(cache, indent=1, sort_keys=True))
        except OSError:
            pass
    return best, times


def best_tiling(form: str, nx: int, ny: int, tune_if_missing: bool = True):
    """Cached best (rows_per_tile, warps_per_block) for this device, form and
    size; tunes (a few hundred ms) when the cache has no entry."""
    default = default_tiling(form, nx, ny)
    e = _load().get(_key(form, nx, ny))
    if e and "%dx%d" % default in e.get("candidates", {}):
        return int(e["rows_per_tile"]), int(e["warps_per_block"])
    if tune_if_missing:
        best, _ = autotune(form, nx, ny)
        return best
    return default


def best_batch_tiling(batch, nx, ny, steps: int = 4, save: bool = True):
    """Cached (rows per item, warps per block, blocks per SM) for a batch of
    these sizes on this device; sweeps the candidates on the batch itself
    (its state is advanced by the sweep: call before uploading)."""
    import hashlib
    key = f"{_device_key()}|batch|{hashlib.sha1(np.asarray([nx, ny]).tobytes()).hexdigest()[:12]}|{len(nx)}"
    cache = _load()
    default = batch.default_tiling() + (0,)
    e = cache.get(key)
    if e and "%dx%dx%d" % default in e.get("candidates", {}):
        return int(e["rows_per_tile"]), int(e["warps_per_block"]), int(e["blocks_per_sm"])
    times = {}
    for shape in dict.fromkeys([default] + [(r, w, bps) for r in (16, 32, 64) for w in (1, 2, 4) for bps in (0, 4)]):
        batch.set_tiling(*shape)
        batch.step_profiled(1, 0.4)
        _, _, tot = batch.step_profiled(steps, 0.4)
        times[shape] = tot / steps
    best = min(times, key=times.get)
    if save:
        cache[key] = {"rows_per_tile": best[0], "warps_per_block": best[1], "blocks_per_sm": best[2],
                      "ms_per_step": times[best],
                      "candidates": {"%dx%dx%d" % k: t for k, t in sorted(times.items())}}
        try:
            CACHE.write_text(json.dumps(cache, indent=1, sort_keys=True))
        except OSError:
            pass
    return best


if __name__ == "__main__":
    import argparse

    ap = argparse.ArgumentParser(description="sweep launch shapes and cache the best")
    ap.add_argument("--sizes", default="4096", help="comma-separated square sizes")
    ap.add_argument("--forms", default="f32,f64")
    ap.add_argument("--out", default="", help="also write the cache to this path")
    a = ap.parse_args()
    for n in [int(x) for x in a.sizes.split(",")]:
        for f in a.forms.split(","):
            best, times = autotune(f, n, n)
            print(f, n, "best", best, "ms/step %.4f" % times[best])
            for k, v in sorted(times.items(), key=lambda kv: kv[1]):
                print("   ", k, "%.4f" % v)
    if a.out:
        Path(a.out).write_text(CACHE.read_text())
