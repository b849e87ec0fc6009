"""The square root of a quotient that the 1D kernels take their sound speeds from
(sqrt_quot_f64 in nest_b200/csrc/f64div.cuh) against IEEE division and square
root, bit for bit wherever the kernels keep it: the roots nearest to midpoints of two
doubles, divided by one, by powers of two and by general divisors, and operands
over the whole range.  Kept is everything but quotients whose significand is next to
a power of two (two arguments come closer to a midpoint than the method's error)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_gpu_div import bits, nearest_to_midpoints

pytestmark = pytest.mark.gpu


def check(a, b):
    import torch
    from nest_b200 import _capi as A
    da, db = (torch.from_numpy(np.ascontiguousarray(v, dtype=np.float64)).cuda() for v in (a, b))
    dr = torch.empty_like(da)
    dok = torch.zeros(da.numel(), dtype=torch.int32, device="cuda")
    st = A.lib.nest_selftest_sqrt_quot_f64(*(C.c_void_p(t.data_ptr()) for t in (da, db, dr, dok)), da.numel())
    assert st == A.NEST_OK, A.last_error()
    ok = dok.cpu().numpy().astype(bool)
    r, q = dr.cpu().numpy(), a / b
    want = np.sqrt(q)
    frac = bits(q) & ((1 << 52) - 1)
    assert np.array_equal(ok, (frac != 1) & (frac != (1 << 52) - 1))
    bad = ok & (bits(r) != bits(want))
    assert not bad.any(), (bad.sum(), list(zip(a[bad][:5], b[bad][:5], r[bad][:5], want[bad][:5])))


def hard_roots():
    """test_gpu_div.py's doubles whose roots come nearest to a midpoint."""
    xs = []
    for c in range(-513, 512):
        if c % 8 != 7:
            continue
        for mod in (54, 55):
            for m in nearest_to_midpoints(c, mod):
                x = m * m + c
                e = x.bit_length() - 53
                if x % (1 << e) == 0 and x.bit_length() in (107, 108):
                    xs.append((x >> e) * 2.0 ** (e - 106))
    return np.unique(np.array(xs))


def test_hard_roots_over_powers_of_two(gpu):
    xs = hard_roots()
    assert len(xs) > 100
    for k in (0, 1, -1, 7, -20, 33, -45, 50):
        for j in (0, 1, -1, 5, -7, 30, -31):
            b = np.full_like(xs, 2.0 ** j)
            check(xs * 4.0 ** k * b, b)


def test_hard_roots_over_general_divisors(gpu):
    """a = RN(x b) for random b, kept where a / b rounds back to x."""
    xs = hard_roots()
    rng = np.random.default_rng(31)
    x = np.tile(xs, 4000) * 4.0 ** rng.integers(-30, 30, 4000 * len(xs)).astype(np.float64)
    b = rng.uniform(1.0, 2.0, len(x)) * 2.0 ** rng.integers(-30, 30, len(x)).astype(np.float64)
    b[: len(x) // 4] = (2.0 - np.spacing(1.0) * rng.integers(1, 64, len(x) // 4))
    a = x * b
    keep = a / b == x
    assert keep.mean() > 0.5
    check(a[keep], b[keep])


@pytest.mark.parametrize("seed", [1, 2])
def test_wide_range(gpu, seed):
    rng = np.random.default_rng(seed)
    n = 4_000_000
    a = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-128, 138, n).astype(np.float64)
    b = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-128, 128, n).astype(np.float64)
    q = n // 4
    a[:q] = 1.4 * rng.uniform(1e-3, 10.0, q)                 # gamma p over rho as solvers meet them
    b[:q] = rng.uniform(1e-3, 10.0, q)
    s = rng.uniform(1.0, 2.0, q)                             # roots next to doubles
    b[q:2 * q] = rng.uniform(1.0, 2.0, q)
    a[q:2 * q] = s * s * b[q:2 * q]
    a[2 * q:3 * q] = np.nextafter(4.0, 0) - np.spacing(2.0) * rng.integers(0, 1 << 20, q)
    b[2 * q:3 * q] = 1.0
    check(a, b)


def test_sound_speed_of_uniform_states(gpu):
    """dt of uniform states at rest whose gamma p / rho rounds to one of the two
    hardest arguments, (1 + ulp) 4^k and (4 - 2 ulp) 4^k: IEEE's sound speed."""
    rng = np.random.default_rng(5)
    n, g, cfl = 8, 1.5, 0.4
    pairs = []
    while len(pairs) < 1500:
        x = (1.0 + 2.0 ** -52, 4.0 - 2.0 ** -51)[len(pairs) % 2] * 4.0 ** int(rng.integers(-20, 20))
        rho = rng.uniform(1.0, 2.0) * 2.0 ** int(rng.integers(-20, 20))
        a = x * rho
        for p in (a / g, np.nextafter(a / g, 0), np.nextafter(a / g, np.inf)):
            if g * p == a and a / rho == x:
                pairs.append((rho, p, x))
                break
    s = gpu.Solver(1, n, bc=gpu.BC_PERIODIC, gamma=g)
    U = np.zeros((3, n + 4))
    wrong = 0
    for rho, p, x in pairs:
        U[0], U[2] = rho, p / (g - 1.0)  # gamma - 1 = 1/2: exact
        s.upload(U)
        wrong += s.compute_dt(cfl) != cfl * (1.0 / n) / np.sqrt(x)
    assert wrong == 0, wrong
