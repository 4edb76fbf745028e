"""The FP64 lane's integer arithmetic as the device runs it (carry chains, approximate
reciprocals, funnel shifts: other code than the host build of the same header) against
IEEE operations, on the operands where rounding goes wrong if it does."""
import ctypes as C

import numpy as np
import pytest

from conformal_cubed_sphere_gb300 import _lib as L

pytestmark = pytest.mark.gpu

(MUL, MUL_UNPACKED, DIV, DIV_UNPACKED, ONE_PLUS_DIV, ADD, SQRT, CURVATURE, GRID_DIV, DIV6, HALF,
 RECONSTRUCTION) = range(12)
N = 5 * (1 << 19)


def check(what, a, b):
    a, b = (np.ascontiguousarray(x, dtype=np.float64) for x in (a, b))
    fast, ieee = np.empty(a.size), np.empty(a.size)
    p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in (a, b, fast, ieee)]
    assert L.lib().ccs_selftest_integer(what, p[0], p[1], a.size, p[2], p[3]) == L.CCS_OK
    nan = np.isnan(ieee)
    bad = np.flatnonzero((fast.view(np.int64) != ieee.view(np.int64)) & ~(nan & np.isnan(fast)))
    assert bad.size == 0, (what, bad.size, a[bad[0]].hex(), b[bad[0]].hex(), fast[bad[0]].hex(), ieee[bad[0]].hex())
    return ieee


def significands(rng, n):
    """random, few leading bits, long runs of ones, powers of two and their neighbours"""
    m = rng.integers(0, 1 << 52, size=n, dtype=np.uint64)
    kind = rng.integers(0, 6, size=n)
    sh = rng.integers(0, 52, size=n).astype(np.uint64)
    ones = np.uint64((1 << 52) - 1)
    m = np.where(kind == 1, m & (ones << sh) & ones, m)
    m = np.where(kind == 2, m | ((np.uint64(1) << sh) - np.uint64(1)), m)
    m = np.where(kind == 3, np.where(m % np.uint64(3) == 0, ones, np.uint64(0)), m)
    m = np.where(kind == 4, m % np.uint64(16), m)
    return np.where(kind == 5, ones - m % np.uint64(16), m)


def doubles(rng, lo, hi, n=N):
    e = rng.integers(1023 + lo, 1023 + hi + 1, size=n).astype(np.uint64)
    return ((e << np.uint64(52)) | significands(rng, n)).view(np.float64)


def nudge(rng, x):
    return (x.view(np.int64) + rng.integers(-2, 3, size=x.size)).view(np.float64)


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_operations(seed):
    rng = np.random.default_rng(seed)
    a, b = doubles(rng, -200, 199), doubles(rng, -200, 199)
    near = nudge(rng, np.where(rng.random(N) < 0.5, b * doubles(rng, -3, 3), b))  # quotients next to representable ones
    for what in (MUL, MUL_UNPACKED):
        assert np.array_equal(check(what, a, b), a * b)
    for what in (DIV, DIV_UNPACKED):
        assert np.array_equal(check(what, a, b), a / b)
        check(what, near, b)
    check(ONE_PLUS_DIV, a, b)
    check(ONE_PLUS_DIV, near, b)
    check(ONE_PLUS_DIV, doubles(rng, -60, 60), doubles(rng, -3, 3))
    c, d = doubles(rng, -70, 70), doubles(rng, -3, 3)
    assert np.array_equal(check(ADD, c, d), c + d)
    check(ADD, d, c)
    assert np.array_equal(check(SQRT, a, b), np.sqrt(a))
    r = doubles(rng, -90, 90)
    check(SQRT, nudge(rng, r * r), b)
    check(SQRT, nudge(rng, np.full(N, 4.0)), b)
    sign = rng.choice([1.0, -1.0], size=N)
    z = np.where(rng.random(N) < 0.01, 0.0, a) * sign
    check(CURVATURE, z, b)
    check(CURVATURE, doubles(rng, -250, 202) * sign, b)


@pytest.mark.parametrize("seed", [4, 5])
def test_quotients_of_any_double(seed):
    """By a grid spacing, by six and by two: every dividend, with zeros, subnormals,
    infinities and NaNs, and divisors on both sides of the integer quotients' range."""
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 1 << 64, size=N, dtype=np.uint64, endpoint=False).view(np.float64).copy()
    a[:N // 2] = doubles(rng, -1022, 1023, N // 2) * rng.choice([1.0, -1.0], size=N // 2)
    a[:8] = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0 ** 1023]
    for b in (doubles(rng, -405, 305), doubles(rng, -40, 40), doubles(rng, -1022, 1023)):
        check(GRID_DIV, a, b)
    check(DIV6, a, a)
    check(HALF, a, a)


@pytest.mark.parametrize("seed", range(6, 12))
def test_reconstructions(seed):
    """Windows of five cells: unrelated values, small variations of one value, straight lines
    and parabolas with noise in the last places, equal cells, steps, mixed signs, zeros, and
    values at the ends of the window."""
    rng = np.random.default_rng(seed)
    m = N // 5
    w = doubles(rng, -199, 198, N).reshape(m, 5) * rng.choice([1.0, -1.0], size=(m, 5))
    kind = rng.integers(0, 8, size=m)
    base = doubles(rng, -60, 60, m)[:, None] * rng.choice([1.0, -1.0], size=(m, 1))
    x = np.arange(-2.0, 3.0)[None, :]
    small = base * (1 + rng.normal(size=(m, 5)) * 2.0 ** rng.integers(-52, 0, size=(m, 1)).astype(float))
    line = nudge(rng, np.ravel(base * (1 + x * 2.0 ** rng.integers(-40, 2, size=(m, 1)).astype(float)))).reshape(m, 5)
    para = nudge(rng, np.ravel(base * (1.5 + 0.1 * x + x * x * 2.0 ** rng.integers(-30, 2, size=(m, 1)).astype(float)))
                 ).reshape(m, 5)
    step = np.where(x < rng.integers(-2, 3, size=(m, 1)), base, base * 2.0 ** rng.integers(-20, 20, size=(m, 1)).astype(float))
    few = base * rng.choice([0.0, 1.0, -1.0, 2.0, 0.5], size=(m, 5))
    for k, v in ((1, small), (2, line), (3, para), (4, step), (5, few), (6, np.repeat(base, 5, axis=1))):
        w = np.where((kind == k)[:, None], v, w)
    near = doubles(rng, -40, 40, N).reshape(m, 5) * rng.choice([1.0, -1.0], size=(m, 5))
    w = np.where((kind == 7)[:, None], near, w)
    # the window, to which zeros belong (a nudged zero may be a NaN)
    w = np.where((np.abs(w) >= 2.0 ** -200) & (np.abs(w) < 2.0 ** 200), w, 0.0)
    ieee = check(RECONSTRUCTION, w.ravel(), w.ravel())
    assert np.isfinite(ieee[:m]).all() and not ieee[m:].any()
