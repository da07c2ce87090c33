"""The branch-free FP64 quotients and reciprocals of csrc/div64.cuh, and the
WENO3/5 faces built on them, against IEEE division: operands next to what their
derivations rest on."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGE = 2.0 - 2.0 ** -15  # significands from here on take IEEE division
INF, NAN = float("inf"), float("nan")


def run(kernel_checks, a, b):
    n = len(a)
    a, b, out = np.ascontiguousarray(a), np.ascontiguousarray(b), np.zeros((7, n))
    assert kernel_checks.run_quotients(n, a.ctypes.data_as(C.c_void_p),
                                       b.ctypes.data_as(C.c_void_p),
                                       out.ctypes.data_as(C.c_void_p)) == 0
    return out


def same(x, y):
    return np.all((x == y) & (np.signbit(x) == np.signbit(y)) | (np.isnan(x) & np.isnan(y)))


def near_midpoints(rng, n):
    """Operands whose quotient lies as close to the midpoint t / 2^54 (t odd, of 54
    bits) of two doubles as quotients of doubles come: with d the odd integer
    significand of b and r small and odd, t = r / d modulo 2^54 makes
    a = (t d - r) / 2^54 an integer, and a / b is off the midpoint by r / (2 d) ulp.
    Significands of b are random, next to 1 or next to the edge."""
    a, b = [], []
    top = 2 ** 53
    while len(a) < n:
        d = [int(rng.integers(top // 2, top - top // 2 ** 16)), top // 2 + int(rng.integers(4096)),
             top - top // 2 ** 16 - 1 - int(rng.integers(4096))][len(a) % 3] | 1
        r = (2 * int(rng.integers(8)) + 1) * (-1 if rng.integers(2) else 1)
        t = r * pow(d, -1, 2 * top) % (2 * top)
        if t >= top and d < top - top // 2 ** 16:
            a.append(math.ldexp((t * d - r) >> 54, -53))
            b.append(math.ldexp(d, -52))
    return np.array(a), np.array(b)


def test_quotients_next_to_midpoints(kernel_checks):
    rng = np.random.default_rng(11)
    a, b = near_midpoints(rng, 60000)
    assert b.max() < EDGE
    for ea, eb in ((0, 0), (-300, 400), (880, 90), (-880, -95)):
        x, d = np.ldexp(a, ea), np.ldexp(b, eb)
        by, divisor, ieee = run(kernel_checks, x, d)[:3]
        assert np.array_equal(by, ieee)
        assert np.array_equal(divisor, ieee)


def test_quotients_of_random_operands(kernel_checks):
    rng = np.random.default_rng(12)
    n = 1 << 22
    d = np.ldexp(1.0 + rng.random(n), rng.integers(-100, 100, n))
    x = np.ldexp((1.0 + rng.random(n)) * rng.choice([-1.0, 1.0], n), rng.integers(-890, 890, n))
    by, divisor, ieee = run(kernel_checks, x, d)[:3]
    ok = np.frexp(d)[0] * 2 < EDGE
    assert np.array_equal(by[ok], ieee[ok]) and not np.all(ok)
    assert np.array_equal(divisor, ieee)


def test_divisor_of_any_operands(kernel_checks):
    """Both sides of every limit, with their neighbours, zeros, infinities and
    NaN, in all pairs and both signs."""
    lim = [2.0 ** -100, 2.0 ** 100, EDGE, 2.0, 1.0, EDGE * 2.0 ** -60, 2.0 ** -900, 2.0 ** 900,
           2.0 ** -1022, 5e-324, 1.7976931348623157e308, 3.0]
    with np.errstate(over="ignore"):
        v = [0.0, INF, NAN] + [w for u in lim for w in (u, np.nextafter(u, 0), np.nextafter(u, INF))]
    v = np.array(v + [-w for w in v])
    x, d = (g.ravel() for g in np.meshgrid(v, v))
    _, divisor, ieee = run(kernel_checks, x, d)[:3]
    assert same(divisor, ieee)


def test_hardware_approximations_and_reciprocals(kernel_checks):
    """Every significand of 20 bits (what the approximations read), with the
    lowest and the highest of the 32 bits below: the residuals stay below
    2^-18, rcp64 within 0.51 ulp and rsqrt64 within 1.2 ulp."""
    hi = np.arange(1 << 20, dtype=np.int64)
    eps = np.finfo(np.longdouble).eps
    assert eps < 2.0 ** -60  # the reference below has bits to spare
    for scale in (0, 1, -1021, 1020):
        for low in (0, 0xFFFFFFFF):
            b = ((1023 + scale << 52) | (hi << 32) | low).view(np.float64)
            _, _, _, rcp, rsqrt, e1, e2 = run(kernel_checks, b, b)
            assert np.abs(e1).max() < 2.0 ** -18 and np.abs(e2).max() < 2.0 ** -18
            exact = np.longdouble(b)
            for got, want, ulps in ((rcp, 1 / exact, 0.51), (rsqrt, 1 / np.sqrt(exact), 1.2)):
                err = np.abs(np.longdouble(got) - want)
                assert np.all(err <= ulps * np.longdouble(np.spacing(np.abs(got))))


@pytest.mark.parametrize("order", [3, 5])
def test_weno_faces(kernel_checks, order):
    """Faces with one operand test and with two, bit for bit those with IEEE
    divisions: smooth, rough and constant stencils of sizes from 1e-30 to 1e70, and
    upwind stencils (0, v, w, ...) whose first eps + beta^2 falls in the edge band."""
    rng = np.random.default_rng(13)
    n = 1 << 20
    v = np.ldexp(rng.random((n, 2 * order)) - 0.5, rng.integers(-100, 230, (n, 1)))
    v[::3] = np.ldexp(1.0 + 1e-5 * v[::3] / np.abs(v[::3]).max(axis=1, keepdims=True),
                      rng.integers(-60, 200, (len(v[::3]), 1)))
    v[::17, :order] = v[::17, :1]
    band = np.arange(5, n, 4)
    beta = {3: 1.0, 5: 10.0 / 3.0}[order]  # beta_0 = this * v^2 with the other cells zero
    q = np.ldexp(EDGE + rng.random(len(band)) * 2.0 ** -15, rng.integers(-20, 400, len(band)))
    up = np.zeros((len(band), order))
    up[:, {3: 1, 5: 2}[order]] = np.sqrt(np.sqrt(q) / beta)
    v[band, :order] = up
    # constructed well: eps + beta^2 has an edge significand for nearly all of them
    b0 = beta * up.max(axis=1) ** 2
    assert np.mean(np.frexp(1e-16 + b0 * b0)[0] * 2 >= EDGE) > 0.9
    v = np.ascontiguousarray(v)
    out = np.zeros((3, n))
    assert kernel_checks.run_faces(order, n, v.ctypes.data_as(C.c_void_p),
                                   out.ctypes.data_as(C.c_void_p)) == 0
    assert same(out[0], out[2]) and same(out[1], out[2])
