"""The ordered sum (residual_ordered_kernel) of given values against numpy's cumsum of their
squares, bit for bit, where the values or the sum leave the ordinary range: NaN and Inf at every
place, sums that overflow or stay subnormal, terms halfway between two multiples of the sum's
last place, values spread over 600 binades, one value that crosses many binades, and sums so
close below a power of two that the approximate prefix lies in another binade.  Sums that are
not finite take no longer than finite ones: their value is known without a walk."""
import ctypes

import numpy as np
import pytest

from nuc3d_b200 import _LIB_PATH


def _sum(v):
    lib = ctypes.CDLL(str(_LIB_PATH.with_name("libnuc3d_probe.so")))
    P = ctypes.POINTER(ctypes.c_double)
    lib.nuc3d_probe_ordered_sum.restype = ctypes.c_int
    lib.nuc3d_probe_ordered_sum.argtypes = [ctypes.c_int, P, ctypes.c_longlong, P, P]
    v = np.ascontiguousarray(v, dtype=np.float64)
    out, ms = np.empty(3), np.empty(1)
    ptr = lambda x: x.ctypes.data_as(P)  # noqa: E731
    assert lib.nuc3d_probe_ordered_sum(0, ptr(v), v.size, ptr(out), ptr(ms)) == 0
    return out, float(ms[0])


def _finite(n):
    return np.random.default_rng(1).standard_normal(n) * 1e-3


def _with(n, **at):
    v = _finite(n)
    for place, x in at.items():
        v[{"first": 0, "middle": n // 2, "last": n - 1}[place]] = x
    return v


def _ties(n):
    # S in [2, 4): its last place is 2^-51, and the squares of odd multiples of 2^-26 lie
    # halfway between two multiples of it; the other values round either way
    rng = np.random.default_rng(2)
    v = rng.choice([1.0, 3.0, 5.0, 7.0], n) * 2.0 ** -26
    other = rng.random(n) < 0.3
    v[other] = rng.uniform(1.0, 9.0, int(other.sum())) * 2.0 ** -26
    v[0] = 1.5
    return v


def _below_power(n):
    # S just below 2; every later term is below half its last place, but not their sum
    v = np.full(n, 3e-9)
    v[0], v[1] = 1.0, np.sqrt(1.0 - 2.0 ** -50)
    return v


def _crossings(n):
    v = _finite(n)
    v[n // 3] = 40.0
    v[n // 3 + 1] = 1e5
    v[2 * n // 3] = 1e20
    return v


def _spread(n):
    rng = np.random.default_rng(3)
    return rng.uniform(1.0, 2.0, n) * 2.0 ** rng.uniform(-300, 300, n)


def _growing(n):
    return 2.0 ** np.linspace(-530.0, 400.0, n)


NAN, INF = float("nan"), float("inf")
CASES = {
    "nan first": lambda n: _with(n, first=NAN), "nan middle": lambda n: _with(n, middle=NAN),
    "nan last": lambda n: _with(n, last=NAN), "all nan": lambda n: np.full(n, NAN),
    "inf first": lambda n: _with(n, first=INF), "inf middle": lambda n: _with(n, middle=-INF),
    "inf last": lambda n: _with(n, last=INF), "all inf": lambda n: np.full(n, INF),
    "inf then nan": lambda n: _with(n, first=INF, last=NAN), "nan then inf": lambda n: _with(n, first=NAN, last=INF),
    "overflow": lambda n: np.full(n, 1e154), "subnormal": lambda n: _finite(n) * 1e-156,
    "subnormal to normal": lambda n: np.full(n, 2.0 ** -515), "zeros": lambda n: np.zeros(n),
    "ties": _ties, "below a power of two": _below_power, "crossings": _crossings, "spread": _spread,
    "growing": _growing, "finite": _finite,
}


@pytest.mark.gpu
@pytest.mark.parametrize("n", [5, 125, 4095, 4100, 40960, 1100000])
@pytest.mark.parametrize("name", CASES)
def test_sum_is_the_sequential_sum(name, n):
    v = CASES[name](n)
    with np.errstate(all="ignore"):
        want = np.cumsum(v * v)[-1]
    got, _ = _sum(v)
    assert np.array_equal(got, np.full(3, want), equal_nan=True), (got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["nan first", "nan middle", "nan last", "all nan", "inf first", "all inf", "overflow"])
def test_a_sum_that_is_not_finite_takes_no_longer(name):
    n = 5 * 64 ** 3
    t = {k: min(_sum(CASES[k](n))[1] for _ in range(5)) for k in (name, "finite")}
    assert t[name] <= 1.2 * t["finite"], t
