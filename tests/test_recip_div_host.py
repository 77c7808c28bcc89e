"""recip_div.h compiled for the host: every quotient and reciprocal that passes the operand checks
is the IEEE one (bit for bit), and the operands the method does not cover are refused."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILD = os.path.join(ROOT, "tests", "_build")
P = ctypes.POINTER(ctypes.c_double)
N = 2_000_000


@pytest.fixture(scope="module")
def h():
    os.makedirs(BUILD, exist_ok=True)
    out = os.path.join(BUILD, "librecip_div_host.so")
    subprocess.run(["g++", "-O2", "-mfma", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "ocotillo_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "recip_div_host.cpp")], check=True, capture_output=True)
    lib = ctypes.CDLL(out)
    lib.recip_div_check.restype = ctypes.c_int64
    lib.recip_div_check.argtypes = [P, P, ctypes.c_int64, ctypes.POINTER(ctypes.c_int64)]
    lib.recip_div_accepts.argtypes = [ctypes.c_double, ctypes.c_double]
    return lib


def _mantissas(rng, n):
    """Significands in [1, 2): random, sparse, next to 1, next to 2 (2^-20 and beyond excluded by
    the check)."""
    k = rng.integers(0, 4, n)
    f = rng.integers(0, 1 << 52, n)
    f = np.where(k == 1, f & (rng.integers(0, 1 << 52, n) & rng.integers(0, 1 << 52, n)), f)
    f = np.where(k == 2, rng.integers(0, 1 << 12, n), f)
    f = np.where(k == 3, (1 << 52) - 1 - rng.integers(0, 1 << 34, n), f)
    return (f.astype(np.uint64) | np.uint64(1023 << 52)).view(np.float64)


def _operands(kind, rng):
    sign = rng.choice([-1.0, 1.0], N)
    b = _mantissas(rng, N)
    if kind == "random":
        a = _mantissas(rng, N)
    elif kind == "exact":  # quotients that are representable
        b = np.ldexp(np.floor(np.ldexp(b, 25)), -25)
        a = b * np.ldexp(np.floor(np.ldexp(_mantissas(rng, N), 25)), -25)
    else:  # dividends next to a midpoint between two quotients
        q = _mantissas(rng, N)
        a = (b.astype(np.longdouble) * (q.astype(np.longdouble) + np.longdouble(2.0) ** -53)).astype(np.float64)
        a = np.nextafter(a, a * rng.choice([0.0, 1.0, 2.0], N))
    return np.ldexp(a * sign, rng.integers(-759, 478, N)), np.ldexp(b, rng.integers(-200, 200, N))


@pytest.mark.parametrize("kind", ["random", "exact", "midpoint"])
def test_checked_quotients_are_ieee(h, kind):
    rng = np.random.default_rng({"random": 1, "exact": 2, "midpoint": 3}[kind])
    a, b = (np.ascontiguousarray(x) for x in _operands(kind, rng))
    used = ctypes.c_int64()
    bad = h.recip_div_check(a.ctypes.data_as(P), b.ctypes.data_as(P), N, ctypes.byref(used))
    assert bad == 0
    assert used.value > 0.6 * N


def test_refused_operands(h):
    ones = 2.0 - 2.0**-52
    inf, nan = float("inf"), float("nan")
    for b in (0.0, -0.0, inf, -inf, nan, 5e-324, 2.0**-201, 2.0**200, ones, -ones, 2.0 - 2.0**-21):
        assert not h.recip_div_accepts(1.0, b), b
    for a in (0.0, -0.0, inf, -inf, nan, 5e-324, 2.0**-761, 2.0**480):
        assert not h.recip_div_accepts(a, 3.0), a
    for a, b in ((1.0, 1.0), (-1.0, 2.0 - 2.0**-19), (2.0**-760, -(2.0**-200)), (1.99 * 2.0**479, 1.99 * 2.0**199)):
        assert h.recip_div_accepts(a, b), (a, b)
