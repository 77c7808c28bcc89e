"""The branch-free logarithm equals oco_log bit for bit on every positive normal argument and refuses
the others."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILD = os.path.join(ROOT, "tests", "_build")
P = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def check():
    os.makedirs(BUILD, exist_ok=True)
    out = os.path.join(BUILD, "libocomath_nb_host.so")
    subprocess.run(["g++", "-O2", "-mfma", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "ocotillo_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "ocomath_nb_host.cpp")], check=True, capture_output=True)
    h = ctypes.CDLL(out)
    h.log_nb_check.restype = ctypes.c_int64
    h.log_nb_check.argtypes = [P, ctypes.c_int64, ctypes.POINTER(ctypes.c_int64)]

    def run(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        used = ctypes.c_int64()
        return h.log_nb_check(x.ctypes.data_as(P), x.size, ctypes.byref(used)), used.value

    return run


def test_equals_log(check):
    rng = np.random.default_rng(1)
    bits = (rng.integers(1, 0x7fe, 1_000_000).astype(np.uint64) << np.uint64(52)) | rng.integers(0, 1 << 52, 1_000_000).astype(np.uint64)
    near = 1.0 + np.arange(-4096, 4097) * 2.0**-52
    edges = np.concatenate([np.nextafter(v, [0, 3]) for v in (0.75, 1.0, 1.5, 2.0)])
    powers = 2.0 ** np.arange(-1022, 1024)
    for x in (bits.view(np.float64), near, edges, powers, rng.uniform(0.5, 2.0, 500_000)):
        bad, used = check(x)
        assert bad == 0 and used == x.size


def test_refuses(check):
    x = [0.0, -0.0, -1.0, 5e-324, 2.0**-1023, np.inf, -np.inf, np.nan]
    assert check(x) == (0, 0)
