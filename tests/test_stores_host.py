"""The ring through which the sweeps store outputs with z fastest (stores.h), with host threads as the
lanes of a warp: no lane writes the ring while another still reads the forward sweep's shared memory
under it, and every level reaches its place at every alignment and remainder, with nothing around the
rows touched."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILD = os.path.join(ROOT, "tests", "_build")
P = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def h():
    os.makedirs(BUILD, exist_ok=True)
    out = os.path.join(BUILD, "libstores_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-I", "/usr/local/cuda/include", "-I",
                    os.path.join(ROOT, "ocotillo_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "stores_host.cpp")], check=True, capture_output=True)
    lib = ctypes.CDLL(out)
    lib.stores_host_item.argtypes = [ctypes.c_int] * 3 + [P] * 3 + [ctypes.c_int64] * 2
    return lib


def test_ring_waits_for_the_forward_sweep(h):
    assert h.stores_host_early_lanes() == 0


@pytest.mark.parametrize("by_rows", [1, 0])
@pytest.mark.parametrize("rows", [1, 13, 32])
def test_levels_reach_their_places(h, by_rows, rows):
    rng = np.random.default_rng(rows)
    for nz in [4, 5, 11, 12, 13, 19, 20, 21, 28, 35, 64]:
        gap, shift = rng.integers(0, 8, 2)  # elements between rows; of the first row past a 64-byte boundary
        n = {"U": nz + 6, "K": nz, "V": nz}
        pitch = {"U": nz + 6 + gap, "K": nz + gap, "V": nz + gap}
        buf = {k: np.full(32 * pitch[k] + 32, -77.0) for k in n}
        at = {}
        for k in n:  # numpy's buffers are 16-byte aligned: count from a boundary
            at[k] = int(8 - buf[k].ctypes.data // 8 % 8 + shift)
        ptr = {k: ctypes.cast(buf[k].ctypes.data + 8 * at[k], P) for k in n}
        h.stores_host_item(by_rows, nz, rows, ptr["U"], ptr["K"], ptr["V"], pitch["U"], pitch["K"])
        for k in n:
            want = np.full_like(buf[k], -77.0)
            for r in range(rows):
                v = r * 1000.0 + np.arange(n[k])
                want[at[k] + r * pitch[k]:][:n[k]] = {"U": v, "K": v + 0.5, "V": -v}[k]
            assert np.array_equal(buf[k], want), (k, nz, gap, shift)
