"""The host copies of large pageable outputs (host_copy.cu) with the CUDA calls replaced by plain copies:
complete at every row pitch, and complete on fewer threads where starting one runs out of memory."""
import ctypes
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILD = os.path.join(ROOT, "tests", "_build")

# A process of its own: a failure of a thread's start must not end the process, which a test can only
# see from outside.
CHILD = """
import ctypes, sys
import numpy as np
h = ctypes.CDLL(sys.argv[1])
h.host_copy_run.argtypes = [ctypes.c_void_p, ctypes.c_void_p] + [ctypes.c_size_t] * 3 + [ctypes.c_long]
row, pitch, rows, allow = (int(x) for x in sys.argv[2:])
src = np.random.default_rng(1).integers(0, 256, row * rows, dtype=np.uint8)
dst = np.full(pitch * rows + 64, 7, dtype=np.uint8)
want = dst.copy()
for r in range(rows):
    want[r * pitch:r * pitch + row] = src[r * row:(r + 1) * row]
assert h.host_copy_run(src.ctypes.data, dst.ctypes.data, row, pitch, rows, allow) == 0
assert np.array_equal(dst, want)
print("complete")
"""


@pytest.fixture(scope="module")
def lib():
    os.makedirs(BUILD, exist_ok=True)
    out = os.path.join(BUILD, "libhost_copy_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-Wl,-Bsymbolic", "-I",
                    "/usr/local/cuda/include", "-I", os.path.join(ROOT, "ocotillo_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "host_copy_host.cpp")], check=True, capture_output=True)
    return out


@pytest.mark.parametrize("row,pitch,rows", [(4096, 4096, 700), (999, 1013, 4001), ((5 << 20) + 3, (5 << 20) + 64, 1)])
@pytest.mark.parametrize("allow", [-1, 0, 1, 3])
def test_copies_are_complete(lib, row, pitch, rows, allow):
    r = subprocess.run([sys.executable, "-c", CHILD, lib] + [str(x) for x in (row, pitch, rows, allow)],
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "complete\n", r.stderr[-500:]


@pytest.mark.parametrize("mb,ready", [
    ([4.2], [0]),  # a process that solves one block pays for no pinned memory
    ([4.2, 4.2, 4.2], [0, 1, 1]), ([31.0], [1]), ([0.5, 2.0] * 8, [0] * 16), ([2.9] * 4 + [4.2, 4.2, 2.0], [0] * 5 + [1, 0])])
def test_pinned_memory_waits_for_enough_outputs(lib, mb, ready):
    h = ctypes.CDLL(lib)
    n = (ctypes.c_size_t * len(mb))(*[int(x * (1 << 20)) for x in mb])
    got = (ctypes.c_int * len(mb))()
    h.host_copy_ready(n, len(mb), got)
    assert list(got) == ready
