"""The kernels' data layouts (oco_internal.h), compiled for the host."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILD = os.path.join(ROOT, "tests", "_build")


@pytest.fixture(scope="module")
def h():
    os.makedirs(BUILD, exist_ok=True)
    out = os.path.join(BUILD, "liblayout_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", "/usr/local/cuda/include", "-I",
                    os.path.join(ROOT, "ocotillo_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "layout_host.cpp")], check=True, capture_output=True)
    lib = ctypes.CDLL(out)
    lib.layout_tile_level.restype = ctypes.c_int64
    lib.layout_split_doubles.restype = ctypes.c_uint64
    lib.layout_split_doubles.argtypes = [ctypes.c_int64, ctypes.c_int]
    return lib


def test_records_hold_aligned_pairs(h):
    """Records are read in 16-byte pairs from shared and local memory: the type that holds one there
    carries the alignment, and records lie one after another."""
    assert h.layout_record_alignment() == 16
    assert h.layout_record_doubles() == h.layout_record_fields()
    assert h.layout_record_fields() % 2 == 0


def test_split_solve_indexes_tall_columns(h):
    """One column of 2^26 levels fits the device (86 GB of the split solve's scratch), and the offsets
    of its levels do not fit 32 bits."""
    for z in (0, 1, (1 << 26) - 1, 1 << 26, (1 << 26) + 1, (1 << 31) - 1):
        assert h.layout_tile_level(z) == 32 * z
    assert 8 * h.layout_split_doubles(1, (1 << 26) + 1) < 180e9
