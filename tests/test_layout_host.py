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
    return ctypes.CDLL(out)


def test_records_hold_aligned_pairs(h):
    """Records are read in 16-byte pairs from shared and local memory: the type that holds one there
    carries the alignment, and records lie one after another."""
    assert h.layout_record_alignment() == 16
    assert h.layout_record_doubles() == h.layout_record_fields()
    assert h.layout_record_fields() % 2 == 0
