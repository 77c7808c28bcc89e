"""The block solves' rules by size (oco_internal.h), compiled for the host.  The split solve takes few tiles
and grey transfer, and never grids beyond the caller's cap, by which a server shares the GPU between jobs;
by-item chunks count as few while their warps fit; the mixed form's ring takes z-fastest outputs above 56 MiB."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILD = os.path.join(ROOT, "tests", "_build")
SMS = 148


@pytest.fixture(scope="module")
def h():
    os.makedirs(BUILD, exist_ok=True)
    out = os.path.join(BUILD, "libsplit_rule_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", "/usr/local/cuda/include", "-I",
                    os.path.join(ROOT, "ocotillo_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "split_rule_host.cpp")], check=True, capture_output=True)
    lib = ctypes.CDLL(out)
    lib.split_rule.argtypes = [ctypes.c_int, ctypes.c_int64] + [ctypes.c_int] * 4
    lib.split_grid.argtypes = [ctypes.c_int64, ctypes.c_int, ctypes.c_int]
    lib.split_grid.restype = ctypes.c_int64
    lib.items_few.argtypes = [ctypes.c_int, ctypes.c_int64, ctypes.c_int]
    lib.mixed_mode.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int64, ctypes.c_int]
    return lib


@pytest.mark.parametrize("cap", [1, 7, 74, 148, 592])
@pytest.mark.parametrize("ncol,nw,nz", [(1, 64, 12), (1, 64, 512), (16, 250, 500), (148, 64, 33), (992, 5, 33), (40, 33, 17)])
def test_the_split_grids_fit_the_cap(h, cap, ncol, nw, nz):
    grid = h.split_grid(ncol, nw, nz)
    assert h.split_rule(0, ncol, nw, nz, SMS, cap) == (grid <= cap)
    assert h.split_rule(0, ncol, nw, nz, SMS, 0) == 1


@pytest.mark.parametrize("ncol,nw,split", [(296, 32, 1), (297, 32, 0), (1894, 5, 1), (1895, 5, 0), (37, 250, 1), (38, 250, 0)])
def test_two_tiles_per_sm(h, ncol, nw, split):
    assert h.split_rule(0, ncol, nw, 100, SMS, 0) == split
    assert h.split_rule(1, ncol, 1, 100, SMS, 0) == 1


@pytest.mark.parametrize("mixed,blocks", [(0, 2), (1, 4)])
def test_few_items(h, mixed, blocks):
    n = SMS * blocks * 128
    assert [h.items_few(mixed, i, SMS) for i in (1, n, n + 1, 1 << 40)] == [1, 1, 0, 0]


def test_mixed_ring_from_a_size_on(h):
    lane, ring, planes = 0, 1, 2
    for arrays in (1, 2, 3):
        points = (56 << 20) // 8 // arrays
        assert h.mixed_mode(arrays, 0, points, 1) == lane and h.mixed_mode(arrays, 0, points + 1, 1) == ring
        assert h.mixed_mode(arrays, 0, points // 7, 7) == lane and h.mixed_mode(arrays, 0, points // 7 + 1, 7) == ring
        assert h.mixed_mode(arrays, 1, 1 << 40, 100) == lane
    assert h.mixed_mode(0, 0, 1 << 40, 100) == planes and h.mixed_mode(0, 1, 1, 1) == planes


def test_short_columns_are_not_split(h):
    assert [h.split_rule(0, 4, 64, nz, SMS, 0) for nz in (2, 11, 12, 13)] == [0, 0, 1, 1]
    assert h.split_rule(1, 4, 1, 2, SMS, 0) == 1
