"""recip_div.h on the device, with the hardware's reciprocal seed: every pattern of a divisor's 20 leading
fraction bits, against the division operator, bit for bit; and the seed's relative error."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BUILD = os.path.join(ROOT, "tests", "_build")


@pytest.fixture(scope="module")
def lib():
    os.makedirs(BUILD, exist_ok=True)
    out = os.path.join(BUILD, "librecip_div_device.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17",
                    "-fmad=false", "-prec-div=true", "-Xcompiler", "-fPIC", "-shared", "-I",
                    os.path.join(ROOT, "ocotillo_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "recip_div_device.cu")], check=True, capture_output=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("seed", [1, 2])
def test_against_the_operator(lib, seed):
    count = (ctypes.c_uint64 * 4)()
    assert lib.recip_div_device(ctypes.c_uint64(seed), count) == 0
    used, recip, quot, seeds = count
    assert used > 15 << 20
    assert (recip, quot, seeds) == (0, 0, 0)
