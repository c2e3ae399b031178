"""The branch-free FP64 reciprocals, quotients and roots (rf_device.cuh) against
IEEE division and root, over random mantissas and the exponents in use."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def helpers(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc to build the test's kernel")
    so = str(tmp_path_factory.mktemp("arith") / "device_arithmetic.so")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", os.path.join(HERE, "..", "rigidfibers_kth_b200", "csrc"), "-o", so,
                    os.path.join(HERE, "device_arithmetic.cu")], check=True)
    return ctypes.CDLL(so).device_arithmetic


# squared distances of 1e-4 .. 1e4 half-lengths, then far wider (the products of
# the last form stay inside the range up to 1e100)
@pytest.mark.parametrize("lo,hi", [(-8, 8), (-30, 30), (-40, 100)])
def test_against_ieee(helpers, lo, hi):
    rng = np.random.default_rng(hi)
    n = 1 << 20
    a = rng.choice([-1, 1], n) * rng.uniform(1, 10, n) * 10.0 ** rng.uniform(lo, hi, n)
    b = rng.uniform(1, 10, n) * 10.0 ** rng.uniform(lo, hi, n)
    out = np.zeros((10, n))
    dp = ctypes.POINTER(ctypes.c_double)
    assert helpers(n, a.ctypes.data_as(dp), b.ctypes.data_as(dp), out.ctypes.data_as(dp)) == 0
    rcp, rsq, root, quo, d3, d5, d7, d10, den, quo6 = out
    L = b.astype(np.longdouble)
    for got, exact in ((rcp, 1 / L), (rsq, 1 / np.sqrt(L))):
        assert np.abs((got - exact) / exact).max() <= 2 * 2.0 ** -53  # two units
    # Correctly rounded but for operands within 2^-45 units of a rounding boundary,
    # which a million random ones hold with a probability below 1e-6
    assert np.array_equal(root, np.sqrt(b))
    assert np.array_equal(quo, a / b)
    assert np.array_equal(quo6, a / den)
    # always correctly rounded
    for got, k in ((d3, 3.0), (d5, -5.0), (d7, 7.0), (d10, -10.0)):
        assert np.array_equal(got, a / k)
