"""The integer long division equals the correctly rounded float64 quotient."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("quot") / "quot.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-o", so,
                           os.path.join(ROOT, "tests", "native", "quot_check.cpp")])
    L = ctypes.CDLL(so)
    L.pgld_check_remainder.restype = ctypes.c_double
    L.pgld_check_remainder.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                                       ctypes.c_double]
    return L


def operands(rng, n):
    """Positive integers below 2^53 over every size, small ones, ratios near a tie."""
    a = np.exp2(rng.uniform(0, 53, n)).astype(np.int64)
    b = np.exp2(rng.uniform(0, 53, n)).astype(np.int64)
    a[:2000], b[2000:4000] = rng.integers(1, 50, 2000), rng.integers(1, 50, 2000)
    b[4000:6000] = 1 << rng.integers(0, 52, 2000)
    a[6000:8000] = (1 << 53) - rng.integers(1, 9, 2000)
    b[7000:9000] = (1 << 53) - rng.integers(1, 9, 2000)
    b[9000:11000] = (1 << 52) + rng.integers(0, 9, 2000)
    a[11000:13000] = b[11000:13000]
    top = (1 << 53) - 1
    return np.clip(a, 1, top), np.clip(b, 1, top)


@pytest.mark.parametrize("seed", range(4))
def test_quotient_is_correctly_rounded(lib, seed):
    rng = np.random.default_rng(seed)
    a, b = operands(rng, 400_000)
    a[::2] *= -1
    a[::97] = 0
    big = rng.random(a.size) < 0.05  # operands above 53 bits: rounded first
    a[big] = rng.integers(-(1 << 62), 1 << 62, big.sum())
    out = np.zeros(a.size)
    lib.pgld_check_quot(a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p),
                        a.size, out.ctypes.data_as(ctypes.c_void_p))
    assert np.array_equal(out, a.astype(np.float64) / b.astype(np.float64))


# the device's reciprocal is within one unit of its last place (2^-23 relative)
@pytest.mark.parametrize("off", [-2.0 ** -23, 0.0, 2.0 ** -23])
def test_remainder_stays_below_two(lib, off):
    a, b = operands(np.random.default_rng(9), 400_000)
    worst = lib.pgld_check_remainder(a.ctypes.data, b.ctypes.data, a.size, off)
    assert 0.0 <= worst < 2.0
