"""The unrolled statistics of two to four populations, built for the host.

pg_gpu_gb300/csrc/pgld_multi.cuh is compiled with g++ and evaluated on count
tables of tiny, odd and large populations.  Haplotype statistics and the
genotype ones of mixed populations are sums of at most 16 non-negative products
of features of one rounding each, or one signed product: within 12 roundings of
their terms' absolute sum.  Each value must lie within 1e-6 of the oracle's,
where the oracle value is at least 1e-3 of the statistic's largest (below it
the two signed products of a Dz term may cancel), and within 1e-9 of that
largest value otherwise.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import ld_oracle as O
from tests.conftest import ROOT

SRC = os.path.join(ROOT, "tests", "native", "multi_check.cpp")


@pytest.fixture(scope="module")
def check_lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("multi") / "multi.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o",
                           so, SRC])
    L = ctypes.CDLL(so)
    L.pgld_check_multi.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                   ctypes.c_void_p, ctypes.c_int]
    L.pgld_check_den.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    return L


@pytest.mark.parametrize("geno", [False, True])
@pytest.mark.parametrize("P", [2, 3, 4])
@pytest.mark.parametrize("nmax", [4, 7, 61, 1000, 2047])
def test_multi_population_statistics_match_oracle(check_lib, P, geno, nmax):
    rng = np.random.default_rng(100 * P + nmax)
    N, K = 2000, 9 if geno else 4
    c = np.zeros((N, P, K), np.int32)
    for k in range(N):
        for p in range(P):
            n = int(rng.integers(4, nmax + 1))
            c[k, p] = rng.multinomial(n, rng.dirichlet(np.full(K, 0.4)))
    cs, nv = [c[:, p] for p in range(P)], [None] * P
    ref = (O.geno_multi_pop_stats if geno else O.multi_pop_stats)(cs, nv)
    out = np.full(ref.shape, np.nan, np.float32)
    check_lib.pgld_check_multi(c.ctypes.data, N, P, int(geno), out.ctypes.data, ref.shape[1])
    big = np.abs(ref).max(0)
    tol = np.where(np.abs(ref) >= 1e-3 * big, 1e-6 * np.abs(ref), 1e-9 * big)
    err = np.abs(out - ref)
    bad = np.argwhere(err > tol)
    assert len(bad) == 0, [(O.ld_names(P)[s], ref[k, s], out[k, s]) for k, s in bad[:5]]


def test_denominators_round_as_the_two_conversions(check_lib):
    n = np.arange(0, 2049, dtype=np.float64)
    rng = np.random.default_rng(5)
    i, j, k = (rng.choice(n, 200_000) for _ in range(3))
    a = np.concatenate([i * (i - 1), n * (n - 1)]).astype(np.float32)
    b = np.concatenate([j * k, np.maximum(n - 2, 0) * np.maximum(n - 3, 0)]).astype(np.float32)
    out = np.empty((len(a), 6), np.float32)
    check_lib.pgld_check_den(a.ctypes.data, b.ctypes.data, len(a), out.ctypes.data)
    np.testing.assert_array_equal(out[:, :3], out[:, 3:])


@pytest.mark.parametrize("P", [3, 4])
def test_too_few_haplotypes_give_zero(check_lib, P):
    rng = np.random.default_rng(P)
    c = np.stack([rng.multinomial(n, np.full(4, 0.25)) for n in rng.integers(0, 5, 4000 * P)])
    c = c.reshape(-1, P, 4).astype(np.int32)
    ref = O.multi_pop_stats([c[:, p] for p in range(P)], [None] * P)
    out = np.full(ref.shape, np.nan, np.float32)
    check_lib.pgld_check_multi(c.ctypes.data, len(c), P, 0, out.ctypes.data, ref.shape[1])
    np.testing.assert_allclose(out, np.nan_to_num(ref, nan=0.0), rtol=1e-6, atol=0)
