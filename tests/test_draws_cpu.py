"""The float32 numerators that count draws, against exact integers.

A numerator that is rounded once has a relative error of at most 2^-24 and, over
many values, a root mean square of about 0.41 units of 2^-24 (a uniform mantissa);
two independent roundings give 0.58.  pi2, pi2_iiij and the shared pi2 round their
main term once and a smaller one by a factor n up to three times: at most three
units, and below 0.5 rms.  pi2_ijij (Kahan's two-product sum) is within two units
and rounds twice, the first time mostly in the smaller product: below 0.5 rms as
well.  DD and its rest together are exact to 2^-40.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests.conftest import ROOT

SRC = os.path.join(ROOT, "tests", "native", "draws_check.cpp")
U = 2.0 ** -24


@pytest.fixture(scope="module")
def check_lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("draws") / "draws.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", so, SRC])
    L = ctypes.CDLL(so)
    for f in (L.pgld_check_hap_draws, L.pgld_check_geno_draws):
        f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    return L


def tables(rng, N, n, cells):
    """Counts of three populations with some linkage and uneven frequencies."""
    pr = rng.dirichlet(np.full(cells, 0.5), N)
    return np.stack([np.array([rng.multinomial(n - rng.integers(0, n // 20 + 1), q) for q in
                               0.7 * pr + 0.3 * rng.dirichlet(np.full(cells, 0.5), N)])
                     for _ in range(3)], 1).astype(np.int32)


def within(got, exact, most, rms):
    # below 2^53: float64 holds the values and their differences
    exact = exact.astype(np.float64)
    err, zero = got.astype(np.float64) - exact, exact == 0
    assert np.all(err[zero] == 0)
    assert np.abs(err[~zero] / exact[~zero]).max() <= most * U
    assert np.sqrt((err ** 2).sum() / (exact ** 2).sum()) <= rms * U


@pytest.mark.parametrize("n", [5, 60, 700, 1000, 2048])
def test_haplotype_numerators(check_lib, n):
    rng = np.random.default_rng(n)
    c = tables(rng, 4000, n, 4)
    # one carrier at each SNP, the same haplotype or not; no variation; perfect linkage
    c[:4, :] = np.array([[1, 0, 0, n - 1], [0, 1, 1, n - 2], [0, 0, 1, n - 1], [2, 0, 0, n - 2]])[:, None]
    out = np.zeros((len(c), 6), np.float32)
    check_lib.pgld_check_hap_draws(c.ctypes.data, len(c), out.ctypes.data)
    c1, c2, c3, c4 = (c[:, :, k].astype(np.int64) for k in range(4))
    pA, qA, pB, qB, m = c1 + c2, c3 + c4, c1 + c3, c2 + c4, c1 + c2 + c3 + c4
    X = [pA * pB - c1, pA * qB - c2, qA * pB - c3, qA * qB - c4]  # ordered draws of two haplotypes
    pi = pA * pB * qB * qA - c1 * c4 * (c1 + 3 * c2 + 3 * c3 + c4 - 1) - c2 * c3 * (3 * c1 + c2 + c3 + 3 * c4 - 1)
    dd = c1 * (c1 - 1) * c4 * (c4 - 1) + c2 * (c2 - 1) * c3 * (c3 - 1) - 2 * c1 * c2 * c3 * c4
    Tb, TB = pA * X[3] - c2 * qA, pA * X[2] - c1 * qA
    within(out[:, 0], pi[:, 0], 3, 0.5)
    within(out[:, 1], Tb[:, 0] * pB[:, 1] + TB[:, 0] * qB[:, 1], 3, 0.5)
    within(out[:, 2], 4 * sum(X[k][:, 0] * X[3 - k][:, 1] for k in range(4)), 2, 0.5)
    x, a, b = [v[:, 0] for v in X], 1, 2
    within(out[:, 3], qA[:, a] * (x[0] * qB[:, b] + x[1] * pB[:, b]) + pA[:, a] * (x[2] * qB[:, b] + x[3] * pB[:, b]),
           3, 0.5)
    split = out[:, 4].astype(np.float64) + out[:, 5].astype(np.float64)
    assert np.all(np.abs(split - dd[:, 0]) <= 2.0 ** -40 * np.abs(dd[:, 0]))


@pytest.mark.parametrize("n", [5, 60, 500, 1000, 2048])
def test_genotype_numerators(check_lib, n):
    rng = np.random.default_rng(n)
    c = tables(rng, 4000, n, 9)
    c[0] = [0, 0, n, 0, 0, 0, 0, 0, 0]
    c[1] = [0, 0, n - 1, 1, 0, 0, 0, 0, 0]
    out = np.zeros((len(c), 2), np.float32)
    check_lib.pgld_check_geno_draws(c.ctypes.data, len(c), out.ctypes.data)
    g = np.array([[i, j] for i in range(3) for j in range(3)], np.int64) - 1
    w = c.astype(np.int64)
    mom = lambda x, y: (w * (g[:, 0] ** x * g[:, 1] ** y)).sum(2)  # noqa: E731
    m, m1, m3, m4 = mom(0, 0), mom(0, 1), mom(1, 0), mom(1, 1)
    # sums over individuals u != v of (1 +- c_I(u)) (1 +- c_J(v))
    X = [(m + p * m3) * (m + q * m1) - (m + p * m3 + q * m1 + p * q * m4) for p in (1, -1) for q in (1, -1)]
    within(4 * out[:, 0], sum(X[k][:, 0] * X[3 - k][:, 1] for k in range(4)), 2, 0.5)
    x, a, b = [v[:, 0] for v in X], 1, 2
    P, R, Q, S = m + m3, m - m3, m + m1, m - m1
    within(4 * out[:, 1], R[:, a] * (x[0] * S[:, b] + x[1] * Q[:, b]) + P[:, a] * (x[2] * S[:, b] + x[3] * Q[:, b]),
           3, 0.5)
