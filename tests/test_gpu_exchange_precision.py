"""The connection probabilities G against the recursions in extended precision.

All beads at one point (every cycle energy 0) and ln xi a whole number: the
weights' exponents (k - 1) ln xi - ln l are then the same doubles here and there.
G is a product of a weight, two unknowns and 1 / X_N: X_N and its
reciprocal are rounded to a double, and so is G (3 2^-53), and the 62-bit numbers
between drop at most 2^-60 a product, N of them in the longest chain.
"""
import ctypes as C
import math

import numpy as np
import pytest

import xmd_x
from gpu_common import random_state

pytestmark = pytest.mark.gpu


def _xi(n):
    v = math.exp(-n)
    for c in (v, np.nextafter(v, 1), np.nextafter(v, 0)):
        if math.log(c) == -float(n):
            return float(c)
    pytest.skip("no double with this logarithm")


@pytest.mark.skipif(np.finfo(np.longdouble).eps > 2e-19, reason="needs a long double wider than a double")
@pytest.mark.parametrize("N,n", [(20, 1), (100, 2), (128, 7), (129, 0), (512, 0), (512, 1), (512, 7), (1000, 3)])
def test_g_against_extended_precision(N, n):
    Q = np.longdouble
    lib = xmd_x.load(3, 4)
    s = xmd_x.PimdSystem(lib, N, 3, _xi(n), 1.0)
    s.set_state(**{**random_state(3, 4, N, 3, 0.5, 10.0, False, seed=N), "x": np.zeros((N, 3, 3))})
    lib.check(lib.md_pimd_fast_fill_ENk_x(s.pimd, 0))
    lib.check(lib.md_pimd_fill_VB_x(s.pimd))
    lib.check(lib.md_pimd_fast_fill_force_VB_x(s.pimd, 0))
    tmp, G = np.zeros(N + 1), np.zeros((N, N))
    dp = C.POINTER(C.c_double)
    lib.check(lib.md_gb300_exchange_tables_x(s.pimd, tmp.ctypes.data_as(dp), G.ctypes.data_as(dp)))
    s.free()
    W = np.zeros((N + 1, N), dtype=Q)
    for l in range(1, N + 1):
        k = np.arange(1, l + 1)
        W[l, l - k] = np.exp(((k - 1) * -float(n) - math.log(l)).astype(Q))
    X, Y = np.zeros(N + 1, dtype=Q), np.zeros(N + 1, dtype=Q)
    X[0] = Y[N] = 1
    for l in range(1, N + 1):
        X[l] = (W[l, :l] * X[:l]).sum()
    for j in range(N - 1, -1, -1):
        Y[j] = (W[j + 1:, j] * Y[j + 1:]).sum()
    R = W[1:] * X[:N] * Y[1:, None] / X[N]
    on = R > 1e-300
    rel = ((G.astype(Q) - R)[on] / R[on]).astype(float)
    print("N = %d, ln xi = -%d: mean %.2e, worst %.2e" % (N, n, rel.mean(), np.abs(rel).max()))
    assert np.abs(rel).max() <= 3 * 2.0 ** -53 + N * 2.0 ** -60
    up = np.arange(N - 1)
    np.testing.assert_allclose(G[up, up + 1], (1 - X[1:N] * Y[1:N] / X[N]).astype(float), rtol=0,
                               atol=4 * 2.0 ** -53 + N * 2.0 ** -60)
