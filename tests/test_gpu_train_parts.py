"""The network's gradient as a sum over CTAs: one tile, every CTA one tile, more
tiles than CTAs, a last tile of one row; and training to the same bits twice.

A gradient is linear in its rows: that of all rows is the row-weighted mean of
those of the pieces (the network's forward and backward products of a row do
not depend on the others).  Each piece's output gradient is scaled by 1 / rows
before it is rounded to BF16, and rounds the same way when the row counts differ
by a power of two: only the FP32 sums' order differs then, of up to R
terms: R 2^-24 of the sum of sizes, taken as the norm of the pieces' gradients.
"""
import math

import numpy as np
import pytest

import xmd_x
from test_gpu_learned import random_params, ueg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small():
    lib = xmd_x.load(3, 4)
    s, *_ = ueg(lib, 64, 4, 4, seed=7)
    m = xmd_x.EwaldModel(lib, s, nsum_cheap=2, capacity=2, seed=3)
    yield lib, s, m
    m.free()
    s.free()


@pytest.mark.parametrize("rows", [2, 256, 2 * 129, 128 * 152, 128 * 304 + 2])
def test_gradient_of_parts(small, rows):
    lib, s, m = small
    m.params(random_params(lib.md_gb300_ewald_model_nparam_x(), 21))
    rng = np.random.default_rng(rows)
    X = rng.standard_normal((rows, 64)).astype(np.float32)
    V = np.zeros((rows, 12), np.float32)
    V[:, :9] = rng.standard_normal((rows, 9))
    V[:, 9] = 1.0
    T = rng.standard_normal((rows, 4)).astype(np.float32)
    g, loss = m.grad(X, V, T, we=0.8, wf=1.2)
    g2, _ = m.grad(X, V, T, we=0.8, wf=1.2)
    np.testing.assert_array_equal(g, g2)
    h = rows // 2
    a, la = m.grad(X[:h], V[:h], T[:h], we=0.8, wf=1.2)
    b, lb = m.grad(X[h:], V[h:], T[h:], we=0.8, wf=1.2)
    a, b = a.astype(np.float64), b.astype(np.float64)
    tol = rows * 2.0 ** -24 * (np.linalg.norm(a) + np.linalg.norm(b))
    assert np.linalg.norm(g - (a + b) / 2) <= tol
    assert math.isclose(float(np.sum(loss)), float(np.sum(la) + np.sum(lb)), rel_tol=rows * 2.0 ** -24)


def test_training_is_reproducible():
    lib = xmd_x.load(3, 4)
    out = []
    for _ in range(2):
        s, *_ = ueg(lib, 100, 8, 4, seed=5)
        m = xmd_x.EwaldModel(lib, s, nsum_cheap=2, capacity=2, seed=3)
        m.collect(s)
        m.train(6, 3, 1e-3)
        out.append(np.array(m.params()))
        m.free()
        s.free()
    np.testing.assert_array_equal(out[0], out[1])
