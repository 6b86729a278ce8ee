"""One training step's gradient over many CTAs against the 64-bit sum of its tiles' gradients.

With 2^k tiles of 128 rows, 1 / rows is a power of two, so a tile's rows give the
same BF16 products in a call of its own and in the call of all tiles, up to
that power of two: only the FP32 additions over tiles differ.

128 tiles are one a CTA.  Their parts are added in two levels, 16 of every
eighth part and then eight sums: no more than 23 additions touch a value, so each
component is within 23 2^-24 of the sum of its parts' sizes.  With 256 tiles
some CTAs add a second tile in the tensor memory first, eight accumulating
products of 16 rows each way; with their rounding taken as 2^-23 (truncation)
that is another 16 2^-23.  The bias gradients add 4 x 2 more sums in FP32.
"""
import numpy as np
import pytest

import xmd_x
from test_gpu_learned import random_params, ueg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles,eps", [(2, 23 * 2.0 ** -24), (128, 23 * 2.0 ** -24), (256, (23 + 2 * 16 + 8) * 2.0 ** -24)])
def test_gradient_is_the_sum_of_its_tiles(tiles, eps):
    lib = xmd_x.load(3, 4)
    s, *_ = ueg(lib, 64, 4, 4, seed=7)
    m = xmd_x.EwaldModel(lib, s, nsum_cheap=2, capacity=2, seed=3)
    m.params(random_params(lib.md_gb300_ewald_model_nparam_x(), 22))
    rng = np.random.default_rng(tiles)
    rows = 128 * tiles
    X = rng.standard_normal((rows, 64)).astype(np.float32)
    V = np.zeros((rows, 12), np.float32)
    V[:, :9] = rng.standard_normal((rows, 9))
    V[:, 9] = 1.0
    T = rng.standard_normal((rows, 4)).astype(np.float32)
    g, loss = m.grad(X, V, T, we=0.8, wf=1.2)
    parts, losses = [], []
    for t in range(tiles):
        r = slice(128 * t, 128 * t + 128)
        a, b = m.grad(X[r], V[r], T[r], we=0.8, wf=1.2)
        parts.append(a.astype(np.float64) / tiles)
        losses.append(b.astype(np.float64))
    m.free()
    s.free()
    exact, size = np.sum(parts, axis=0), np.sum(np.abs(parts), axis=0)
    off = np.abs(g - exact)
    print("gradient of %d tiles: %.2e of its norm, worst %.2f of its bound" %
          (tiles, np.linalg.norm(off) / np.linalg.norm(exact), np.max(off / np.maximum(eps * size, 1e-30))))
    assert np.all(off <= eps * size)
    assert np.linalg.norm(off) <= 3e-6 * np.linalg.norm(exact)
    # the losses: one FP32 addition a tile, in any order
    total = np.sum(losses, axis=0)
    np.testing.assert_allclose(loss, total, rtol=tiles * 2.0 ** -24)
