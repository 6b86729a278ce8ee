"""Small structure factors in the learned residual's shell features, and positions that are no number.

Two particles half a box diagonal and 2^-20 of an edge apart: for a wave vector with an
odd n_x + n_y + n_z = s the phases cancel to |S|^2 = 4 sin^2(s pi 2^-20), 1e-11 of the largest, and every
number on the way is exact in FP32 or good to a few ulps of itself: the phases' harmonics are
products, |n_i| <= 6 of them, so a feature is good to 64 ulps.
"""
import numpy as np
import pytest

import xmd_x

pytestmark = pytest.mark.gpu

BOX = 8.0


def _features(lib, x):
    N, P = x.shape[:2]
    xmd_x.set_potentials(lib, coul_s=1.0, alpha=5.6 / BOX, nsum=4)
    s = xmd_x.PimdSystem(lib, N, P, 0.5, 1.0, box=BOX)
    s.set_state(m=np.ones(N * P), x=x, v=np.zeros(x.size), f=np.zeros(x.size))
    m = xmd_x.EwaldModel(lib, s, nsum_cheap=2, capacity=1, seed=3)
    F, V = m.features(s)
    m.free()
    s.free()
    return F, V


def test_small_structure_factors():
    lib = xmd_x.load(3, 4)
    x = np.zeros((2, 3, 3))
    x[1] = BOX / 2 + BOX * 2.0 ** -20
    F, _ = _features(lib, x)
    r = np.arange(-6, 7)
    n = np.stack(np.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)
    n2, total = (n ** 2).sum(1), n.sum(1)
    odd = 0
    for i, s2 in enumerate(sorted(set(n2[n2 > 0]))[:32]):
        on = n2 == s2  # both halves: twice the vectors, each twice
        if s2 % 2 == 0:
            continue
        odd += 1
        v = (4 * np.sin(np.pi * total[on] * 2.0 ** -20) ** 2).sum() / (2 * on.sum())
        np.testing.assert_allclose(F[:, 32 + i], np.sqrt(v), rtol=64 * 2.0 ** -24, err_msg=f"|n|^2 = {s2}")
    assert odd >= 10


def test_not_a_number():
    lib = xmd_x.load(3, 4)
    rng = np.random.default_rng(5)
    x = rng.uniform(0, BOX, (300, 2, 3))
    x[250, 1, 2] = np.nan
    F, _ = _features(lib, x)  # rows: slice by slice
    assert np.isfinite(F[:300]).all()
    # of the broken slice, every shell with a wave vector across that coordinate: all of them
    assert np.isnan(F[300:, 32:]).all()
