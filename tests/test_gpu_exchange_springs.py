"""Exchange spring forces at the edges of the 32 x 32 tiles and of their parts,
against the definition in numpy with the library's own cycle probabilities.

Bounds: a spring difference is good to 2 ulps of the box (the nearest image), a
product and a sum of at most 2 N + 4 terms add one ulp of the terms' sizes each:
(2 N + 16) 2^-53 times w2 times the sum of weighted sizes (each at least the
box's where images are taken) covers both.
"""
import numpy as np
import pytest

import xmd_x

pytestmark = pytest.mark.gpu


def _reference(x, G, L, w2, image):
    def near(c):
        return c - L * np.rint(c / L) if image else c

    N, P, D = x.shape
    x1, xP = x[:, 0], x[:, -1]
    f, size = np.zeros((N, P, D)), np.zeros((N, P, D))
    for a, b in ((1, 0), (-1, 1)):
        for j in range(1, P - 1):
            c = near(x[:, j] - x[:, j + a])
            f[:, j] -= w2 * c
            size[:, j] += w2 * (np.abs(c) + L)
    c = near(xP[:, None] - x1[None])
    gc = G[..., None] * c
    gs = np.abs(G)[..., None] * (np.abs(c) + L)
    for j, k, W, S, z in ((0, 1, G.sum(0), -gc.sum(0), gs.sum(0)), (P - 1, P - 2, G.sum(1), gc.sum(1), gs.sum(1))):
        r = near(x[:, j] - x[:, k])
        f[:, j] = -w2 * (W[:, None] * r + S)
        size[:, j] = w2 * (np.abs(W)[:, None] * (np.abs(r) + L) + z)
    return f, size


@pytest.mark.parametrize("image", [0, 1])
@pytest.mark.parametrize("D,N,P", [(3, 1, 2), (2, 2, 3), (3, 31, 2), (2, 32, 3), (3, 33, 5), (2, 64, 4), (3, 65, 3),
                                   (2, 97, 2), (3, 128, 3), (3, 129, 7), (2, 512, 3), (3, 545, 2)])
def test_against_definition(D, N, P, image):
    lib = xmd_x.load(D, 4)
    L, T = 2.5, 0.4
    rng = np.random.default_rng(1000 * D + N + P)
    x = rng.uniform(0.0, L, (N, 1, D)) + 0.2 * rng.standard_normal((N, P, D))
    if image:
        x = np.mod(x, L)
    s = xmd_x.PimdSystem(lib, N, P, 0.7, T, box=L)
    try:
        s.set_state(m=np.full(N * P, 2.0), x=x, v=np.zeros(x.size), f=np.zeros(x.size))
        for step in range(2):  # G from the solves' numbers, then read
            lib.check(lib.md_reset_force_x(s.sim))
            lib.check(lib.md_pimd_fast_fill_ENk_x(s.pimd, image))
            lib.check(lib.md_pimd_fill_VB_x(s.pimd))
            if step:  # another xi than the solves': G by the fallback, read by the springs
                s.pimd.contents.vi = 0.6
            lib.check(lib.md_pimd_fast_fill_force_VB_x(s.pimd, image))
            f = s.state()["f"].reshape(N, P, D)
            tmpV, G = np.zeros(N + 1), np.zeros((N, N))
            lib.check(lib.md_gb300_exchange_tables_x(s.pimd, tmpV.ctypes.data_as(xmd_x._dp), G.ctypes.data_as(xmd_x._dp)))
            assert (np.triu(G, 2) == 0).all()
            if not step:
                np.testing.assert_allclose(G.sum(1), 1.0, rtol=0, atol=1e-9)
            F, size = _reference(x, G, L, s.pimd.contents.omegaP ** 2, image)
            assert (np.abs(f - F) <= (2 * N + 16) * 2.0 ** -53 * size).all()
    finally:
        s.free()
