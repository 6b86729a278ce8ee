"""The virial estimator's cycle table at sizes around a warp, a block and more
than one row a thread, against the definition's running sums in extended
precision.

Bound: a nearest image is good to an ulp of |difference| + box, so a term
1/2 m w2 sum_d t_d u_d is good to 2 D + 4 <= 10 roundings of
size = 1/2 m w2 sum_d (|t_d| + L)(|u_d| + L); an entry is one such term and the
difference of two prefix sums whose rounding errors are kept, which adds the
terms' own errors and three roundings of results no larger than the terms'
sizes: 16 2^-53 times the sum of the sizes.
"""
import numpy as np
import pytest

import xmd_x

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("image", [0, 1])
@pytest.mark.parametrize("D,N,P", [(3, 1, 2), (2, 2, 3), (3, 32, 2), (2, 33, 3), (3, 34, 2), (3, 129, 3), (2, 1025, 2),
                                   (3, 1026, 2), (3, 1203, 2)])
def test_enk2_against_definition(D, N, P, image):
    lib = xmd_x.load(D, 4)
    L, T = 2.5, 0.4
    rng = np.random.default_rng(77 * D + N + P)
    x = rng.uniform(0.0, L, (N, 1, D)) + 0.3 * rng.standard_normal((N, P, D))
    if image:
        x = np.mod(x, L)
    s = xmd_x.PimdSystem(lib, N, P, 0.7, T, box=L)
    try:
        s.set_state(m=np.full(N * P, 2.0), x=x, v=np.zeros(x.size), f=np.zeros(x.size))
        lib.check(lib.md_pimd_fast_fill_ENk2_x(s.pimd, image))
        got = s.exchange()["ENk2"]
        w2 = np.longdouble(s.pimd.contents.omegaP ** 2)
        x1, xP = x[:, 0].astype(np.longdouble), x[:, -1].astype(np.longdouble)

        def near(c):
            return c - L * np.rint(c / L) if image else c

        term, size = np.zeros((N, N), np.longdouble), np.zeros((N, N))
        for d in range(D):
            t, u = near(x1[:, None, d] - xP[None, :, d]), near(x1[:, None, d] - x1[None, :, d])
            term += w2 * t * u  # half of mass 2
            size += np.float64(w2) * ((np.abs(t) + L) * (np.abs(u) + L)).astype(np.float64)
        for l in range(N):
            c = np.arange(l - 1, -1, -1)
            inc = np.concatenate([[term[l, l]], term[l, c] - term[l, c + 1] + term[c, c + 1]])
            sizes = size[l, l::-1] + np.concatenate([[0.0], np.cumsum(size[c, c + 1])])
            row = got[l * (l + 1) // 2:(l + 1) * (l + 2) // 2]
            assert (np.abs(row - np.cumsum(inc)) <= 16 * 2.0 ** -53 * sizes).all()
    finally:
        s.free()
