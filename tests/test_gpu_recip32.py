"""FP32 reciprocal Ewald sums of the mixed form at the edges of particle blocks,
items and columns, against the strict FP64 form.

Positions are multiples of box / 4096, so their FP32 copies are exact; alpha L =
9 keeps every vector of the cube in weight.  Bounds, with u = 2^-24: a first
harmonic good to 2 u, a product to 2 u more, so a term of a sum to
(2 |n|_1 + 4) u <= (6 nsum + 4) u, S the same per particle, the FP32 partial sums
16 u; twice (6 nsum + 16) u of sum |G| c N covers the reciprocal force.  The FP32
real space leaves out images whose h is below 1e-5 (at most one image a pair
here has more than half of that) and rounds 64 u of the largest force.
"""
import math

import numpy as np
import pytest

import xmd_x

pytestmark = pytest.mark.gpu

U, XCUT = 2.0 ** -24, 3.6


def _weight_sum(box, alpha, ns, s):
    n = np.stack(np.meshgrid(*[np.arange(-ns, ns + 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
    g2 = ((n / np.asarray(box)) ** 2).sum(1)
    g2 = g2[g2 > 0]
    c = s / g2 * np.exp(-math.pi ** 2 * g2 / alpha ** 2) / (math.pi * np.prod(box))
    return (c * np.sqrt(g2)).sum() / 2


@pytest.mark.parametrize("N,P,nsum", [(2, 2, 1), (7, 3, 6), (8, 2, 7), (32, 2, 8), (33, 5, 9), (64, 2, 11), (127, 2, 5),
                                      (128, 3, 10), (129, 2, 11), (300, 2, 10), (512, 2, 3)])
def test_forces_against_strict_form(N, P, nsum):
    lib = xmd_x.load(3, 4)
    box, s, m = np.array([6.0, 6.5, 7.0]), 1.5, 1.25
    alpha = 9.0 / box.min()
    rng = np.random.default_rng(N + 10 * P + nsum)
    x = rng.integers(0, 4096, (N, P, 3)) * (box / 4096)
    xmd_x.set_potentials(lib, coul_s=s, alpha=alpha, nsum=nsum)
    u = xmd_x.PimdSystem(lib, N, P, 0.5, 1.0, box=1.0)
    try:
        lib.md_init_nd_rect_box_x(u.sim.contents.box, box.ctypes.data_as(xmd_x._dp))
        f = []
        for mode in (1, 2):
            u.set_state(m=np.full(N * P, m), x=x, v=np.zeros(x.size), f=np.zeros(x.size))
            lib.check(lib.md_gb300_set_precision_x(mode))
            lib.check(lib.md_pimd_calc_pair_force_x(u.pimd, lib.fn("md_coulomb_3d_ewald_force_x")))
            lib.check(lib.md_gb300_set_precision_x(0))
            f.append(np.asarray(u.state()["f"]))
        tol = (4 * math.pi * _weight_sum(box, alpha, nsum, s) * N * 2 * (6 * nsum + 16) * U
               + N * s * 1e-5 * alpha ** 2 / XCUT ** 2) / (m * P) + 64 * U * np.abs(f[1]).max()
        assert np.abs(f[0] - f[1]).max() <= tol
    finally:
        lib.check(lib.md_gb300_set_precision_x(0))
        u.free()
