"""FP64 Gaussian and Coulomb pair forces and energies at the edges of tiles and
of their parts, against the definitions in numpy.

Bounds: a pair's force and energy are good to 16 ulps (a separation, its
square, one division, the exponential of a number up to about 30 in size, a
product), their sums of N terms to N more of the sum of sizes: N + 64 times
2^-53 times the sum of the pairs' sizes covers both.
"""
import math

import numpy as np
import pytest

import xmd_x

pytestmark = pytest.mark.gpu

KINDS = {"gaussian": False, "periodic_gaussian": True, "coulomb": False, "coulomb_periodic": True}


def _reference(x, L, kind, g, s, q):
    """forces (N, P, D) / P, energy, and the sums of the pairs' sizes"""
    N, P, D = x.shape
    d = x[:, None] - x[None]
    if KINDS[kind]:
        d = d - L * np.rint(d / L)
    r2 = (d ** 2).sum(-1) + np.eye(N)[:, :, None]
    if "gaussian" in kind:
        e = g / (math.pi * s * s) * np.exp(-r2 / (s * s))
        w = e * 2 / (s * s)
    else:
        e = q / np.sqrt(r2)
        w = q / (r2 * np.sqrt(r2))
    off = 1 - np.eye(N)[:, :, None]
    e, w = e * off, w * off
    F = w[..., None] * d / P
    return F.sum(1), e.sum() / 2 / P, np.abs(F).sum(1), np.abs(e).sum() / 2 / P


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("N,P", [(1, 2), (2, 1), (4, 32), (17, 3), (31, 2), (32, 5), (33, 2), (61, 45), (64, 64), (130, 3)])
def test_against_definition(D, N, P):
    lib = xmd_x.load(D, 4)
    L, g, s, q = 3.0, 2.4, 0.7, 1.3
    rng = np.random.default_rng(100 * N + P)
    x = rng.uniform(-1.0, 4.0, (N, P, D))
    xmd_x.set_potentials(lib, gauss_g=g, gauss_s=s, coul_s=q)
    u = xmd_x.PimdSystem(lib, N, P, 0.5, 1.0, box=L)
    try:
        u.set_state(m=np.full(N * P, 2.0), x=x, v=np.zeros(x.size), f=np.zeros(x.size))
        for kind in KINDS:
            lib.check(lib.md_reset_force_x(u.sim))
            lib.check(lib.md_pimd_calc_pair_force_x(u.pimd, lib.fn(f"md_{kind}_force_x")))
            f = u.state()["f"].reshape(N, P, D) * 2.0
            lib.check(lib.md_pimd_calc_pair_energy_x(u.pimd, lib.fn(f"md_{kind}_energy_x"), u.stats))
            e = u.take_energy()
            F, E, sF, sE = _reference(x, L, kind, g, s, q)
            tol = (N + 64) * 2.0 ** -53
            assert (np.abs(f - F) <= tol * (sF + sF.max())).all(), kind
            assert abs(e - E) <= tol * (sE + 1e-300), kind
    finally:
        u.free()
