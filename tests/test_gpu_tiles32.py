"""FP32 pair tiles at the edges of tiles, on both sides of the single-shift rule
(no image shifted along two axes inside 3.6 / alpha) and with the image cube cut
to n_sum 1, against the strict FP64 form.

Positions are multiples of box / 4096 (exact in FP32).  Each pair's FP32 force
is good to about 32 u = 32 2^-24 of itself (reciprocal square root, reciprocal,
exponential at 2 u each with arguments up to 13, a polynomial, a dozen products),
a tile's partial sums to 32 u more, the images left out have h below 1e-5 each
(at most 27 a pair): 64 u of the pair sizes, taken as N times the largest force,
plus N 27 1e-5 s alpha^2 / 3.6^2.
"""
import numpy as np
import pytest

import xmd_x

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alphaL,nsum", [(5.6, 4), (5.6, 1), (5.12, 3), (5.05, 3), (4.6, 1), (4.0, 2)])
@pytest.mark.parametrize("N,P", [(2, 2), (31, 3), (32, 2), (33, 2), (64, 3), (65, 2), (161, 2)])
def test_ewald_against_strict_form(N, P, alphaL, nsum):
    lib = xmd_x.load(3, 4)
    box = np.array([5.0, 5.0, 5.0]) if N % 2 else np.array([5.0, 5.25, 5.5])
    s, m, u = 1.5, 1.25, 2.0 ** -24
    alpha = alphaL / box.min()
    rng = np.random.default_rng(N + P + int(100 * alphaL))
    x = rng.integers(0, 4096, (N, P, 3)) * (box / 4096)
    xmd_x.set_potentials(lib, coul_s=s, alpha=alpha, nsum=nsum)
    sys = xmd_x.PimdSystem(lib, N, P, 0.5, 1.0, box=1.0)
    try:
        lib.md_init_nd_rect_box_x(sys.sim.contents.box, box.ctypes.data_as(xmd_x._dp))
        f = []
        for mode in (1, 2):
            sys.set_state(m=np.full(N * P, m), x=x, v=np.zeros(x.size), f=np.zeros(x.size))
            lib.check(lib.md_gb300_set_precision_x(mode))
            lib.check(lib.md_pimd_calc_pair_force_x(sys.pimd, lib.fn("md_coulomb_3d_ewald_force_x")))
            lib.check(lib.md_gb300_set_precision_x(0))
            f.append(np.asarray(sys.state()["f"]))
        tol = 64 * u * N * np.abs(f[1]).max() + N * 27e-5 * s * alpha ** 2 / 3.6 ** 2 / (m * P)
        assert np.abs(f[0] - f[1]).max() <= tol
    finally:
        lib.check(lib.md_gb300_set_precision_x(0))
        sys.free()


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("N,P", [(2, 2), (31, 3), (32, 2), (33, 2), (64, 3), (65, 2)])
@pytest.mark.parametrize("masses", ["one", "several"])
def test_gaussian_against_strict_form(D, N, P, masses):
    """one mass for all beads, and one a particle (divided by the higher-index particle's)"""
    lib = xmd_x.load(D, 4)
    rng = np.random.default_rng(N + P + D)
    x = rng.integers(0, 4096, (N, P, D)) * (4.0 / 4096)
    m = np.full((N, P), 2.0) if masses == "one" else np.repeat(rng.uniform(0.5, 3.0, (N, 1)), P, 1)
    xmd_x.set_potentials(lib, gauss_g=2.4, gauss_s=0.7)
    sys = xmd_x.PimdSystem(lib, N, P, 0.5, 1.0, box=4.0)
    try:
        f = []
        for mode in (1, 2):
            sys.set_state(m=m.reshape(-1), x=x, v=np.zeros(x.size), f=np.zeros(x.size))
            lib.check(lib.md_gb300_set_precision_x(mode))
            lib.check(lib.md_pimd_calc_pair_force_x(sys.pimd, lib.fn("md_gaussian_force_x")))
            lib.check(lib.md_gb300_set_precision_x(0))
            f.append(np.asarray(sys.state()["f"]))
        assert np.abs(f[0] - f[1]).max() <= 64 * 2.0 ** -24 * N * np.abs(f[1]).max()
    finally:
        lib.check(lib.md_gb300_set_precision_x(0))
        sys.free()
