"""The double-float Ewald kernels of the FP64 form against the strict form,
whose every term is FP64, at the edges of tiles, boxes and image cubes.

Bounds.  Both forms leave out the same images (alpha R >= 5.2); an image
within FP32 rounding of the cut-off may be taken by one of them only, and
adds h(5.2) / 5.2^3 = 8e-14 in units of s alpha^2.  Double-float rounding
is 2^-45 of each pair's force at most, the FP32 part of the reciprocal sum
below 1e-12 of a bead's own force.  Together below 2e-12 of the largest
force for forces of the order of the largest pair's, which every state here
has; energies, sums of terms good to 2^-46 with random signs of rounding,
below 1e-13 of themselves plus the same of the largest part.
"""
import numpy as np
import pytest

import xmd_x

pytestmark = pytest.mark.gpu

TOL_F, TOL_E = 2e-12, 2e-13


@pytest.fixture(scope="module")
def lib():
    return xmd_x.load(3, 4)


def _system(lib, N, P, box, seed, spread):
    rng = np.random.default_rng(seed)
    s = xmd_x.PimdSystem(lib, N, P, 0.5, 1.0, box=1.0)
    b = np.asarray(box, dtype=np.float64)
    lib.md_init_nd_rect_box_x(s.sim.contents.box, b.ctypes.data_as(xmd_x._dp))
    # spread > 1 puts beads outside the box, up to (spread - 1) / 2 boxes
    x = rng.uniform(0.5 - spread / 2, 0.5 + spread / 2, (N, P, 3)) * b
    s.set_state(m=np.full(N * P, 1.25), x=x, v=np.zeros((N * P, 3)), f=np.zeros((N * P, 3)))
    return s


def _forces(lib, systems, mode):
    lib.check(lib.md_gb300_set_precision_x(mode))
    pair = lib.fn("md_coulomb_3d_ewald_force_x")
    for s in systems:
        lib.check(lib.md_reset_force_x(s.sim))
        lib.check(lib.md_pimd_calc_pair_force_x(s.pimd, pair))
    if len(systems) == 2:
        lib.check(lib.md_pimd_calc_pair_force_2_x(systems[0].pimd, systems[1].pimd, pair))
    lib.check(lib.md_gb300_set_precision_x(0))
    return np.concatenate([s.state()["f"] for s in systems])


def _energy(lib, s, mode):
    lib.check(lib.md_gb300_set_precision_x(mode))
    lib.check(lib.md_pimd_calc_pair_energy_x(s.pimd, lib.fn("md_coulomb_3d_ewald_energy_x"), s.stats))
    lib.check(lib.md_gb300_set_precision_x(0))
    return s.take_energy()


@pytest.mark.parametrize("N,P,box,alphaL,nsum,spread", [
    (2, 2, (3.0, 3.0, 3.0), 5.6, 6, 1.0),
    (31, 3, (5.0, 5.0, 5.0), 5.6, 8, 1.0),
    (32, 2, (5.0, 5.0, 5.0), 5.25, 5, 1.0),
    (33, 2, (5.0, 6.0, 7.5), 5.6, 8, 1.0),      # alpha L = 5.6 on the shortest edge
    (65, 3, (6.0, 6.0, 6.0), 7.0, 10, 2.4),     # beads outside the box
    (40, 2, (5.0, 5.0, 5.0), 5.6, 1, 3.0),      # the image cube cuts candidates off
    (40, 2, (5.0, 5.0, 5.0), 5.6, 2, 5.0),
    (257, 2, (9.0, 9.0, 9.0), 5.6, 9, 1.0),
    (20, 2, (5.0, 5.0, 5.0), 4.2, 4, 1.0),      # cut-off beyond the box: the FP64 tiles
])
def test_forces_and_energy_against_strict_form(lib, N, P, box, alphaL, nsum, spread):
    xmd_x.set_potentials(lib, coul_s=1.5, alpha=alphaL / min(box), nsum=nsum)
    s = _system(lib, N, P, box, N + P, spread)
    try:
        f, f0 = _forces(lib, [s], 0), _forces(lib, [s], 2)
        assert np.abs(f - f0).max() <= TOL_F * np.abs(f0).max()
        e, e0 = _energy(lib, s, 0), _energy(lib, s, 2)
        pairs = 1.5 * N * N / 2 / min(box)  # the size of the parts that cancel in e
        assert abs(e - e0) <= TOL_E * (abs(e0) + pairs)
    finally:
        s.free()


@pytest.mark.parametrize("Na,Nb,P,spread", [(1, 33, 2, 1.0), (32, 31, 3, 1.0), (65, 40, 2, 2.2)])
def test_two_species_against_strict_form(lib, Na, Nb, P, spread):
    box = (5.0, 5.5, 6.0)
    xmd_x.set_potentials(lib, coul_s=1.0, alpha=5.6 / 5.0, nsum=7)
    a, b = _system(lib, Na, P, box, 1, spread), _system(lib, Nb, P, box, 2, spread)
    try:
        f, f0 = _forces(lib, [a, b], 0), _forces(lib, [a, b], 2)
        assert np.abs(f - f0).max() <= TOL_F * np.abs(f0).max()
    finally:
        a.free()
        b.free()


def test_close_pair_keeps_its_relative_accuracy(lib):
    """two beads 1e-5 of the box apart across its edge: the Coulomb force 1/r^2 to 1e-12"""
    L, r = 4.0, 4e-5
    xmd_x.set_potentials(lib, coul_s=1.0, alpha=5.6 / L, nsum=6)
    s = xmd_x.PimdSystem(lib, 2, 2, 0.5, 1.0, box=L)
    try:
        x = np.full((2, 2, 3), 1.0)
        x[0, :, 0], x[1, :, 0] = r / 4, L - 3 * r / 4
        s.set_state(m=np.ones(4), x=x, v=np.zeros((4, 3)), f=np.zeros((4, 3)))
        f = _forces(lib, [s], 0).reshape(2, 2, 3)
        sep = x[0, 0, 0] - (x[1, 0, 0] - L)
        assert np.abs(f[0, :, 0] * 2 * sep * sep - 1.0).max() < 1e-12
    finally:
        s.free()


@pytest.mark.parametrize("N,P,nsum", [(2, 2, 1), (7, 3, 4), (64, 2, 6), (65, 5, 11), (300, 2, 9)])
def test_reciprocal_sums_alone(lib, N, P, nsum):
    """a large alpha L makes the real-space part vanish beside the reciprocal one; every wave vector of the cube is
    kept then, most of them double-float"""
    box = (6.0, 6.5, 7.0)
    xmd_x.set_potentials(lib, coul_s=1.0, alpha=9.0 / 6.0, nsum=nsum)
    s = _system(lib, N, P, box, 3 * N + P, 1.7)
    try:
        f, f0 = _forces(lib, [s], 0), _forces(lib, [s], 2)
        assert np.abs(f - f0).max() <= TOL_F * np.abs(f0).max()
        e, e0 = _energy(lib, s, 0), _energy(lib, s, 2)
        assert abs(e - e0) <= TOL_E * (abs(e0) + N * N / 2 / 6.0)
    finally:
        s.free()
