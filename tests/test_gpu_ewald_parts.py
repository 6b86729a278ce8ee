"""Real-space Ewald tiles in eight, four, two parts and whole (the number of
tiles decides), against the strict FP64 form; bounds as for the other sizes.
"""
import pytest

import numpy as np
import xmd_x
from test_gpu_ewald_df import TOL_E, TOL_F, _energy, _forces, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [2, 101, 102, 810, 811, 1621, 1622])  # 3 tiles a bead slice
def test_forces_and_energy(P):
    lib = xmd_x.load(3, 4)
    N, L = 40, 5.0
    xmd_x.set_potentials(lib, coul_s=1.5, alpha=5.6 / L, nsum=4)
    s = _system(lib, N, P, (L, L, L), P, 1.3)
    try:
        f, f0 = _forces(lib, [s], 0), _forces(lib, [s], 2)
        assert np.abs(f - f0).max() <= TOL_F * np.abs(f0).max()
        e, e0 = _energy(lib, s, 0), _energy(lib, s, 2)
        assert abs(e - e0) <= TOL_E * (abs(e0) + 1.5 * N * N / 2 / L)
    finally:
        s.free()


@pytest.mark.parametrize("P", [3, 77, 609, 1215, 1216])  # 4 cross tiles a bead slice
def test_cross_pairs(P):
    lib = xmd_x.load(3, 4)
    xmd_x.set_potentials(lib, coul_s=1.0, alpha=5.6 / 5.0, nsum=4)
    a, b = (_system(lib, N, P, (5.0, 5.5, 6.0), N, 1.0) for N in (40, 33))
    try:
        f, f0 = _forces(lib, [a, b], 0), _forces(lib, [a, b], 2)
        assert np.abs(f - f0).max() <= TOL_F * np.abs(f0).max()
    finally:
        a.free()
        b.free()
