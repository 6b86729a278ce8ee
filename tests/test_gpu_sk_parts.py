"""Structure factors with 16 and with 8 threads an item (the number of bead
slices decides): the same slices give the same reciprocal forces and energies,
to the rounding of sums of N double-float terms in another order; the bounds
are those against the strict form.
"""
import numpy as np
import pytest

import xmd_x
from test_gpu_ewald_df import TOL_E, TOL_F, _energy, _forces, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 15, 64, 65, 131])
@pytest.mark.parametrize("nsum,P", [(2, 266), (2, 267), (6, 88), (6, 89), (10, 19), (10, 20)])
def test_against_strict_form(N, nsum, P):
    lib = xmd_x.load(3, 4)
    box = (6.0, 6.5, 7.0)
    # alpha L large: the reciprocal sums are the larger part, and no vector of the cube is dropped
    xmd_x.set_potentials(lib, coul_s=1.0, alpha=9.0 / 6.0, nsum=nsum)
    s = _system(lib, N, P, box, 5 * N + P, 1.5)
    try:
        f, f0 = _forces(lib, [s], 0), _forces(lib, [s], 2)
        assert np.abs(f - f0).max() <= TOL_F * np.abs(f0).max()
        e, e0 = _energy(lib, s, 0), _energy(lib, s, 2)
        assert abs(e - e0) <= TOL_E * (abs(e0) + (N * N + N) / 2 / 6.0)
    finally:
        s.free()
