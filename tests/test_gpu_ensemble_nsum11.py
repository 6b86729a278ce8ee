"""The persistent ensemble step at the largest wave-vector cubes it takes: at
n_sum = 11 a longer Ewald range keeps more columns than one block's shared memory
holds (263 of 265 at alpha L = 9; the reciprocal forces then take them in parts):
bit for bit the states of stepping each system on its own.
"""
import pytest

import test_gpu_ensemble_nsum as base

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsum", [9, 10, 11])
@pytest.mark.parametrize("alphaL", [5.6, 6.8, 9.0])
def test_matches_individual_steps(nsum, alphaL, monkeypatch):
    # one, two and five tiles of particles to a slice
    monkeypatch.setattr(base, "SPECS", [("ueg", 16, 4, 0.5, 1.0), ("ueg", 33, 3, 0.75, 3.0), ("ueg", 130, 2, 1.0, 2.0)])
    base.test_matches_individual_steps(nsum, alphaL)
