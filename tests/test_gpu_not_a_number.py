"""A position that is no number, or infinite, shows in what is formed from it: the
exchange recursions' V_B from its row of cycle energies on, the exchange forces,
Gaussian energies.  And V_B before that row keeps its bits.
"""
import numpy as np
import pytest

import xmd_x
from gpu_common import random_state

pytestmark = pytest.mark.gpu


def _system(lib, N, P, xi, st):
    s = xmd_x.PimdSystem(lib, N, P, xi, 0.5)
    s.set_state(**st)
    return s


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("N,p", [(5, 2), (40, 36), (40, 0), (128, 63), (200, 130), (1000, 961)])
@pytest.mark.parametrize("xi", [1.0, 0.4, 0.0])
def test_recursions(N, p, xi, bad):
    lib = xmd_x.load(3, 4)
    st = random_state(3, 4, N, 3, 0.5, 10.0, False, seed=N + p)
    vb, f = [], []
    for broken in (False, True):
        x = np.array(st["x"], dtype=np.float64).reshape(N, 3, 3)
        if broken:
            x[p, 1, 2] = bad
        s = _system(lib, N, 3, xi, {**st, "x": x})
        lib.check(lib.md_reset_force_x(s.sim))
        lib.check(lib.md_pimd_fast_fill_ENk_x(s.pimd, 0))
        lib.check(lib.md_pimd_fill_VB_x(s.pimd))
        lib.check(lib.md_pimd_fast_fill_force_VB_x(s.pimd, 0))
        f.append(s.state()["f"].reshape(N, 3, 3))
        ex = s.exchange()
        vb.append(ex["VBN"])
        # the first row of cycle energies with one that is no number (the energies' prefix sums come in runs of
        # ceil((N - 1) / 256) particles, which may bring it up to a run forward)
        # (xi = 0: only one-particle cycles have a weight)
        row = next((l for l in range(1, N + 1)
                    if not np.isfinite(ex["ENk"][l * (l - 1) // 2:][:l if xi else 1]).all()), None)
        s.free()
    assert np.isfinite(vb[0]).all() and np.isfinite(f[0]).all()
    assert p + 1 - (N - 1) // 256 <= row <= p + 1
    np.testing.assert_array_equal(vb[1][:row], vb[0][:row])
    assert np.isnan(vb[1][row:]).all()
    assert np.isnan(f[1][:, [0, 2]]).any(axis=(0, 1, 2))
    assert not np.isfinite(f[1][p, 1, 2])


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("kind", ["gaussian", "periodic_gaussian"])
def test_gaussian_energy(D, kind):
    lib = xmd_x.load(D, 4)
    N, P = 37, 2
    xmd_x.set_potentials(lib, gauss_g=2.0, gauss_s=0.5)
    st = random_state(D, 4, N, P, 1.0, 10.0, False, seed=3)
    x = np.array(st["x"], dtype=np.float64).reshape(N, P, D)

    def energy(x):
        s = xmd_x.PimdSystem(lib, N, P, 0.5, 1.0, box=10.0)
        s.set_state(**{**st, "x": x})
        lib.check(lib.md_pimd_calc_pair_energy_x(s.pimd, lib.fn(f"md_{kind}_energy_x"), s.stats))
        e = s.take_energy()
        s.free()
        return e

    assert np.isfinite(energy(x))
    y = x.copy()
    y[11, 1, 0] = np.nan
    assert np.isnan(energy(y))
    if kind == "gaussian":  # a bead beyond every other's reach, its square beyond the largest double
        far, gone = x.copy(), x.copy()
        far[11, 1, 0], gone[11, 1, 0] = 1e3, 1e160
        assert energy(far) == energy(gone)


def test_ranges_beyond_a_doubles_square():
    """s^2 overflows: the potential's strength over it is zero, and so is everything else"""
    lib = xmd_x.load(3, 4)
    N, P = 9, 2
    st = random_state(3, 4, N, P, 1.0, 10.0, False, seed=4)
    xmd_x.set_potentials(lib, gauss_g=2.0, gauss_s=1e170)
    s = xmd_x.PimdSystem(lib, N, P, 0.5, 1.0)
    s.set_state(**st)
    lib.check(lib.md_reset_force_x(s.sim))
    lib.check(lib.md_pimd_calc_pair_force_x(s.pimd, lib.fn("md_gaussian_force_x")))
    assert not s.state()["f"].any()
    lib.check(lib.md_pimd_calc_pair_energy_x(s.pimd, lib.fn("md_gaussian_energy_x"), s.stats))
    assert s.take_energy() == 0.0
    s.free()
