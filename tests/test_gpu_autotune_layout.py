"""The FP64 autotuner times the structure-factor layouts with the kernels that
have them (FP64 sums), also where the form set takes the double-float ones: in
its sweep the structure factors take as long as in the strict form's sweep,
ten times what the double-float kernel takes.
"""
import ctypes as C

import pytest

import xmd_x
from test_gpu_ensemble import make

pytestmark = pytest.mark.gpu


def test_layouts_are_timed():
    lib = xmd_x.load(3, 4)
    s, box = make(lib, ("ueg", 512, 8, 0.5, 1.0), 9)
    pf = lib.fn("md_coulomb_3d_ewald_force_x")
    xmd_x.set_potentials(lib, coul_s=1.0, alpha=5.6 / box, nsum=10)
    spent, chosen = {}, {}
    try:
        for mode in (2, 0, 2, 0):  # strict, FP64; the first pair warms up
            lib.check(lib.md_gb300_set_precision_x(mode))
            bps, lay, ms = C.c_int(), C.c_int(), C.c_double()
            lib.check(lib.md_gb300_profile_x(1))
            lib.check(lib.md_gb300_autotune_fp64_x(s.pimd, pf, 3, C.byref(bps), C.byref(lay), C.byref(ms)))
            spent[mode] = lib.profile_report()["sk"]
            lib.check(lib.md_gb300_profile_x(0))
            chosen[mode] = lay.value
            assert ms.value > 0
    finally:
        lib.check(lib.md_gb300_set_precision_x(0))
        s.free()
    print(spent, chosen)
    assert spent[0][0] >= 0.6 * spent[2][0]  # (milliseconds, launches)
    assert chosen[0] in (1, 2, 3)
