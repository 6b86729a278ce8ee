"""The persistent ensemble step for every wave-vector cube it takes, odd and even
(its reciprocal forces take harmonics two at a time): bit for bit the states
of stepping each system on its own.
"""
import ctypes as C

import numpy as np
import pytest

import xmd_x
from test_gpu_ensemble import STEP_FN, make

pytestmark = pytest.mark.gpu

SPECS = [("ueg", 16, 4, 0.5, 1.0), ("ueg", 33, 3, 0.75, 3.0)]


@pytest.mark.parametrize("nsum", range(1, 9))
@pytest.mark.parametrize("alphaL", [5.6, 9.0])  # the longer columns' last vectors dropped, all kept
def test_matches_individual_steps(nsum, alphaL):
    lib = xmd_x.load(3, 4)
    ens, ref = ([make(lib, sp, 40 + i) for i, sp in enumerate(SPECS)] for _ in range(2))

    def one(s, box):
        xmd_x.set_potentials(lib, coul_s=1.0, alpha=alphaL / box, nsum=nsum)
        xmd_x.md_step(lib, s, 0.05, image=1, pair=lib.fn("md_coulomb_3d_ewald_force_x"), pbc=True)

    def cb(i, ctx):
        try:
            one(*ens[i])
            return 0
        except Exception:
            return -1

    graph = C.c_void_p()
    lib.check(lib.md_gb300_set_precision_x(1))
    try:
        for s, box in ens + ref:
            one(s, box)
        fn = STEP_FN(cb)
        lib.check(lib.md_gb300_capture_ensemble_persistent_x(len(ens), C.cast(fn, C.c_void_p), None, C.byref(graph)))
        lib.check(lib.md_gb300_graph_launch_x(graph, 2))
        lib.check(lib.md_gb300_ensemble_status_x(graph))
        for s, box in ref:
            one(s, box)
            one(s, box)
        for (a, _), (b, _) in zip(ens, ref):
            sa, sb = a.state(), b.state()
            for k in ("x", "v", "f", "theta", "vtheta"):
                assert np.array_equal(sa[k], sb[k]), k
    finally:
        lib.check(lib.md_gb300_set_precision_x(0))
        if graph:
            lib.md_gb300_graph_free_x(graph)
        for s, _ in ens + ref:
            s.free()
