"""The persistent ensemble step for systems whose own calls take the cluster solve
of the exchange recursions (N > 128; sixteen blocks from N = 929 on), beside a small
one: bit for bit the states of stepping each system on its own, signless weights of
every kind (xi = 0, between and 1), with and without the Ewald sums.
"""
import ctypes as C

import numpy as np
import pytest

import xmd_x
from test_gpu_ensemble import STEP_FN, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,P,xi", [(129, 3, 1.0), (160, 2, 0.0), (200, 4, 0.5), (500, 2, 1.0), (928, 2, 0.3), (1000, 2, 1.0)])
@pytest.mark.parametrize("kind", ["ueg", "trap"])
def test_matches_individual_steps(kind, N, P, xi):
    lib = xmd_x.load(3, 4)
    specs = [(kind, N, P, xi, 2.0), (kind, 40, 3, 0.5, 1.0)]
    ens, ref = ([make(lib, sp, 70 + i) for i, sp in enumerate(specs)] for _ in range(2))

    def one(s, box):
        if kind == "ueg":
            xmd_x.set_potentials(lib, coul_s=1.0, alpha=5.6 / box, nsum=4)
            xmd_x.md_step(lib, s, 0.05, image=1, pair=lib.fn("md_coulomb_3d_ewald_force_x"), pbc=True)
        else:
            xmd_x.set_potentials(lib, trap_w=1.0, gauss_g=0.75 * np.pi, gauss_s=0.5)
            xmd_x.md_step(lib, s, 0.005, trap=lib.fn("md_harmonic_trap_force_x"), pair=lib.fn("md_gaussian_force_x"))

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
                assert np.isfinite(sb[k]).all()
                assert np.array_equal(sa[k], sb[k]), k
    finally:
        lib.check(lib.md_gb300_set_precision_x(0))
        if graph:
            lib.md_gb300_graph_free_x(graph)
        for s, _ in ens + ref:
            s.free()
