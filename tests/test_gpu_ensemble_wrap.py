"""The persistent ensemble step with beads that cross the box faces: the end
beads' own ring springs belong to the positions before the periodic wrap, which the
same phase applies.  Short rings (P = 2, 3: every bead is an end bead or beside
one), image on and off, run three times: bit for bit the states of stepping each
system on its own, every time.
"""
import ctypes as C

import numpy as np
import pytest

import xmd_x
from test_gpu_ensemble import STEP_FN, make

pytestmark = pytest.mark.gpu

SPECS = [("ueg", 33, 2, 0.5, 1.0), ("ueg", 64, 3, 0.75, 2.0), ("ueg", 100, 2, 1.0, 1.0), ("ueg", 17, 5, 0.25, 3.0)] * 4


def near_faces(s, box, seed):
    """whole rings within a few hundredths of a face, moving across it"""
    rng = np.random.default_rng(seed)
    n, P, D = s.N, s.P, 3
    centre = rng.uniform(0, box, (n, 1, D))
    axis = rng.integers(0, D, n)
    centre[np.arange(n), 0, axis] = rng.integers(0, 2, n) * box
    x = np.mod(centre + 0.02 * rng.standard_normal((n, P, D)), box)
    s.set_state(x=x, v=4 * rng.standard_normal((n, P, D)))


@pytest.mark.parametrize("image,dt", [(1, 0.02), (0, 0.002)])
def test_end_beads_at_the_faces(image, dt):
    lib = xmd_x.load(3, 4)

    def one(s, box):
        xmd_x.set_potentials(lib, coul_s=1.0, alpha=5.6 / box, nsum=4)
        xmd_x.md_step(lib, s, dt, image=image, pair=lib.fn("md_coulomb_3d_ewald_force_x"), pbc=True)

    lib.check(lib.md_gb300_set_precision_x(1))
    ens, ref = ([make(lib, sp, 60 + i) for i, sp in enumerate(SPECS)] for _ in range(2))
    graph = C.c_void_p()

    def cb(i, ctx):
        try:
            one(*ens[i])
            return 0
        except Exception:
            return -1

    try:
        for s, box in ens + ref:
            one(s, box)
        fn = STEP_FN(cb)
        lib.check(lib.md_gb300_capture_ensemble_persistent_x(len(ens), C.cast(fn, C.c_void_p), None, C.byref(graph)))
        for rep in range(3):
            for i, ((a, box), (b, _)) in enumerate(zip(ens, ref)):
                for s in (a, b):
                    near_faces(s, box, 100 * rep + i)
                    lib.check(lib.md_pimd_fast_fill_ENk_x(s.pimd, image))  # uploads the state
            crossed = sum(np.count_nonzero(np.minimum(s.state()["x"], box - s.state()["x"]) < 0.05) for s, box in ref)
            assert crossed > 100
            lib.check(lib.md_gb300_graph_launch_x(graph, 4))
            lib.check(lib.md_gb300_ensemble_status_x(graph))
            for s, box in ref:
                for _ in range(4):
                    one(s, box)
            for (a, _), (b, _) in zip(ens, ref):
                sa, sb = a.state(), b.state()
                for k in ("x", "v", "f", "theta", "vtheta"):
                    assert np.isfinite(sb[k]).all()
                    assert np.array_equal(sa[k], sb[k]), (rep, k)
    finally:
        lib.check(lib.md_gb300_set_precision_x(0))
        if graph:
            lib.md_gb300_graph_free_x(graph)
        for s, _ in ens + ref:
            s.free()
