"""Estimators after a replayed graph use what the replay left, not what the last
call made by hand left: the same numbers as the calls made by hand, bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

import xmd_x

pytestmark = pytest.mark.gpu


def _capture(lib, calls):
    g = C.c_void_p()
    lib.check(lib.md_gb300_capture_begin_x())
    calls()
    lib.check(lib.md_gb300_capture_end_x(C.byref(g)))
    return g


@pytest.mark.parametrize("N", [5, 64, 160])
@pytest.mark.parametrize("left", ["energies", "recursions", "forces", "forces only"])
def test_estimator_after_replay(N, left):
    lib = xmd_x.load(3, 4)
    P, T = 3, 0.5
    rng = np.random.default_rng(N)
    x0, x1 = (rng.standard_normal((N, 1, 3)) + 0.2 * rng.standard_normal((N, P, 3)) for _ in range(2))
    s = xmd_x.PimdSystem(lib, N, P, 0.8, T)

    def exchange(forces):
        lib.check(lib.md_pimd_fast_fill_ENk_x(s.pimd, 0))
        lib.check(lib.md_pimd_fill_VB_x(s.pimd))
        if forces:
            lib.check(lib.md_pimd_fast_fill_force_VB_x(s.pimd, 0))

    calls = {"energies": lambda: lib.check(lib.md_pimd_fast_fill_ENk_x(s.pimd, 0)),
             "recursions": lambda: exchange(False), "forces": lambda: exchange(True),
             "forces only": lambda: lib.check(lib.md_pimd_fast_fill_force_VB_x(s.pimd, 0))}[left]

    def estimate():
        lib.check(lib.md_gb300_profile_x(1))
        lib.check(lib.md_pimd_calc_VBN_energy_x(s.pimd, s.stats))
        e = s.take_energy()
        prof = lib.profile_report()
        lib.check(lib.md_gb300_profile_x(0))
        return e, "est_rows" in prof

    graph = None
    try:
        zero = np.zeros(x0.size)
        s.set_state(m=np.ones(N * P), x=x0, v=zero, f=zero)
        exchange(True)  # every buffer is there
        graph = _capture(lib, calls)
        got = []
        for replay in (False, True):
            for after in (False, True):  # what was made by hand before: the energies alone, or G too
                s.set_state(x=x0, v=zero, f=zero)
                exchange(after)
                if not after:
                    lib.check(lib.md_pimd_fast_fill_ENk_x(s.pimd, 0))
                s.set_state(x=x1, v=zero, f=zero)
                if left == "forces only":
                    exchange(False)  # a replay takes the recursions by the address they had
                else:
                    lib.check(lib.md_reset_force_x(s.sim))
                lib.check(lib.md_gb300_graph_launch_x(graph, 1)) if replay else calls()
                got.append(estimate())
        assert [r for _, r in got] == [left.startswith("forces")] * 2 + [left == "forces"] * 2
        if left == "forces only":  # by hand from G, after the replay from the recursion: 1e-10 as everywhere
            np.testing.assert_allclose([e for e, _ in got], got[0][0], rtol=1e-10)
        else:
            assert len({e for e, _ in got}) == 1
    finally:
        if graph:
            lib.md_gb300_graph_free_x(graph)
        s.free()
