"""Gaussian pair forces and energies at a negative range: the range enters squared
only, so they are those of the positive one, bit for bit, through every entry point
(own pairs in FP64 and in the mixed form, cross pairs, the call without allocations),
and the oracle's.
"""
import numpy as np
import pytest

import orc
import xmd_x
from gpu_common import PARITY, random_state
from helpers import assert_close

pytestmark = pytest.mark.gpu

N, NB, P, BOX = 45, 20, 4, 3.0


def _all(lib, kind, s):
    """every Gaussian result at range s"""
    D = lib.D
    xmd_x.set_potentials(lib, gauss_g=2.4, gauss_s=s)
    pf, pe = lib.fn(f"md_{kind}_force_x"), lib.fn(f"md_{kind}_energy_x")
    a, b = xmd_x.PimdSystem(lib, N, P, 0.5, 1.0, box=BOX), xmd_x.PimdSystem(lib, NB, P, 0.5, 1.0, box=BOX)
    out = {}
    try:
        for u, n, seed in ((a, N, 1), (b, NB, 2)):
            u.set_state(**random_state(D, 4, n, P, 1.0, BOX, True, seed))
        for name, mixed in (("own", 0), ("mixed", 1)):
            lib.check(lib.md_gb300_set_precision_x(mixed))
            lib.check(lib.md_reset_force_x(a.sim))
            lib.check(lib.md_pimd_calc_pair_force_x(a.pimd, pf))
            out[name] = a.state()["f"]
        lib.check(lib.md_gb300_set_precision_x(0))
        lib.check(lib.md_pimd_calc_pair_energy_x(a.pimd, pe, a.stats))
        out["energy"] = np.array([a.take_energy()])
        for u in (a, b):
            lib.check(lib.md_reset_force_x(u.sim))
        lib.check(lib.md_pimd_calc_pair_force_2_x(a.pimd, b.pimd, pf))
        out["cross a"], out["cross b"] = a.state()["f"], b.state()["f"]
        lib.check(lib.md_pimd_calc_pair_energy_2_x(a.pimd, b.pimd, pe, a.stats))
        out["cross energy"] = np.array([a.take_energy()])
        x = a.state()["x"]
    finally:
        lib.check(lib.md_gb300_set_precision_x(0))
        a.free()
        b.free()
    torch = pytest.importorskip("torch")
    soa = np.ascontiguousarray(x.reshape(N, P, D).transpose(1, 2, 0))
    xd, m = torch.tensor(soa, device="cuda"), torch.ones((P, N), dtype=torch.float64, device="cuda")
    f = torch.zeros_like(xd)
    lib.check(lib.md_gb300_pair_force_noalloc_x(pf, xd.data_ptr(), m.data_ptr(), f.data_ptr(), N, P, N,
                                                np.full(D, BOX).ctypes.data_as(xmd_x._dp),
                                                torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    out["noalloc"] = f.cpu().numpy()
    return out


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("kind", ["gaussian", "periodic_gaussian"])
def test_sign_of_the_range(D, kind):
    lib = xmd_x.load(D, 4)
    plus, minus = _all(lib, kind, 0.5), _all(lib, kind, -0.5)
    for k in plus:
        assert np.any(plus[k] != 0), k
        np.testing.assert_array_equal(plus[k], minus[k], err_msg=k)
    if kind == "gaussian":
        st = random_state(D, 4, N, P, 1.0, BOX, True, 1)
        o = orc.OrcSim(D, 4, N * P, st["m"], st["x"], st["v"], np.zeros(N * P * D), st["cf"], st["theta"], st["vtheta"],
                       st["Q"], 1.0, [BOX] * 3)
        prm = orc.params(gauss_g=2.4, gauss_s=-0.5)
        assert orc.lib().orc_pair_force(o.ref, N, P, orc.PAIR_GAUSSIAN, orc.C.byref(prm)) == 0
        assert_close(minus["own"], o.f, PARITY, "forces at a negative range")
