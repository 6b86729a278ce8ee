"""Performance cases of the path-integral MD framework.

Each case is work that a program built on this library has it do through the
public entry points (the C ABI by way of md-lab_gb300/xmd_x.py):

  steps      `steps` MD steps in the reference driver's call order, then the
             primitive estimator and the state read back, as a run does that
             samples every `steps` steps; as plain calls or as a replayed
             CUDA graph; 2D/3D trap with Gaussian repulsion, ideal trapped
             bosons, electron gas (Ewald), electron gas with the learned
             residual, and two species
  ensemble   the same for many independent systems, one persistent launch
             per step
  sample     the estimators of one configuration: pair or trap energy,
             primitive and virial exchange energies, g(r)
  train      Adam steps of the residual network on collected configurations

Inputs come from the seed alone: ring polymers drawn from the free (electron
gas) or harmonic (trap) path distribution, electron centres on a jittered
lattice so that no two start on top of each other, thermal velocities and
thermostat momenta.

The mixed and learned forms compute forces in FP32, so their state is handed
over as FP32 values; the FP64 form's state comes back as the library's own
host records.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "md-lab_gb300"))
import xmd_x  # noqa: E402

GAUSS_G, GAUSS_S = 0.75 * math.pi, 0.5  # V(r) = 3 exp(-r^2/0.25)
GAUSS_G_2D = 0.5 * math.pi  # V(r) = 2 exp(-r^2/0.25)
ALPHA_L = 5.6
_LIBS = {}


def _lib(D):
    if D not in _LIBS:
        _LIBS[D] = xmd_x.load(D, 4)
    return _LIBS[D]


# ---------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------
def listed():
    return [
        # the smallest run: four bosons in a 2D trap, plain calls, where
        # launches and latency are all there is
        {"name": "trap2d_n4_p32_fp64", "what": "steps", "system": "trap", "form": "fp64", "D": 2, "N": 4, "P": 32,
         "xi": 1.0, "beta": 2.0, "dt": 0.01, "steps": 10, "graph": False},
        # xi extrapolation in a 3D trap: N=64, P=64, beta=4, FP32 forces
        {"name": "trap3d_n64_p64_mixed", "what": "steps", "system": "trap", "form": "mixed", "D": 3, "N": 64, "P": 64,
         "xi": 0.5, "beta": 4.0, "dt": 0.005, "steps": 10, "graph": True},
        # the same kind of run in FP64, at sizes that no tile divides
        {"name": "trap3d_n61_p45_fp64", "what": "steps", "system": "trap", "form": "fp64", "D": 3, "N": 61, "P": 45,
         "xi": 0.25, "beta": 4.0, "dt": 0.005, "steps": 10, "graph": True},
        # electron gas of ordinary size, rs=2, FP64
        {"name": "ueg_n128_p32_fp64", "what": "steps", "system": "ueg", "form": "fp64", "D": 3, "N": 128, "P": 32,
         "xi": 0.6, "rs": 2.0, "theta": 0.5, "nsum": 8, "dt": 0.05, "steps": 10, "graph": True},
        # the benchmark's electron gas in each arithmetic form
        {"name": "ueg_n512_p64_fp64", "what": "steps", "system": "ueg", "form": "fp64", "D": 3, "N": 512, "P": 64,
         "xi": 0.5, "rs": 1.0, "theta": 0.5, "nsum": 10, "dt": 0.01, "steps": 10, "graph": True},
        {"name": "ueg_n512_p64_mixed", "what": "steps", "system": "ueg", "form": "mixed", "D": 3, "N": 512, "P": 64,
         "xi": 0.5, "rs": 1.0, "theta": 0.5, "nsum": 10, "dt": 0.01, "steps": 10, "graph": True},
        {"name": "ueg_n512_p64_learned", "what": "steps", "system": "ueg", "form": "learned", "D": 3, "N": 512,
         "P": 64, "xi": 0.5, "rs": 1.0, "theta": 0.5, "nsum": 10, "nsum_cheap": 3, "dt": 0.01, "steps": 10,
         "graph": True},
        # ideal trapped bosons, the size of the published timings: all
        # exchange recursion and thermostat
        {"name": "ideal_n1600_p72_fp64", "what": "steps", "system": "ideal", "form": "fp64", "D": 3, "N": 1600,
         "P": 72, "xi": 1.0, "beta": 6.0, "dt": 0.01, "steps": 10, "graph": True},
        # unpolarised electron gas: two species and their cross pairs
        {"name": "two_species_n256_p64_fp64", "what": "steps", "system": "two", "form": "fp64", "D": 3, "N": 256,
         "N2": 256, "P": 64, "xi": 0.5, "rs": 1.0, "theta": 0.5, "nsum": 10, "dt": 0.01, "steps": 4, "graph": True},
        # extrapolation over xi and temperature: 64 uneven systems, half
        # traps, half electron gases, one persistent launch per step
        {"name": "ensemble_64", "what": "ensemble", "systems": 64, "nmin": 16, "nmax": 128, "pmin": 16, "pmax": 64,
         "nsum": 8, "form": "mixed", "steps": 20},
        # what a sampling run evaluates on one configuration
        {"name": "sample_ueg_n128_p32", "what": "sample", "system": "ueg", "form": "fp64", "D": 3, "N": 128, "P": 32,
         "xi": 0.6, "rs": 2.0, "theta": 0.5, "nsum": 8, "points": 200},
        # training of the residual network: forward, backward and Adam
        {"name": "train_n256_p16", "what": "train", "system": "ueg", "form": "mixed", "D": 3, "N": 256, "P": 16,
         "xi": 0.5, "rs": 1.0, "theta": 0.5, "nsum": 8, "nsum_cheap": 3, "configs": 8, "steps": 20, "tiles": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trap", "trap", "ueg", "ueg", "ueg", "learned", "ideal", "two", "ensemble", "sample", "train"])
    xi = rng.choice([0.0, 0.2, 0.4, 0.5, 0.6, 0.75, 0.8, 1.0])
    gas = {"rs": rng.choice([1.0, 2.0, 4.0]), "theta": rng.choice([0.5, 0.75, 1.0]), "dt": 0.01}
    if kind == "trap":
        return {"what": "steps", "system": "trap", "form": rng.choice(["fp64", "mixed"]), "D": rng.choice([2, 3, 3]),
                "N": _log(rng, 3, 300), "P": _log(rng, 8, 72), "xi": xi, "beta": rng.choice([1.0, 2.0, 4.0]),
                "dt": 0.005, "steps": 10, "graph": rng.random() < 0.7}
    if kind == "ueg":
        return {"what": "steps", "system": "ueg", "form": rng.choice(["fp64", "mixed"]), "D": 3,
                "N": _log(rng, 12, 512), "P": _log(rng, 8, 64), "xi": xi, "nsum": rng.randint(6, 10), "steps": 10,
                "graph": rng.random() < 0.7, **gas}
    if kind == "learned":
        return {"what": "steps", "system": "ueg", "form": "learned", "D": 3, "N": _log(rng, 64, 512),
                "P": _log(rng, 8, 64), "xi": xi, "nsum": rng.randint(8, 10), "nsum_cheap": 3, "steps": 10,
                "graph": True, **gas}
    if kind == "ideal":
        return {"what": "steps", "system": "ideal", "form": "fp64", "D": rng.choice([2, 3]),
                "N": _log(rng, 100, 1600), "P": _log(rng, 12, 72), "xi": xi, "beta": rng.choice([1.0, 6.0]),
                "dt": 0.01, "steps": 10, "graph": True}
    if kind == "two":
        n = _log(rng, 16, 256)
        return {"what": "steps", "system": "two", "form": "fp64", "D": 3, "N": n, "N2": rng.randint(max(8, n // 2), n),
                "P": _log(rng, 8, 64), "xi": xi, "nsum": rng.randint(6, 10), "steps": 4, "graph": True, **gas}
    if kind == "ensemble":
        return {"what": "ensemble", "systems": rng.randint(6, 64), "nmin": 16, "nmax": rng.choice([32, 64, 128]),
                "pmin": 16, "pmax": rng.choice([32, 64]), "nsum": rng.randint(6, 8), "form": "mixed", "steps": 20}
    if kind == "sample":
        system = rng.choice(["ueg", "trap"])
        case = {"what": "sample", "system": system, "form": "fp64", "D": 3, "N": _log(rng, 16, 300),
                "P": _log(rng, 8, 64), "xi": xi, "points": rng.randint(50, 400)}
        case.update({"nsum": rng.randint(6, 10), "rs": gas["rs"], "theta": gas["theta"]} if system == "ueg" else
                    {"beta": rng.choice([1.0, 2.0, 4.0])})
        return case
    return {"what": "train", "system": "ueg", "form": "mixed", "D": 3, "N": _log(rng, 64, 256), "P": _log(rng, 8, 24),
            "xi": 0.5, "rs": gas["rs"], "theta": gas["theta"], "nsum": 8, "nsum_cheap": 3, "configs": rng.randint(2, 8),
            "steps": 20, "tiles": rng.choice([32, 64, 100, 128])}


# ---------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------
def _physics(case):
    """box edge (0: none), temperature"""
    if case["system"] in ("trap", "ideal"):
        return 0.0, 1.0 / case["beta"]
    n = case["N"] + case.get("N2", 0)
    box = (4 * math.pi * n / 3) ** (1 / 3) * case["rs"]
    spins = 2 if "N2" in case else 1
    return box, case["theta"] * 0.5 * (6 * math.pi ** 2 * n / spins / box ** 3) ** (2 / 3)


def _rmax(case):
    return (_physics(case)[0] or 8.0) / 2


def _paths(rng, N, P, D, beta, w):
    """ring polymers of the action beta sum (omega_P^2 (x_j - x_j+1)^2 + w^2 x_j^2 / P) / 2, centred on 0 for w = 0"""
    lam = P / beta ** 2 * 4 * np.sin(math.pi * np.arange(P) / P) ** 2 + w * w / P
    amp = np.zeros(P)
    amp[lam > 1e-12] = 1 / np.sqrt(beta * lam[lam > 1e-12])
    z = np.fft.fft(rng.standard_normal((N, P, D)), axis=1)
    return np.real(np.fft.ifft(z * amp[None, :, None], axis=1))


def _inputs(case, seed):
    """one dict of x, v, theta, vtheta, Q per species"""
    rng = np.random.default_rng(seed)
    box, T = _physics(case)
    D, P, beta = case["D"], case["P"], 1 / T
    sizes = [case["N"]] + ([case["N2"]] if "N2" in case else [])
    if box:
        m = math.ceil(sum(sizes) ** (1 / 3))
        sites = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
        sites = rng.permutation(sites)[:sum(sizes)] + 0.5 + 0.25 * rng.uniform(-1, 1, (sum(sizes), 3))
        centre = sites * (box / m)
    out, n0 = [], 0
    omega = math.sqrt(P) / beta
    for n in sizes:
        x = _paths(rng, n, P, D, beta, 0.0 if box else 1.0)
        if box:
            x = np.mod(x + centre[n0:n0 + n, None, :], box)
        n0 += n
        out.append({"N": n, "x": x, "v": rng.standard_normal((n, P, D)) * math.sqrt(T),
                    "vtheta": rng.standard_normal((n, P, D, 4)) * omega, "Q": T / omega ** 2})
    return out


def _ensemble(case, seed):
    """the systems of an ensemble case, each a steps case of its own with its seed; shapes do not depend on the seed"""
    rng = np.random.default_rng(case["systems"])
    ns = [n for n in (16, 24, 32, 48, 64, 96, 128) if case["nmin"] <= n <= case["nmax"]]
    ps = [p for p in (16, 32, 64) if case["pmin"] <= p <= case["pmax"]]
    out = []
    for i in range(case["systems"]):
        c = {"system": "ueg" if i % 2 else "trap", "form": case["form"], "D": 3, "N": int(rng.choice(ns)),
             "P": int(rng.choice(ps)), "xi": (i // 8) % 8 / 7.0, "steps": case["steps"]}
        beta = i % 8 + 1.0
        if c["system"] == "ueg":
            # theta chosen so that the temperature is 1 / beta
            t_f = 0.5 * (6 * math.pi ** 2 * 3 / (4 * math.pi * 8.0)) ** (2 / 3)
            c.update({"rs": 2.0, "theta": 1 / (beta * t_f), "nsum": case["nsum"], "dt": 0.05})
        else:
            c.update({"beta": beta, "dt": 0.005})
        out.append((c, seed * 1000 + i))
    return out


# ---------------------------------------------------------------------
# through the framework
# ---------------------------------------------------------------------
def _potentials(lib, case, box):
    if box:
        xmd_x.set_potentials(lib, coul_s=1.0, alpha=ALPHA_L / box, nsum=case["nsum"])
    else:
        xmd_x.set_potentials(lib, trap_w=1.0, gauss_g=GAUSS_G_2D if case["D"] == 2 else GAUSS_G, gauss_s=GAUSS_S)


def _systems(lib, case, seed):
    box, T = _physics(case)
    out = []
    for s in _inputs(case, seed):
        u = xmd_x.PimdSystem(lib, s["N"], case["P"], case["xi"], T, box=box or 10.0)
        u.set_state(m=np.ones(s["N"] * case["P"]), x=s["x"], v=s["v"], f=np.zeros(s["x"].size),
                    theta=np.zeros(s["vtheta"].size), vtheta=s["vtheta"], Q=np.full(s["vtheta"].size, s["Q"]),
                    cf=np.ones(s["x"].size))
        out.append(u)
    return out


def _restore(systems, case, seed):
    """the initial state again, on the device"""
    for u, s in zip(systems, _inputs(case, seed)):
        u.set_state(x=s["x"], v=s["v"], f=np.zeros(s["x"].size), theta=np.zeros(s["vtheta"].size), vtheta=s["vtheta"])
        u.lib.check(u.lib.md_pimd_fast_fill_ENk_x(u.pimd, 1 if _physics(case)[0] else 0))


def _stepper(lib, case, systems):
    box, _ = _physics(case)
    image, pbc = (1, True) if box else (0, False)
    trap = lib.fn("md_harmonic_trap_force_x") if not box else None
    pair = {"trap": "md_gaussian_force_x", "ideal": None}.get(case["system"], "md_coulomb_3d_ewald_force_x")
    pair = lib.fn(pair) if pair else None
    if case["system"] == "two":
        return lambda: xmd_x.two_species_step(lib, *systems, case["dt"], image=image, pair=pair, pbc=pbc)
    return lambda: xmd_x.md_step(lib, systems[0], case["dt"], image=image, trap=trap, pair=pair, pbc=pbc)


class State:
    """what a program keeps between calls; device memory is given back with it"""

    def __init__(self, case):
        self.case, self.systems, self.graph, self.model, self.gr = case, [], None, None, None
        self.lib = _lib(case.get("D", 3))
        self.lib.check(self.lib.md_gb300_set_precision_x(0 if case["form"] == "fp64" else 1))

    def capture(self, step):
        self.graph = C.c_void_p()
        self.lib.check(self.lib.md_gb300_capture_begin_x(), "capture")
        step()
        self.lib.check(self.lib.md_gb300_capture_end_x(C.byref(self.graph)), "capture")

    def __del__(self):
        self.lib.md_gb300_synchronize_x()
        if self.graph:
            self.lib.md_gb300_graph_free_x(self.graph)
        if self.model:
            if self.case["what"] == "steps":
                self.model.detach(self.systems[0])
            self.model.free()
        if self.gr:
            self.lib.md_gb300_free_stats_x(self.gr)
        for u in self.systems:
            u.free()


def _prepare_model(st, case, seed, configs):
    """network with data of short converged runs, its weights from the seed"""
    lib, u = st.lib, st.systems[0]
    st.model = xmd_x.EwaldModel(lib, u, nsum_cheap=case["nsum_cheap"], capacity=configs, seed=7)
    step = _stepper(lib, {**case, "dt": 0.01}, st.systems)
    for _ in range(configs):
        step()
        st.model.collect(u)
    rng = np.random.default_rng(seed + 1)
    shapes = ((128, 64), (128,), (128, 128), (128,), (4, 128), (4,))
    st.model.params(np.concatenate([(rng.standard_normal(s) / math.sqrt(s[-1]) if len(s) > 1 else np.zeros(s)).ravel()
                                    for s in shapes]).astype(np.float32))


def _prepare_ensemble(case, seed):
    st = State(case)
    lib = st.lib
    parts = _ensemble(case, seed)
    for c, s in parts:
        st.systems += _systems(lib, c, s)
    steps = [_stepper(lib, c, [u]) for (c, _), u in zip(parts, st.systems)]

    def one(i, ctx=None):
        try:
            _potentials(lib, parts[i][0], _physics(parts[i][0])[0])
            steps[i]()
            return 0
        except RuntimeError:
            return -1

    for i in range(len(steps)):
        one(i)
    fn = C.CFUNCTYPE(C.c_int, C.c_int, C.c_void_p)(one)
    st.graph = C.c_void_p()
    lib.check(lib.md_gb300_capture_ensemble_persistent_x(len(steps), C.cast(fn, C.c_void_p), None, C.byref(st.graph)),
              "ensemble capture")
    for (c, s), u in zip(parts, st.systems):
        _potentials(lib, c, _physics(c)[0])
        _restore([u], c, s)
    _buffers(st)
    return st


def prepare(case, seed):
    if case["what"] == "ensemble":
        return _prepare_ensemble(case, seed)
    st = State(case)
    lib, box = st.lib, _physics(case)[0]
    _potentials(lib, case, box)
    st.systems = _systems(lib, case, seed)
    if case["what"] == "train":
        _prepare_model(st, case, seed, case["configs"])
        return st
    if case["what"] == "sample":
        # the configuration, its exchange tables and its forces
        u = st.systems[0]
        st.gr = lib.md_alloc_stats_x(case["points"])
        image, pair = (1, "md_coulomb_3d_ewald_force_x") if box else (0, "md_gaussian_force_x")
        lib.check(lib.md_pimd_fast_fill_ENk_x(u.pimd, image))
        lib.check(lib.md_pimd_fill_VB_x(u.pimd))
        lib.check(lib.md_pimd_fast_fill_force_VB_x(u.pimd, image))
        if not box:
            lib.check(lib.md_pimd_calc_trap_force_x(u.pimd, lib.fn("md_harmonic_trap_force_x")))
        lib.check(lib.md_pimd_calc_pair_force_x(u.pimd, lib.fn(pair)))
        return st
    st.step = _stepper(lib, case, st.systems)
    if case["form"] == "learned":
        _prepare_model(st, case, seed, 1)
        st.model.attach(st.systems[0], judge_every=0)
    if case["graph"]:
        st.step()
        st.capture(st.step)
    _restore(st.systems, case, seed)
    if case["form"] != "fp64":
        _buffers(st)
    return st


class _Records:
    """a view of the state's own host records that keeps the state alive"""

    def __init__(self, st, a):
        self.st, self.__array_interface__ = st, a.__array_interface__


def _read(st):
    """the states after a host sync, one dict per system: {m, x, v, f} records, thermostat positions and momenta"""
    out = []
    for i, u in enumerate(st.systems):
        if not st.lib.md_simulation_sync_host_x(u.sim, 1):
            raise RuntimeError("sync failed: " + st.lib.err())
        p, c = u._particles(), u._chains()
        if st.case["form"] == "fp64":
            views = {"particles": p, "theta": c["theta"], "vtheta": c["vtheta"]}
            out.append({k: np.asarray(_Records(st, v)) for k, v in views.items()})
        else:
            # a chain record is 1 + 3 L doubles: the count, theta, vtheta, Q
            st.particles[i].copy_(torch.from_numpy(p))
            st.chains[i].copy_(torch.from_numpy(c.view(np.float64).reshape(len(c), -1)))
            out.append({"particles": st.particles[i], "theta": st.chains[i][:, 1:5], "vtheta": st.chains[i][:, 5:9]})
    return out


def _buffers(st):
    """FP32 host memory for the states of the mixed forms, all systems in one piece"""
    nb = [u.nb for u in st.systems]
    st.all_particles, st.all_chains = torch.zeros(sum(nb), 1 + 3 * st.lib.D), torch.zeros(sum(nb) * st.lib.D, 13)
    st.particles, st.chains = st.all_particles.split(nb), st.all_chains.split([n * st.lib.D for n in nb])


def _run_sample(st):
    lib, case, u = st.lib, st.case, st.systems[0]
    ck, image = lib.check, 1 if _physics(case)[0] else 0
    out = {}
    if image:
        ck(lib.md_pimd_calc_pair_energy_x(u.pimd, lib.fn("md_coulomb_3d_ewald_energy_x"), u.stats))
    else:
        ck(lib.md_pimd_calc_trap_energy_x(u.pimd, lib.fn("md_harmonic_trap_energy_x"), u.stats))
        out["trap"] = u.take_energy()
        ck(lib.md_pimd_calc_pair_energy_x(u.pimd, lib.fn("md_gaussian_energy_x"), u.stats))
    out["pair"] = u.take_energy()
    ck(lib.md_pimd_calc_VBN_energy_x(u.pimd, u.stats))
    out["primitive"] = u.take_energy()
    ck(lib.md_pimd_fast_fill_ENk2_x(u.pimd, image))
    ck(lib.md_pimd_calc_vi_virial_energy_x(u.pimd, u.stats, image))
    out["virial"] = u.take_energy()
    ck(lib.md_reset_stats_f_x(st.gr, 0.0))
    ck(lib.md_pimd_calc_pair_correlation_x(u.pimd, st.gr, _rmax(case), case["N"] * (case["N"] - 1) / 2.0, 1, image))
    out["gr"] = np.ctypeslib.as_array(st.gr.contents.fxs[0], (case["points"],)).copy()
    return {k: np.float64(v) if np.ndim(v) == 0 else v for k, v in out.items()}


def run(st):
    case, lib = st.case, st.lib
    if case["what"] == "sample":
        return _run_sample(st)
    if case["what"] == "train":
        loss = st.model.train(case["steps"], case["tiles"], 1e-3)
        return {"params": st.model.params(), "loss": np.float32(loss)}
    if st.graph:
        lib.check(lib.md_gb300_graph_launch_x(st.graph, case["steps"]))
    else:
        for _ in range(case["steps"]):
            st.step()
    if case["what"] == "ensemble":
        _read(st)
        return {"particles": st.all_particles, "theta": st.all_chains[:, 1:5], "vtheta": st.all_chains[:, 5:9]}
    energies = []
    for u in st.systems:
        lib.check(lib.md_pimd_calc_VBN_energy_x(u.pimd, u.stats))
        e = u.take_energy()
        energies.append(np.float64(e) if case["form"] == "fp64" else np.float32(e))
    return {str(i): {"primitive": e, **r} for i, (e, r) in enumerate(zip(energies, _read(st)))}


# ---------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------
def _kept_nz(nsum):
    """+-nz pairs of the half-space wave vectors whose force weight reaches 1e-17 of the largest"""
    n = np.arange(-nsum, nsum + 1)
    nx, ny, nz = np.meshgrid(n, n, np.arange(1, nsum + 1), indexing="ij")
    g2 = nx * nx + ny * ny + nz * nz
    w = np.exp(-math.pi ** 2 * g2 / ALPHA_L ** 2) / np.sqrt(g2)
    return int((w >= 1e-17 * math.exp(-math.pi ** 2 / ALPHA_L ** 2)).sum()) // 2 + nsum


def _work_step(case):
    """flops of one step: springs and exchange tables (40 per entry), recursions (2 x 20), thermostat (120 per
    coordinate), pair forces (a Gaussian 30; an Ewald pair 39 plus 47 per image inside the form's cut-off, and 26 per
    wave vector and particle)"""
    N, P, D = case["N"] + case.get("N2", 0), case["P"], case["D"]
    ex = sum(n * n / 2 * 100.0 for n in (case["N"], case.get("N2", 0)))
    fl = ex + 120.0 * N * P * D + 12.0 * N * P * D
    pairs = P * N * (N - 1) / 2
    if case["system"] == "trap":
        fl += 30.0 * pairs
    elif case["system"] != "ideal":
        cut = 5.2 if case["form"] == "fp64" else 3.6
        nsum = case["nsum_cheap"] if case["form"] == "learned" else case["nsum"]
        fl += pairs * (39 + 47 * 4 / 3 * math.pi * (cut / ALPHA_L) ** 3) + 26.5 * _kept_nz(nsum) * N * P
        if case["form"] == "learned":
            fl += 2.0 * N * P * (64 * 128 + 128 * 128 + 128 * 16) + 2 * pairs * 38 + N * P * (4096 + 474 * 14)
    return fl


def _work_bytes(case):
    """positions, velocities, forces and chains, read and written once (Q and masses only read)"""
    ndof = (case["N"] + case.get("N2", 0)) * case["P"] * case["D"]
    return 8.0 * ndof * (2 * (3 + 8) + 4 + 1 / case["D"])


def work(case):
    if case["what"] == "ensemble":
        parts = [c for c, _ in _ensemble(case, 0)]
        return {"bytes": sum(map(_work_bytes, parts)), "flops": case["steps"] * sum(map(_work_step, parts))}
    N, P, D = case["N"], case["P"], case["D"]
    if case["what"] == "train":
        rows = case["steps"] * case["tiles"] * 128
        return {"bytes": rows * (64 * 2 + 12 * 4 + 4 * 4.0), "flops": 6.0 * rows * (64 * 128 + 128 * 128 + 128 * 4)}
    if case["what"] == "sample":
        pairs = P * N * (N - 1) / 2
        fl = 8.0 * N * P * D + 30 * N * N
        fl += pairs * (25 + 40 * 4 / 3 * math.pi * (5.8 / ALPHA_L) ** 3) + 9.0 * _kept_nz(case["nsum"]) * N * P \
            if case["system"] == "ueg" else 25.0 * pairs
        return {"bytes": 8.0 * (2 * N * P * D + 2 * N * N), "flops": fl}
    return {"bytes": _work_bytes(case), "flops": case["steps"] * _work_step(case)}


# ---------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------
class _Plain:
    """the textbook formulas of one system; positions (N, P, D)"""

    def __init__(self, case, box, T, inp):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        self.case, self.box, self.T, self.beta = case, box, T, 1 / T
        self.N, self.P, self.D = inp["N"], case["P"], case["D"]
        self.w2 = self.P * T * T
        self.x, self.v, self.vt = self.t(inp["x"]), self.t(inp["v"]), self.t(inp["vtheta"])
        self.f, self.th, self.Q = torch.zeros_like(self.x), torch.zeros_like(self.vt), inp["Q"]
        l, s = torch.meshgrid(*[torch.arange(1, self.N + 1, device=dev)] * 2, indexing="ij")
        self.l, self.low = l.to(torch.float64), s <= l
        # ln of xi^(l - s), -inf where the cycle s..l does not exist
        steps = torch.where(self.low, l - s, 0).to(torch.float64)
        lnxi = steps * math.log(case["xi"]) if case["xi"] > 0 else torch.where(l == s, 0.0, -math.inf).to(self.x)
        self.lnxi = torch.where(self.low, lnxi, -math.inf)

    def image(self, a):
        return a - self.box * torch.round(a / self.box) if self.box else a

    def link(self):
        """[a, b]: spring from the last bead of a to the first of b"""
        return 0.5 * self.w2 * self.image(self.x[:, None, -1] - self.x[None, :, 0]).square().sum(-1)

    def exchange(self):
        """cycle energies E[l, s], V_B, backward potentials, connection probabilities G[l, j]"""
        N, beta, x = self.N, self.beta, self.x
        inner = 0.5 * self.w2 * self.image(x[:, 1:] - x[:, :-1]).square().sum((1, 2))
        link = self.link()
        c = torch.cat([torch.zeros_like(inner[:1]), inner.cumsum(0)])
        g = torch.cat([torch.zeros_like(inner[:1]), torch.diagonal(link, 1).cumsum(0)])
        self.E = (c[1:, None] - c[None, :-1]) + (g[:, None] - g[None, :]) + link
        lnw = self.lnxi - beta * torch.where(self.low, self.E, 0.0)
        # the two recursions, row by row on the host: they are short and sequential
        lnb = lnw - self.l.log()
        wf, wb = lnw.cpu().numpy(), np.ascontiguousarray(lnb.T.cpu().numpy())
        V, B = np.zeros(N + 1), np.zeros(N + 1)

        def lse(t):
            top = t.max()
            return top + math.log(np.exp(t - top).sum())

        for l in range(1, N + 1):
            V[l] = (math.log(l) - lse(wf[l - 1, :l] - beta * V[:l])) / beta
        for s in range(N, 0, -1):
            B[s - 1] = -lse(wb[s - 1, s - 1:] - beta * B[s:]) / beta
        V, B = self.t(V), self.t(B)
        self.V, self.p = V, torch.exp(lnb - beta * (V[None, :-1] + B[1:, None] - V[N]))
        self.G = self.p.clone()
        nxt = 1 - torch.exp(-beta * (V[1:N] + B[1:N] - V[N]))
        self.G += torch.diag(nxt, 1)

    def spring_forces(self):
        x, w2 = self.x, self.w2
        f = torch.zeros_like(x)
        d = self.image(x[:, 1:] - x[:, :-1])
        f[:, 1:-1] = w2 * (d[:, 1:] - d[:, :-1])
        ends = self.image(x[:, None, 0] - x[None, :, -1])  # [l, j]: first bead of l from the last of j
        f[:, 0] = w2 * (d[:, 0] * self.G.sum(0)[:, None] - (self.G.T[..., None] * ends).sum(1))
        f[:, -1] += w2 * (-d[:, -1] * self.G.sum(1)[:, None] + (self.G[..., None] * ends.transpose(0, 1)).sum(1))
        return f

    def nhc_force(self, k):
        if k == 0:
            return (self.v * self.v - self.T) / self.Q
        return (self.Q * self.vt[..., k - 1] ** 2 - self.T) / self.Q

    def kick(self, h):
        e = torch.exp(-0.25 * h * self.vt[..., 0])
        self.v = self.v * e * e + 0.5 * h * self.f * e
        for k in (0, 2):
            self.th[..., k] += 0.5 * h * self.vt[..., k]

    def odd(self, h, force):
        for k, nxt in ((1, self.vt[..., 2]), (3, torch.zeros_like(self.v))):
            e = torch.exp(-0.25 * h * nxt)
            self.vt[..., k] = self.vt[..., k] * e * e + 0.5 * h * force[k] * e

    def first_half(self, h):
        force = {k: self.nhc_force(k) for k in (1, 3)}
        self.kick(h)
        self.odd(h, force)
        self.x = self.x + h * self.v
        for k in (1, 3):
            self.th[..., k] += h * self.vt[..., k]
        force = {k: self.nhc_force(k) for k in (0, 2)}
        for k in (0, 2):
            e = torch.exp(-0.5 * h * self.vt[..., k + 1])
            self.vt[..., k] = self.vt[..., k] * e * e + h * force[k] * e

    def second_half(self, h):
        self.kick(h)
        self.odd(h, {k: self.nhc_force(k) for k in (1, 3)})
        if self.box:
            self.x = torch.where(self.x < 0, self.x + self.box, torch.where(self.x > self.box, self.x - self.box, self.x))

    def estimator(self, E):
        """expectation of -E over the cycles the recursion draws"""
        return -float((self.p * torch.where(self.low, E, 0.0)).sum())

    def primitive(self):
        return np.float64(self.estimator(self.E) + self.D * self.N * self.P / (2 * self.beta))

    def virial(self):
        x, D = self.x, self.D
        # [b, i]: (x1_b - xP_i) . (x1_b - x1_i)
        t = 0.5 * self.w2 * (self.image(x[:, None, 0] - x[None, :, -1]) * self.image(x[:, None, 0] - x[None, :, 0])).sum(-1)
        c = torch.cat([torch.zeros_like(t[:1, 0]), torch.diagonal(t, 1).cumsum(0)])
        E2 = t + c[:, None] - c[None, :]
        kin = -(self.image(x[:, 1:] - x[:, :1]) * self.f[:, 1:]).sum() / 2
        return np.float64(self.estimator(E2) + D * self.N / (2 * self.beta) + float(kin))

    def read(self):
        one = torch.ones_like(self.x[..., :1])
        parts = torch.cat([one, self.x, self.v, self.f], -1).reshape(self.N * self.P, -1)
        flat = lambda a: a.reshape(-1, 4).cpu().numpy()  # noqa: E731
        return {"particles": parts.cpu().numpy(), "theta": flat(self.th), "vtheta": flat(self.vt)}


def _slices(x):
    """(bead slice range, positions (slices, N, D)) in pieces of at most 2^22 pairs"""
    N, P, _ = x.shape
    step = max(1, (1 << 22) // (N * N))
    for j in range(0, P, step):
        yield slice(j, j + step), x[:, j:j + step].transpose(0, 1)


def _plain_gauss(x, g, s, energy=False):
    """forces / P, or the mean energy, of V(r) = g / (pi s^2) exp(-r^2 / s^2)"""
    N, P, _ = x.shape
    f, e = torch.zeros_like(x), 0.0
    for at, y in _slices(x):
        d = y[:, :, None] - y[:, None]
        u = g / (math.pi * s * s) * torch.exp(-d.square().sum(-1) / (s * s))
        f[:, at] = (u[..., None] * 2 * d / (s * s)).sum(2).transpose(0, 1) / P
        e += float(u.sum() - u.diagonal(dim1=1, dim2=2).sum()) / 2 / P
    return e if energy else f


def _plain_ewald(x, box, nsum, energy=False):
    """Ewald forces / P or mean energy of unit charges: 27 boxes and the cube |n| <= nsum"""
    N, P, _ = x.shape
    a, vol = ALPHA_L / box, box ** 3
    n = torch.arange(-nsum, nsum + 1, dtype=torch.float64, device=x.device)
    nx, ny, nz = torch.meshgrid(n, n, n, indexing="ij")
    g2 = (nx * nx + ny * ny + nz * nz) / box ** 2
    g2[nsum, nsum, nsum] = 1.0
    c = torch.exp(-math.pi ** 2 * g2 / a ** 2) / g2 / (vol * math.pi)
    c[nsum, nsum, nsum] = 0.0
    m = 2 * nsum + 1
    c, k = c.reshape(-1, m), torch.stack([nx, ny, nz]).reshape(3, m * m, m)
    f, e = torch.zeros_like(x), 0.0
    eye = torch.eye(N, dtype=torch.bool, device=x.device)
    for at, y in _slices(x):
        ph = torch.exp(2j * math.pi / box * (y[..., None] * n))
        A = (ph[:, :, 0, :, None] * ph[:, :, 1, None, :]).reshape(len(y), N, -1)
        S = A.transpose(1, 2) @ ph[:, :, 2]
        d0 = y[:, :, None] - y[:, None]
        d0 = d0 - box * torch.round(d0 / box)
        if energy:
            e += (float((c * S.abs().square()).sum()) - len(y) * N * float(c.sum())) / 2 / P
            e -= len(y) * N * (N - 1) / 2 * math.pi / (a * a * vol) / P
        else:
            T = c * S.conj() * (2 * math.pi / box)
            for q in range(3):
                f[:, at, q] = ((A @ (k[q] * T)) * ph[:, :, 2]).sum(2).imag.T / P
        for i in range(27):
            d = d0 + box * torch.tensor([i // 9 - 1, i // 3 % 3 - 1, i % 3 - 1], dtype=torch.float64, device=x.device)
            r2 = d.square().sum(-1).masked_fill(eye, 1.0)
            r = r2.sqrt()
            if energy:
                e += float((torch.erfc(a * r) / r).masked_fill(eye, 0.0).sum()) / 2 / P
            else:
                w = 2 * a / math.sqrt(math.pi) * torch.exp(-a * a * r2) / r2 + torch.erfc(a * r) / (r2 * r)
                f[:, at] += (w.masked_fill(eye, 0.0)[..., None] * d).sum(2).transpose(0, 1) / P
    return e if energy else f


def _plain_pairs(case, systems, box):
    """trap and pair forces added to f"""
    x = torch.cat([s.x for s in systems])
    f = torch.zeros_like(x)
    if box:
        f += _plain_ewald(x, box, case["nsum"])
    else:
        f -= x / case["P"]
        if case["system"] == "trap":
            f += _plain_gauss(x, GAUSS_G_2D if case["D"] == 2 else GAUSS_G, GAUSS_S)
    n0 = 0
    for s in systems:
        s.f = s.spring_forces() + f[n0:n0 + s.N]
        n0 += s.N


def _exact_steps(case, seed):
    box, T = _physics(case)
    systems = [_Plain(case, box, T, inp) for inp in _inputs(case, seed)]
    for _ in range(case["steps"]):
        for s in systems:
            s.first_half(case["dt"])
            s.exchange()
        _plain_pairs(case, systems, box)
        for s in systems:
            s.second_half(case["dt"])
    # the estimator belongs to the cycle energies and probabilities of the last step's forces
    return {str(i): {"primitive": s.primitive(), **s.read()} for i, s in enumerate(systems)}


def _exact_sample(case, seed):
    box, T = _physics(case)
    s = _Plain(case, box, T, _inputs(case, seed)[0])
    s.exchange()
    _plain_pairs(case, [s], box)
    out = {}
    if box:
        out["pair"] = _plain_ewald(s.x, box, case["nsum"], energy=True)
    else:
        out["trap"] = 0.5 * float(s.x.square().sum()) / case["P"]
        out["pair"] = _plain_gauss(s.x, GAUSS_G, GAUSS_S, energy=True)
    out["primitive"], out["virial"] = s.primitive(), s.virial()
    r = s.image(s.x[:, None, 0] - s.x[None, :, 0]).square().sum(-1).sqrt()
    k = (r / (_rmax(case) / case["points"])).to(torch.int64).fill_diagonal_(case["points"])
    n = torch.bincount(k.clamp(max=case["points"]).reshape(-1), minlength=case["points"] + 1)[:case["points"]]
    out["gr"] = n.cpu().numpy() / (case["N"] * (case["N"] - 1) / 2.0)
    return {k: np.float64(v) if np.ndim(v) == 0 else v for k, v in out.items()}


def exact(case, seed):
    """None for what the network takes part in: its weights, its descriptors and its BF16 products have no 64-bit form"""
    if case["what"] == "train" or case["form"] == "learned":
        return None
    if case["what"] == "sample":
        return _exact_sample(case, seed)
    if case["what"] == "steps":
        return _exact_steps(case, seed)
    got = [_exact_steps(c, s)["0"] for c, s in _ensemble(case, seed)]
    return {k: np.concatenate([g[k] for g in got]) for k in ("particles", "theta", "vtheta")}
