"""The measured cases: what users of this framework have it do.

A user advances disks DT by DT (one DT = one AlgoGas call with all its CFL
substeps), from the smallest test disks, where launches and host round trips
count, through the 128x384 gas disk and the 1024x3072 pebble + embryo disk to
2048x6144; on the host path (``algogas``), as one CUDA graph per DT
(``algogas_graph``), in ensembles of uneven disks, and with the two SOR warm
starts.  One pass takes a disk's state from pinned host arrays (as the C
boundary has it: PolarGrid arrays of the caller), advances one DT and brings
the new state back, so every pass does the same substeps and SOR sweeps.  The
conservation integrals (the reference's -a option) are a call of their own.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from fargo_thorin_gb300 import _lib, workloads
from fargo_thorin_gb300 import warmstart as WS
from fargo_thorin_gb300.disk import GpuDisk
from fargo_thorin_gb300.ensemble import Ensemble

DT = 0.0314159265358979                     # the workloads' DT, 1/200 of an orbit at r = 1
RMIN, RMAX = 0.4, 2.5
GAS = {"dens": 0, "vrad": 1, "vtheta": 2, "energy": 3, "temper": 8}
PEBBLES = {"pebdens": 4, "pebvrad": 5, "pebvtheta": 6}
SOUNDSPEED = 9                              # part of the state a DT starts from
NETWORK = "fargo_thorin_gb300/warmnet_disk1_1024x3072.npy"
ENSEMBLE_SIZES = (128, 192, 256, 384)       # rings; the drawn ensembles' sizes below 512


def listed():
    return [
        # a test-sized gas disk: launches, synchronisations and the graph's restarts
        {"name": "gas_24x72", "kind": "disk0", "nrad": 24, "nsec": 72, "mode": "host", "start": "plain", "eps": 1e-6},
        # the default gas disk of the plain method (reference's SOR tolerance)
        {"name": "gas_128x384", "kind": "disk0", "nrad": 128, "nsec": 384, "mode": "host", "start": "plain",
         "eps": 1e-6},
        # an isothermal disk (the reference's default: no energy equation, no SOR)
        {"name": "isothermal_256x768", "kind": "disk0", "nrad": 256, "nsec": 768, "mode": "host", "start": "plain",
         "eps": 1e-6, "isothermal": True},
        # a disk of the ensembles' sizes, alone, as one graph per DT
        {"name": "pebbles_192x576_graph", "kind": "disk1", "nrad": 192, "nsec": 576, "mode": "graph",
         "start": "plain", "eps": 1e-8},
        # a grid that is no multiple of anything the kernels tile by
        {"name": "pebbles_333x1002", "kind": "disk1", "nrad": 333, "nsec": 1002, "mode": "host", "start": "plain",
         "eps": 1e-8},
        # Zhu et al. opacities with stellar irradiation, the settings of the shipped relaxation runs
        {"name": "irradiated_384x1152", "kind": "disk1", "nrad": 384, "nsec": 1152, "mode": "host", "start": "plain",
         "eps": 1e-8, "opacity": "ZHU12", "irradiation": True},
        # the learned SOR start (the network inside the DT graph)
        {"name": "learned_512x1536_graph", "kind": "disk1", "nrad": 512, "nsec": 1536, "mode": "graph",
         "start": "learned", "eps": 1e-8},
        # the measured workload: the large pebble + embryo disk
        {"name": "pebbles_1024x3072", "kind": "disk1", "nrad": 1024, "nsec": 3072, "mode": "host", "start": "plain",
         "eps": 1e-8},
        # the same disk as production runs advance it: one graph per DT, extrapolated SOR start
        {"name": "extrapolated_1024x3072_graph", "kind": "disk1", "nrad": 1024, "nsec": 3072, "mode": "graph",
         "start": "extrapolated", "eps": 1e-8},
        # the largest grid of the combined workload, a quarter of its DT
        {"name": "pebbles_2048x6144", "kind": "disk1", "nrad": 2048, "nsec": 6144, "mode": "host", "start": "plain",
         "eps": 1e-8, "dt_fraction": 0.25},
        # an ensemble of uneven disks, all DT graphs launched together
        {"name": "ensemble_8_disks", "mode": "ensemble", "disks": 8, "eps": 1e-8},
        # the conservation integrals of a large disk
        {"name": "integrals_1024x3072", "mode": "integrals", "nrad": 1024, "nsec": 3072},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.08:
        return {"mode": "ensemble", "disks": rng.randint(2, 8), "eps": 1e-8}
    nrad = _log_int(rng, 24, 1200)
    nsec = 2 * int(round(nrad * rng.uniform(2.6, 3.4) / 2))      # red-black SOR wants an even count
    if pick < 0.16:
        return {"mode": "integrals", "nrad": nrad, "nsec": nsec}
    case = {"kind": rng.choice(["disk0", "disk1", "disk1"]), "nrad": nrad, "nsec": nsec,
            "mode": rng.choice(["host", "graph"]), "start": rng.choice(["plain", "plain", "extrapolated"]),
            "eps": rng.choice([1e-6, 1e-8])}
    if case["kind"] == "disk0" and case["mode"] == "host" and rng.random() < 0.4:
        case.update(isothermal=True, start="plain")
    elif rng.random() < 0.2:
        case.update(opacity="ZHU12", irradiation=True)
    if case["kind"] == "disk1":
        case["planet_mass"] = rng.choice([1.0e-6, 1.0e-5, 3.0e-5, 6.0e-5])
    return case


def _omega(nrad):
    """About the SOR parameter that the calibration of a disk's first solve
    settles on (1.00 at 24 rings, 1.31 at 128, 1.64 at 512, 1.77 at 1024); a
    program that restarts a disk hands its schedule over in the same way."""
    return max(1.001, 2.0 - 7.7 / math.sqrt(nrad))


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _params(case):
    over = {}
    if case.get("opacity"):
        over["OpacityTable"] = case["opacity"]
    if case.get("irradiation"):
        over["StellarIrradiation"] = "YES"
    if case.get("isothermal"):
        over["EnergyEquation"] = "NO"
    if case.get("dt_fraction"):
        over["DT"] = DT * case["dt_fraction"]
    return workloads.params_for(case["kind"], case["nrad"], case["nsec"], sor_eps=case["eps"], **over)


class _Run:
    """A disk, its planets and the host copy of the state each pass starts from."""

    def __init__(self, disk, params, system, warm=None):
        self.disk, self.system, self.warm = disk, system, warm
        self.outputs = {k: f for k, f in GAS.items() if params.energy_eq or k != "energy"}
        if params.pebbles:
            self.outputs.update(PEBBLES)
        self.isothermal = not params.energy_eq
        self.cells = params.nrad * params.nsec
        self.shape = (params.nrad, params.nsec)

    def keep(self):
        """The state now on the device becomes the start of every pass."""
        n = self.cells + self.shape[1]
        self.up = {}
        for f in list(self.outputs.values()) + [SOUNDSPEED]:
            self.up[f] = _pinned(n)
            self._copy(self.disk.L.thorin_gpu_download, f, self.up[f])
        self.out = {k: _pinned(n) for k in self.outputs}
        self.start = self.system.copy()
        self.sor, self.time = self.disk.sor_state()[:3], self.disk.stats().physical_time
        self.dt_stellar = self.disk.dt_stellar()

    def _copy(self, call, field, array):
        _lib.check(call(self.disk.h, field, array.ctypes.data_as(C.POINTER(C.c_double))), "copy of a field")

    def upload(self):
        d = self.disk
        for f, a in self.up.items():
            self._copy(d.L.thorin_gpu_upload, f, a)
        if not self.isothermal:
            d.set_sor_state(*self.sor)
        d.set_time(self.time)
        d.set_dt_stellar(self.dt_stellar)
        d.refresh(4)                                  # the ring means of c_s
        if self.warm is not None:
            WS.attach(d, *self.warm)                  # without the updates recorded after this state
        C.memmove(C.byref(self.system), C.byref(self.start), C.sizeof(self.start))

    def download(self):
        d, s = self.disk, self.system
        for k, f in self.outputs.items():
            self._copy(d.L.thorin_gpu_download, f, self.out[k])
        r = {k: a[:self.cells].reshape(self.shape) for k, a in self.out.items()}
        r["planet"] = np.array([s.x[0], s.y[0], s.vx[0], s.vy[0], s.mass[0]])
        r["substeps"] = d.stats().substeps
        if not self.isothermal:
            r["sor_omega"], _, r["sor_sweeps"], _ = d.sor_state()
        return r


def _start(disk, params, seed):
    """The measured initial state: Sigma perturbed by 1e-4 u, v_r = 0."""
    disk.init_default()
    st = workloads.perturbed_state(params, {"dens": disk.get(0), "temper": disk.get(8)}, seed=seed)
    disk.set(0, st["dens"])
    disk.set(1, st["vrad"])
    if params.energy_eq:
        disk.set(3, st["energy"])
    if params.pebbles:
        disk.set(4, st["pebdens"])
        disk.set(7, st["pebsize"])
    disk.refresh(2 if params.pebbles else 1)


def _prepare_dt(case, seed):
    p = _params(case)
    d = GpuDisk(p)
    _start(d, p, seed)
    planet = list(workloads.PLANET1 if case["kind"] == "disk1" else workloads.PLANET0)
    if case.get("planet_mass"):
        planet[0] = case["planet_mass"]
    system = workloads.make_planets(p, [tuple(planet)])
    if p.energy_eq:
        d.set_sor_state(_omega(case["nrad"]), 4.9e-4, 50)
    warm = None
    if case["start"] == "extrapolated":
        warm = (None, WS.EXTRAPOLATE)
    elif case["start"] == "learned":
        warm = (WS.WarmNet(case["nrad"], case["nsec"], params=WS.WarmNet.load_params(NETWORK)), WS.PREDICT)
    if warm is not None:
        WS.attach(d, *warm)
    r = _Run(d, p, system, warm)
    step = d.algogas_graph if case["mode"] == "graph" else d.algogas
    for _ in range(1 if case.get("dt_fraction") else 2):      # past the first DT, whose steps are shorter
        step(system)
    r.keep()
    r.step = step
    return r


def _prepare_ensemble(case, seed):
    rng = np.random.default_rng(seed)
    specs = []
    for k in range(case["disks"]):
        specs.append({"nrad": ENSEMBLE_SIZES[k % len(ENSEMBLE_SIZES)], "alpha": 1e-3, "aspect": 0.05,
                      "sigma_scale": float(rng.uniform(0.8, 1.2)), "mplanet": float(rng.uniform(1e-6, 6e-5))})
    ens = Ensemble(specs, seed=seed)
    for d in ens.disks:
        d.set_sor_state(_omega(d.nr), 4.9e-4, 50)
    runs = [_Run(d, p, s) for d, p, s in zip(ens.disks, ens.params, ens.systems)]
    ens.step_graph()
    ens.step_graph()
    for r in runs:
        r.keep()
    return {"ensemble": ens, "runs": runs}


def _fields(case, seed):
    """Gas and pebble fields of a disk with a spiral perturbation."""
    nr, ns = case["nrad"], case["nsec"]
    g = np.random.default_rng(seed)
    r = RMIN * (RMAX / RMIN) ** ((np.arange(nr) + 0.5) / nr)
    u = g.uniform(-1.0, 1.0, (5, nr, ns))
    dens = 5e-4 * r[:, None] ** -0.5 * (1.0 + 0.05 * u[0])
    return {0: dens, 1: 1e-3 * u[1], 2: r[:, None] ** -0.5 * (1.0 + 1e-3 * u[2]),
            3: dens * 2.5e-3 / r[:, None] / 0.4 * (1.0 + 0.02 * u[3]),
            4: 0.01 * dens * (1.0 + 0.1 * u[4]), 6: r[:, None] ** -0.5 * (1.0 + 1e-3 * u[1])}


def _prepare_integrals(case, seed):
    d = GpuDisk(workloads.params_for("disk1", case["nrad"], case["nsec"]))
    for f, a in _fields(case, seed).items():
        d.set(f, a)
    return d


def prepare(case, seed):
    if case["mode"] == "ensemble":
        return _prepare_ensemble(case, seed)
    if case["mode"] == "integrals":
        return _prepare_integrals(case, seed)
    return _prepare_dt(case, seed)


def run(state):
    if isinstance(state, GpuDisk):
        return np.array(state.integrals())
    if isinstance(state, dict):
        for r in state["runs"]:
            r.upload()
        state["ensemble"].step_graph()
        # every disk's gas, its pebble density and its planet
        keep = tuple(GAS) + ("pebdens", "planet")
        return [{k: v for k, v in r.download().items() if k in keep} for r in state["runs"]]
    state.upload()
    state.step(state.system)
    return state.download()


def _exact_integrals(case, seed):
    f = _fields(case, seed)
    nr, ns = case["nrad"], case["nsec"]
    edge = RMIN * np.exp(np.arange(nr + 1) / nr * math.log(RMAX / RMIN))
    rin, rout = edge[:-1, None], edge[1:, None]
    rmed = 2.0 / 3.0 * (rout ** 3 - rin ** 3) / (rout ** 2 - rin ** 2)
    surf = math.pi * (rout ** 2 - rin ** 2) / ns
    dens, vr, vt, e = f[0], np.vstack([f[1], np.zeros((1, ns))]), f[2], f[3]

    def momentum(rho, v):
        return float(0.5 * np.sum(surf * (rho + np.roll(rho, 1, axis=1)) * rmed * v))

    vrc = ((rmed - rin) * vr[1:] + (rout - rmed) * vr[:-1]) / (rout - rin)
    vtc = 0.5 * (vt + np.roll(vt, -1, axis=1))
    energy = float(np.sum(0.5 * surf * dens * (vrc ** 2 + vtc ** 2) + surf * e))
    return np.array([float(np.sum(surf * dens)), momentum(dens, vt), energy, float(np.sum(surf * f[4])),
                     momentum(f[4], f[6])])


def exact(case, seed):
    """The integrals as numpy sums.  A DT has no such value: it is FP64
    throughout, and a restatement of the scheme in FP64 rounds no better."""
    return _exact_integrals(case, seed) if case["mode"] == "integrals" else None


def _dt_work(nrad, nsec, pebbles, energy, dt_fraction=1.0):
    """Bytes and operations of one DT: the state in and out, per CFL substep
    the gas and pebble state (64 and 56 bytes a cell) and per SOR sweep the
    temperature, five coefficients and the right-hand side (64 bytes, 14
    operations).  Substeps and sweeps are those of the settled disks: nrad /
    128 substeps of a whole DT, 1.2 sqrt(nrad) + 8 sweeps a solve."""
    cells = nrad * nsec
    substeps = max(1.0, nrad / 128.0 * dt_fraction)
    sweeps = (1.2 * math.sqrt(nrad) + 8.0) if energy else 0.0
    state = 64.0 + (56.0 if pebbles else 0.0)
    per_cell = 400.0 + (250.0 if pebbles else 0.0) + (150.0 if energy else 0.0)
    return {"bytes": cells * (substeps * (state + 64.0 * sweeps) + 2.0 * state),
            "flops": cells * substeps * (per_cell + 14.0 * sweeps)}


def work(case):
    if case["mode"] == "integrals":
        cells = case["nrad"] * case["nsec"]
        return {"bytes": 48.0 * cells, "flops": 30.0 * cells}
    if case["mode"] == "ensemble":
        w = [_dt_work(n, 3 * n, True, True)
             for n in (ENSEMBLE_SIZES[k % len(ENSEMBLE_SIZES)] for k in range(case["disks"]))]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    return _dt_work(case["nrad"], case["nsec"], case["kind"] == "disk1", not case.get("isothermal"),
                    case.get("dt_fraction", 1.0))
