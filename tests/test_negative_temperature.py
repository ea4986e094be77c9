"""A cell whose energy has turned negative (the crash test of a disk with
pebbles looks at their density alone) shows in the opacity and is left out of
the diffusion time step, as in the reference: T^(1/2) of the Bell & Lin grains
is not a number there, and no comparison with it holds."""
import numpy as np
import pytest

import harness as H
import oracle as O
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu
NR, NS = 16, 96
T2SI = 1.32712440018e20 / (8.3144598 / (2.4 * 0.001)) / 149597870700.0       # K of a code unit
UT = (149597870700.0 ** 3 / 1.32712440018e20) ** 0.5                          # s of a code unit


def _step(cells):
    """One short DT of a GPU disk and the oracle with a negative energy in the
    given cells; the solve is cut off, as no sweep converges on such a state."""
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk1", NR, NS, DT=1.0e-9)
    p.sor_maxiters = 5
    d, o = GpuDisk(p), O.OracleDisk(p)
    o.init_default()
    init = {"dens": o.get(H.FIELD_IDS["dens"]).copy(), "temper": o.get(H.FIELD_IDS["temper"]).copy()}
    d.init_default()
    for x in (d, o):
        H.start_state(x, p, init)
        e = np.array(x.get(H.FIELD_IDS["energy"]))
        for i, j in cells:
            e[i * NS + j] *= -1.0
        x.set(H.FIELD_IDS["energy"], e[:NR * NS])
        x.set_sor_state(1.0, 1e-3, 50)
    sg, so = (workloads.make_planets(p, [workloads.PLANET1]) for _ in range(2))
    d.algogas(sg)
    o.algogas(so)
    assert d.stats().substeps == 1 and o.stats().substeps == 1
    return d, o


def test_opacity_of_a_negative_temperature():
    cells = [(3, 0), (8, 40), (NR - 4, NS - 1)]
    d, o = _step(cells)
    bad = np.zeros((NR, NS), bool)
    bad[tuple(zip(*cells))] = True
    for f in ("opacity", "qminus"):
        a, b = (np.asarray(x.get(H.FIELD_IDS[f])[:NR * NS]).reshape(NR, NS) for x in (d, o))
        np.testing.assert_array_equal(np.isnan(b), bad)
        np.testing.assert_array_equal(np.isnan(a), bad, err_msg=f)
        # the tolerance of the oracle comparisons (test_gpu_parity)
        assert H.rel_l2(a[~bad], b[~bad]) < 1e-11, f
    d.close()


@pytest.mark.parametrize("factor", [-1.0, np.nan])
def test_diffusion_time_step_without_the_cells_that_are_not_numbers(factor):
    """DiffusionTimestep's minimum over the other cells, whichever ring the bad
    one lies in: dr^2 / (2 D) restated from the state (FluxLimiterValue and
    DiffusionCoefs, EnergySources.c:556-605, 684-696, 833-856).  One short
    hydro substep; what it changes of the state is of order 1e-9."""
    from fargo_thorin_gb300 import _lib
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk1", NR, NS)
    p.sor_maxiters = 5
    sig = 5.670367e-8 / 1.98855e30 * UT ** 3 * T2SI ** 4
    for i in range(NR):
        d = GpuDisk(p)
        d.init_default()
        H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
        rho, e = (np.array(d.get(H.FIELD_IDS[f])[:NR * NS]).reshape(NR, NS) for f in ("dens", "energy"))
        e[i, 37] *= factor
        d.set(H.FIELD_IDS["energy"], e)
        d.set_sor_state(1.0, 1e-3, 50)
        _lib.check(d.L.thorin_gpu_stokes(d.h), "stokes")
        _lib.check(d.L.thorin_gpu_hydro(d.h, 1.0e-9), "hydro", ok=(0, 4))
        T = e * (p.adiabind - 1.0) / rho
        rin, rout, rmed, _ = (np.asarray(a)[:, None] for a in d.rings())
        kap = np.asarray(d.get(H.FIELD_IDS["opacity"])[:NR * NS]).reshape(NR, NS)
        fac = np.sqrt(2.0 * np.pi) * np.sqrt(np.abs(T)) * rmed ** 1.5 / (rho * kap)
        gr = np.vstack([np.zeros((1, NS)), np.diff(T, axis=0) / np.diff(rmed, axis=0)])
        gt = (T - np.roll(T, 1, axis=1)) / (2.0 * np.pi / NS * rmed)
        grad = np.zeros((NR, NS))
        grad[1:-1] = np.hypot(0.5 * (gr[2:] + gr[1:-1]), 0.5 * (np.roll(gt, -1, axis=1) + gt)[1:-1])
        grad[0], grad[-1] = grad[1], grad[-2]
        s = 4.0 * grad * fac / T
        lim = np.where(s <= 2.0, 2.0 / (3.0 + np.sqrt(9.0 + 10.0 * s * s)),
                       10.0 / (10.0 * s + 9.0 + np.sqrt(np.abs(81.0 + 180.0 * s))))
        dt = 0.5 * (rout - rin) ** 2 / (lim * 16.0 * sig * T ** 3 * fac)
        assert np.isnan(dt[i, 37])
        assert abs(d.dt_stellar() / np.nanmin(dt) - 1.0) < 1e-6, i
        d.close()
