"""The Zhu et al. opacity (its T^1.5 regimes without logarithms) and the stellar
irradiation against the oracle: temperatures swept across the regimes and
finely across the thresholds that FP32 logarithms decide, over one DT."""
import numpy as np
import pytest

import harness as H
import oracle as O
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu
T2SI = 1.32712440018e20 / (8.3144598 / (2.4 * 0.001)) / 149597870700.0       # K of a code unit


@pytest.mark.parametrize("lo,hi,irr", [(60.0, 130.0, "YES"), (120.0, 175.0, "YES"), (150.0, 170.0, "NO"),
                                       (560.0, 720.0, "YES"), (620.0, 640.0, "YES"), (1400.0, 1900.0, "NO")])
def test_zhu_opacity_across_its_regimes(lo, hi, irr):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk0", 24, 96, OpacityTable="ZHU12", StellarIrradiation=irr)
    d, o = GpuDisk(p), O.OracleDisk(p)
    nr, ns = p.nrad, p.nsec
    n = nr * ns
    o.init_default()
    init = {"dens": o.get(H.FIELD_IDS["dens"]).copy(), "temper": o.get(H.FIELD_IDS["temper"]).copy()}
    d.init_default()
    i, j = np.meshgrid(np.arange(nr), np.arange(ns), indexing="ij")
    kelvin = lo + (hi - lo) * (0.5 + 0.45 * np.sin(2 * np.pi * (j / ns + 0.31 * i / nr)) + 0.05 * i / nr)
    for x in (d, o):
        H.start_state(x, p, init)
        dens = np.asarray(x.get(H.FIELD_IDS["dens"]))[:n].reshape(nr, ns)
        x.set(H.FIELD_IDS["energy"], dens * kelvin / T2SI / (p.adiabind - 1.0))
        x.refresh(1)
    sg, so = (workloads.make_planets(p, [workloads.PLANET0]) for _ in range(2))
    d.algogas(sg)
    o.algogas(so)
    assert d.stats().substeps == o.stats().substeps
    for f in ("opacity", "qminus", "temper", "dens"):
        # the tolerance of the oracle comparisons (test_gpu_parity)
        assert H.rel_l2(d.get(H.FIELD_IDS[f])[:n], o.get(H.FIELD_IDS[f])[:n]) < 1e-11, f
    d.close()
