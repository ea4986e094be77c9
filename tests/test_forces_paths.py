"""The force kernels' branches against the oracle: no planet, one planet per
template of k_forces (1, 2, 3) and the generic one, inclined planets (nodes on
both sides of the midplane), light planets next to the thin disk's scale height
and heavy ones whose Hill sphere holds 30-node and tapered cells, thin and thick
columns (the star's series and its node-by-node sum)."""
import numpy as np
import pytest

import harness as H
import oracle as O
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu

ROWS = [(1.0e-4, 0., 0., 1.00, 0.00, 0.0, 0., 0., 20.), (3.0e-5, 0., 0., 0.70, 0.02, 0.4, 30., 10., 200.),
        (1.0e-3, 0., 0., 1.60, 0.01, 3.0, 60., 0., 100.), (1.0e-6, 0., 0., 0.55, 0.05, 0.0, 0., 0., 300.),
        (5.0e-5, 0., 0., 2.10, 0.00, 1.0, 10., 5., 150.)]


@pytest.mark.parametrize("kind,rows,aspect", [("disk0", [], 0.05), ("disk0", [0], 0.05), ("disk1", [0], 0.10),
                                              ("disk1", [0, 1], 0.05), ("disk1", [2], 0.05), ("disk1", [0, 2, 3], 0.05),
                                              ("disk1", [0, 1, 2, 3, 4], 0.06), ("disk0", [1, 2, 3, 4], 0.03)])
def test_forces_match_the_oracle(kind, rows, aspect):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for(kind, 48, 200, AspectRatio=aspect, PlanetsFeelDisk="YES")
    d, o = GpuDisk(p), O.OracleDisk(p)
    o.init_default()
    init = {"dens": o.get(H.FIELD_IDS["dens"]).copy(), "temper": o.get(H.FIELD_IDS["temper"]).copy()}
    d.init_default()
    for x in (d, o):
        H.start_state(x, p, init)
        x.set_time(1.0)                               # the mass taper is over
    sg, so = (workloads.make_planets(p, [ROWS[k] for k in rows]) for _ in range(2))
    n = p.nrad * p.nsec
    for step in range(1, 3):
        d.algogas(sg)
        o.algogas(so)
        assert d.stats().substeps == o.stats().substeps
        for f in H.GAS + (H.PEB if p.pebbles else []):
            # the tolerance of the oracle comparisons (test_gpu_parity)
            assert H.rel_l2(d.get(H.FIELD_IDS[f])[:n], o.get(H.FIELD_IDS[f])[:n]) < 1e-11, f"{f} at DT {step}"
        for k in range(len(rows)):
            a = np.hypot(so.ax[k], so.ay[k])
            assert np.hypot(sg.ax[k] - so.ax[k], sg.ay[k] - so.ay[k]) <= 1e-9 * a
            assert abs(sg.x[k] - so.x[k]) < 1e-13 and abs(sg.vy[k] - so.vy[k]) < 1e-13
    d.close()
