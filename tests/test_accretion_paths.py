"""Pebble accretion in three launches: spheres of no cell, one cell and many,
inclined orbits (a column not symmetric about the midplane), planets at both
edges of the grid (no second ring for the flow's mean outside), several
planets and none inside, against the oracle after each DT."""
import numpy as np
import pytest

import harness as H
import oracle as O
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu
EARTH = 3.0e-6


@pytest.mark.parametrize("nr,ns,rows", [
    (24, 72, [(1e-4 * EARTH, 1.03, 0.0)]), (24, 72, [(20 * EARTH, 1.03, 0.0)]), (48, 144, [(300 * EARTH, 0.9, 0.0)]),
    (48, 144, [(20 * EARTH, 1.1, 1.5)]), (33, 130, [(5 * EARTH, 0.81, 0.0), (60 * EARTH, 1.26, 3.0)]),
    (40, 120, [(20 * EARTH, None, 0.0)]), (64, 1030, [(100 * EARTH, 1.0, 0.4)])])
def test_accretion_matches_the_oracle(nr, ns, rows):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk1", nr, ns)
    d, o = GpuDisk(p), O.OracleDisk(p)
    o.init_default()
    init = {"dens": o.get(H.FIELD_IDS["dens"]).copy(), "temper": o.get(H.FIELD_IDS["temper"]).copy()}
    d.init_default()
    for x in (d, o):
        H.start_state(x, p, init)
    rsup = np.asarray(d.rings()[1])
    systems = []
    for _ in range(2):
        s = workloads.make_planets(p, [tuple([m] + list(workloads.PLANET1)[1:]) for m, _, _ in rows])
        for k, (m, a, inc) in enumerate(rows):
            a = a if a is not None else float(rsup[nr - 1]) * 0.9995        # the last ring
            el = workloads.planet_from_elements(m, 0.0, 0.0, a, 0.01, inc, 20.0, 10.0, 40.0 + 100.0 * k)
            for key, v in el.items():
                getattr(s, key)[k] = v
        systems.append(s)
    sg, so = systems
    n = nr * ns
    for step in range(1, 4):
        d.algogas(sg)
        o.algogas(so)
        assert d.stats().substeps == o.stats().substeps
        for f in H.GAS + H.PEB:
            # the tolerance of the oracle comparisons (test_gpu_parity)
            assert H.rel_l2(d.get(H.FIELD_IDS[f])[:n], o.get(H.FIELD_IDS[f])[:n]) < 1e-11, f"{f} at DT {step}"
        for k in range(sg.nb):
            assert abs(sg.mass[k] - so.mass[k]) <= 1e-11 * so.mass[k], f"mass of planet {k} at DT {step}"
            assert abs(sg.solid[k] - so.solid[k]) <= 1e-9 * so.mass[k], f"accreted mass of planet {k} at DT {step}"
    d.close()
