"""A cell whose energy has turned negative (the crash test of a disk with
pebbles looks at their density alone) shows in the opacity, as in the reference: T^(1/2) of the
Bell & Lin grains is not a number there."""
import numpy as np
import pytest

import harness as H
import oracle as O
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu
NR, NS = 16, 96


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
