"""The device's N-body step (two warps, a lane per body and component) against
the host's, for every number of lanes in use: one to eight planets, eccentric
and inclined, through DTs of the graph and the host path."""
import ctypes as C

import numpy as np
import pytest

import harness as H
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npl", [1, 2, 3, 5, 8])
def test_planets_of_the_graph_match_the_host(npl):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk0", 24, 72)
    out = []
    for graph in (False, True):
        d = GpuDisk(p)
        d.init_default()
        H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
        d.set_sor_state(1.3, 1e-3, 50)
        s = workloads.make_planets(p, [workloads.PLANET0] * npl)
        for k in range(npl):
            el = workloads.planet_from_elements(1e-4 / (k + 1), 0.0, 0.0, 0.5 + 0.21 * k, 0.05 * (k % 3), 2.0 * k,
                                                15.0 * k, 10.0, 77.0 * k)
            for key, v in el.items():
                getattr(s, key)[k] = v
        d.algogas(s)
        for _ in range(2):
            (d.algogas_graph if graph else d.algogas)(s)
        out.append([(s.x[k], s.y[k], s.z[k], s.vx[k], s.vy[k], s.vz[k]) for k in range(npl)])
        d.close()
    # the N-body steps are the same operations; pow and atan2 of the planet
    # side differ between device and host (1e-13, as in test_graph_dt)
    np.testing.assert_allclose(np.array(out[1]), np.array(out[0]), rtol=0, atol=1e-13)
