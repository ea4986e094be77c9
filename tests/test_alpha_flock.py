"""The temperature-dependent alpha (AlphaFlock): the initial radial velocity, the
pebbles' equilibrium and the parametric cooling's heating profile use it too,
as FViscosity does for every caller in the reference (Viscosity.c:26-54)."""
import numpy as np
import pytest

import harness as H
import oracle as O
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu
FLOCK = {"AlphaFlock": "YES", "AlphaMRI": 1e-2, "AlphaDead": 1e-3, "TMRI": 400.0}


@pytest.mark.parametrize("kind,over", [("disk0", {}), ("disk1", {}), ("disk1", {"EnergyEquation": "NO"}),
                                       ("disk0", {"CoolingTime": 10.0}), ("disk1", {"AlphaViscosity": 0.0})])
def test_alpha_flock_matches_the_oracle(kind, over):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for(kind, 32, 96, **FLOCK, **over)
    d, o = GpuDisk(p), O.OracleDisk(p)
    n = 32 * 96
    for x in (d, o):
        x.init_default()
    fields = H.GAS + (H.PEB if p.pebbles else [])
    for f in fields:
        assert H.rel_l2(d.get(H.FIELD_IDS[f])[:n], o.get(H.FIELD_IDS[f])[:n]) < 1e-13, f"initial {f}"
    init = {"dens": o.get(0).copy(), "temper": o.get(8).copy()}
    for x in (d, o):
        H.start_state(x, p, init)
    row = workloads.PLANET1 if kind == "disk1" else workloads.PLANET0
    sg, so = (workloads.make_planets(p, [row]) for _ in range(2))
    for step in range(1, 4):
        d.algogas(sg)
        o.algogas(so)
        assert d.stats().substeps == o.stats().substeps
        for f in fields:
            # the tolerance of the oracle comparisons (test_gpu_parity)
            assert H.rel_l2(d.get(H.FIELD_IDS[f])[:n], o.get(H.FIELD_IDS[f])[:n]) < 1e-11, f"{f} at DT {step}"
    d.close()
