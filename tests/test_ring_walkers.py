"""The kernels that walk rings (sources, forces, diffusion, matrix, radial
transport, viscosity) take blocks of 128 columns and chunks of rings: grids at
and around those edges, remainders in both directions and the fewest rings,
against the oracle after each DT."""
import numpy as np
import pytest

import harness as H
import oracle as O
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nr,ns,over", [
    ("disk1", 33, 128, {}), ("disk1", 41, 130, {}), ("disk0", 57, 126, {}), ("disk1", 24, 258, {}),
    ("disk0", 19, 514, {}), ("disk1", 8, 64, {}), ("disk0", 6, 10, {}),
    ("disk1", 43, 254, {"OpacityTable": "ZHU12", "StellarIrradiation": "YES"}),
    ("disk0", 35, 132, {"OpacityTable": "LP85"}), ("disk0", 29, 130, {"EnergyEquation": "NO"}),
    ("disk1", 27, 384, {"LabelAdvection": "YES", "OmegaFrame": 0.5})])
def test_grids_at_the_edges_of_the_tiles(kind, nr, ns, over):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for(kind, nr, ns, **over)
    d, o = GpuDisk(p), O.OracleDisk(p)
    o.init_default()
    init = {"dens": o.get(H.FIELD_IDS["dens"]).copy(), "temper": o.get(H.FIELD_IDS["temper"]).copy()}
    d.init_default()
    for x in (d, o):
        H.start_state(x, p, init)
    row = workloads.PLANET1 if kind == "disk1" else workloads.PLANET0
    sg, so = (workloads.make_planets(p, [row]) for _ in range(2))
    n = nr * ns
    for step in range(1, 4):
        d.algogas(sg)
        o.algogas(so)
        assert d.stats().substeps == o.stats().substeps
        np.testing.assert_array_equal(d.nshift(), o.nshift())
        if p.energy_eq:
            assert d.stats().sor_last_niter == o.stats().sor_last_niter
        for f in H.GAS + (H.PEB if p.pebbles else []) + (["energy"] if p.energy_eq else []) + \
                (["label"] if p.label_advection else []):
            # the tolerance of the oracle comparisons (test_gpu_parity)
            assert H.rel_l2(d.get(H.FIELD_IDS[f])[:n], o.get(H.FIELD_IDS[f])[:n]) < 1e-11, f"{f} at DT {step}"
    d.close()


@pytest.mark.parametrize("nr,ns", [(4, 6), (6, 10), (24, 72), (97, 366), (6, 4000), (700, 40), (400, 804), (560, 1230)])
def test_solve_in_one_launch_matches_the_launched_passes(nr, ns, monkeypatch):
    """A solve is one cooperative launch; THORIN_SOR_DIRECT runs a launch per
    colour pass.  Same updates, so the same bits and sweep counts, on the host
    path and in the DT graph: fewer pairs than blocks, rings longer than a
    block's share and shorter than it, one and several rows a thread, and
    coefficients partly in shared memory (560x1230)."""
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk0", nr, ns)
    out = []
    for direct in ("0", "1"):
        monkeypatch.setenv("THORIN_SOR_DIRECT", direct)
        d = GpuDisk(p)
        d.init_default()
        H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
        d.set_sor_state(1.3, 1e-3, 50)
        s = workloads.make_planets(p, [workloads.PLANET0])
        n = []
        for k in range(3):
            (d.algogas_graph if direct == "0" and k else d.algogas)(s)
            n.append((d.stats().sor_last_niter, d.stats().substeps))
        out.append((n, [d.get(f).copy() for f in (0, 1, 2, 3, 8)]))
        d.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b)
