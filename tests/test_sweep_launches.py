"""Sweeps as launches inside WHILE nodes (disks above 2.4 million cells, and any
disk with THORIN_SOR_PASSES=1): the sweep loop of the host path, the sweep loop
inside the substep loop of a DT graph, and the launch shapes, bit for bit
against plain launches of the passes (THORIN_SOR_DIRECT) and the solve in one
launch."""
import numpy as np
import pytest

import harness as H
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu
GAS, PEB = (0, 1, 2, 3, 8), (4, 5, 6)


def _run(monkeypatch, p, kind, form, dts, graph, shape=None):
    from fargo_thorin_gb300.disk import GpuDisk
    monkeypatch.setenv("THORIN_SOR_PASSES", "1" if form == "passes" else "0")
    monkeypatch.setenv("THORIN_SOR_DIRECT", "1" if form == "direct" else "0")
    d = GpuDisk(p)
    d.init_default()
    H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
    d.set_sor_state(1.3, 1e-3, 50)
    if shape is not None:
        d.set_launch_shape(*shape)
        assert d.launch_shape() == shape
    s = workloads.make_planets(p, [workloads.PLANET1 if kind == "disk1" else workloads.PLANET0])
    counts = []
    for k in range(dts):
        (d.algogas_graph if graph else d.algogas)(s)
        st = d.stats()
        counts.append((st.substeps, st.sor_sweeps, st.sor_last_niter))
    out = [d.get(f).copy() for f in GAS + (PEB if p.pebbles else ())]
    if not graph:
        out.append(np.array([s.x[0], s.y[0], s.vx[0], s.vy[0]]))
    d.close()
    return counts, out


def _same(a, b):
    assert a[0] == b[0]
    for x, y in zip(a[1], b[1]):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("kind,nr,ns", [("disk0", 4, 6), ("disk0", 24, 72), ("disk1", 33, 130), ("disk1", 97, 366)])
def test_sweep_loops_match_the_launched_passes(monkeypatch, kind, nr, ns):
    p = workloads.params_for(kind, nr, ns)
    direct = _run(monkeypatch, p, kind, "direct", 3, False)
    _same(direct, _run(monkeypatch, p, kind, "passes", 3, False))
    _same(direct, _run(monkeypatch, p, kind, "one", 3, False))
    # DT graphs: the planets' transcendental functions are the device's, so
    # the two forms are compared with one another
    _same(_run(monkeypatch, p, kind, "passes", 3, True), _run(monkeypatch, p, kind, "one", 3, True))


def test_launch_shapes_of_launched_sweeps(monkeypatch):
    p = workloads.params_for("disk1", 64, 600)
    for graph in (False, True):
        ref = _run(monkeypatch, p, "disk1", "one", 3, graph)
        for shape in ((8, 1536), (4, 256), (1, 512), (16, 2048), (64, 1024)):
            _same(ref, _run(monkeypatch, p, "disk1", "passes", 3, graph, shape))


@pytest.mark.parametrize("nr", [896, 898])
def test_solves_on_either_side_of_the_cell_limit(monkeypatch, nr):
    """894 and 896 rings of 2684 unknowns: 2,399,496 cells are solved in one
    launch, 2,404,864 by launched sweeps."""
    p = workloads.params_for("disk0", nr, 2684, DT=0.004)
    direct = _run(monkeypatch, p, "disk0", "direct", 2, False)
    _same(direct, _run(monkeypatch, p, "disk0", "one", 2, False))
    _same(_run(monkeypatch, p, "disk0", "passes", 2, True), _run(monkeypatch, p, "disk0", "one", 2, True))
