"""A disk advanced as a DT graph alone and beside other disks keeps one graph
for each: neither call runs the solve's launch shape of the other, neither
rebuilds the other's graph, and the state goes from one to the other and the
host path bit for bit."""
import ctypes as C

import numpy as np
import pytest

from fargo_thorin_gb300 import _lib

FIELDS = (0, 1, 2, 3, 4, 5, 6, 8)
SPECS = [{"nrad": 48, "alpha": 1e-3, "sigma_scale": 1.0, "aspect": 0.05, "mplanet": 3e-5},
         {"nrad": 32, "alpha": 3e-4, "sigma_scale": 2.0, "aspect": 0.04, "mplanet": 1e-5}]


def test_arguments():
    n = C.c_int()
    assert _lib.load().thorin_selftest_graph_builds(None, C.byref(n), C.byref(n)) == 1


def _builds(d):
    a, b = C.c_int(), C.c_int()
    _lib.check(d.L.thorin_selftest_graph_builds(d.h, C.byref(a), C.byref(b)), "graph_builds")
    return a.value, b.value


@pytest.mark.gpu
@pytest.mark.parametrize("first", ["alone", "beside"])
def test_one_graph_alone_and_one_beside_others(first):
    from fargo_thorin_gb300.ensemble import Ensemble
    ens, ref = Ensemble(SPECS, seed=3), Ensemble(SPECS[:1], seed=3)
    d, s = ens.disks[0], ens.systems[0]
    r, rs = ref.disks[0], ref.systems[0]
    ens.step(1)                                           # DT 1 calibrates omega on the host path
    r.algogas(rs)
    order = ["alone", "beside", "host", "beside", "alone", "alone", "host", "alone", "beside"]
    if first == "beside":
        order = order[1:2] + order
    seen = set()
    for how in order:
        if how == "alone":
            d.algogas_graph(s)
        elif how == "beside":
            assert ens.step_graph() == [0, 0]
        else:
            d.algogas(s)
        seen.add(how)
        r.algogas_graph(rs)
        assert _builds(d) == (int("alone" in seen), int("beside" in seen)), order
        assert d.stats().sor_sweeps == r.stats().sor_sweeps and d.stats().substeps == r.stats().substeps
    # the host path's DTs agree with the graph's to rounding (test_graph_dt)
    for f in FIELDS:
        a, b = d.get(f), r.get(f)
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b), f
    ens.close()
    ref.close()


@pytest.mark.gpu
def test_graphs_alone_and_beside_give_the_same_bits():
    from fargo_thorin_gb300.ensemble import Ensemble
    out = []
    for how in ((0, 0, 0, 0), (1, 1, 1, 1), (0, 1, 0, 1), (1, 0, 0, 1)):
        ens = Ensemble(SPECS, seed=4)
        ens.step(1)
        for beside in how:
            if beside:
                assert ens.step_graph() == [0, 0]
            else:
                for d, s in zip(ens.disks, ens.systems):
                    d.algogas_graph(s)
        out.append([d.get(f) for d in ens.disks for f in FIELDS])
        ens.close()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
