"""The schedule tuner times only launch shapes that change a launch.

CPU: which candidates it runs, with disks that stand in for the GPU's.  GPU: a
disk's launches by shape, and a DT graph that holds no sweeps outliving a
change of the shape."""
import ctypes as C

import pytest

from fargo_thorin_gb300 import _lib
from fargo_thorin_gb300.ensemble import Ensemble


class _Disk:
    def __init__(self, nr, one):
        self.nr, self.one = nr, one

    def sweep_launches(self, sweeps, threads):
        return None if self.one else (sweeps, min(threads, 1024) // 256 * 152)


def _ensemble(disks, ms):
    ens = Ensemble.__new__(Ensemble)
    ens.disks = disks
    ens.restore = lambda snaps: None
    ens.run_schedule = lambda sched, ndt=1: {"seconds": 1e-3 * ms(sched)}
    return ens


def test_sizes_solved_in_one_launch_try_no_shapes():
    ens = _ensemble([_Disk(128, True), _Disk(256, True)], lambda s: 5.0 if s["mode"] == "graph" else 6.0)
    r = ens.tune_schedule([], pool_workers=(2, 4))
    assert [t["schedule"]["mode"] for t in r["trials"]] == ["graph", "pool", "pool"]
    assert r["schedule"] == {"mode": "graph", "shapes": {}} and r["ms_per_dt"] == 5.0


def test_shapes_with_the_same_launches_are_tried_once():
    def ms(s):
        return 5.0 - sum(0.5 for k in s["shapes"].values() if k[0] == 16)
    ens = _ensemble([_Disk(128, True), _Disk(1200, False)], ms)
    r = ens.tune_schedule([], pool_workers=(2,))
    # of the default shapes only 16 sweeps differ from 8: 1024 threads are the most a pass holds
    assert [t["shapes"] for t in r["trials"]] == [{}, {}, {"1200": [16, 1536]}]
    assert r["schedule"]["shapes"] == {1200: (16, 1536)} and r["ms_per_dt"] < 5.0
    r = ens.tune_schedule([], shapes=((8, 1536), (8, 512), (8, 640), (4, 2048)), pool_workers=())
    assert [t["shapes"] for t in r["trials"]] == [{}, {"1200": [8, 512]}, {"1200": [4, 2048]}]


def test_arguments():
    n = C.c_int()
    assert _lib.load().thorin_gpu_sweep_blocks(None, 1024, C.byref(n)) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("passes", [False, True])
def test_launch_shape_and_the_graphs(monkeypatch, passes):
    import harness as H
    from fargo_thorin_gb300 import workloads
    from fargo_thorin_gb300.disk import GpuDisk
    monkeypatch.setenv("THORIN_SOR_PASSES", "1" if passes else "0")
    p = workloads.params_for("disk0", 200, 2400)
    d = GpuDisk(p)
    d.init_default()
    H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
    d.set_sor_state(1.3, 1e-3, 50)
    s = workloads.make_planets(p, [workloads.PLANET0])
    a, b = C.c_int(), C.c_int()
    for shape in ((8, 1536), (16, 1024), (8, 512)):
        d.set_launch_shape(*shape)
        d.algogas_graph(s)
        _lib.check(d.L.thorin_selftest_graph_builds(d.h, C.byref(a), C.byref(b)), "graph_builds")
    assert (a.value, b.value) == ((3, 0) if passes else (1, 0))
    k = d.sweep_launches(8, 512)
    if passes:                                            # 928 blocks of 256 cells a colour
        sms = k[1] // 2
        assert k == (8, 2 * sms) and d.sweep_launches(4, 2048) == d.sweep_launches(4, 1024) == (4, 4 * sms)
        assert d.sweep_launches(8, 128) == (8, sms)
    else:
        assert k is None
    assert d.L.thorin_gpu_sweep_blocks(d.h, 100, C.byref(a)) == 1
    d.close()
