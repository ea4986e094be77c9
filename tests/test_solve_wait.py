"""A wait of the solve in one launch that runs out: the blocks give up, the
caller gets an error, and the disk goes on from a state put back.  With a
limit of one load the first value that a neighbouring block has not yet
posted is waited for in vain."""
import ctypes as C

import numpy as np
import pytest

import harness as H
from fargo_thorin_gb300 import _lib, workloads

FIELDS = (0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 11)
TIMEOUT = 5


def test_arguments():
    assert _lib.load().thorin_selftest_solve_wait(None, 1) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("nr,ns", [(24, 72), (128, 384), (333, 1002)])
def test_wait_that_runs_out_is_an_error(nr, ns, graph):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk1", nr, ns)
    d = GpuDisk(p)
    d.init_default()
    H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
    d.set_sor_state(1.3, 1e-3, 50)
    s = workloads.make_planets(p, [workloads.PLANET1])
    step = d.algogas_graph if graph else d.algogas
    step(s)
    snap, s0 = d.snapshot(FIELDS), s.copy()
    step(s)
    want = [d.get(f) for f in FIELDS] + [np.array([s.x[0], s.vy[0], s.mass[0]]), np.array(d.sor_state()[:3])]
    for _ in range(2):
        d.restore(snap)
        C.memmove(C.byref(s), C.byref(s0), C.sizeof(s))
        _lib.check(d.L.thorin_selftest_solve_wait(d.h, 1), "solve_wait")
        with pytest.raises(_lib.ThorinError, match="a wait of the SOR solve ran out") as e:
            step(s)
        assert e.value.code == TIMEOUT
        _lib.check(d.L.thorin_selftest_solve_wait(d.h, 0), "solve_wait")
        d.restore(snap)
        C.memmove(C.byref(s), C.byref(s0), C.sizeof(s))
        step(s)
        got = [d.get(f) for f in FIELDS] + [np.array([s.x[0], s.vy[0], s.mass[0]]), np.array(d.sor_state()[:3])]
        for a, b in zip(want, got):
            np.testing.assert_array_equal(a, b)
    d.close()
