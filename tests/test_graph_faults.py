"""Failures while a DT graph is built, by faked return codes of host calls: the
disk keeps its state and its buffers, the error reaches the caller, and only
a refused cooperative launch makes the graph fall back on launched sweeps."""
import ctypes as C

import numpy as np
import pytest

import harness as H
from fargo_thorin_gb300 import _lib, workloads

REFUSED, COPY = 1, 2
FIELDS = (0, 1, 2, 3, 4, 5, 6, 8, 9)


def test_fault_arguments():
    lib = _lib.load()
    assert lib.thorin_selftest_graph_fault(None, COPY) == 1


def _disk():
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk1", 32, 96)
    d = GpuDisk(p)
    d.init_default()
    H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
    s = workloads.make_planets(p, [workloads.PLANET1])
    d.algogas(s)                                          # calibrates omega on the host path
    return d, s


def _state(d, s):
    return [d.get(f).copy() for f in FIELDS] + [np.array([s.x[0], s.y[0], s.vx[0], s.vy[0], s.mass[0]]),
                                                np.array(d.sor_state()[:3]), np.array([d.stats().physical_time])]


def _same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("built", [False, True])
def test_failed_capture_reaches_the_caller_and_keeps_the_disk(built):
    a, sa = _disk()
    b, sb = _disk()
    if built:                                             # a graph was there before
        a.algogas_graph(sa)
        b.algogas_graph(sb)
    before = _state(b, sb)
    _lib.check(b.L.thorin_selftest_graph_fault(b.h, COPY), "graph_fault")
    with pytest.raises(_lib.ThorinError, match="state back into its buffers"):
        b.algogas_graph(sb)
    _same(before, _state(b, sb))
    for _ in range(2):
        a.algogas_graph(sa)
        b.algogas_graph(sb)
        assert a.stats().substeps == b.stats().substeps
        _same(_state(a, sa), _state(b, sb))
    a.algogas(sa)
    b.algogas(sb)
    _same(_state(a, sa), _state(b, sb))
    a.close()
    b.close()


@pytest.mark.gpu
def test_refused_solve_launch_falls_back_on_launched_sweeps():
    """The sweeps' updates are the same bits in either form."""
    a, sa = _disk()
    b, sb = _disk()
    _lib.check(b.L.thorin_selftest_graph_fault(b.h, REFUSED), "graph_fault")
    for _ in range(3):
        a.algogas_graph(sa)
        b.algogas_graph(sb)
        assert a.stats().sor_sweeps == b.stats().sor_sweeps
        _same(_state(a, sa), _state(b, sb))
    a.algogas(sa)                                         # and the host path solves in one launch again
    b.algogas(sb)
    _same(_state(a, sa), _state(b, sb))
    a.close()
    b.close()
