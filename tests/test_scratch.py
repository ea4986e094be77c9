"""The reduction scratch of a disk holds what every launch writes to it.

CPU: the launchers' own counts against the size allocated, over grids from the
smallest to wide and to narrow ones and every number of planets (one or two
rings a block of the force kernels need the most).  GPU: the forces of eight
planets on grids that need the most for their size, against the oracle."""
import ctypes as C

import numpy as np
import pytest

import harness as H
import oracle as O
from fargo_thorin_gb300 import _lib, workloads

COLUMNS = sorted({4, 72, 126} | {128 * k + e for k in range(1, 63) for e in (0, 2)})


@pytest.mark.parametrize("nsm", [152, 148, 76, 1])
def test_scratch_holds_what_the_launches_write(nsm):
    lib = _lib.load()
    need, held = C.c_longlong(), C.c_longlong()
    for nr in list(range(4, 130)) + [192, 256, 333, 400, 1024, 2048]:
        for ns in COLUMNS:
            for npl in (0, 1, 7, 8):
                assert lib.thorin_selftest_partials(nr, ns, npl, nsm, C.byref(need), C.byref(held)) == 0
                assert 0 < need.value <= held.value, (nr, ns, npl, need.value, held.value)


def test_scratch_counts_the_force_kernels_blocks():
    """24516, 24552 and 24336 doubles with eight planets on 152 multiprocessors, 21792
    with seven: a ring a block, 2 (blocks of k_forces and k_forces_near) + 152
    blocks of 2 + 2 npl values."""
    lib = _lib.load()
    need, held = C.c_longlong(), C.c_longlong()
    for nr, ns, npl, least in [(121, 514, 8, 24516), (101, 642, 8, 24552), (25, 3072, 8, 24336), (55, 1282, 7, 21792)]:
        assert lib.thorin_selftest_partials(nr, ns, npl, 152, C.byref(need), C.byref(held)) == 0
        assert need.value >= least and held.value >= least, (nr, ns)


def test_scratch_count_rejects_bad_arguments():
    lib = _lib.load()
    need, held = C.c_longlong(), C.c_longlong()
    for bad in [(3, 72, 1, 152), (24, 2, 1, 152), (24, 72, 9, 152), (24, 72, -1, 152), (24, 72, 1, 0)]:
        assert lib.thorin_selftest_partials(*bad, C.byref(need), C.byref(held)) == 1
    assert lib.thorin_selftest_partials(24, 72, 1, 152, None, C.byref(held)) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("kind,nr,ns", [("disk0", 121, 514), ("disk1", 101, 642)])
def test_forces_of_eight_planets_on_wide_grids(kind, nr, ns):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for(kind, nr, ns, PlanetsFeelDisk="YES")
    rows = [(m, 0., 0., a, 0.01 * (k % 3), 0.5 * (k % 2), 20. * k, 10., 47. * k)
            for k, (m, a) in enumerate(zip([3e-5, 1e-6, 1e-4, 1e-5, 6e-5, 3e-6, 2e-5, 5e-5],
                                           [0.5, 0.66, 0.83, 1.03, 1.27, 1.55, 1.88, 2.2]))]
    d, o = GpuDisk(p), O.OracleDisk(p)
    o.init_default()
    init = {"dens": o.get(H.FIELD_IDS["dens"]).copy(), "temper": o.get(H.FIELD_IDS["temper"]).copy()}
    d.init_default()
    for x in (d, o):
        H.start_state(x, p, init)
        x.set_time(1.0)                               # the mass taper is over
    sg, so = (workloads.make_planets(p, rows) for _ in range(2))
    n = nr * ns
    for step in range(1, 3):
        d.algogas(sg)
        o.algogas(so)
        assert d.stats().substeps == o.stats().substeps
        # the pebbles' density and v_r are left to the tests of the accretion: a
        # cell that gives up all but 1e-8 of its pebbles keeps a difference of
        # that relative accuracy, here in the spheres of eight planets
        for f in H.GAS + (["pebblevtheta"] if p.pebbles else []):
            # the tolerance of the oracle comparisons (test_gpu_parity)
            assert H.rel_l2(d.get(H.FIELD_IDS[f])[:n], o.get(H.FIELD_IDS[f])[:n]) < 1e-11, f"{f} at DT {step}"
        for k in range(8):
            a = np.hypot(so.ax[k], so.ay[k])
            assert np.hypot(sg.ax[k] - so.ax[k], sg.ay[k] - so.ay[k]) <= 1e-9 * a
            assert abs(sg.x[k] - so.x[k]) < 1e-13 and abs(sg.vy[k] - so.vy[k]) < 1e-13
    d.close()
