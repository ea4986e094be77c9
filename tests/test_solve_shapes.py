"""The solve in one launch has two shapes, for a disk alone and beside others; a
disk takes it only where both are within the limits.

CPU: the shared memory of the larger one over grids and numbers of
multiprocessors.  GPU: the shape beside others at the largest disks it takes
and above the size from which a block no longer fits twice, bit for bit
against plain launches of the passes."""
import ctypes as C

import numpy as np
import pytest

from fargo_thorin_gb300 import _lib

SMEM = 227 * 1024 - 256


def _shape(nr, ns, nsm):
    w, b = C.c_int(), C.c_longlong()
    assert _lib.load().thorin_selftest_solve_shape(nr, ns, nsm, C.byref(w), C.byref(b)) == 0
    return w.value, b.value


@pytest.mark.parametrize("nsm", [152, 148, 132, 114, 76, 20])
def test_both_shapes_are_within_the_limits(nsm):
    for nr, ns in [(4, 4), (24, 72), (128, 384), (333, 1002), (512, 1536), (700, 2100), (800, 2400), (850, 2550),
                   (896, 2684), (898, 2684), (1024, 3072), (6, 40000), (40000, 60)]:
        within, smem = _shape(nr, ns, nsm)
        np_, sms = ns // 2 * (nr - 2), (3 * nsm + 3) // 4
        pm = -(-np_ // min(-(-np_ // 32), sms))              # pairs a block beside others
        if 2 * np_ > 2400000:
            assert not within
        else:
            assert smem >= 20 * pm
            assert bool(within) == (smem <= SMEM), (nr, ns, smem)


def test_the_whole_range_fits_on_this_gpu():
    for nr, ns in [(896, 2684), (850, 2550), (400, 6030), (1550, 1550)]:
        assert _shape(nr, ns, 152)[0] == 1


def test_arguments():
    w, b = C.c_int(), C.c_longlong()
    lib = _lib.load()
    assert lib.thorin_selftest_solve_shape(3, 72, 152, C.byref(w), C.byref(b)) == 1
    assert lib.thorin_selftest_solve_shape(24, 72, 0, C.byref(w), C.byref(b)) == 1
    assert lib.thorin_selftest_solve_shape(24, 72, 152, None, C.byref(b)) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("nr,ns", [(24, 72), (560, 1680), (700, 2100), (896, 2684)])
def test_solve_beside_other_disks_matches_the_launched_passes(monkeypatch, nr, ns):
    import harness as H
    from fargo_thorin_gb300 import workloads
    from fargo_thorin_gb300.disk import GpuDisk
    out = []
    for form in ("direct", "pool", "graph"):
        monkeypatch.setenv("THORIN_SOR_DIRECT", "1" if form == "direct" else "0")
        disks, systems = [], []
        for n, m in ((nr, ns), (40, 120)):
            p = workloads.params_for("disk0", n, m, DT=0.004)
            d = GpuDisk(p)
            d.init_default()
            H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
            d.set_sor_state(1.3, 1e-3, 50)
            disks.append(d)
            systems.append(workloads.make_planets(p, [workloads.PLANET0]))
        dp = (C.c_void_p * 2)(*[d.h.value for d in disks])
        sp = (C.c_void_p * 2)(*[C.cast(C.pointer(s), C.c_void_p).value for s in systems])
        st = (C.c_int * 2)()
        lib = _lib.load()
        counts = []
        for _ in range(2):
            if form == "graph":
                _lib.check(lib.thorin_ensemble_algogas_graph(dp, sp, 2, st), "graph")
            else:
                _lib.check(lib.thorin_ensemble_algogas(dp, sp, 2, 2 if form == "pool" else 1, 0, st), "pool")
            counts.append([(d.stats().substeps, d.stats().sor_last_niter) for d in disks])
        out.append((counts, [d.get(f).copy() for d in disks for f in (0, 1, 2, 3, 8)]))
        for d in disks:
            d.close()
    assert out[0][0] == out[1][0] == out[2][0]
    for a, b, c in zip(out[0][1], out[1][1], out[2][1]):
        np.testing.assert_array_equal(a, b)
        # the graph's planet side is the device's (test_graph_dt)
        assert np.linalg.norm(a - c) <= 1e-12 * np.linalg.norm(a)
