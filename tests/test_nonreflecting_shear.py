"""The non-reflecting boundaries copy the ring next to the edge, turned by the
Keplerian shear over a cell: by whole turns and more in thin disks, always
within the ring."""
import numpy as np
import pytest

import harness as H
from fargo_thorin_gb300 import _lib, workloads

pytestmark = pytest.mark.gpu


def _shear(rinf, dr, cs, ns):
    # (int) of the shear in cells (NonReflectingBoundary, SideEuler.c:234-337)
    return int(((rinf ** -1.5 - 1.0) / cs * dr) / 2.0 / np.pi * ns + 0.5)


@pytest.mark.parametrize("aspect,nr,ns,turns", [(0.05, 24, 72, 0), (0.01, 24, 72, 1), (0.003, 12, 36, 8), (0.001, 12, 130, 20)])
def test_edges_are_turned_within_their_rings(aspect, nr, ns, turns):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk0", nr, ns, InnerBoundary="NONREFLECTING", EnergyEquation="NO", AspectRatio=aspect)
    d = GpuDisk(p)
    d.init_default()
    H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
    rho = np.array(d.get(0)[:nr * ns]).reshape(nr, ns)
    rho *= 1.0 + 0.01 * np.random.default_rng(1).uniform(-1, 1, rho.shape)
    d.set(0, rho)
    d.refresh(1)                                          # the targets are the rings' means
    cs = np.asarray(d.get(9)[:nr * ns]).reshape(nr, ns).mean(axis=1)
    rin, _, rmed, _ = (np.asarray(a) for a in d.rings())
    inner = _shear(rin[1], rmed[1] - rmed[0], 0.5 * (cs[0] + cs[1]), ns)
    outer = _shear(rin[nr - 2], rmed[nr - 1] - rmed[nr - 2], 0.5 * (cs[nr - 2] + cs[nr - 1]), ns)
    assert max(abs(inner), abs(outer)) >= turns * ns
    _lib.check(d.L.thorin_gpu_hydro(d.h, 1.0e-9), "hydro")
    out = np.asarray(d.get(0)[:nr * ns]).reshape(nr, ns)
    want = rho.copy()
    want[0] = np.roll(rho[1], inner) + rho[0].mean() - rho[1].mean()
    want[nr - 1] = np.roll(rho[nr - 2], outer) + rho[nr - 1].mean() - rho[nr - 2].mean()
    # the substep itself changes the densities by of order 1e-9 of the shear
    assert np.abs(out / want - 1.0).max() < 1e-6
    d.close()
