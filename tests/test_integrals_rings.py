"""The conservation integrals (a block per ring, the rings' sums by the last
block) against exactly rounded sums (math.fsum) of the reference's terms, at
rings shorter than a block, at its edges and at ring counts around a warp."""
import math

import numpy as np
import pytest

from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nr,ns", [("disk1", 5, 10), ("disk0", 33, 126), ("disk1", 31, 128), ("disk1", 64, 130),
                                        ("disk0", 97, 514), ("disk1", 129, 1030)])
def test_integrals_of_every_shape(kind, nr, ns):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for(kind, nr, ns, OmegaFrame=0.7)
    d = GpuDisk(p)
    d.init_default()
    peb = kind == "disk1"
    g = np.random.default_rng(nr * ns)
    rin, rout, rmed, surf = (np.asarray(a)[:nr, None] for a in d.rings())
    f = {0: g.uniform(0.5, 1.5, (nr, ns)), 1: 1e-2 * g.uniform(-1, 1, (nr, ns)),
         2: rmed ** -0.5 * g.uniform(0.9, 1.1, (nr, ns)), 3: g.uniform(1e-3, 2e-3, (nr, ns))}
    if peb:
        f[4], f[6] = g.uniform(0.0, 0.1, (nr, ns)), rmed ** -0.5 * g.uniform(0.9, 1.1, (nr, ns))
    for k, a in f.items():
        d.set(k, a)
    vr = np.vstack([f[1], np.asarray(d.get(1)).reshape(-1)[nr * ns:].reshape(-1, ns)[:1]
                    if np.asarray(d.get(1)).size > nr * ns else np.zeros((1, ns))])
    w = p.omega_frame
    terms = [surf * f[0], 0.5 * surf * (f[0] + np.roll(f[0], 1, 1)) * rmed * (f[2] + w * rmed),
             0.5 * surf * f[0] * ((((rmed - rin) * vr[1:] + (rout - rmed) * vr[:-1]) / (rout - rin)) ** 2 +
                                  (0.5 * (f[2] + np.roll(f[2], -1, 1)) + rmed * w) ** 2) + surf * f[3]]
    if peb:
        terms += [surf * f[4], 0.5 * surf * (f[4] + np.roll(f[4], 1, 1)) * rmed * (f[6] + w * rmed)]
    for q, (got, t) in enumerate(zip(d.integrals(), terms)):
        # a sum passes through ns / 128 + nr / 64 + 20 roundings at most, a
        # term (here and there) through 16
        bound = (ns / 128 + nr / 64 + 36) * 2.0 ** -53 * float(np.abs(t).sum())
        assert abs(got - math.fsum(t.ravel())) <= bound, q
    d.close()
