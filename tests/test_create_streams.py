"""A disk is made and advanced on its own stream alone: work of the program that
is still queued on the default stream neither delays nor overwrites it."""
import numpy as np
import pytest

import harness as H
from fargo_thorin_gb300 import workloads

pytestmark = pytest.mark.gpu


def _run(queued=None):
    from fargo_thorin_gb300.disk import GpuDisk
    p = workloads.params_for("disk1", 48, 144)
    d = GpuDisk(p)
    d.init_default()
    H.start_state(d, p, {"dens": d.get(0), "temper": d.get(8)})
    d.set_sor_state(1.1, 1e-3, 50)
    s = workloads.make_planets(p, [workloads.PLANET1])
    for k in range(4):
        (d.algogas_graph if k > 1 else d.algogas)(s)
    if queued is not None:
        print("default stream still busy after the DTs:", not queued.query())
    out = [d.get(f) for f in (0, 1, 2, 3, 4, 5, 6, 8)] + [np.array(d.sor_state()[:3])]
    d.close()
    return out


def test_disk_beside_a_busy_default_stream():
    import torch
    quiet = _run()
    a = torch.full((8192, 8192), 1e-4, device="cuda")
    a @ a
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    b = a
    for _ in range(40):                                   # some tenths of a second
        b = b @ a
    done.record()
    busy = _run(done)
    torch.cuda.synchronize()
    for x, y in zip(quiet, busy):
        np.testing.assert_array_equal(x, y)
