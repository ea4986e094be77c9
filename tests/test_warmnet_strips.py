"""The network's convolutions walk strips of rings: grids whose units of work
take several rings (with a remainder, also across a batch) at one or more
levels, and widths around the strip of 128 cells, against the oracle."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "oracle"))

import warmnet_oracle as WO  # noqa: E402
from test_warmnet import _inputs, _params  # noqa: E402
from fargo_thorin_gb300 import warmstart as WS  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 16, 16), (1, 1000, 16), (2, 648, 16), (1, 344, 264), (1, 56, 128), (1, 632, 136)])
def test_forward_matches_oracle_on_strips(B, H, W):
    p = _params(31)
    x, _ = _inputs(32, B, H, W)
    net = WS.WarmNet(H, W, max_batch=B, params=p.astype(np.float32))
    y = net.forward(WO.bf16_bits(x))
    yo, _ = WO.forward(p.astype(np.float32), x, bf=True)
    # the tolerance of test_forward_matches_oracle, ring by ring
    err = np.linalg.norm(y - yo, axis=-1) / np.linalg.norm(yo, axis=-1)
    assert err.max() < 2e-2, err.max()
    assert np.linalg.norm(y - yo) / np.linalg.norm(yo) < 1e-2
