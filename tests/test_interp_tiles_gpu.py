"""Which GridInterpolater calls are staged by tiles: the same bits on either side of the line, tiles of any size of call."""
import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg
from libmolgrid_b200 import _cabi
from libmolgrid_b200 import synthetic as cases

pytestmark = pytest.mark.gpu


# batch, channels, input and output points: tiny, ragged tiles, and just below and above the lines of the choice
@pytest.mark.parametrize("shape", [(1, 1, 8, 4), (1, 7, 24, 24), (3, 8, 12, 25), (2, 33, 16, 13), (49, 2, 8, 8), (2, 12, 28, 36),
                                   (2, 13, 28, 36), (13, 27, 24, 24), (13, 28, 24, 24), (2, 10, 28, 36), (2, 11, 28, 36),
                                   (8, 1, 28, 36), (9, 1, 28, 36), (26, 2, 24, 36), (27, 2, 24, 36)])
@pytest.mark.parametrize("identity", [False, True])
def test_tiles_and_direct_reads_agree(shape, identity):
    B, K, n, m = shape
    rng = np.random.default_rng(n * m + K)
    gi = lmg.GridInterpolater(0.5, (n - 1) * 0.5, 0.5, (m - 1) * 0.5)
    src = torch.randn(B, K, n, n, n, device="cuda")
    q = cases.random_quaternion(rng, B)
    trs = [lmg.Transform(lmg.Quaternion(1, 0, 0, 0) if identity else lmg.Quaternion(*[float(v) for v in q[b]]), (0.0, 0.0, 0.0),
                         tuple(float(v) for v in rng.uniform(-1, 1, 3))) for b in range(B)]
    out = []
    try:
        for mode in (0, 1, 2):
            _cabi.lib().lmg_set_interp_tiled(mode)
            out.append(torch.full((B, K, m, m, m), float(7 + mode), device="cuda"))
            gi.forward(src, trs, out[-1])
    finally:
        _cabi.lib().lmg_set_interp_tiled(1)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
    assert _cabi.lib().lmg_tma_timeouts() == 0
