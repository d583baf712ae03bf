"""GridInterpolater at the sizes where its launches divide differently: channels shared among blocks, one
channel, more than a block takes, ragged grids, outputs much finer than the input."""
import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg
from libmolgrid_b200 import _cabi
from libmolgrid_b200 import synthetic as cases

pytestmark = pytest.mark.gpu

# batch, channels, input and output points, resolutions
SHAPES = [(1, 1, 5, 4, 0.5, 0.5), (1, 7, 24, 24, 0.5, 0.5), (3, 8, 12, 25, 0.5, 0.5), (1, 9, 13, 12, 0.375, 0.375),
          (2, 33, 16, 13, 1.0, 1.0), (1, 17, 20, 9, 0.375, 1.0), (1, 3, 8, 40, 1.0, 0.125), (49, 2, 8, 8, 0.5, 0.5),
          (1, 5, 20, 39, 0.5, 0.25), (2, 3, 28, 28, 0.75, 0.75)]


def transforms(rng, B, kind):
    if kind == "identity":
        return [lmg.Transform(lmg.Quaternion(1, 0, 0, 0))] * B
    q = cases.random_quaternion(rng, B)
    far = 1e7 if kind == "far" else 0.0
    return [lmg.Transform(lmg.Quaternion(*[float(v) for v in q[b]]), (0.5, -1, 0.25),
                          tuple(float(v) + far for v in rng.uniform(-1, 1, 3))) for b in range(B)]


@pytest.mark.parametrize("kind", ["random", "identity", "far"])
@pytest.mark.parametrize("shape", SHAPES)
def test_forward_both_ways_and_backward_is_its_adjoint(shape, kind):
    B, K, n, m, rin, rout = shape
    rng = np.random.default_rng(n * m + K)
    gi = lmg.GridInterpolater(rin, (n - 1) * rin, rout, (m - 1) * rout)
    torch.manual_seed(K)
    src = torch.randn(B, K, n, n, n, device="cuda")
    trs = transforms(rng, B, kind)
    out = torch.full((B, K, m, m, m), 7.0, device="cuda")
    gi.forward(src, trs, out)
    try:
        for mode in (0, 2):                  # read directly, staged wherever the input allows it
            _cabi.lib().lmg_set_interp_tiled(mode)
            other = torch.full_like(out, 8.0)
            gi.forward(src, trs, other)
            assert torch.equal(out, other)   # the same roundings
    finally:
        _cabi.lib().lmg_set_interp_tiled(1)
    gout = torch.randn_like(out)
    gin, again = torch.full_like(src, 7.0), torch.full_like(src, 8.0)
    gi.backward(gout, trs, gin)
    gi.backward(gout, trs, again)
    assert torch.equal(gin, again)           # sums in a fixed order
    # <out, gout> = <src, gin>: 2^-24 for each of the eight products and sums behind a term
    left, right = (out.double() * gout.double()).sum(), (src.double() * gin.double()).sum()
    scale = float((out.double() * gout.double()).abs().sum() + (src.double() * gin.double()).abs().sum())
    assert abs(float(left - right)) <= 16 * 2.0 ** -24 * scale
    if kind == "far":
        assert not out.any() and not gin.any()
    assert _cabi.lib().lmg_tma_timeouts() == 0
