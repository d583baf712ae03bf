"""GridInterpolater at its limits: more channels than a launch has blocks, maps that have no use."""
import ctypes

import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg

pytestmark = pytest.mark.gpu


def test_a_refused_launch_is_not_found_again(lib):
    """2^21 channels ask for a launch of more blocks than an axis has unless they are shared out; refused or not, the next
    call is none the worse."""
    K = 65535 * 32 + 40
    gi = lmg.GridInterpolater(1.0, 1.0, 1.0, 1.0)
    a, b = torch.zeros((K, 2, 2, 2), device="cuda"), torch.zeros((K, 2, 2, 2), device="cuda")
    try:
        gi.backward(a, lmg.Transform(), b)
    except RuntimeError:
        pass
    x = torch.rand((10, 3), device="cuda")
    y = torch.empty_like(x)
    from libmolgrid_b200 import _cabi
    t = lmg.Transform().struct()
    _cabi.check(lib.lmg_transform_forward(ctypes.byref(t), 10, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(y.data_ptr()), 1, None))
    torch.cuda.synchronize()
    assert torch.equal(x, y)


@pytest.mark.parametrize("more", [-40, 0, 1, 40])
def test_backward_of_many_channels(more):
    """Channels beyond 65535 blocks of 32: all of them come through, with the identity unchanged."""
    K = 65535 * 32 + more
    gi = lmg.GridInterpolater(1.0, 1.0, 1.0, 1.0)
    g = torch.rand((K, 2, 2, 2), device="cuda")
    out = torch.full_like(g, 7.0)
    gi.backward(g, lmg.Transform(), out)
    assert torch.equal(g, out)


@pytest.mark.parametrize("odd", ["zero", "far", "infinite", "nan"])
def test_backward_of_maps_without_use(odd):
    """A quaternion of length zero, positions far beyond the numbers between voxels and none at all, beside an example as usual:
    the adjoint of the forward pass, in milliseconds (a search of every pair of voxels takes seconds)."""
    n, K = 96, 3
    gi = lmg.GridInterpolater(0.5, (n - 1) * 0.5, 0.5, (n - 1) * 0.5)
    t = {"zero": lmg.Transform(lmg.Quaternion(0, 0, 0, 0)), "far": lmg.Transform(lmg.Quaternion(1, 0, 0, 0), (0, 0, 0), (3e7, 0, 0)),
         "infinite": lmg.Transform(lmg.Quaternion(1, 0, 0, 0), (0, 0, 0), (float("inf"), 0, 0)),
         "nan": lmg.Transform(lmg.Quaternion(float("nan"), 0, 0, 0))}[odd]
    trs = [lmg.Transform(lmg.Quaternion(0.6, 0, 0.8, 0)), t]
    src = torch.rand((2, K, n, n, n), device="cuda") + 0.5
    # sums of 96^3 small whole numbers in one voxel are exact
    g = torch.randint(0, 8, src.shape, device="cuda").float()
    out, back = torch.empty_like(src), torch.full_like(src, 7.0)
    gi.forward(src, trs, out)
    gi.backward(g, trs, back)
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    gi.backward(g, trs, back)
    end.record()
    end.synchronize()
    assert start.elapsed_time(end) < 200.0
    for b in range(2):
        left, right = (out[b].double() * g[b].double()).sum(), (src[b].double() * back[b].double()).sum()
        scale = float((out[b].double() * g[b].double()).abs().sum() + (src[b].double() * back[b].double()).abs().sum())
        assert abs(float(left - right)) <= 16 * 2.0 ** -24 * scale
    if odd == "far":
        assert not out[1].any() and not back[1].any()


@pytest.mark.parametrize("odd", ["infinite", "nan", "far", "zero", "distant"])
@pytest.mark.parametrize("rout,K", [(0.5, 3), (0.5, 40), (1.0, 9), (0.45, 9)])
def test_gradients_do_not_depend_on_the_other_examples(odd, rout, K):
    """The same bits alone and beside an example whose map has no use, or whose positions are rounded so far from the origin
    (a rotation about a point 3000 cells away) that the sums take another order for it."""
    n, m = 18, 17
    gi = lmg.GridInterpolater(0.5, (n - 1) * 0.5, rout, (m - 1) * rout)
    inf, nan = float("inf"), float("nan")
    one = lmg.Quaternion(1, 0, 0, 0)
    t = {"infinite": lmg.Transform(one, (0, 0, 0), (inf, 0, 0)), "nan": lmg.Transform(lmg.Quaternion(nan, 0, 0, 0)),
         "far": lmg.Transform(one, (0, 0, 0), (3e7, 0, 0)), "zero": lmg.Transform(lmg.Quaternion(0, 0, 0, 0)),
         "distant": lmg.Transform(lmg.Quaternion(0.8, 0.6, 0, 0), (1500.0, 0, 0), (0.25, -0.5, 0))}[odd]
    trs = [lmg.Transform(lmg.Quaternion(0.6, 0, 0.8, 0), (0, 0, 0), (0.3, -0.2, 0.1)), t,
           lmg.Transform(lmg.Quaternion(0.5, -0.5, 0.1, 0.7), (0.25, 1, -0.5), (0.7, 0.1, -0.4))]
    cen = np.zeros((3, 3), np.float32)
    g = torch.randn((3, K, m, m, m), device="cuda")
    together = torch.full((3, K, n, n, n), 7.0, device="cuda")
    gi.backward(cen, g, trs, cen, together)
    for b in range(3):
        if b == 1 and odd not in ("far", "distant"):
            continue  # positions that are no numbers: added up by reductions, in no fixed order
        alone = torch.full((1, K, n, n, n), 8.0, device="cuda")
        gi.backward(cen[b:b + 1], g[b:b + 1].clone(), trs[b:b + 1], cen[b:b + 1], alone)
        assert torch.equal(alone[0], together[b])
        assert bool(alone.any()) == (b != 1 or odd == "distant")


def _adjoint_axis(din, dout, f, shift):
    """The weights of an axis without rotation: output voxel o at input index f * (o - (dout - 1) / 2) - shift + (din - 1) / 2."""
    g = f * (np.arange(dout) - (dout - 1) / 2) - shift + (din - 1) / 2
    return np.maximum(0.0, 1.0 - np.abs(np.arange(din)[:, None] - g[None, :]))


@pytest.mark.parametrize("rout", [0.5, 0.25])
def test_backward_from_a_grid_of_more_voxels_than_32_bits_count(rout):
    """1626^3 output voxels, of which the last planes lie in the input grid (a translation by whole quarters of a voxel, so
    that every weight and sum is exact): by cells, and by the search for a finer output."""
    din, m = 9, 1626
    gi = lmg.GridInterpolater(0.5, (din - 1) * 0.5, rout, (m - 1) * rout)
    rng = np.random.default_rng(3)
    keep = 24
    corner = rng.integers(-8, 8, (keep,) * 3).astype(np.float32)
    g = torch.zeros((1, m, m, m), device="cuda")
    g[0, -keep:, -keep:, -keep:] = torch.from_numpy(corner).cuda()
    shift = rout / 0.5 * (m - 1) / 2 - (din - 1) / 2  # the last output voxel on the last of the input
    back = torch.full((1, din, din, din), 7.0, device="cuda")
    gi.backward(g, lmg.Transform(lmg.Quaternion(1, 0, 0, 0), (0, 0, 0), (shift * 0.5,) * 3), back)
    w = _adjoint_axis(din, m, rout / 0.5, shift)[:, -keep:]
    assert w.sum() > din - 1
    want = np.einsum("ai,bj,ck,ijk->abc", w, w, w, corner.astype(float))
    assert np.array_equal(back[0].cpu().numpy(), want)


def test_forward_to_a_grid_of_2048_voxels_a_side():
    """2^33 output voxels, a count of zero in 32 bits."""
    din, m = 5, 2048
    gi = lmg.GridInterpolater(0.5, (din - 1) * 0.5, 0.5, (m - 1) * 0.5)
    src = torch.rand((1, din, din, din), device="cuda")
    out = torch.full((1, m, m, m), 7.0, device="cuda")
    gi.forward(src, lmg.Transform(lmg.Quaternion(1, 0, 0, 0), (0, 0, 0), (0.25, 0.25, 0.25)), out)
    lo = (m - din) // 2  # an odd difference: half a voxel that the translation makes up for
    inside = out[0, lo - 1:lo + din + 2, lo - 1:lo + din + 2, lo - 1:lo + din + 2].clone()
    assert torch.equal(inside[inside != 0].sort().values, src[0].flatten().sort().values)
    out[0, lo - 1:lo + din + 2, lo - 1:lo + din + 2, lo - 1:lo + din + 2] = 0
    assert not out.any()
