"""GPU parity of Transform forward/backward and GridInterpolater against the CPU oracle,
through the C ABI.  Coordinates are bit-exact (same operation order, no fused multiply-add);
interpolated grids are held to rel 1e-4 as the path states, and checked for exact equality too
since the kernel keeps the reference's operation order."""
import numpy as np
import pytest
import torch

from tests import cases

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.fixture(autouse=True)
def _no_copy_timeouts():
    """No block of the tiled interpolation ever gave up waiting for its staged box."""
    yield
    from libmolgrid_b200 import _cabi
    torch.cuda.synchronize()
    assert _cabi.lib().lmg_tma_timeouts() == 0


def make_transform(q, c, t):
    import libmolgrid_b200 as lmg
    return lmg.Transform(lmg.Quaternion(*q), tuple(c), tuple(t))


@pytest.mark.parametrize("dotranslate", [True, False])
def test_transform_bit_exact(port, dotranslate):
    rng = np.random.default_rng(2)
    pts = (rng.normal(size=(1000, 3)) * 8).astype(np.float32)
    for q in (cases.random_quaternion(rng, 1)[0], rng.normal(size=4).astype(np.float32)):  # unit and not
        c, t = rng.uniform(-3, 3, 3).astype(np.float32), rng.uniform(-2, 2, 3).astype(np.float32)
        tr = make_transform(q, c, t)
        otr = port.tr(q, c, t)
        out = torch.empty((1000, 3), device="cuda")
        tr.forward(dev(pts), out, dotranslate)
        assert np.array_equal(out.cpu().numpy(), port.transform_forward(otr, pts, dotranslate))
        tr.backward(dev(pts), out, dotranslate)
        assert np.array_equal(out.cpu().numpy(), port.transform_backward(otr, pts, dotranslate))


def test_transform_known_points():
    """test/test_transform.py:30-97 of the reference: rotations by 90 degrees about axes."""
    import libmolgrid_b200 as lmg
    s = float(np.sqrt(0.5))
    pts = dev(np.array([[1, 1, 1]], np.float32))
    out = torch.empty_like(pts)
    tr = lmg.Transform(lmg.Quaternion(s, 0, 0, s), (0, 1, 1), (2, 2, -3))
    tr.forward(pts, out)
    # rotate (1,0,0) about z by 90 degrees around centre (0,1,1) -> (0,1,0)+(0,1,1), then translate
    assert np.allclose(out.cpu().numpy(), [[2, 4, -2]], atol=1e-6)
    back = torch.empty_like(pts)
    tr.backward(out, back)
    assert np.allclose(back.cpu().numpy(), [[1, 1, 1]], atol=1e-5)
    # in place is allowed
    tr.forward(pts, pts)
    assert torch.equal(pts, out)


def test_transform_roundtrip_large():
    import libmolgrid_b200 as lmg
    lmg.set_random_seed(0)
    rng = np.random.default_rng(1)
    pts = dev((rng.normal(size=(200000, 3)) * 10).astype(np.float32))
    tr = lmg.Transform((1.0, -2.0, 0.5), 3.0, True)
    a = torch.empty_like(pts)
    b = torch.empty_like(pts)
    tr.forward(pts, a)
    tr.backward(a, b)
    assert torch.allclose(b, pts, atol=1e-4)


@pytest.mark.usefixtures("interpolation")
@pytest.mark.parametrize("gi", [(0.5, 11.5, 0.5, 11.5), (0.5, 11.5, 0.25, 8.0), (0.25, 6.0, 0.5, 9.5)])
def test_interpolate(port, gi):
    import libmolgrid_b200 as lmg
    rng = np.random.default_rng(4)
    g = lmg.GridInterpolater(*gi)
    din, dout = g.s.in_dim, g.s.out_dim
    K = 5
    grid = rng.uniform(size=(K, din, din, din)).astype(np.float32)
    for q, c, t, ic, oc in [
        ((1, 0, 0, 0), (0, 0, 0), (0, 0, 0), (0, 0, 0), (0, 0, 0)),
        (cases.random_quaternion(rng, 1)[0], (0.5, 0, -1), (1, -0.5, 0.25), (0.5, 0, -1), (0.5, 0, -1)),
        (cases.random_quaternion(rng, 1)[0], (0, 0, 0), (0, 2, 0), (1, 0, 0), (0, 0.5, 0)),
    ]:
        want = port.interpolate(gi, ic, grid, port.tr(q, c, t), oc)
        out = torch.full((K, dout, dout, dout), -3.0, device="cuda")
        g.forward(ic, dev(grid), make_transform(q, c, t), oc, out)
        got = out.cpu().numpy()
        assert np.allclose(got, want, rtol=1e-4, atol=1e-6)
        assert np.array_equal(got, want)


@pytest.mark.usefixtures("interpolation")
def test_interpolate_batched_and_identity(port):
    import libmolgrid_b200 as lmg
    rng = np.random.default_rng(9)
    gi = (0.5, 5.5, 0.5, 5.5)
    g = lmg.GridInterpolater(*gi)
    B, K, d = 60, 3, 12   # more examples than one launch carries
    grids = rng.uniform(size=(B, K, d, d, d)).astype(np.float32)
    qs = cases.random_quaternion(rng, B)
    ts = rng.uniform(-1, 1, (B, 3)).astype(np.float32)
    trs = [make_transform(qs[b], (0, 0, 0), ts[b]) for b in range(B)]
    out = torch.empty((B, K, d, d, d), device="cuda")
    g.forward(dev(grids), trs, out)
    got = out.cpu().numpy()
    for b in (0, 17, 47, 48, 59):
        want = port.interpolate(gi, (0, 0, 0), grids[b], port.tr(qs[b], (0, 0, 0), ts[b]), (0, 0, 0))
        assert np.array_equal(got[b], want)
    # identity transform reproduces the input (test/test_gridinterp.py:15-30)
    one = torch.empty((K, d, d, d), device="cuda")
    g.forward(dev(grids[0]), lmg.Transform(), one)
    assert np.array_equal(one.cpu().numpy(), grids[0])
    with pytest.raises(ValueError):
        g.forward(one, lmg.Transform(), one)


def test_interpolate_tiled_equals_direct_at_benchmark_shape():
    """28x48^3 grids under random rotations: the kernel that stages input boxes with tensor copies
    and the direct-read kernel give identical bits, and no staged copy ever timed out."""
    import libmolgrid_b200 as lmg
    from libmolgrid_b200 import _cabi
    rng = np.random.default_rng(21)
    B, K, d = 6, 28, 48
    g = lmg.GridInterpolater(0.5, 23.5, 0.5, 23.5)
    src = torch.rand((B, K, d, d, d), device="cuda")
    qs = cases.random_quaternion(rng, B)
    qs[0] = (1, 0, 0, 0)
    qs[1] = np.array([0.5, 0.5, 0.5, 0.5], np.float32)   # 120 degrees about the diagonal
    ts = rng.uniform(-2, 2, (B, 3)).astype(np.float32)
    ts[2] = (40, 0, 0)                                    # mostly outside the input
    trs = [make_transform(qs[b], (0, 0, 0), ts[b]) for b in range(B)]
    tiled, direct = torch.full_like(src, -2.0), torch.empty_like(src)
    lib = _cabi.lib()
    g.forward(src, trs, tiled)
    try:
        lib.lmg_set_interp_tiled(0)
        g.forward(src, trs, direct)
    finally:
        lib.lmg_set_interp_tiled(1)
    torch.cuda.synchronize()
    assert torch.equal(tiled, direct)
    assert float(tiled[3].abs().sum()) > 0 and float(tiled[2].abs().sum()) < float(tiled[3].abs().sum())
    assert lib.lmg_tma_timeouts() == 0
    # an unaligned view of the same data takes the direct kernel and agrees as well
    shifted = torch.empty(src[0].numel() + 1, device="cuda")[1:].view_as(src[0])
    shifted.copy_(src[3])
    one = torch.empty_like(src[0])
    g.forward(shifted, trs[3], one)
    assert torch.equal(one, tiled[3])


@pytest.mark.usefixtures("interpolation")
@pytest.mark.parametrize("gi", [(0.5, 23.5, 0.6, 21.0), (0.5, 23.5, 0.41, 15.17), (0.5, 15.5, 1.5, 30.0)])
def test_interpolate_staged_resampling(port, gi):
    """Coarser and finer output grids than the input (input rows 16-byte aligned: the finer one
    takes the staged kernel, the coarser ones the direct kernel), against the oracle."""
    import libmolgrid_b200 as lmg
    rng = np.random.default_rng(33)
    g = lmg.GridInterpolater(*gi)
    din, dout = g.s.in_dim, g.s.out_dim
    assert din % 4 == 0
    K = 3
    grid = rng.uniform(size=(K, din, din, din)).astype(np.float32)
    q = cases.random_quaternion(rng, 1)[0]
    c, t = (0.25, -0.5, 0.75), (1.0, -2.0, 0.5)
    want = port.interpolate(gi, c, grid, port.tr(q, c, t), (0.0, 0.5, 0.0))
    out = torch.full((K, dout, dout, dout), -3.0, device="cuda")
    g.forward(c, dev(grid), make_transform(q, c, t), (0.0, 0.5, 0.0), out)
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("gi", [(0.5, 11.5, 0.5, 11.5), (0.5, 11.5, 0.25, 8.0), (0.25, 6.0, 0.5, 9.5)])
def test_interpolate_backward_is_the_adjoint(gi):
    """<forward(x), y> == <x, backward(y)> for random x, y, and backward of a one-hot output gradient
    reproduces the forward pass's weights (checked through a finite difference of the forward)."""
    import libmolgrid_b200 as lmg
    rng = np.random.default_rng(41)
    torch.manual_seed(41)          # the random grids below: the same on every run
    g = lmg.GridInterpolater(*gi)
    din, dout = g.s.in_dim, g.s.out_dim
    K = 3
    tr = make_transform(cases.random_quaternion(rng, 1)[0], (0.5, 0, -1), (1, -0.5, 0.25))
    x = torch.rand((K, din, din, din), device="cuda", dtype=torch.float32)
    y = torch.randn((K, dout, dout, dout), device="cuda", dtype=torch.float32)
    fx = torch.empty_like(y)
    g.forward(x, tr, fx)
    by = torch.full_like(x, 5.0)   # must be overwritten
    g.backward(y, tr, by)
    lhs = float((fx.double() * y.double()).sum())
    rhs = float((x.double() * by.double()).sum())
    # float32 accumulation on both sides: the bound is relative to the size of the terms, since
    # y has both signs and the sums may cancel
    scale = float((fx.double() * y.double()).abs().sum())
    assert scale > 1.0 and abs(lhs - rhs) <= 1e-5 * scale
    # linearity in x: forward(x + h e) - forward(x) = h * forward(e); <that, y> = h * by[e]
    e = (1, din // 2, din // 2 - 1, din // 2)
    x2 = x.clone()
    x2[e] += 1.0
    fx2 = torch.empty_like(y)
    g.forward(x2, tr, fx2)
    assert float(((fx2 - fx).double() * y.double()).sum()) == pytest.approx(float(by[e]), rel=1e-3, abs=1e-4)
    # batched, five-argument form
    xb = torch.rand((2, K, din, din, din), device="cuda")
    yb = torch.randn((2, K, dout, dout, dout), device="cuda")
    trs = [tr, make_transform(cases.random_quaternion(rng, 1)[0], (0, 0, 0), (0, 1, 0))]
    cen = np.zeros((2, 3), np.float32)
    fb, bb = torch.empty_like(yb), torch.empty_like(xb)
    g.forward(cen, xb, trs, cen, fb)
    g.backward(cen, yb, trs, cen, bb)
    scale = float((fb.double() * yb.double()).abs().sum())
    assert abs(float((fb.double() * yb.double()).sum()) - float((xb.double() * bb.double()).sum())) <= 1e-5 * scale
    with pytest.raises(ValueError):
        g.backward(y, tr, torch.empty_like(y) if din != dout else y)


def _adjoint64(y, din, res_in, res_out, q, c, t):
    """The adjoint of the trilinear resample in 64 bits, by scattering."""
    dout = y.shape[-1]
    w, v = q[0], np.asarray(q[1:], float)
    n = w * w + v @ v
    S = np.array([[0, -v[2], v[1]], [v[2], 0, -v[0]], [-v[1], v[0], 0]])
    R = ((w * w - v @ v) * np.eye(3) + 2 * np.outer(v, v) - 2 * w * S) / n     # the inverse rotation
    ax = (np.arange(dout) - (dout - 1) / 2) * res_out
    p = np.stack(np.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    g = ((p - t - c) @ R.T + c) / res_in + (din - 1) / 2
    lo = np.floor(g).astype(int)
    fr = g - lo
    out = np.zeros((y.shape[0], din, din, din))
    for k in range(8):
        up = np.array([k >> 2, k >> 1 & 1, k & 1])
        wt = np.where(up, fr, 1 - fr).prod(1)
        idx = lo + up
        ok = ((idx >= 0) & (idx < din)).all(1)
        i, j, l = idx[ok].T
        for ch in range(y.shape[0]):
            np.add.at(out[ch], (i, j, l), wt[ok] * y[ch].reshape(-1)[ok])
    return out


@pytest.mark.parametrize("din,dout,rin,rout", [(16, 16, 0.5, 0.5), (17, 23, 0.5, 0.5), (9, 4, 0.5, 0.5), (3, 30, 0.5, 0.5),
                                               (25, 13, 0.5, 1.0), (33, 31, 0.375, 0.375), (20, 18, 0.5, 0.45), (1, 1, 0.5, 0.5)])
@pytest.mark.parametrize("K", [1, 8, 9])
def test_interpolate_backward_against_64_bits(din, dout, rin, rout, K):
    """Tiles with and without remainders, output grids as fine, coarser and finer, shares of eight channels with and
    without a rest, positions on the planes of the input grid (no rotation, and a quarter turn).  A position is off by a
    few roundings of some ten Angstrom, 1e-6 cells or so, and a weight by as much: 2e-5 of the sum's own norm."""
    import libmolgrid_b200 as lmg
    rng = np.random.default_rng(din * 100 + dout)
    g = lmg.GridInterpolater(rin, (din - 1) * rin, rout, (dout - 1) * rout)
    turns = [(cases.random_quaternion(rng, 1)[0], (0.25, -0.5, 1.0), (0.75, -0.3, 0.2)), ((1, 0, 0, 0), (0, 0, 0), (0, 0, 0)),
             ((0.5 ** 0.5, 0, 0, 0.5 ** 0.5), (0, 0, 0), (rin, 0, -rin))]
    y = rng.normal(size=(len(turns), K, dout, dout, dout)).astype(np.float32)
    cen = np.zeros((len(turns), 3), np.float32)
    out = torch.full((len(turns), K, din, din, din), 7.0, device="cuda")
    trs = [make_transform(*t) for t in turns]
    g.backward(cen, dev(y), trs, cen, out)
    for b, (q, c, t) in enumerate(turns):
        want = _adjoint64(y[b].astype(float), din, rin, rout, np.asarray(q, float), np.asarray(c, float), np.asarray(t, float))
        assert np.linalg.norm(out[b].cpu().numpy() - want) <= 2e-5 * np.linalg.norm(want) + 1e-6
    again = torch.full_like(out, 3.0)
    g.backward(cen, dev(y), trs, cen, again)
    assert torch.equal(out, again)


# either side of every line between the two kernels: outputs a little finer, centres far away (in cells), outputs coarser by
# more and less than 2.5 and, in grids of many tiles, twice as coarse with channels that make whole groups and others
@pytest.mark.parametrize("din,dout,rin,rout,far,K,B", [
    (17, 18, 0.5, 0.499, 0, 1, 24), (17, 18, 0.5, 0.498, 0, 1, 24), (17, 18, 0.5, 0.5, 2580, 1, 24), (17, 18, 0.5, 0.5, 2720, 1, 24),
    (30, 12, 0.5, 1.24, 0, 2, 24), (30, 12, 0.5, 1.25, 0, 2, 24), (30, 13, 0.5, 0.87, 0, 32, 2), (61, 14, 0.5, 0.875, 0, 32, 2),
    (61, 14, 0.5, 0.875, 0, 33, 1), (29, 5, 0.5, 0.7, 0, 9, 8), (29, 5, 0.5, 0.8, 0, 9, 8)])
def test_interpolate_backward_on_either_side_of_the_lines(din, dout, rin, rout, far, K, B):
    """Random rotations of grids of several tiles.  Positions of `far` cells are off by a few roundings of that size, and
    the weights by as much."""
    import libmolgrid_b200 as lmg
    rng = np.random.default_rng(din + 7 * dout + far)
    g = lmg.GridInterpolater(rin, (din - 1) * rin, rout, (dout - 1) * rout)
    center = np.array([far * rin, 0, 0], np.float32)
    q, t = cases.random_quaternion(rng, B), rng.uniform(-1, 1, (B, 3)).astype(np.float32)
    y = rng.normal(size=(B, K, dout, dout, dout)).astype(np.float32)
    out = torch.full((B, K, din, din, din), 7.0, device="cuda")
    cen = np.tile(center, (B, 1))
    g.backward(cen, dev(y), [make_transform(q[b], center, t[b]) for b in range(B)], cen, out)
    # one rounding of a position for each of about sixteen operations, in the worst case along all axes
    for b in range(B):
        want = _adjoint64(y[b].astype(float), din, rin, rout, q[b].astype(float), np.zeros(3), t[b].astype(float))
        assert np.linalg.norm(out[b].cpu().numpy() - want) <= (2e-5 + 16 * 2.0 ** -24 * far) * np.linalg.norm(want) + 1e-6


@pytest.mark.parametrize("layer", ["python", "compiled"])
def test_transform_known_answers_on_host_arrays_and_in_place(layer):
    """The reference's worked example (test/test_transform.py:65-140): a quarter turn about z through
    (0,1,1) then a shift by (2,0,-3), on numpy arrays and MGrids, the input left unchanged; a random
    transform undone in place."""
    if layer == "python":
        import libmolgrid_b200 as mg
    else:
        import molgrid as mg
    from math import sqrt
    q = mg.Quaternion(sqrt(0.5), 0, 0, sqrt(0.5))
    nr = mg.Transform(q, mg.float3(0, 1, 1), mg.float3(2, 0, -3))
    data = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1], [-1, .5, 3], [1, 1, 1], [0, 1, 1], [.333, .75, -9]],
                    np.float32)
    coords, out = data.copy(), np.zeros((8, 3), np.float32)
    nr.forward(coords, out)
    assert tuple(out[6]) == (2, 1, -2) and tuple(out[2]) == (2, 1, -3) and tuple(out[5]) == (2, 2, -2)
    assert np.array_equal(coords, data)
    m_in, m_out = mg.MGrid2f(8, 3), mg.MGrid2f(8, 3)
    m_in.copyFrom(data)
    nr.forward(m_in, m_out)
    assert np.array_equal(m_out.tonumpy(), out)
    r = mg.Transform(mg.float3(0, 1, 1), 10.0, True)
    r.forward(coords, out)
    assert not np.isclose(out, coords, atol=1e-5).all(axis=1).any()
    r.backward(out, out)                                   # in place
    assert np.allclose(out, coords, atol=1e-5)
