"""Gradients of type vectors with radii by channel where a warp takes several channels of an atom: against the CPU oracle, at the
edges of the channels a warp takes, for atoms with no, one and all channels weighted."""
import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg
from libmolgrid_b200 import _cabi, api

pytestmark = pytest.mark.gpu


def _case(seed, N, T, side):
    rng = np.random.default_rng(seed)
    coords = rng.uniform(-side / 2 - 2, side / 2 + 2, (N, 3)).astype(np.float32)
    radii = rng.uniform(0.6, 2.6, T).astype(np.float32)
    radii[T // 2] = 0.0  # a channel that reaches nothing
    types = np.zeros((N, T), np.float32)
    for a in range(N):
        k = (0, 1, T // 2 + 1, T)[a % 4]
        types[a, rng.permutation(T)[:k]] = rng.uniform(0.1, 1, k)
    return coords, types, radii


def _close(got, want):
    np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(want).max())))


# channels, atoms, points, resolution: one warp an atom to four, footprints of more columns than are held at a time
@pytest.mark.parametrize("T,N,points,res", [(4, 160, 24, 1.0), (5, 2000, 16, 1.0), (16, 700, 24, 1.0), (16, 9000, 12, 1.0), (17, 100, 24, 1.0),
                                            (17, 9000, 12, 1.0), (33, 60, 24, 1.0), (64, 20, 24, 1.0), (64, 3000, 8, 1.0), (28, 440, 32, 0.5),
                                            (9, 40000, 16, 0.25), (14, 50, 36, 0.75)])
@pytest.mark.parametrize("multiple", [1.0, 0.4, 2.5])
def test_gradients(port, T, N, points, res, multiple):
    side = (points - 1) * res
    coords, types, radii = _case(T * points, N, T, side)
    g, og = lmg.GridMaker(res, side, False, True, 1.0, multiple), port.gm(res, side, False, True, 1.0, multiple)
    diff = torch.randn(g.grid_dimensions(T), device="cuda")
    dc, dt, dr = (torch.from_numpy(x).cuda() for x in (coords, types, radii))
    out = []
    for _ in range(2):
        ag, tg = torch.full((N, 3), 7.0, device="cuda"), torch.full((N, T), 7.0, device="cuda")
        g.backward((0, 0, 0), dc, dt, dr, diff, ag, tg)
        out.append((ag, tg))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    m = min(N, 40)
    wag, wtg = port.backward_vector(og, (0, 0, 0), coords[:m], types[:m], radii, diff.cpu().numpy())
    _close(out[0][0][:m].cpu().numpy(), wag)
    _close(out[0][1][:m].cpu().numpy(), wtg)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("weighted", [(3,), (0, 1, 2, 4, 5, 6, 7, 8, 9, 10)])
def test_channels_without_weight_do_not_reach_the_atoms(value, weighted):
    T, N = 11, 200
    coords, types, radii = _case(7, N, T, 20.0)
    types[:] = 0
    types[:, weighted] = np.random.default_rng(1).uniform(0.1, 1, (N, len(weighted)))
    g = lmg.GridMaker(1.0, 23.0, False, True)
    diff = torch.randn(g.grid_dimensions(T), device="cuda")
    data = [torch.from_numpy(x.astype(np.float32)).cuda() for x in (coords, types, radii)]
    grads = []
    for v in (0.0, value):
        diff[[t for t in range(T) if t not in weighted]] = v
        grads.append((torch.empty(N, 3, device="cuda"), torch.empty(N, T, device="cuda")))
        g.backward((0, 0, 0), *data, diff, *grads[-1])
    _close(grads[1][0].cpu().numpy(), grads[0][0].cpu().numpy())
    assert torch.equal(grads[0][1][:, list(weighted)], grads[1][1][:, list(weighted)])


@pytest.mark.parametrize("T,N,points,res", [(4, 160, 24, 1.0), (16, 60, 24, 1.0), (17, 60, 24, 1.0), (33, 60, 24, 1.0), (64, 20, 24, 1.0),
                                            (28, 440, 32, 0.5), (14, 50, 36, 0.75)])
@pytest.mark.parametrize("multiple", [1.0, 2.0])
@pytest.mark.parametrize("infinite", [False, True])
def test_second_derivatives(port, T, N, points, res, multiple, infinite):
    side = (points - 1) * res
    coords, types, radii = _case(T + points, N, T, side)
    rng = np.random.default_rng(T)
    ca, ct = rng.normal(size=(N, 3)).astype(np.float32), rng.normal(size=(N, T)).astype(np.float32)
    diff = rng.normal(size=(T, points, points, points)).astype(np.float32)
    if infinite:  # an incoming gradient that is no number stays within its atom's reach
        coords[5] = 0.0
        ca[5, 1] = np.inf
    g, og = lmg.GridMaker(res, side, False, True, 1.0, multiple), port.gm(res, side, False, True, 1.0, multiple)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii, diff, ca, ct)]
    dd, da, dt = torch.full(diff.shape, 7.0, device="cuda"), torch.full((N, 3), 7.0, device="cuda"), torch.full((N, T), 7.0, device="cuda")
    g.backward_gradients((0, 0, 0), *data, dd, da, dt)
    wd, wa, wt = port.backward_gradients(og, (0, 0, 0), coords, types, radii, diff, ca, ct)
    got, keep = dd.cpu().numpy(), np.isfinite(wd)
    if infinite:
        assert keep.mean() > 0.5 and np.isfinite(got[keep]).all()
    _close(got[keep], wd[keep])
    rows = [a for a in range(N) if not (infinite and a == 5)]
    _close(da.cpu().numpy()[rows], wa[rows])
    assert not dt.any()


# Radii so small that an atom's own footprint is empty beside its coordinates, and others that reach one voxel at most, for
# atoms on grid points and off them.
@pytest.mark.parametrize("T,N,points,res", [(4, 160, 24, 1.0), (16, 60, 24, 1.0), (33, 60, 24, 1.0), (28, 440, 32, 0.5)])
@pytest.mark.parametrize("multiple", [1.0, 2.5])
@pytest.mark.parametrize("on_points", [False, True])
def test_radii_below_a_voxel(port, T, N, points, res, multiple, on_points):
    side = (points - 1) * res
    coords, types, radii = _case(T * points + 1, N, T, side)
    if on_points:
        coords = (np.round((coords + side / 2) / res) * res - side / 2).astype(np.float32)
    rng = np.random.default_rng(T)
    small = rng.choice([1e-38, 1e-20, 1e-12, 1e-7, 4e-7, 1e-6, 2e-6, 1e-4, 0.03, 0.15], T).astype(np.float32)
    radii = np.where(np.arange(T) % 3 == 1, radii, small).astype(np.float32)
    ca, ct = rng.normal(size=(N, 3)).astype(np.float32), rng.normal(size=(N, T)).astype(np.float32)
    diff = rng.normal(size=(T, points, points, points)).astype(np.float32)
    g, og = lmg.GridMaker(res, side, False, True, 1.0, multiple), port.gm(res, side, False, True, 1.0, multiple)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii, diff)]
    ag, tg = torch.full((N, 3), 7.0, device="cuda"), torch.full((N, T), 7.0, device="cuda")
    g.backward((0, 0, 0), *data, ag, tg)
    wag, wtg = port.backward_vector(og, (0, 0, 0), coords, types, radii, diff)
    _close(ag.cpu().numpy(), wag)
    _close(tg.cpu().numpy(), wtg)
    dd, da, dt = torch.empty_like(data[3]), torch.empty_like(ag), torch.empty_like(tg)
    g.backward_gradients((0, 0, 0), *data, torch.from_numpy(ca).cuda(), torch.from_numpy(ct).cuda(), dd, da, dt)
    wd, wa, _ = port.backward_gradients(og, (0, 0, 0), coords, types, radii, diff, ca, ct)
    _close(dd.cpu().numpy(), wd)
    _close(da.cpu().numpy(), wa)


@pytest.mark.parametrize("weight", [float("inf"), -3.4e38, 1e37])
@pytest.mark.parametrize("by_channel,T,N,points", [(True, 16, 60, 24), (True, 17, 60, 24), (True, 28, 60, 24), (False, 14, 1200, 25)])
def test_infinite_and_huge_weights(port, weight, by_channel, T, N, points):
    """An atom's gradient is the weighted sum of its channels' own: infinite, not undefined, where a weight is."""
    side = points - 1.0
    coords, types, radii = _case(T + 3 * points, N, T, side)
    # huge ones in a single channel: sums of several may overflow on the way or not, as they are added up
    rows = types[::2] if np.isinf(weight) else types[1::4]
    rows[rows != 0] = weight
    if not by_channel:
        radii = np.random.default_rng(1).uniform(0.8, 2.2, N).astype(np.float32)
    g, og = lmg.GridMaker(1.0, side, False, by_channel), port.gm(1.0, side, False, by_channel)
    diff = np.random.default_rng(T).normal(size=(T, points, points, points)).astype(np.float32)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii, diff)]
    ag, tg = torch.full((N, 3), 7.0, device="cuda"), torch.full((N, T), 7.0, device="cuda")
    g.backward((0, 0, 0), *data, ag, tg)
    m = min(N, 200)
    wag, wtg = port.backward_vector(og, (0, 0, 0), coords[:m], types[:m], radii if by_channel else radii[:m], diff)
    ag, keep = ag[:m].cpu().numpy(), np.isfinite(wag)
    assert np.array_equal(np.isnan(ag), np.isnan(wag)) and np.array_equal(ag[~keep & ~np.isnan(wag)], wag[~keep & ~np.isnan(wag)])
    # gradients of weights that differ by up to 1e38: each against its own atom's
    scale = np.maximum(np.nanmax(np.where(keep, np.abs(wag), 0), axis=1, keepdims=True), 1.0) + np.zeros((1, 3))
    np.testing.assert_array_less(np.abs(ag[keep] / scale[keep] - wag[keep] / scale[keep]), 2e-4)
    _close(tg[:m].cpu().numpy(), wtg)


@pytest.mark.parametrize("soft", [False, True])
def test_large_spheres_against_64_bits(soft):
    """Some thousand voxels an atom and channel, 28 distinct atoms of many: a lane's sums are as near to 64 bits as those of a warp
    for each channel, whose relative error (2-norm) here is 2.2e-7 with one weighted channel and 2.4e-7 with all."""
    points, res, T, grm, N, k = 96, 0.25, 14, 2.0, 28, 800
    torch.manual_seed(1)
    coords = (torch.rand(N, 3, device="cuda") - 0.5) * 16
    types = torch.rand(N, T, device="cuda") ** 4 if soft else torch.nn.functional.one_hot(torch.arange(N, device="cuda") % T, T).float()
    radii = 1.2 + torch.rand(T, device="cuda")
    g = lmg.GridMaker(res, (points - 1) * res, False, True, 1.0, grm)
    diff = torch.randn(g.grid_dimensions(T), device="cuda")
    ag, tg = torch.empty(N * k, 3, device="cuda"), torch.empty(N * k, T, device="cuda")
    g.backward((0, 0, 0), coords.repeat(k, 1), types.repeat(k, 1), radii, diff, ag, tg)
    assert torch.equal(ag[:N], ag[-N:]) and torch.equal(tg[:N], tg[-N:])
    e = np.exp(-2 * grm * grm)
    A, B, C = 4 * grm ** 2 * e, -e * (4 * grm + 8 * grm ** 3), e * (4 * grm ** 4 + 4 * grm ** 2 + 1)
    axis = torch.arange(points, device="cuda", dtype=torch.float64) * res - (points - 1) * res / 2
    wag, wtg = torch.zeros(N, 3, dtype=torch.float64, device="cuda"), torch.zeros(N, T, dtype=torch.float64, device="cuda")
    for a in range(N):
        d = [(axis - coords[a, c].double()).reshape([-1 if i == c else 1 for i in range(3)]) for c in range(3)]
        r = (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).sqrt()
        for t in range(T):
            ar = radii[t].double()
            q = r / ar
            gauss, inside = torch.exp(-2 * q * q), q <= (1 + 2 * grm * grm) / (2 * grm)
            wtg[a, t] = (torch.where(q <= grm, gauss, (A * q + B) * q + C) * inside * diff[t].double()).sum()
            f = torch.where(q <= grm, 4 * gauss / ar ** 2, -(2 * A * q + B) / ar / r) * inside * diff[t].double() * types[a, t].double()
            wag[a] += torch.stack([(f * x).sum() for x in d])
    assert ((ag[:N].double() - wag).norm() / wag.norm()).item() < 2.4e-7
    assert ((tg[:N].double() - wtg).norm() / wtg.norm()).item() < 3.1e-7  # 2.6e-7 measured, 3.0e-7 a warp for each channel


def _batch(seed, B, N, T, side):
    """Examples of their own, with a centre, a rotation and a translation each."""
    from libmolgrid_b200 import synthetic
    rng = np.random.default_rng(seed)
    coords, types, radii = (np.stack(x) for x in zip(*(_case(seed + b, N, T, side) for b in range(B))))
    q = synthetic.random_quaternion(rng, B)
    rows = np.concatenate([q, rng.uniform(-1, 1, (B, 6)).astype(np.float32)], 1).astype(np.float32)
    return coords, types, radii, rng.uniform(-1, 1, (B, 3)).astype(np.float32), rows


class _Room:
    """Workspaces of at most this many bytes."""
    def __init__(self, nbytes):
        self.nbytes = nbytes

    def __enter__(self):
        self.old, api.MAX_WORKSPACE_BYTES = api.MAX_WORKSPACE_BYTES, self.nbytes
        api._workspaces.clear()

    def __exit__(self, *a):
        api.MAX_WORKSPACE_BYTES = self.old
        api._workspaces.clear()


def _bytes(g, op, B, N, T):
    import ctypes
    return _cabi.lib().lmg_workspace_bytes(ctypes.byref(g.s), op, B, N, T, 1)


# one warp an atom and several; in one pass and in passes of two and one
@pytest.mark.parametrize("T,N,points,res", [(5, 160, 16, 1.0), (14, 3000, 12, 1.0), (17, 60, 24, 1.0), (28, 160, 32, 0.5)])
@pytest.mark.parametrize("passes", [False, True])
def test_batches(port, T, N, points, res, passes):
    """Examples with a centre, a transform and a count each: every one against the oracle, with nothing behind the counts."""
    B, side = 5, (points - 1) * res
    coords, types, radii, centers, rows = _batch(T * N, B, N, T, side)
    n = np.array([N, N - 7, N // 2, 1, 0], np.int32)
    rng = np.random.default_rng(N)
    diff = rng.normal(size=(B, T, points, points, points)).astype(np.float32)
    ca, ct = rng.normal(size=(B, N, 3)).astype(np.float32), rng.normal(size=(B, N, T)).astype(np.float32)
    g, og = lmg.GridMaker(res, side, False, True), port.gm(res, side, False, True)
    d = [torch.from_numpy(x).cuda() for x in (centers, coords, types, radii, diff, ca, ct)]
    more = dict(transforms=torch.from_numpy(rows).cuda(), n_atoms=torch.from_numpy(n).cuda())
    shapes = (B, N, 3), (B, N, T), diff.shape, (B, N, 3), (B, N, T)
    rooms = [torch.full((int(np.prod(x)) + 64,), 7.0, device="cuda") for x in shapes]
    ag, tg, dd, da, dt = (r[32:-32].view(x) for r, x in zip(rooms, shapes))
    launches = [_cabi.lib().lmg_launch_count()]
    with _Room(_bytes(g, _cabi.OP_BACKWARD, 2, N, T) if passes else api.MAX_WORKSPACE_BYTES):
        g.backward(*d[:5], ag, tg, **more)
    launches.append(_cabi.lib().lmg_launch_count())
    with _Room(_bytes(g, _cabi.OP_BACKWARD_GRADIENTS, 2, N, T) if passes else api.MAX_WORKSPACE_BYTES):
        g.backward_gradients(*d[:5], d[5], d[6], dd, da, dt, **more)
    launches.append(_cabi.lib().lmg_launch_count())
    # constants, records and sums, and the parts of atoms that several warps share
    assert all((b - a) in ((9, 12) if passes else (3, 4)) for a, b in zip(launches, launches[1:]))
    assert all(bool((r[:32] == 7.0).all() and (r[-32:] == 7.0).all()) for r in rooms)  # nothing beside the outputs
    for b in range(B):
        m = int(n[b])
        assert not ag[b, m:].any() and not tg[b, m:].any() and not da[b, m:].any()
        if m == 0:
            assert not dd[b].any()
            continue
        k = min(m, 60)
        moved = port.transform_forward(port.tr(rows[b, :4], rows[b, 4:7], rows[b, 7:]), coords[b, :m])
        wag, wtg = port.backward_vector(og, centers[b], moved[:k], types[b, :k], radii[b], diff[b])
        _close(ag[b, :k].cpu().numpy(), wag)
        _close(tg[b, :k].cpu().numpy(), wtg)
        wd, wa, _ = port.backward_gradients(og, centers[b], moved, types[b, :m], radii[b], diff[b], ca[b, :m], ct[b, :m])
        _close(dd[b].cpu().numpy(), wd)
        _close(da[b, :m].cpu().numpy(), wa)


@pytest.mark.parametrize("T,N,points,res", [(8, 50, 24, 1.0), (16, 130, 24, 1.0), (28, 160, 32, 0.5)])
def test_passes_of_a_call_take_the_same_kernel(T, N, points, res):
    """Five times the same example, two a pass: the last one alone has the bits of the others."""
    side = (points - 1) * res
    coords, types, radii = (torch.from_numpy(x).cuda()[None].repeat(5, *[1] * x.ndim) for x in _case(T, N, T, side))
    g = lmg.GridMaker(res, side, False, True)
    diff = torch.randn(g.grid_dimensions(T), device="cuda")[None].repeat(5, 1, 1, 1, 1)
    ca, ct = torch.randn(N, 3, device="cuda")[None].repeat(5, 1, 1), torch.randn(N, T, device="cuda")[None].repeat(5, 1, 1)
    centers = torch.zeros(5, 3, device="cuda")
    ag, tg = torch.empty_like(coords), torch.empty_like(types)
    with _Room(_bytes(g, _cabi.OP_BACKWARD, 2, N, T)):
        g.backward(centers, coords, types, radii, diff, ag, tg)
    dd, da, dt = torch.empty_like(diff), torch.empty_like(coords), torch.empty_like(types)
    with _Room(_bytes(g, _cabi.OP_BACKWARD_GRADIENTS, 2, N, T)):
        g.backward_gradients(centers, coords, types, radii, diff, ca, ct, dd, da, dt)
    for x in (ag, tg, da):
        assert all(torch.equal(x[0], x[b]) for b in range(1, 5))


# by (atom, channel) or by atom: records (and the channels' constants), sums, their reduction if there is one
@pytest.mark.parametrize("by_channel,quads,T,N,first,second", [(True, 1, 16, 9000, 3, 3), (True, 1, 17, 100, 4, 4), (True, 0, 17, 100, 4, 5),
                                                               (True, 1, 3, 100, 4, 4), (False, 1, 5, 100, 2, 2), (False, 0, 5, 100, 3, 4)])
def test_launches_are_counted(by_channel, quads, T, N, first, second):
    lib, side = _cabi.lib(), 23.0
    coords, types, radii = _case(3, N, T, side)
    if not by_channel:
        radii = np.ones(N, np.float32)
    g = lmg.GridMaker(1.0, side, False, by_channel)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii)]
    diff, ag, tg = torch.randn(g.grid_dimensions(T), device="cuda"), torch.empty_like(data[0]), torch.empty_like(data[1])
    outs = torch.empty_like(diff), torch.empty_like(ag), torch.empty_like(tg)
    lib.lmg_set_quads(quads)
    try:
        n = [lib.lmg_launch_count()]
        g.backward((0, 0, 0), *data, diff, ag, tg)
        n.append(lib.lmg_launch_count())
        g.backward_gradients((0, 0, 0), *data, diff, ag, tg, *outs)
        n.append(lib.lmg_launch_count())
    finally:
        lib.lmg_set_quads(1)
    assert (n[1] - n[0], n[2] - n[1]) == (first, second)
