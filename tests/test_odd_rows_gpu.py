"""Grids whose rows lie on no 16-byte boundary: quads that reach into neighbouring rows and to the end of the
tensor, footprints of one to several passes, each pass of index and vector types, against the CPU checker."""
import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg
from libmolgrid_b200 import synthetic as cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def port():
    from oracle.oracle import CpuOracle
    return CpuOracle("port")


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def inside(shape, value, shift):
    """A tensor in the middle of a larger one that is NaN; `shift` floats off a 16-byte boundary."""
    n = int(np.prod(shape))
    big = torch.full((n + 64,), float("nan"), device="cuda")
    view = big[16 + shift:16 + shift + n].view(shape)
    view.copy_(value if torch.is_tensor(value) else torch.full(shape, value))
    return big, view


def untouched(big, view, shift):
    n = view.numel()
    assert bool(torch.isnan(big[:16 + shift]).all()) and bool(torch.isnan(big[16 + shift + n:]).all())


# footprints of 1 to 35 voxels on rows of every remainder; the largest counts go through records
@pytest.mark.parametrize("res,points,N", [(1.0, 3, 6), (2.0, 2, 4), (0.5, 13, 9), (0.5, 14, 300), (0.5, 15, 1300), (0.5, 11, 4096), (0.5, 11, 4097),
                                          (0.125, 43, 8), (0.1, 45, 5), (0.5, 13, 9000), (1.0, 9, 33000)])
@pytest.mark.parametrize("shift", [0, 1])
def test_index_types(port, res, points, N, shift):
    T, B = 3, 1 if N > 1300 else 3
    g, og = lmg.GridMaker(res, (points - 1) * res), port.gm(res, (points - 1) * res)
    extent = (points - 1) * res / 2
    ex = [cases.index_case(7 + b, N, T, max(extent, 1.0)) for b in range(B)]
    coords, types, radii = (np.stack([e[k] for e in ex]) for k in range(3))
    coords[0, 0], coords[-1, -1] = -extent, extent  # the first and the last voxel of a channel
    types[0, 0], types[-1, -1] = 0, T - 1
    cen = torch.zeros((B, 3), device="cuda")
    big, out = inside((B,) + g.grid_dimensions(T), 7.0, shift)
    g.forward(cen, dev(coords), dev(types), dev(radii), out)
    untouched(big, out, shift)
    diff_np = np.random.default_rng(N).normal(size=tuple(out.shape)).astype(np.float32)
    _, diff = inside(out.shape, dev(diff_np), shift)
    ag, rel = torch.full((B, N, 3), 7.0, device="cuda"), torch.full((B, N), 7.0, device="cuda")
    g.backward(cen, dev(coords), dev(types), dev(radii), diff, ag)
    g.backward_relevance(cen, dev(coords), dev(types), dev(radii), out, diff, rel)
    for b in range(B):
        want = port.forward_index(og, (0, 0, 0), coords[b], types[b], radii[b], T)
        got = out[b].cpu().numpy()
        # up to N / T terms a voxel in any order: a rounding of the running sum each
        np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-6 * max(1.0, N / T / 50))
        wag = port.backward_index(og, (0, 0, 0), coords[b], types[b], radii[b], diff_np[b])
        np.testing.assert_allclose(ag[b].cpu().numpy(), wag, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wag).max())))
        wrel = port.backward_relevance(og, (0, 0, 0), coords[b], types[b], radii[b], got, diff_np[b])
        np.testing.assert_allclose(rel[b].cpu().numpy(), wrel, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wrel).max())))


# gradients on either side of the line between the two kernels, for tails of other shapes and none (a negative multiple)
@pytest.mark.parametrize("multiple", [1.0, 0.7, 2.5, -1.5])
@pytest.mark.parametrize("N", [4096, 4097])
def test_gradients_of_any_tail(port, multiple, N):
    T = 3
    g = lmg.GridMaker(0.5, 6.0, gaussian_radius_multiple=multiple)
    og = port.gm(0.5, 6.0, gaussian_radius_multiple=multiple)
    coords, types, radii = cases.index_case(5, N, T, 4.0)
    diff_np = np.random.default_rng(N).normal(size=g.grid_dimensions(T)).astype(np.float32)
    _, diff = inside(diff_np.shape, dev(diff_np), 0)
    ag = torch.full((N, 3), 7.0, device="cuda")
    g.backward((0, 0, 0), dev(coords), dev(types), dev(radii), diff, ag)
    want = port.backward_index(og, (0, 0, 0), coords, types, radii, diff_np)
    np.testing.assert_allclose(ag.cpu().numpy(), want, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(want).max())))


@pytest.mark.parametrize("res,points,T", [(0.5, 13, 1), (0.5, 14, 9), (0.1, 45, 2), (1.0, 3, 35)])
@pytest.mark.parametrize("binary", [False, True])
@pytest.mark.parametrize("rti", [False, True])
def test_vector_types(port, res, points, T, binary, rti):
    N = 9
    extent = (points - 1) * res / 2
    coords, tv, radii = cases.vector_case(points + T, N, T, extent, rti=rti)
    coords[0], coords[-1] = -extent, extent
    g, og = lmg.GridMaker(res, (points - 1) * res, binary, rti), port.gm(res, (points - 1) * res, binary, rti)
    big, out = inside(g.grid_dimensions(T), 7.0, 0)
    g.forward((0, 0, 0), dev(coords), dev(tv), dev(radii), out)
    untouched(big, out, 0)
    want = port.forward_vector(og, (0, 0, 0), coords, tv, radii)
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-5, atol=2e-6)
    diff_np = np.random.default_rng(N).normal(size=tuple(out.shape)).astype(np.float32)
    _, diff = inside(out.shape, dev(diff_np), 0)
    for with_types in (True, False):
        ag = torch.full((N, 3), 7.0, device="cuda")
        tg = torch.full((N, T), 7.0, device="cuda") if with_types else None
        g.backward_arrays((0, 0, 0), dev(coords), dev(tv), dev(radii), diff, ag, tg, want_type_gradients=with_types)
        wag, wtg = port.backward_vector(og, (0, 0, 0), coords, tv, radii, diff_np)
        np.testing.assert_allclose(ag.cpu().numpy(), wag, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wag).max())))
        if with_types:
            np.testing.assert_allclose(tg.cpu().numpy(), wtg, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wtg).max())))


# radii so small that 1 / radius^2 or 4 / radius^2 is infinite, and one with finite factors, between the grid's points: the
# kernel that prepares its own atoms, the one with records, rows of any and of 16-byte alignment
@pytest.mark.parametrize("radius", [1e-20, 1e-19, 1e-15])
@pytest.mark.parametrize("points,N,shift", [(13, 9, 0), (13, 4097, 0), (13, 9, 1), (16, 9, 0), (16, 9, 1)])
def test_gradients_of_vanishing_radii(port, radius, points, N, shift):
    T, extent = 3, (points - 1) * 0.25
    g, og = lmg.GridMaker(0.5, 2 * extent), port.gm(0.5, 2 * extent)
    coords, types, radii = cases.index_case(11, N, T, extent, ties=False)
    on = np.abs(((coords + extent) * 2) % 1 - 0.5).max(axis=1) < 0.5
    assert on.all()  # no coordinate on a plane of the grid
    radii[::2] = radius
    diff_np = np.random.default_rng(N).normal(size=g.grid_dimensions(T)).astype(np.float32)
    _, diff = inside(diff_np.shape, dev(diff_np), shift)
    ag = torch.full((N, 3), 7.0, device="cuda")
    g.backward((0, 0, 0), dev(coords), dev(types), dev(radii), diff, ag)
    assert not ag[::2].any()
    want = port.backward_index(og, (0, 0, 0), coords, types, radii, diff_np)
    np.testing.assert_allclose(ag.cpu().numpy(), want, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(want).max())))
