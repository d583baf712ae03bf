"""backward_gradients at the edges of its sweep (footprints of one to several passes of quads, partial columns,
many channels, grids without aligned rows), against the CPU checker."""
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


# resolution and points: footprints of 3 to 40 voxels; rows of 16 bytes, or not
@pytest.mark.parametrize("res,points", [(1.0, 8), (0.5, 24), (0.125, 44), (0.5, 13)])
@pytest.mark.parametrize("T,rti", [(1, False), (5, True), (35, False), (35, True)])
def test_both_terms(port, res, points, T, rti):
    N = 7
    extent = (points - 1) * res / 2
    coords, tv, radii = cases.vector_case(points * T + rti, N, T, extent, rti=rti)
    coords[0] = extent          # on a corner of the grid, on a grid point
    if T == 1:
        tv[2] = 0.0             # an atom without weight
    g = lmg.GridMaker(res, (points - 1) * res, False, rti)
    og = port.gm(res, (points - 1) * res, False, rti)
    rng = np.random.default_rng(5)
    diff = rng.normal(size=(T,) + (points,) * 3).astype(np.float32)
    ag, tg = rng.normal(size=(N, 3)).astype(np.float32), rng.normal(size=(N, T)).astype(np.float32)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dd, add, tdd = (torch.full(x.shape, 7.0, device="cuda") for x in (diff, ag, tg))
    g.backward_gradients((0, 0, 0), d(coords), d(tv), d(radii), d(diff), d(ag), d(tg), dd, add, tdd)
    want = port.backward_gradients(og, (0, 0, 0), coords, tv, radii, diff, ag, tg)
    for got, w in zip((dd, add, tdd), want):
        scale = max(1.0, float(np.abs(w).max()))
        np.testing.assert_allclose(got.cpu().numpy(), w, rtol=1e-4, atol=1e-5 * scale)


def beyond(coords, radii, res, points, channels):
    """[atom, channel] voxels that the atom's density does not reach, of a multiple of 1 (cut-off 1.5 radii)."""
    ax = torch.arange(points, dtype=torch.float64) * res - (points - 1) * res / 2
    x = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1)
    d = torch.stack([(x - torch.tensor(c, dtype=torch.float64)).norm(dim=-1) for c in coords])
    if len(radii) == channels:   # by type
        return torch.stack([(d > 1.5 * float(r) * 1.0001) for r in radii], 1)
    return torch.stack([(d[a] > 1.5 * float(radii[a]) * 1.0001) for a in range(len(coords))])[:, None].expand(-1, channels, -1, -1, -1)


# sweeps of quads per (atom, channel) and per atom, and single voxels; values that are not finite next to a footprint
@pytest.mark.parametrize("points", [24, 13])
@pytest.mark.parametrize("rti", [False, True])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_values_beyond_the_cut_off_do_not_matter(points, rti, bad):
    N, T, res = 5, 7, 0.5
    coords, tv, radii = cases.vector_case(points + rti, N, T, points * res / 4, rti=rti)
    tv = np.maximum(tv, 0.05).astype(np.float32)
    out = beyond(coords, radii, res, points, T)
    g = lmg.GridMaker(res, (points - 1) * res, False, rti)
    rng = np.random.default_rng(7)
    diff = torch.from_numpy(rng.normal(size=(T,) + (points,) * 3).astype(np.float32))
    ag, tg = (torch.from_numpy(rng.normal(size=s).astype(np.float32)).cuda() for s in ((N, 3), (N, T)))
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()

    def run(diff, ag):
        dd, add, tdd = (torch.full(x.shape, 7.0, device="cuda") for x in (diff, ag, tg))
        g.backward_gradients((0, 0, 0), d(coords), d(tv), d(radii), diff.cuda(), ag, tg, dd, add, tdd)
        return dd.cpu(), add.cpu()

    free = out.all(0)   # voxels that no atom reaches
    assert bool(free.any()) and not bool(free.all())
    ok, want = run(torch.where(free, 0.0, diff), ag)
    _, got = run(torch.where(free, bad, diff), ag)
    assert bool(torch.isfinite(got).all()) and torch.equal(got, want)
    wild = ag.clone()
    wild[2] = bad       # and an atom's gradient where the atom does not reach
    dd, _ = run(diff, wild)
    assert bool(torch.isfinite(dd[out[2]]).all()) and torch.allclose(dd[out[2]], ok[out[2]], rtol=1e-5, atol=1e-5)


def test_grid_term_against_64_bits():
    """Radii by atom, all channels weighted.  The density from a root of its own and the slope in one rounding: 1.705e-7,
    2-norm; from the reciprocal root that the second derivative needs: 1.807e-7."""
    N, T, P = 200, 4, 24
    gen = torch.Generator().manual_seed(0)
    coords, w = (torch.randn(N, 3, generator=gen) * 3).cuda(), torch.rand(N, T, generator=gen).cuda()
    radii = (torch.rand(N, generator=gen) + 1.2).cuda()
    torch.rand(T, generator=gen)
    diff, ag, tg = (torch.randn(*s, generator=gen).cuda() for s in ((T, P, P, P), (N, 3), (N, T)))
    dd, add, tdd = (torch.empty_like(x) for x in (diff, ag, tg))
    lmg.GridMaker(0.5, (P - 1) * 0.5).backward_gradients((0.0, 0.0, 0.0), coords, w, radii, diff, ag, tg, dd, add, tdd)
    ax = torch.arange(P, device="cuda", dtype=torch.float64) * 0.5 - (P - 1) * 0.25
    x = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    want = torch.zeros(T, P ** 3, device="cuda", dtype=torch.float64)
    e2 = float(np.exp(-2.0))
    for a in range(N):
        ar, delta = radii[a].double(), x - coords[a].double()
        dist = delta.norm(dim=1)
        r = dist / ar
        v = torch.where(r <= 1, torch.exp(-2 * r * r), torch.where(r <= 1.5, e2 * (2 * r - 3) ** 2, 0.0))
        slope = torch.where(r <= 1, 4 * v / ar ** 2, torch.where(r <= 1.5, -4 * e2 * (2 * r - 3) / (ar * dist), 0.0))
        want += v * tg[a].double()[:, None] + w[a].double()[:, None] * (slope * (delta @ ag[a].double()))
    assert float((dd.reshape(T, -1).double() - want).norm() / want.norm()) < 1.75e-7
