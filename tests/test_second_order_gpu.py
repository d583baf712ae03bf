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
