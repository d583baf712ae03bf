"""Type vectors with radii by atom and one, two, a few and all channels weighted: which of them the forward pass adds one
by one or together, and from what the backward pass takes the atom gradient, against the CPU oracle."""
import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg
from libmolgrid_b200 import synthetic as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [3, 4, 5, 7, 8, 14, 15, 33])
@pytest.mark.parametrize("weighted", [0, 1, 2, 3, 13, 40])
@pytest.mark.parametrize("binary,multiple", [(False, 1.0), (True, 1.0), (False, 3.0), (False, -1.5)])
def test_weighted_channels(T, weighted, binary, multiple):
    from oracle.oracle import CpuOracle
    port, N = CpuOracle("port"), 21
    coords, tv, radii = cases.vector_case(T + weighted, N, T, 4.0, rti=False)
    rng = np.random.default_rng(T * 50 + weighted)
    tv[:] = 0
    for a in range(N):  # neighbouring channels, so that several fall into one round, from any first one
        first = int(rng.integers(T))
        for k in range(min(weighted, T)):
            tv[a, (first + k) % T] = rng.uniform(0.1, 1)
    assert ((tv != 0).sum(axis=1) == min(weighted, T)).all()
    g = lmg.GridMaker(0.5, 7.5, binary, gaussian_radius_multiple=multiple)
    og = port.gm(0.5, 7.5, binary, gaussian_radius_multiple=multiple)
    assert g.grid_dimensions(T)[1] % 4 == 0
    dc, dt, dr = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (coords, tv, radii))
    out = torch.full(g.grid_dimensions(T), 7.0, device="cuda")
    g.forward((0, 0, 0), dc, dt, dr, out)
    want = port.forward_vector(og, (0, 0, 0), coords, tv, radii)
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-5, atol=2e-6)
    diff = rng.normal(size=want.shape).astype(np.float32)
    ag, tg = torch.full((N, 3), 7.0, device="cuda"), torch.full((N, T), 7.0, device="cuda")
    g.backward((0, 0, 0), dc, dt, dr, torch.from_numpy(diff).cuda(), ag, tg)
    wag, wtg = port.backward_vector(og, (0, 0, 0), coords, tv, radii, diff)
    np.testing.assert_allclose(ag.cpu().numpy(), wag, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wag).max())))
    np.testing.assert_allclose(tg.cpu().numpy(), wtg, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wtg).max())))


@pytest.mark.parametrize("T,weighted", [(14, (3, 4)), (15, (0, 13)), (28, (2, 9, 11)), (16, (5,))])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), -3.4e38])
@pytest.mark.parametrize("binary", [False, True])
def test_unweighted_channels_do_not_reach_the_atoms(T, weighted, value, binary):
    """Gradients of the grid that are no numbers, in the channels without weight beside those with one: the atom gradients and
    the weighted channels' type gradients are those of a grid with zeros there."""
    from oracle.oracle import CpuOracle
    port, N = CpuOracle("port"), 13
    coords, tv, radii = cases.vector_case(T, N, T, 4.0, rti=False)
    rng = np.random.default_rng(T)
    tv[:] = 0
    tv[:, weighted] = rng.uniform(0.1, 1, (N, len(weighted)))
    g, og = lmg.GridMaker(0.5, 7.5, binary), port.gm(0.5, 7.5, binary)
    diff = np.zeros(g.grid_dimensions(T), np.float32)
    diff[list(weighted)] = rng.normal(size=(len(weighted),) + diff.shape[1:])
    wag, wtg = port.backward_vector(og, (0, 0, 0), coords, tv, radii, diff)
    diff[[t for t in range(T) if t not in weighted]] = value
    dc, dt, dr = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (coords, tv, radii))
    ag, tg = torch.full((N, 3), 7.0, device="cuda"), torch.full((N, T), 7.0, device="cuda")
    g.backward((0, 0, 0), dc, dt, dr, torch.from_numpy(diff).cuda(), ag, tg)
    np.testing.assert_allclose(ag.cpu().numpy(), wag, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wag).max())))
    tg, wtg = tg.cpu().numpy()[:, weighted], wtg[:, weighted]
    np.testing.assert_allclose(tg, wtg, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wtg).max())))


# densities in the reference's order of operations: few and many atoms, with few, more and many weighted channels of a round
@pytest.mark.parametrize("N,weighted", [(30, 12), (30, 13), (1200, 12), (1201, 6), (1201, 7)])
@pytest.mark.parametrize("points", [12, 40])
def test_precise_densities_of_weighted_channels(N, weighted, points):
    from oracle.oracle import CpuOracle
    port, T = CpuOracle("port"), 16
    res = 0.5 if points < 20 else 0.125  # footprints of one and of two passes along z
    if points > 20 and N > 1000:
        pytest.skip("one size of grid is enough for many atoms")
    coords, tv, radii = cases.vector_case(N, N, T, (points - 1) * res / 2, rti=False)
    rng = np.random.default_rng(N)
    tv[:] = 0
    for a in range(N):
        tv[a, rng.permutation(T)[:weighted]] = rng.uniform(0.1, 1, weighted)
    g = lmg.GridMaker(res, (points - 1) * res, gaussian_radius_multiple=2.5)
    og = port.gm(res, (points - 1) * res, gaussian_radius_multiple=2.5)
    out = torch.full(g.grid_dimensions(T), 7.0, device="cuda")
    g.forward((0, 0, 0), *(torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (coords, tv, radii)), out)
    want = port.forward_vector(og, (0, 0, 0), coords, tv, radii)
    # N terms of at most one a voxel in any order: a rounding of the running sum each
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-5, atol=2e-6 * max(1.0, N / 50))
