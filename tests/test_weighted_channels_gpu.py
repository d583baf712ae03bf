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
