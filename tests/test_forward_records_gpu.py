"""Densities of index types at the atom counts from which they are gridded from records instead of by warps that prepare their
own atom: against the CPU oracle and against the sums by single voxels."""
import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg
from libmolgrid_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,B,N,ragged", [(13, 6, 1999, False), (13, 6, 2000, False), (13, 4, 5000, True), (13, 4, 4999, True),
                                               (12, 7, 2000, False), (12, 7, 1999, False), (17, 4, 3000, False), (18, 12, 1000, False),
                                               (13, 10, 1999, False), (13, 10, 2000, False), (14, 5, 4000, False),
                                               (13, 6, 4000, True), (13, 6, 3999, True)])
def test_densities_at_the_lines(port, points, B, N, ragged):
    T, res = 5, 0.5 if ragged and N in (3999, 4000) else 1.0
    side = (points - 1) * res
    rng = np.random.default_rng(points * N)
    coords = rng.uniform(-side / 2 - 1, side / 2 + 1, (B, N, 3)).astype(np.float32)
    types = rng.integers(-1, T, (B, N)).astype(np.float32)
    radii = rng.uniform(1.0, 2.0, (B, N)).astype(np.float32)
    n = [N - 1700 * b if ragged else N for b in range(B)]
    more = dict(n_atoms=torch.tensor(n, dtype=torch.int32, device="cuda").clamp_min(0)) if ragged else {}
    g, og = lmg.GridMaker(res, side), port.gm(res, side)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii)]
    out = []
    for quads in (1, 0):
        api._cabi.lib().lmg_set_quads(quads)
        try:
            out.append(torch.full((B,) + tuple(g.grid_dimensions(T)), 7.0, device="cuda"))
            g.forward(torch.zeros(B, 3, device="cuda"), *data, out[-1], **more)
        finally:
            api._cabi.lib().lmg_set_quads(1)
    # up to some hundred densities a voxel, each within 3e-7, summed in any order
    scale = float(out[1].max())
    assert torch.allclose(out[0], out[1], rtol=1e-5, atol=1e-6 * scale)
    for b in (0, B - 1):
        m = max(n[b], 0)
        want = port.forward_index(og, (0, 0, 0), coords[b, :m], types[b, :m], radii[b, :m], T)
        np.testing.assert_allclose(out[0][b].cpu().numpy(), want, rtol=1e-5, atol=1e-6 * scale)
