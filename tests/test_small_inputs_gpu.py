"""Passes whose warps prepare their own atoms, and the status flags they leave: sizes on both sides of
the limits between the kernels, against the CPU checker or the same input in a larger batch."""
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


# one atom; four warps an atom up to 1200 slots, one beyond; relevance changes at 2560, gradients at 8192
@pytest.mark.parametrize("B,N", [(1, 1), (3, 5), (1, 1200), (1, 1201), (8, 320), (8, 321), (8, 1024), (8, 1025)])
@pytest.mark.parametrize("binary", [False, True])
def test_every_size_against_the_checker(port, B, N, binary):
    T, P = 4, 12
    g, og = lmg.GridMaker(0.5, (P - 1) * 0.5, binary), port.gm(0.5, (P - 1) * 0.5, binary)
    ex = [cases.index_case(100 + b, N, T, 4.0) for b in range(B)]
    coords, types, radii = (np.stack([e[k] for e in ex]) for k in range(3))
    out = torch.full((B,) + g.grid_dimensions(T), 7.0, device="cuda")
    cen = torch.zeros((B, 3), device="cuda")
    g.forward(cen, dev(coords), dev(types), dev(radii), out)
    rng = np.random.default_rng(N)
    diff = rng.normal(size=out.shape).astype(np.float32)
    ag, rel = torch.full((B, N, 3), 7.0, device="cuda"), torch.full((B, N), 7.0, device="cuda")
    g.backward(cen, dev(coords), dev(types), dev(radii), dev(diff), ag)
    g.backward_relevance(cen, dev(coords), dev(types), dev(radii), out, dev(diff), rel)
    g.check_types()
    for b in (0, B - 1):
        want = port.forward_index(og, (0, 0, 0), coords[b], types[b], radii[b], T)
        got = out[b].cpu().numpy()
        if binary:
            np.testing.assert_array_equal(got, want)
        else:
            # up to N / T terms a voxel in any order: a rounding of the running sum each
            np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-6 * max(1.0, N / T / 50))
        wag = port.backward_index(og, (0, 0, 0), coords[b], types[b], radii[b], diff[b])
        np.testing.assert_allclose(ag[b].cpu().numpy(), wag, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wag).max())))
        wrel = port.backward_relevance(og, (0, 0, 0), coords[b], types[b], radii[b], got, diff[b])
        np.testing.assert_allclose(rel[b].cpu().numpy(), wrel, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(wrel).max())))


@pytest.mark.parametrize("N", [3, 1300, 9000])
@pytest.mark.parametrize("at", [0, 1, -1])
def test_status_of_every_pass(N, at):
    """A type beyond the channels is reported wherever it is, by the call that met it and by no later
    one, also when a workspace makes the call run in passes of unequal size."""
    import libmolgrid_b200.api as api
    B, T = 5, 3
    g = lmg.GridMaker(0.5, 5.5)
    coords = torch.zeros((B, N, 3), device="cuda")
    good = torch.ones((B, N), device="cuda")
    radii = torch.ones((B, N), device="cuda")
    cen = torch.zeros((B, 3), device="cuda")
    out = torch.empty((B,) + g.grid_dimensions(T), device="cuda")
    ag = torch.empty((B, N, 3), device="cuda")
    old = api.MAX_WORKSPACE_BYTES
    one = api._cabi.lib().lmg_workspace_bytes(g.s, 0, 1, N, T, 0)
    try:
        for limit in (old, 2 * one):
            api.MAX_WORKSPACE_BYTES = limit
            api._workspaces.clear()
            for b in (0, B - 1):
                bad = good.clone()
                bad[b, at] = T
                g.forward(cen, coords, bad, radii, out)
                with pytest.raises(IndexError):
                    g.check_types()
                g.forward(cen, coords, good, radii, out)
                g.check_types()
                g.backward(cen, coords, bad, radii, out, ag)
                with pytest.raises(ValueError):
                    g.check_types()
                g.backward(cen, coords, good, radii, out, ag)
                g.check_types()
    finally:
        api.MAX_WORKSPACE_BYTES = old
        api._workspaces.clear()


# whole channels, parts of channels and single planes per block; runs of more than one and two words of the mask;
# rows that start anywhere; atoms of one channel in several chunks of the search
@pytest.mark.parametrize("B,N,T,points,res", [(1, 40, 3, 24, 1.0), (3, 100, 50, 13, 0.5), (30, 9, 5, 11, 0.5), (1, 128, 2, 65, 0.0625),
                                              (75, 2100, 2, 10, 0.5), (1, 20, 2, 200, 0.1)])
@pytest.mark.parametrize("shift", [0, 1])
def test_occupancy_in_one_launch(port, B, N, T, points, res, shift):
    side = (points - 1) * res
    g, og = lmg.GridMaker(res, side, True), port.gm(res, side, True)
    ex = [cases.index_case(7 * b + N, N, T, 0.6 * side) for b in range(B)]
    coords, types, radii = (np.stack([e[k] for e in ex]) for k in range(3))
    if N > 2000:
        types[:] = 1.0                      # every atom in one channel
    ns = np.full(B, N, np.int32)
    ns[-1] = N - 1
    buf = torch.full((B * T * points ** 3 + shift,), 7.0, device="cuda")
    out = buf[shift:].view((B,) + g.grid_dimensions(T))
    g.forward(torch.zeros((B, 3), device="cuda"), dev(coords), dev(types), dev(radii), out, n_atoms=dev(ns))
    for b in {0, B - 1}:
        want = port.forward_index(og, (0, 0, 0), coords[b][:ns[b]], types[b][:ns[b]], radii[b][:ns[b]], T)
        np.testing.assert_array_equal(out[b].cpu().numpy(), want)
    assert shift == 0 or float(buf[0]) == 7.0


@pytest.mark.parametrize("B,N,P", [(1, 40, 12), (2, 900, 48), (3, 11000, 24), (2, 500, 41), (1, 7, 13)])
@pytest.mark.parametrize("binary", [False, True])
def test_calls_of_one_stream_keep_their_order(B, N, P, binary):
    """Kernels begin while the one before them drains: a chain of passes, each on the results of the one before,
    gives the same as with a synchronisation after every pass."""
    T = 4
    g = lmg.GridMaker(0.5, (P - 1) * 0.5, binary)
    gen = torch.Generator(device="cuda").manual_seed(N)
    start = torch.randn((B, N, 3), device="cuda", generator=gen) * 3
    types = torch.randint(T, (B, N), device="cuda", generator=gen).float()
    radii = torch.rand((B, N), device="cuda", generator=gen) + 1
    cen = torch.zeros((B, 3), device="cuda")
    results = []
    for between in (torch.cuda.synchronize, lambda: None):
        coords, out = start.clone(), torch.empty((B,) + g.grid_dimensions(T), device="cuda")
        ag, rel = torch.empty((B, N, 3), device="cuda"), torch.empty((B, N), device="cuda")
        grids = []
        torch.cuda.synchronize()
        for step in range(6):
            g.forward(cen, coords, types, radii, out)
            between()
            g.backward(cen, coords, types, radii, out, ag)
            between()
            g.backward_relevance(cen, coords, types, radii, out, out, rel)
            between()
            coords = coords + 1e-3 * torch.tanh(ag) + 1e-3 * torch.tanh(rel)[..., None]
            grids.append(out.clone())
            between()
        results.append((grids, coords))
    for a, b in zip(*[r[0] for r in results]):
        # sums of a voxel in any order; a voxel of occupancy may change sides by the rounding of the steps before
        off = (a - b).abs() > 1e-4 * (1 + a.abs())
        assert float(off.float().mean()) <= (1e-4 if binary else 0.0)
    assert float((results[0][1] - results[1][1]).abs().max()) < 1e-4


# flags of the first pass run past 256 bytes: 20 examples and 1, 500 and 24 of them to a pass
@pytest.mark.parametrize("B,N,fit", [(21, 4000, 20), (524, 4000, 500)])
def test_status_when_the_last_pass_is_small(B, N, fit):
    """The records of a small last pass stay clear of the flags of the passes before it: valid types give no
    error, and a bad one of the first pass is still reported after the last."""
    import libmolgrid_b200.api as api
    T = 2
    g = lmg.GridMaker(1.0, 3.0)
    gen = torch.Generator(device="cuda").manual_seed(B)
    coords = torch.rand((B, N, 3), device="cuda", generator=gen) * 3 - 1.5
    good = torch.randint(T, (B, N), device="cuda", generator=gen).float()
    radii = torch.ones((B, N), device="cuda")
    cen = torch.zeros((B, 3), device="cuda")
    out = torch.empty((B,) + g.grid_dimensions(T), device="cuda")
    ag = torch.empty((B, N, 3), device="cuda")
    old = api.MAX_WORKSPACE_BYTES
    try:
        api.MAX_WORKSPACE_BYTES = api._cabi.lib().lmg_workspace_bytes(g.s, 0, fit, N, T, 0)
        api._workspaces.clear()
        for b, a in ((None, None), (fit - 1, N - 1), (B - 1, 0)):
            types = good.clone()
            if b is not None:
                types[b, a] = T
            for call, error in ((lambda: g.forward(cen, coords, types, radii, out), IndexError),
                                (lambda: g.backward(cen, coords, types, radii, out, ag), ValueError)):
                call()
                if b is None:
                    g.check_types()
                else:
                    with pytest.raises(error):
                        g.check_types()
    finally:
        api.MAX_WORKSPACE_BYTES = old
        api._workspaces.clear()


def test_occupancy_of_large_spheres(port):
    """Radii of 155 to 192 voxels, where the exact test's roundings reach further along a grazed column than the
    positions' do: these four atoms have a column each that ends within that reach of a voxel."""
    P, res = 401, 0.1
    g, og = lmg.GridMaker(res, (P - 1) * res, True), port.gm(res, (P - 1) * res, True)
    assert g.grid_dimensions(1)[1] == P
    atoms = np.array([[-2.6152842044830322, -1.7248189449310303, 2.2062289714813232, 15.479239463806152],
                      [0.5863897800445557, 2.7818641662597656, 1.3268423080444336, 16.368009567260742],
                      [2.0464634895324707, -2.813606023788452, 1.333905577659607, 19.232105255126953],
                      [-2.0822806358337402, 1.2371628284454346, 2.695906639099121, 18.976465225219727]], np.float32)
    for a in atoms:
        coords, types, radii = a[None, :3], np.zeros(1, np.float32), a[3:]
        out = torch.empty(g.grid_dimensions(1), device="cuda")
        g.forward((0.0, 0.0, 0.0), dev(coords), dev(types), dev(radii), out)
        np.testing.assert_array_equal(out.cpu().numpy(), port.forward_index(og, (0, 0, 0), coords, types, radii, 1))


@pytest.mark.parametrize("full", [127, 128, 129, 400])
@pytest.mark.parametrize("passes", [False, True])
def test_occupancy_with_full_channels(port, full, passes):
    """Channels with more atoms than their blocks take (128 for passes this small), beside others that have few or
    none, in batches that run at once or in passes, with types beyond the channels and below them."""
    import libmolgrid_b200.api as api
    B, N, T, P = 40, 420, 9, 12
    g, og = lmg.GridMaker(0.5, (P - 1) * 0.5, True), port.gm(0.5, (P - 1) * 0.5, True)
    ex = [cases.index_case(31 * b + full, N, T, 4.0) for b in range(B)]
    coords, types, radii = (np.stack([e[k] for e in ex]) for k in range(3))
    types = np.where(types == 3, 4, types)
    for b in range(0, B, 3):
        where = np.random.default_rng(b).permutation(N - 15)
        types[b] = np.where(types[b] == 7, 8, types[b])
        types[b, where[:full]] = 7
    types[:, N - 15] = -1.0
    ns = np.full(B, N, np.int32)
    ns[1:] -= np.arange(B - 1, dtype=np.int32) % 5
    out = torch.full((B,) + g.grid_dimensions(T), 7.0, device="cuda")
    old = api.MAX_WORKSPACE_BYTES
    try:
        if passes:
            api.MAX_WORKSPACE_BYTES = api._cabi.lib().lmg_workspace_bytes(g.s, 0, 17, N, T, 0)
            api._workspaces.clear()
        args = (torch.zeros((B, 3), device="cuda"), dev(coords), dev(types), dev(radii), out)
        g.forward(*args, n_atoms=dev(ns))
        g.check_types()
        for b in range(B):
            want = port.forward_index(og, (0, 0, 0), coords[b][:ns[b]], types[b][:ns[b]], radii[b][:ns[b]], T)
            np.testing.assert_array_equal(out[b].cpu().numpy(), want)
        types[B - 1, 0] = T
        g.forward(args[0], args[1], dev(types), args[3], out, n_atoms=dev(ns))
        with pytest.raises(IndexError):
            g.check_types()
    finally:
        api.MAX_WORKSPACE_BYTES = old
        api._workspaces.clear()
