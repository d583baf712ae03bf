"""Gradients of type vectors with radii by atom where the grid gradient is copied with the channels of a voxel next to each
other (many atoms a grid): against the CPU oracle and against the kernels that read it where it lies, at the edges of the
copy's channels and voxels, for atoms with none to many weighted channels."""
import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg
from libmolgrid_b200 import api

pytestmark = pytest.mark.gpu


def _batch(seed, B, N, T, side):
    rng = np.random.default_rng(seed)
    coords = rng.uniform(-side / 2 - 1, side / 2 + 1, (B, N, 3)).astype(np.float32)
    radii = rng.uniform(1.0, 2.2, (B, N)).astype(np.float32)
    types = np.zeros((B, N, T), np.float32)
    for b in range(B):
        for a in range(N):
            k = (0, 1, 2, 4, 5, T)[a % 6]
            types[b, a, rng.permutation(T)[:k]] = rng.uniform(0.1, 1, k)
    return coords, types, radii


def _close(got, want):
    # sums of up to some hundred terms in another order, as for the other gradients
    np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(want).max())))


def _between_guards(shape):
    """A tensor of sevens and the floats around it, which no call writes."""
    n = int(np.prod(shape))
    room = torch.full((n + 64,), 7.0, device="cuda")
    return room[32:32 + n].view(shape), (room[:32], room[32 + n:])


def _gradients(g, data, diff, quads=1, **more):
    lib = api._cabi.lib()
    ag, around_ag = _between_guards(data[0].shape)
    tg, around_tg = _between_guards(data[1].shape)
    lib.lmg_set_quads(quads)
    try:
        g.backward(torch.zeros(len(ag), 3, device="cuda"), *data, diff, ag, tg, **more)
    finally:
        lib.lmg_set_quads(1)
    assert all(bool((x == 7.0).all()) for x in around_ag + around_tg)
    return ag.cpu().numpy(), tg.cpu().numpy()


def _copied(g, B, N, T, counted):
    """Whether the call is one that goes by copies: then its scratch has room for them."""
    from libmolgrid_b200 import _cabi
    return g._bytes(_cabi.OP_BACKWARD_TYPES_COUNTED if counted else _cabi.OP_BACKWARD_TYPES, B, N, T, True) > g._bytes(_cabi.OP_BACKWARD, B, N, T, True)


@pytest.mark.parametrize("points,T,B,N", [(25, 8, 10, 200), (25, 9, 9, 200), (25, 16, 7, 200), (25, 17, 5, 200), (25, 24, 4, 200),
                                          (25, 25, 4, 200), (25, 32, 4, 200), (24, 29, 15, 700), (24, 25, 8, 1700), (24, 28, 7, 1700),
                                          (13, 31, 9, 200), (25, 32, 3, 200), (24, 17, 7, 2800), (13, 31, 3, 200)])
@pytest.mark.parametrize("binary,multiple", [(False, 1.0), (True, 1.0), (False, -1.5)])
def test_copies(port, points, T, B, N, binary, multiple):
    coords, types, radii = _batch(points * T, B, N, T, points - 1.0)
    g = lmg.GridMaker(1.0, points - 1.0, binary, gaussian_radius_multiple=multiple)
    og = port.gm(1.0, points - 1.0, binary, gaussian_radius_multiple=multiple)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii)]
    shape = (B,) + tuple(g.grid_dimensions(T))
    diff = torch.randn(shape, device="cuda")
    assert _copied(g, B, N, T, True) == ((points, T, B) not in ((25, 32, 3), (24, 17, 7), (13, 31, 3)))
    n = torch.tensor([N - 3 * b for b in range(B)], dtype=torch.int32, device="cuda")
    ag, tg = _gradients(g, data, diff, n_atoms=n)
    for a, b in zip((ag, tg), _gradients(g, data, diff, quads=0, n_atoms=n)):
        _close(a, b)
    for b in (0, B - 1):
        m = N - 3 * b
        wag, wtg = port.backward_vector(og, (0, 0, 0), coords[b, :m], types[b, :m], radii[b, :m], diff[b].cpu().numpy())
        _close(ag[b, :m], wag)
        _close(tg[b, :m], wtg)
        assert not ag[b, m:].any() and not tg[b, m:].any()
    again = _gradients(g, data, diff, n_atoms=n)
    assert np.array_equal(ag, again[0]) and np.array_equal(tg, again[1])
    # the same floats off a 16-byte boundary, and a workspace that has no room for copies
    loose = torch.empty(diff.numel() + 1, device="cuda")[1:].view(shape).copy_(diff)
    old = api.MAX_WORKSPACE_BYTES
    try:
        for d, room in ((loose, old), (diff, 2 * (N * (64 + 12 * T) + 4096))):
            api.MAX_WORKSPACE_BYTES = room
            api._workspaces.clear()
            for a, b in zip(_gradients(g, data, d, n_atoms=n), (ag, tg)):
                _close(a, b)
    finally:
        api.MAX_WORKSPACE_BYTES = old
        api._workspaces.clear()


def test_several_copies_and_one_example_more():
    """More examples than are copied at a time, the last copy of a single one."""
    points, T, N = 65, 32, 1400
    each = (points ** 3 + 1) * 128
    B = (256 << 20) // each + 1
    coords, types, radii = _batch(3, B, N, T, 32.0)
    g = lmg.GridMaker(0.5, 32.0)
    assert _copied(g, B, N, T, False)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii)]
    diff = torch.randn((B,) + tuple(g.grid_dimensions(T)), device="cuda")
    for a, b in zip(_gradients(g, data, diff), _gradients(g, data, diff, quads=0)):
        _close(a, b)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_values_beyond_reach_and_without_weight(value):
    """Values that are no numbers, in voxels that no atom reaches and in channels without weight."""
    points, T, B, N = 25, 14, 6, 200
    coords, types, radii = _batch(5, B, N, T, 8.0)
    types[:, :, 3] = 0
    g = lmg.GridMaker(1.0, points - 1.0)
    assert _copied(g, B, N, T, False)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii)]
    diff = torch.randn((B,) + tuple(g.grid_dimensions(T)), device="cuda")
    ag, tg = _gradients(g, data, diff)
    diff[:, :, :2], diff[:, :, :, :2], diff[..., :2], diff[..., -2:] = value, value, value, value
    diff[:, 3] = value
    ag2, tg2 = _gradients(g, data, diff)
    assert np.isfinite(ag2).all()
    _close(ag2, ag)
    keep = [t for t in range(T) if t != 3]
    _close(tg2[..., keep], tg[..., keep])
    assert not np.isfinite(tg2[..., 3]).any()


@pytest.mark.parametrize("points,T,B,N", [(25, 8, 10, 200), (25, 14, 6, 200), (24, 29, 15, 700)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_atoms_without_weight_take_no_channel(points, T, B, N, value):
    """The first channel is no number anywhere and carries no weight: atoms without any weight have exactly no gradient."""
    coords, types, radii = _batch(points + T, B, N, T, points - 1.0)
    types[:, :, 0] = 0
    g = lmg.GridMaker(1.0, points - 1.0)
    assert _copied(g, B, N, T, False)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii)]
    diff = torch.randn((B,) + tuple(g.grid_dimensions(T)), device="cuda")
    ag, tg = _gradients(g, data, diff)
    diff[:, 0] = value
    ag2, tg2 = _gradients(g, data, diff)
    assert not ag2[~types.any(-1)].any()
    _close(ag2, ag)
    _close(tg2[..., 1:], tg[..., 1:])


def test_workspace_off_the_boundary_of_the_copies():
    """A workspace 16 bytes off a 32-byte boundary takes the kernels that need no copies."""
    import ctypes
    from libmolgrid_b200 import _cabi
    lib, points, T, B, N = _cabi.lib(), 25, 16, 7, 200
    coords, types, radii = _batch(11, B, N, T, points - 1.0)
    g = lmg.GridMaker(1.0, points - 1.0)
    assert _copied(g, B, N, T, False)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii)]
    diff = torch.randn((B,) + tuple(g.grid_dimensions(T)), device="cuda")
    want = _gradients(g, data, diff)
    a = _cabi.AtomsStruct()
    a.batch, a.max_atoms, a.ntypes = B, N, T
    a.coords, a.type_vector, a.radii = (t.data_ptr() for t in data)
    need = lib.lmg_workspace_bytes(ctypes.byref(g.s), _cabi.OP_BACKWARD_TYPES, B, N, T, 1)
    room = torch.empty(need + 64, dtype=torch.uint8, device="cuda")
    for off in (0, 16):
        ag, tg = torch.full((B, N, 3), 7.0, device="cuda"), torch.full((B, N, T), 7.0, device="cuda")
        rc = lib.lmg_backward(ctypes.byref(g.s), ctypes.byref(a), diff.data_ptr(), ag.data_ptr(), tg.data_ptr(),
                              room.data_ptr() + off, need, torch.cuda.current_stream().cuda_stream)
        assert rc == 0, lib.lmg_last_error()
        _close(ag.cpu().numpy(), want[0])
        _close(tg.cpu().numpy(), want[1])


@pytest.mark.parametrize("T", [17, 32])
def test_a_grid_without_points(T):
    """No voxel: every gradient is zero, whatever the number of atoms."""
    import ctypes
    from libmolgrid_b200 import _cabi
    lib, N = _cabi.lib(), 20000
    g = lmg.GridMaker(1.0, -1.0)
    assert g.s.dim == 0
    data = [torch.randn(1, N, 3, device="cuda"), torch.rand(1, N, T, device="cuda"), torch.rand(1, N, device="cuda") + 1]
    a = _cabi.AtomsStruct()
    a.batch, a.max_atoms, a.ntypes = 1, N, T
    a.coords, a.type_vector, a.radii = (t.data_ptr() for t in data)
    need = lib.lmg_workspace_bytes(ctypes.byref(g.s), _cabi.OP_BACKWARD_TYPES, 1, N, T, 1)
    room, ag, tg = torch.empty(need, dtype=torch.uint8, device="cuda"), torch.full_like(data[0], 7.0), torch.full_like(data[1], 7.0)
    rc = lib.lmg_backward(ctypes.byref(g.s), ctypes.byref(a), room.data_ptr(), ag.data_ptr(), tg.data_ptr(), room.data_ptr(), need,
                          torch.cuda.current_stream().cuda_stream)
    assert rc == 0, lib.lmg_last_error()
    assert not ag.any() and not tg.any()


def test_room_for_copies_short_by_a_byte():
    """Copies are made where they fit and nowhere else: nothing is written behind the workspace, and one byte less takes the
    kernels that need none (records and two launches more by copies, records, sums and their reduction without)."""
    import ctypes
    from libmolgrid_b200 import _cabi
    lib, points, T, B, N = _cabi.lib(), 25, 16, 7, 200
    coords, types, radii = _batch(12, B, N, T, points - 1.0)
    g = lmg.GridMaker(1.0, points - 1.0)
    assert _copied(g, B, N, T, False)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii)]
    diff = torch.randn((B,) + tuple(g.grid_dimensions(T)), device="cuda")
    a = _cabi.AtomsStruct()
    a.batch, a.max_atoms, a.ntypes = B, N, T
    a.coords, a.type_vector, a.radii = (t.data_ptr() for t in data)
    need = lib.lmg_workspace_bytes(ctypes.byref(g.s), _cabi.OP_BACKWARD_TYPES, B, N, T, 1)
    assert need > lib.lmg_workspace_bytes(ctypes.byref(g.s), _cabi.OP_BACKWARD, B, N, T, 1)
    out = []
    for size in (need, need - 1):
        room = torch.full((need + 4096,), 0xAB, dtype=torch.uint8, device="cuda")
        ag, tg = torch.full((B, N, 3), 7.0, device="cuda"), torch.full((B, N, T), 7.0, device="cuda")
        rc = lib.lmg_backward(ctypes.byref(g.s), ctypes.byref(a), diff.data_ptr(), ag.data_ptr(), tg.data_ptr(), room.data_ptr(), size,
                              torch.cuda.current_stream().cuda_stream)
        assert rc == 0, lib.lmg_last_error()
        assert bool((room[size:] == 0xAB).all())
        out.append((ag.cpu().numpy(), tg.cpu().numpy()))
    _close(out[0][0], out[1][0])
    _close(out[0][1], out[1][1])
    assert not np.array_equal(out[0][1], out[1][1])  # other kernels, other last bits


def test_no_memory_for_copies(monkeypatch):
    """Where the scratch of the copies cannot be had, that of the kernels that need none is enough."""
    points, T, B, N = 25, 16, 7, 200
    coords, types, radii = _batch(13, B, N, T, points - 1.0)
    g = lmg.GridMaker(1.0, points - 1.0)
    assert _copied(g, B, N, T, False)
    data = [torch.from_numpy(x).cuda() for x in (coords, types, radii)]
    diff = torch.randn((B,) + tuple(g.grid_dimensions(T)), device="cuda")
    want = _gradients(g, data, diff)
    from libmolgrid_b200 import _cabi
    least, real = g._bytes(_cabi.OP_BACKWARD, B, N, T, True), torch.empty

    def empty(*a, **k):
        if k.get("dtype") is torch.uint8 and a[0] > least:
            raise torch.OutOfMemoryError("no room")
        return real(*a, **k)
    api._workspaces.clear()
    monkeypatch.setattr(torch, "empty", empty)
    try:
        for _ in range(2):
            got = _gradients(g, data, diff)
            _close(got[0], want[0])
            _close(got[1], want[1])
    finally:
        api._workspaces.clear()
