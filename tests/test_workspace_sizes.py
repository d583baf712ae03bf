"""Scratch sizes that the Python layer asks for: those of the settings at the time of the call."""
import ctypes

import pytest

import libmolgrid_b200 as lmg
from libmolgrid_b200 import _cabi, api


def test_sizes_follow_the_resolution(monkeypatch):
    """Type gradients by copies go by the resolution too: two resolutions of the same points do not share a size."""
    monkeypatch.setattr(api, "_workspace", lambda device, nbytes, *more: nbytes)
    g, B, N, T = lmg.GridMaker(1.0, 23.0), 8, 2000, 28
    ops = range(6)
    sizes = []
    for res in (1.0, 2.0, 1.0):
        g.set_resolution(res)
        g.set_dimension(23.0 * res)
        assert g.s.dim == 24
        sizes.append([g._ws("cuda:0", op, B, N, T, True) for op in ops])
        assert sizes[-1] == [_cabi.lib().lmg_workspace_bytes(ctypes.byref(g.s), op, B, N, T, 1) for op in ops]
    assert sizes[0] == sizes[2] != sizes[1]


def test_only_type_gradients_have_room_for_copies():
    """The scratch of atom gradients alone is that of records and partial sums, whatever the type gradients would take."""
    lib, g, B, N, T = _cabi.lib(), lmg.GridMaker(0.5, 23.5), 50, 3000, 28
    size = lambda op: lib.lmg_workspace_bytes(ctypes.byref(g.s), op, B, N, T, 1)
    assert size(_cabi.OP_BACKWARD) < B * N * (64 + 12 * T) + (1 << 20)
    assert size(_cabi.OP_BACKWARD) < size(_cabi.OP_BACKWARD_TYPES) < size(_cabi.OP_BACKWARD) + (257 << 20)
    few = [lib.lmg_workspace_bytes(ctypes.byref(g.s), op, 1, 20, T, 1) for op in (_cabi.OP_BACKWARD, _cabi.OP_BACKWARD_TYPES)]
    assert few[0] == few[1]


# points, resolution, channels, examples, slots; copies without and with counts
@pytest.mark.parametrize("points,res,T,B,N,plain,counted", [
    (41, 0.5, 14, 40, 1500, True, True), (41, 0.5, 14, 1, 1500, True, False), (41, 0.5, 14, 8, 207, True, False), (41, 0.5, 14, 8, 206, False, False),
    (41, 0.5, 14, 8, 345, True, True), (41, 0.5, 14, 8, 340, True, False), (41, 0.5, 7, 40, 1500, False, False), (57, 0.5, 28, 1, 2223, True, True), (57, 0.5, 28, 1, 2222, True, False), (57, 0.5, 28, 1, 926, False, False),
    (48, 0.5, 28, 50, 3000, True, False), (24, 1.0, 28, 8, 2000, True, True), (48, 0.5, 32, 8, 700, True, True), (48, 0.5, 32, 8, 690, False, False), (48, 0.5, 24, 50, 3000, False, False),
    (48, 0.5, 33, 50, 3000, False, False)])
def test_which_calls_go_by_copies(points, res, T, B, N, plain, counted):
    """Copies of examples whose slots may be empty pay later: the slots a voxel count, on aligned rows and on others."""
    lib, g = _cabi.lib(), lmg.GridMaker(res, (points - 1) * res)
    size = lambda op: lib.lmg_workspace_bytes(ctypes.byref(g.s), op, B, N, T, 1)
    assert (size(_cabi.OP_BACKWARD_TYPES) > size(_cabi.OP_BACKWARD)) == plain
    assert (size(_cabi.OP_BACKWARD_TYPES_COUNTED) > size(_cabi.OP_BACKWARD)) == counted
