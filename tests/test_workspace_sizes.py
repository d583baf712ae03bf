"""Scratch sizes that the Python layer asks for: those of the settings at the time of the call."""
import ctypes

import libmolgrid_b200 as lmg
from libmolgrid_b200 import _cabi, api


def test_sizes_follow_the_resolution(monkeypatch):
    """Type gradients by copies go by the resolution too: two resolutions of the same points do not share a size."""
    monkeypatch.setattr(api, "_workspace", lambda device, nbytes, *more: nbytes)
    g, B, N, T = lmg.GridMaker(1.0, 23.0), 8, 2000, 28
    ops = range(5)
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
