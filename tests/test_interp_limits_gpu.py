"""GridInterpolater at its limits: more channels than a launch has blocks, maps that have no use."""
import ctypes

import pytest
import torch

import libmolgrid_b200 as lmg

pytestmark = pytest.mark.gpu


def test_a_refused_launch_is_not_found_again(lib):
    """2^21 channels ask for a launch of more blocks than an axis has unless they are shared out; refused or not, the next
    call is none the worse."""
    K = 65535 * 32 + 40
    gi = lmg.GridInterpolater(1.0, 1.0, 1.0, 1.0)
    a, b = torch.zeros((K, 2, 2, 2), device="cuda"), torch.zeros((K, 2, 2, 2), device="cuda")
    try:
        gi.backward(a, lmg.Transform(), b)
    except RuntimeError:
        pass
    x = torch.rand((10, 3), device="cuda")
    y = torch.empty_like(x)
    from libmolgrid_b200 import _cabi
    t = lmg.Transform().struct()
    _cabi.check(lib.lmg_transform_forward(ctypes.byref(t), 10, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(y.data_ptr()), 1, None))
    torch.cuda.synchronize()
    assert torch.equal(x, y)


@pytest.mark.parametrize("more", [-40, 0, 1, 40])
def test_backward_of_many_channels(more):
    """Channels beyond 65535 blocks of 32: all of them come through, with the identity unchanged."""
    K = 65535 * 32 + more
    gi = lmg.GridInterpolater(1.0, 1.0, 1.0, 1.0)
    g = torch.rand((K, 2, 2, 2), device="cuda")
    out = torch.full_like(g, 7.0)
    gi.backward(g, lmg.Transform(), out)
    assert torch.equal(g, out)
