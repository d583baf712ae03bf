"""What the native route of calls on resident tensors leaves to the general one."""
import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg
import molgrid
from libmolgrid_b200 import api

pytestmark = pytest.mark.gpu
N, T = 5, 3


def inputs(vec=False):
    c = torch.rand(N, 3, device="cuda")
    t = torch.rand(N, T, device="cuda") if vec else torch.zeros(N, device="cuda")
    return [(0.0, 0.0, 0.0), c, t, torch.ones(N, device="cuda")]


@pytest.mark.parametrize("module", [lmg, molgrid])
def test_tensors_without_memory_of_their_own_are_refused(module):
    """An error, not the end of the process: nested tensors, those inside vmap, fake ones."""
    gm = module.GridMaker(0.5, 5.5)
    out = torch.empty(gm.grid_dimensions(T), device="cuda")
    good = inputs()
    nested = torch.nested.nested_tensor([torch.rand(2, 3, device="cuda"), torch.rand(3, 3, device="cuda")])
    with pytest.raises((RuntimeError, TypeError, ValueError, IndexError)):
        gm.forward(good[0], nested, *good[2:], out)
    with pytest.raises((RuntimeError, TypeError, ValueError, IndexError)):
        torch.vmap(lambda c: gm.forward(good[0], c, good[2], good[3], out) or c)(torch.rand(4, N, 3, device="cuda"))
    with torch._subclasses.FakeTensorMode():
        fake = torch.empty(N, 3, device="cuda")
    with pytest.raises((RuntimeError, TypeError, ValueError, IndexError)):
        gm.forward(good[0], fake, *good[2:], out)
    gm.forward(*good, out)
    torch.cuda.synchronize()


def test_numbers_beyond_a_double():
    gm = lmg.GridMaker(0.5, 5.5)
    out = torch.empty(gm.grid_dimensions(T), device="cuda")
    with pytest.raises((OverflowError, RuntimeError, TypeError, ValueError)):
        gm.forward((10 ** 400, 0.0, 0.0), *inputs()[1:], out)
