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


@pytest.mark.parametrize("module", [lmg, molgrid])
@pytest.mark.parametrize("yes", [1, np.True_, np.bool_(True), "yes", [0]])
@pytest.mark.parametrize("no", [0, np.False_, ""])
def test_want_type_gradients_is_a_truth_value(module, yes, no):
    gm = module.GridMaker(0.5, 5.5)
    diff = torch.rand(gm.grid_dimensions(T), device="cuda")
    want = [torch.empty(N, 3, device="cuda"), torch.empty(N, T, device="cuda")]
    args = inputs(True)
    lmg.GridMaker(0.5, 5.5).backward_arrays(*args, diff, *want)
    for flag, filled in ((yes, True), (no, False)):
        ag, tg = torch.full((N, 3), 7.0, device="cuda"), torch.full((N, T), 7.0, device="cuda")
        call = gm.backward if module is lmg else gm.backward_arrays
        call(*args, diff, ag, tg, want_type_gradients=flag)
        assert torch.allclose(ag, want[0], rtol=1e-5, atol=1e-6)
        assert torch.allclose(tg, want[1], rtol=1e-5, atol=1e-6) if filled else bool((tg == 7.0).all())


def test_words_that_a_call_does_not_know_are_refused():
    gm = lmg.GridMaker(0.5, 5.5)
    grid = torch.rand(gm.grid_dimensions(T), device="cuda")
    args, vec = inputs(), inputs(True)
    ag, tg, rel = torch.empty(N, 3, device="cuda"), torch.empty(N, T, device="cuda"), torch.empty(N, device="cuda")
    for word in ("want_type_gradients", "type_gradients"):
        for value in (None, True):
            with pytest.raises(TypeError):
                gm.forward(*args, grid, **{word: value})
            with pytest.raises(TypeError):
                gm.backward_relevance(*args, grid, grid, rel, **{word: value})
    with pytest.raises(TypeError):
        gm.backward(*vec, grid, ag, tg, type_gradients=tg)
    with pytest.raises(TypeError):
        gm.backward(*vec, grid, ag, None, type_gradients=tg)
