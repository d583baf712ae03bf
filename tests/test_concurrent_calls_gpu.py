"""Calls of the array interface that are under way together: several streams of a thread, several threads of a stream, and
scratch memory that is given up meanwhile."""
import threading

import pytest
import torch

import libmolgrid_b200 as lmg
import libmolgrid_b200.api as api
import molgrid

pytestmark = pytest.mark.gpu
T = 6


class Work(object):
    """Inputs of one caller, what they give when nothing else is under way, and a pass over them."""

    def __init__(self, seed, N, vec):
        g = torch.Generator(device="cuda").manual_seed(seed)
        B = 3
        self.gm = (molgrid if vec else lmg).GridMaker(0.5, 11.5)
        self.c = torch.randn(B, N, 3, device="cuda", generator=g) * 3
        self.t = torch.rand(B, N, T, device="cuda", generator=g) if vec else torch.randint(T, (B, N), device="cuda", generator=g).float()
        self.r = torch.rand(B, N, device="cuda", generator=g) + 1
        self.d = torch.randn((B,) + tuple(self.gm.grid_dimensions(T)), device="cuda", generator=g)
        self.vec = vec
        torch.cuda.synchronize()
        self.want = self.run()
        torch.cuda.synchronize()

    def run(self):
        out, ag, tg = torch.empty_like(self.d), torch.empty_like(self.c), torch.empty_like(self.t)
        self.gm.forward((0.0, 0.0, 0.0), self.c, self.t, self.r, out)
        if self.vec:
            self.gm.backward((0.0, 0.0, 0.0), self.c, self.t, self.r, self.d, ag, tg)
            return out, ag, tg
        self.gm.backward((0.0, 0.0, 0.0), self.c, self.t, self.r, self.d, ag)
        return out, ag

    def check(self, got):
        for a, b in zip(got, self.want):  # sums of a voxel in any order
            assert torch.allclose(a, b, rtol=1e-4, atol=1e-4)


# beyond the sizes whose warps prepare their own atoms, so that the calls have records in scratch memory
@pytest.mark.parametrize("vec", [False, True])
def test_streams_of_a_thread(vec):
    works = [Work(s, n, vec) for s, n in ((1, 12000), (2, 15000), (3, 13000))]
    streams = [torch.cuda.Stream() for _ in works]
    got = []
    for _ in range(6):
        for w, s in zip(works, streams):
            with torch.cuda.stream(s):
                got.append((w, w.run()))
    torch.cuda.synchronize()
    for w, out in got:
        w.check(out)


@pytest.mark.parametrize("own_streams", [False, True])
def test_threads(own_streams):
    """Each drops its scratch memory now and then, as one that needs more does."""
    works = [Work(4 + i, n, i == 2) for i, n in enumerate((12000, 15000, 13000))]
    errors = []

    def loop(w):
        try:
            with torch.cuda.stream(torch.cuda.Stream() if own_streams else torch.cuda.default_stream()):
                got = []
                for i in range(8):
                    if i % 3 == 2:
                        api._workspaces.clear()
                    got.append(w.run())
                torch.cuda.current_stream().synchronize()
                for out in got:
                    w.check(out)
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(w,)) for w in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_scratch_memory_is_bounded():
    w = Work(9, 12000, False)
    streams = [torch.cuda.Stream() for _ in range(20)]
    for s in streams:
        with torch.cuda.stream(s):
            w.run()
    torch.cuda.synchronize()
    assert 1 <= len(api._workspaces.by) <= api._Workspaces.KEPT
    other = []
    t = threading.Thread(target=lambda: other.append(len(api._workspaces.by)))
    t.start()
    t.join()
    assert other == [0]


def test_captured_calls_have_their_own():
    """A graph's scratch memory is not that of later calls on the stream it was captured on."""
    w, x = Work(10, 12000, False), Work(11, 15000, False)
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(s):
        w.run()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        out = w.run()
    with torch.cuda.stream(s):
        later = x.run()
    g.replay()
    torch.cuda.synchronize()
    w.check(out)
    x.check(later)


def test_threads_that_end_give_their_scratch_memory_back():
    """Calls of the compiled module on the default stream, from threads that come and go."""
    gm = molgrid.GridMaker(0.5, 11.5)
    N, B = 40000, 8
    c, t, r = torch.zeros(B, N, 3, device="cuda"), torch.zeros(B, N, device="cuda"), torch.ones(B, N, device="cuda")
    out, cen = torch.empty((B,) + tuple(gm.grid_dimensions(2)), device="cuda"), torch.zeros(B, 3, device="cuda")

    def call():
        gm.forward(cen, c, t, r, out)
        torch.cuda.synchronize()

    def once():
        w = threading.Thread(target=call)
        w.start()
        w.join()

    once()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(20):
        once()
    assert free - torch.cuda.mem_get_info()[0] < 3 * B * N * 64    # each call takes 64 bytes an atom
