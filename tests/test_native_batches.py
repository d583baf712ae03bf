"""Batches of examples made by the compiled module from raw records, against the Python layer's
typing of the same files; and the pinned route of GridMaker.forward(ExampleVec) on the GPU."""
import numpy as np
import pytest


def _lists(tmp_path, natoms, lines):
    from libmolgrid_b200.coord_cache import write_gninatypes
    rng = np.random.default_rng(natoms)
    rows = []
    for i in range(lines):
        for kind, n in (("r", natoms), ("l", max(natoms // 8, 0))):
            # all record types, unknown ones (above 27) and types the default groupings leave out
            write_gninatypes(tmp_path / ("%s%d.gninatypes" % (kind, i)), rng.normal(size=(n, 3)) * 4, rng.integers(0, 33, n))
        rows.append("%d %.2f r%d.gninatypes %s" % (i % 2, i * 0.5, i, "none" if i == 1 else "l%d.gninatypes" % i))
    (tmp_path / "s.types").write_text("\n".join(rows) + "\n")


# no atoms, one, sizes on both sides of where a batch is shared among threads (8192 records)
@pytest.mark.parametrize("natoms,lines", [(0, 2), (1, 3), (1200, 6), (1300, 6)])
def test_examples_from_records(tmp_path, natoms, lines):
    import libmolgrid_b200 as lmg
    import molgrid
    _lists(tmp_path, natoms, lines)
    pn, pp = molgrid.ExampleProvider(data_root=str(tmp_path)), lmg.ExampleProvider(data_root=str(tmp_path))
    for p in (pn, pp):
        p.populate(str(tmp_path / "s.types"))
    for _ in range(2):
        bn, bp = pn.next_batch(lines), pp.next_batch(lines)
        for a, b in zip(bn, bp):
            assert list(a.labels) == [np.float32(v) for v in b.labels] and len(a.coord_sets) == len(b.coord_sets)
            for s, t in zip(a.coord_sets, b.coord_sets):
                assert (s.size(), s.max_type) == (t.size(), t.max_type)
                if t.size():
                    np.testing.assert_array_equal(s.coords.tonumpy(), t.coords.tonumpy())
                    np.testing.assert_array_equal(s.type_index.tonumpy(), t.type_index.tonumpy())
                    np.testing.assert_array_equal(s.radii.tonumpy(), t.radii.tonumpy())
        if natoms:  # an example's arrays are its own
            before = pn._native_line(0)
            bn[0].coord_sets[0].coords[0, 0] = 99.0
            again = molgrid.native._make_examples([before])
            assert again[0].coord_sets[0].coords[0, 0] != 99.0


@pytest.mark.gpu
@pytest.mark.parametrize("stream", [False, True])
def test_example_batches_on_a_stream(tmp_path, stream):
    """Batches of changing size in a row, nothing waited for in between, on torch's default stream and
    on another one: every grid and label as from one example at a time."""
    import torch
    import molgrid
    _lists(tmp_path, 400, 6)
    gm = molgrid.GridMaker(0.5, 11.5)
    prov = molgrid.ExampleProvider(data_root=str(tmp_path))
    prov.populate(str(tmp_path / "s.types"))
    s = torch.cuda.Stream() if stream else torch.cuda.current_stream()
    got = []
    with torch.cuda.stream(s):
        for size in (1, 6, 3, 6, 2, 6, 5):
            batch = prov.next_batch(size)
            out = torch.full((size,) + gm.grid_dimensions(prov.num_types()), 7.0, device="cuda")
            lab = torch.full((size, 2), 7.0, device="cuda")
            batch.extract_labels(lab)
            gm.forward(batch, out, 0.0, False)
            got.append((batch, out.clone(), lab.clone()))
    torch.cuda.synchronize()
    for batch, out, lab in got:
        for i, ex in enumerate(batch):
            one = torch.zeros(out.shape[1:], device="cuda")
            gm.forward(ex, one)
            # reductions of the same terms in another order: a few roundings of the largest value
            assert torch.allclose(out[i], one, rtol=1e-5, atol=1e-6)
            assert lab[i].tolist() == list(ex.labels)


def _provider(tmp_path):
    import molgrid
    p = molgrid.ExampleProvider(data_root=str(tmp_path))
    p.populate(str(tmp_path / "s.types"))
    return p


def test_batches_follow_settings_typers_and_caches(tmp_path):
    """What a provider's settings, typers, lines and loaded structures are when a batch is asked for, not when its lines were
    first seen."""
    import libmolgrid_b200 as lmg
    import molgrid
    _lists(tmp_path, 40, 3)
    p = _provider(tmp_path)
    before = p.next_batch(3)
    # structures loaded after the first use take the place of those read before
    (tmp_path / "other").mkdir()
    _lists(tmp_path / "other", 16, 3)
    q = molgrid.ExampleProvider(data_root=str(tmp_path / "other"))
    q.populate(str(tmp_path / "other" / "s.types"))
    theirs = q.next_batch(3)
    q.save_mem_caches(str(tmp_path / "mem"))
    p.load_mem_caches(str(tmp_path / "mem"))
    now = p.next_batch(3)
    for a, b, c in zip(now, theirs, before):
        assert a.num_coordinates() == b.num_coordinates() != c.num_coordinates()
    # labels of a line
    p.refs[0].labels = [5.0, 6.0]
    p.reset()
    assert list(p.next_batch(3)[0].labels) == [5.0, 6.0]
    # another typer
    p.caches[0].typer = lmg.GninaIndexTyper()
    p.reset()
    assert p.next_batch(3)[0].coord_sets[0].max_type == 28
    # type vectors from now on
    p.settings.make_vector_types = True
    p.reset()
    batch = p.next_batch(3)
    assert batch[0].coord_sets[0].type_vector.size() > 0 and batch[0].coord_sets[0].type_index.size() == 0


def test_a_provider_of_ones_own(tmp_path):
    """Examples that a derived class makes are in its batches too."""
    import molgrid

    class Relabelled(molgrid.ExampleProvider):
        def _make(self, ref):
            ex = molgrid.ExampleProvider._make(self, ref)
            ex.labels = [42.0]
            return ex

    class Every(molgrid.ExampleProvider):
        def next(self):
            ex = molgrid.ExampleProvider.next(self)
            ex.group = 9
            return ex

    _lists(tmp_path, 10, 3)
    for cls in (Relabelled, Every):
        p = cls(data_root=str(tmp_path))
        p.populate(str(tmp_path / "s.types"))
        for ex in p.next_batch(3):
            assert list(ex.labels) == [42.0] if cls is Relabelled else ex.group == 9


def test_a_line_that_cannot_be_read_is_not_skipped_with_others(tmp_path):
    """The example after a missing file is the next one."""
    _lists(tmp_path, 10, 4)
    (tmp_path / "r1.gninatypes").unlink()
    p = _provider(tmp_path)
    with pytest.raises(ValueError):
        p.next_batch(3)
    assert list(p.next_batch(1)[0].labels) == [0.0, 1.0]     # line 2
