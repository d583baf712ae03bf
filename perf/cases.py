"""The gridding path's workloads for timing: what users of this package have it do, one pass each.

A case is a dict of plain values; ``path`` says which part of the interface it goes through:

* ``grid``: atoms with index types through ``GridMaker`` - ``op`` is ``forward`` (one density grid per
  example), ``train`` (forward, then the atom gradients of a grid gradient) or ``relevance``.  ``batch`` 0
  is the one-example overload of ``molgrid``, a positive one the batched call with a random rotation and
  translation per example and ragged atom counts.
* ``autograd``: type vectors through ``Coords2Grid`` - first derivatives, or second ones too.
* ``interpolate``: ``GridInterpolater``, with its backward pass or without.
* ``provider``: example lists on disk through ``ExampleProvider`` to grids, as ``device`` batches or as
  ``objects`` (``next_batch``, the reference's way).

Grids have ``points`` voxels a side, ``resolution`` Angstrom apart.  Atoms lie in a ball of 12 A about the
centre, ``blob`` of them (a share) in a pocket of 4 A; radii are per type, uniform in [1.2, 2.2] A.
"""
import math
import os
import tempfile

import numpy as np
import torch

import libmolgrid_b200 as lmg
import molgrid
from libmolgrid_b200.coord_cache import write_gninatypes


def listed():
    grid = dict(path="grid", op="train", batch=50, min_atoms=2000, max_atoms=4000, types=28, points=48,
                resolution=0.5, binary=False, blob=0.7)
    auto = dict(path="autograd", batch=50, atoms=3000, types=28, points=48, resolution=0.5, soft=False,
                radii_by_type=False, second=False, blob=0.7)
    interp = dict(path="interpolate", batch=48, channels=28, in_points=48, out_points=48, resolution=0.5,
                  backward=False)
    return [
        # one ligand on a coarse grid: scoring a pose at a time, nothing but latency
        dict(grid, name="ligand", op="forward", batch=0, min_atoms=40, max_atoms=40, types=14, points=24,
             resolution=1.0, blob=1.0),
        # one small complex, forward and atom gradients: optimising a pose
        dict(grid, name="pose", batch=0, min_atoms=300, max_atoms=300, blob=0.0),
        # the training batch of a docking network with gradients to the atoms
        dict(grid, name="train batch"),
        # occupancy grids of the same batch
        dict(grid, name="binary batch", op="forward", binary=True),
        # per-atom relevance for the same batch: what a network looked at
        dict(grid, name="relevance batch", op="relevance"),
        # a box of 20 A: 41 points a side, rows of no convenient alignment, ligands beside pockets
        dict(grid, name="odd box", batch=17, min_atoms=37, max_atoms=1503, types=22, points=41, blob=0.4),
        # rescoring a library: as many examples as one call gets
        dict(grid, name="large batch", batch=1024),
        # atom types that a network learns: gradients to coordinates and to every type
        dict(auto, name="learned types"),
        # soft types with radii by type on a fine grid, with the second derivatives of a force match
        dict(auto, name="soft types", batch=4, points=96, resolution=0.25, soft=True, radii_by_type=True,
             second=True),
        # augmenting stored grids: a random rotation and translation each
        dict(interp, name="augment grids"),
        # one grid to a smaller odd one and the gradient back
        dict(interp, name="odd resample", batch=1, channels=14, in_points=49, out_points=41, backward=True),
        # example lists to input grids, the input side of a training step
        dict(path="provider", name="example lists", mode="objects", batch=50, examples=100, min_atoms=2000,
             max_atoms=3900, points=48, resolution=0.5),
    ]


def _spread(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["grid", "grid", "grid", "grid", "autograd", "autograd", "interpolate", "provider"])
    res = rng.choice([0.375, 0.5, 0.5, 0.5, 0.75, 1.0])
    points = rng.choice([24, 32, 40, 48, 48, 56, rng.randint(17, 65)])
    if path == "grid":
        batch = rng.choice([0, _spread(rng, 2, 256)])
        hi = _spread(rng, 16, 4000)
        op = rng.choice(["forward", "train", "train", "relevance"])
        return dict(path=path, op=op, batch=batch, min_atoms=max(8, hi // 2) if batch else hi, max_atoms=hi,
                    types=rng.randint(4, 36), points=points, resolution=res,
                    binary=op == "forward" and rng.random() < 0.4, blob=round(rng.uniform(0, 0.8), 2))
    if path == "autograd":
        soft = rng.random() < 0.5
        return dict(path=path, batch=_spread(rng, 1, 8 if soft else 50), atoms=_spread(rng, 16, 1500 if soft else 3000),
                    types=rng.randint(4, 32), points=points, resolution=max(res, 0.5), soft=soft,
                    radii_by_type=soft and rng.random() < 0.5, second=rng.random() < 0.4,
                    blob=round(rng.uniform(0, 0.8), 2))
    if path == "interpolate":
        return dict(path=path, batch=_spread(rng, 1, 64), channels=rng.randint(4, 32), in_points=points,
                    out_points=rng.choice([points, rng.randint(17, 57)]), resolution=res,
                    backward=rng.random() < 0.4)
    hi = _spread(rng, 100, 4000)
    return dict(path=path, mode=rng.choice(["device", "objects"]), batch=rng.randint(4, 64), examples=rng.randint(64, 100),
                min_atoms=hi // 2, max_atoms=hi, points=points, resolution=res)


# ---- inputs --------------------------------------------------------------------------------------

def _ball(g, shape, radius):
    v = torch.randn(*shape, 3, generator=g, device="cuda")
    r = torch.rand(*shape, 1, generator=g, device="cuda") ** (1 / 3)
    return v / v.norm(dim=-1, keepdim=True) * r * radius


def _positions(g, batch, n, blob):
    """(batch, n, 3): a share ``blob`` of each example in a 4 A pocket, the rest in the 12 A ball."""
    pocket = _ball(g, (batch, 1), 6.0)
    inside = torch.rand(batch, n, 1, generator=g, device="cuda") < blob
    return torch.where(inside, _ball(g, (batch, n), 4.0) + pocket, _ball(g, (batch, n), 12.0)).contiguous()


def _transforms(g, batch):
    """(batch, 10): unit quaternion, centre 0, translation within 2 A."""
    tr = torch.zeros(batch, 10, device="cuda")
    q = torch.randn(batch, 4, generator=g, device="cuda")
    tr[:, :4] = q / q.norm(dim=1, keepdim=True)
    tr[:, 7:] = torch.rand(batch, 3, generator=g, device="cuda") * 4 - 2
    return tr


def _prepare_grid(case, g, host):
    batch, single = max(1, case["batch"]), case["batch"] == 0
    counts = host.integers(case["min_atoms"], case["max_atoms"] + 1, batch)
    n = case["max_atoms"]
    na = torch.tensor(counts, dtype=torch.int32, device="cuda")
    valid = torch.arange(n, device="cuda")[None, :] < na[:, None]
    coords = _positions(g, batch, n, case["blob"]) * valid[..., None]
    kind = torch.randint(case["types"], (batch, n), generator=g, device="cuda")
    radius = torch.rand(case["types"], generator=g, device="cuda") + 1.2
    types, radii = kind.float() * valid, radius[kind] * valid
    module = molgrid if single else lmg
    maker = module.GridMaker(case["resolution"], (case["points"] - 1) * case["resolution"], case["binary"])
    s = dict(case=case, maker=maker)
    shape = (batch,) + tuple(maker.grid_dimensions(case["types"]))
    arrays = dict(coords=coords, types=types, radii=radii, grid=torch.empty(shape, device="cuda"))
    if case["op"] == "train":
        arrays.update(diff=torch.randn(shape, generator=g, device="cuda"), grads=torch.empty_like(coords))
    if case["op"] == "relevance":
        arrays.update(diff=torch.randn(shape, generator=g, device="cuda"), relevance=torch.empty_like(types))
    s.update({k: v[0] for k, v in arrays.items()} if single else arrays)
    if single:
        s.update(center=(0.0, 0.0, 0.0), more={})
    else:
        s.update(center=torch.zeros(batch, 3, device="cuda"), more=dict(transforms=_transforms(g, batch), n_atoms=na))
    if case["op"] == "relevance":
        # the network's input as it was stored, in steps of 2^-14
        maker.forward(s["center"], s["coords"], s["types"], s["radii"], s["grid"], **s["more"])
        s["grid"].mul_(16384).round_().div_(16384)
    return s


def _prepare_autograd(case, g, host):
    shape = (case["batch"], case["atoms"])
    if case["soft"]:
        w = torch._standard_gamma(torch.full(shape + (case["types"],), 0.3, device="cuda"), generator=g)
        types = w / w.sum(dim=-1, keepdim=True)
    else:
        kind = torch.randint(case["types"], shape, generator=g, device="cuda")
        types = torch.nn.functional.one_hot(kind, case["types"]).float()
    if case["radii_by_type"]:
        radii = 1.7 * (0.8 + 0.4 * torch.rand(case["batch"], case["types"], generator=g, device="cuda"))
    else:
        radii = 1.2 + torch.rand(*shape, generator=g, device="cuda")
    maker = lmg.GridMaker(case["resolution"], (case["points"] - 1) * case["resolution"],
                          radius_type_indexed=case["radii_by_type"])
    diff = torch.randn((case["batch"],) + tuple(maker.grid_dimensions(case["types"])), generator=g, device="cuda")
    s = dict(case=case, layer=lmg.Coords2Grid(maker), radii=radii, types=types.requires_grad_(),
             coords=_positions(g, case["batch"], case["atoms"], case["blob"]).requires_grad_(), diff=diff)
    if case["second"]:
        s["diff"].requires_grad_()
        s["vcoords"] = torch.randn(s["coords"].shape, generator=g, device="cuda")
        s["vtypes"] = torch.randn(types.shape, generator=g, device="cuda")
    return s


def _prepare_interpolate(case, g, host):
    single = case["batch"] == 1
    module = molgrid if single else lmg
    res, n, m = case["resolution"], case["in_points"], case["out_points"]
    rows = _transforms(g, case["batch"]).tolist()
    trs = [module.Transform(module.Quaternion(*r[:4]), (0.0, 0.0, 0.0), tuple(r[7:])) for r in rows]
    a = torch.rand(case["batch"], case["channels"], n, n, n, generator=g, device="cuda")
    b = torch.empty(case["batch"], case["channels"], m, m, m, device="cuda")
    s = dict(case=case, inter=module.GridInterpolater(res, (n - 1) * res, res, (m - 1) * res))
    arrays = dict(a=a, b=b)
    if case["backward"]:
        arrays.update(gb=torch.randn(b.shape, generator=g, device="cuda"), ga=torch.empty_like(a))
    s.update({k: v[0] for k, v in arrays.items()} if single else arrays)
    s["transforms"] = trs[0] if single else trs
    return s


def _prepare_provider(case, g, host, seed):
    folder = tempfile.TemporaryDirectory()

    def structure(name, n, kinds, center, radius):
        v = host.normal(size=(n, 3))
        v *= radius * host.uniform(size=(n, 1)) ** (1 / 3) / np.linalg.norm(v, axis=1, keepdims=True)
        write_gninatypes(os.path.join(folder.name, name), (v + center).astype(np.float32), host.integers(2, kinds, n))

    lines = []
    for i in range(case["examples"]):
        center = host.uniform(-20, 20, 3)
        structure("r%d.gninatypes" % i, int(host.integers(case["min_atoms"], case["max_atoms"] + 1)), 28, center, 14.0)
        structure("l%d.gninatypes" % i, int(host.integers(20, 60)), 21, center, 4.0)
        lines.append("%d %.3f r%d.gninatypes l%d.gninatypes" % (i % 2, host.uniform(2, 11), i, i))
    with open(os.path.join(folder.name, "train.types"), "w") as f:
        f.write("\n".join(lines) + "\n")
    molgrid.set_random_seed(seed % (1 << 31))
    provider = molgrid.ExampleProvider(data_root=folder.name)
    provider.populate(os.path.join(folder.name, "train.types"))
    maker = molgrid.GridMaker(case["resolution"], (case["points"] - 1) * case["resolution"])
    shape = (case["batch"],) + tuple(maker.grid_dimensions(provider.num_types()))
    return dict(case=case, folder=folder, provider=provider, maker=maker, grid=torch.empty(shape, device="cuda"),
                labels=torch.empty(case["batch"], provider.num_labels(), device="cuda"))


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    host = np.random.default_rng(seed)
    if case["path"] == "grid":
        return _prepare_grid(case, g, host)
    if case["path"] == "autograd":
        return _prepare_autograd(case, g, host)
    if case["path"] == "interpolate":
        return _prepare_interpolate(case, g, host)
    return _prepare_provider(case, g, host, seed)


# ---- one pass ------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    if case["path"] == "grid":
        atoms = (s["center"], s["coords"], s["types"], s["radii"])
        if case["op"] == "relevance":
            s["maker"].backward_relevance(*atoms, s["grid"], s["diff"], s["relevance"], **s["more"])
            return s["relevance"]
        s["maker"].forward(*atoms, s["grid"], **s["more"])
        if case["op"] == "forward":
            return s["grid"]
        s["maker"].backward(*atoms, s["diff"], s["grads"], **s["more"])
        return s["grid"], s["grads"]
    if case["path"] == "autograd":
        out = s["layer"](s["coords"], s["types"], s["radii"])
        first = torch.autograd.grad(out, (s["coords"], s["types"]), s["diff"], create_graph=case["second"])
        if not case["second"]:
            return (out.detach(),) + first
        second = torch.autograd.grad(first, (s["coords"], s["diff"]), (s["vcoords"], s["vtypes"]))
        return (out.detach(),) + tuple(t.detach() for t in first) + second
    if case["path"] == "interpolate":
        s["inter"].forward(s["a"], s["transforms"], s["b"])
        if not case["backward"]:
            return s["b"]
        s["inter"].backward(s["gb"], s["transforms"], s["ga"])
        return s["b"], s["ga"]
    if case["mode"] == "device":
        batch = s["provider"].next_device_batch(case["batch"])
        labels = batch.labels
    else:
        batch, labels = s["provider"].next_batch(case["batch"]), s["labels"]
        batch.extract_labels(labels)
    s["maker"].forward(batch, s["grid"], 2.0, True)
    return s["grid"], labels


# ---- what a pass cannot do without -----------------------------------------------------------------

def _pairs(case, atoms, r3):
    """(atom, voxel) pairs inside the cut-off of 1.5 radii (1 radius for occupancy), r3 the mean cubed
    radius; an atom near the wall of a small box has fewer."""
    reach = 1.0 if case.get("binary") else 1.5
    side = (case["points"] - 1) * case["resolution"]
    share = min(1.0, side ** 3 / (4 / 3 * math.pi * 12.0 ** 3))
    return atoms * share * 4 / 3 * math.pi * reach ** 3 * r3 / case["resolution"] ** 3


def work(case):
    if case["path"] == "interpolate":
        cells = 4 * case["batch"] * case["channels"]
        nbytes = cells * (case["in_points"] ** 3 + case["out_points"] ** 3)
        ops = cells / 4 * case["out_points"] ** 3 * 21
        return {"bytes": nbytes * (2 if case["backward"] else 1), "flops": ops * (2 if case["backward"] else 1)}
    if case["path"] == "provider":
        atoms = case["batch"] * ((case["min_atoms"] + case["max_atoms"]) / 2 + 40)
        return {"bytes": 4 * case["batch"] * 28 * case["points"] ** 3 + 16 * atoms, "flops": 10 * _pairs(case, atoms, 5.6)}
    if case["path"] == "grid":
        batch = max(1, case["batch"])
        atoms = batch * (case["min_atoms"] + case["max_atoms"]) / 2
        grid = 4 * batch * case["types"] * case["points"] ** 3
        pairs = _pairs(case, atoms, 5.3)
        if case["op"] == "forward":
            return {"bytes": grid + 20 * atoms, "flops": 10 * pairs}
        if case["op"] == "relevance":
            return {"bytes": 2 * grid + 24 * atoms, "flops": 12 * pairs}
        return {"bytes": 2 * grid + 52 * atoms, "flops": 22 * pairs}
    atoms = case["batch"] * case["atoms"]
    grid = 4 * case["batch"] * case["types"] * case["points"] ** 3
    pairs = _pairs(case, atoms, 5.3)
    weighted = case["types"] if case["soft"] else 1
    # forward: a density per pair and a multiply-add per weighted channel; backward: a multiply-add per
    # channel for the type gradients; densities per channel where the radii differ by channel
    each = case["types"] if case["radii_by_type"] else 1
    ops = pairs * (22 * each + 2 * weighted + 2 * case["types"] + 2 * weighted)
    nbytes = 2 * grid + atoms * (28 + 8 * case["types"])
    if case["second"]:
        ops += pairs * (60 * each + 8 * weighted)
        nbytes += 2 * grid + atoms * (40 + 12 * case["types"])
    return {"bytes": nbytes, "flops": ops}


def tolerance(case):
    if case["path"] == "interpolate":
        # the forward pass promises the reference's own roundings; its adjoint sums in any order
        return {"rel": 1e-5} if case["backward"] else "exact"
    if case["path"] == "grid" and case["binary"]:
        return "exact"
    if case["path"] == "grid" and case["op"] == "relevance":
        # a quotient of two densities, which are small differences of 32-bit numbers near the cut-off
        return {"rel": 1e-4}
    if case["path"] == "autograd" and case["second"]:
        return {"rel": 3e-5}
    return {"rel": 1e-5}
