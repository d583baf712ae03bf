"""Relevance near the limits of 32 bits, against 64-bit sums, and the quotients and roots it is made of, against
the device's own."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

import libmolgrid_b200 as lmg

pytestmark = pytest.mark.gpu
P, N, T = 24, 400, 3


def terms(multiple, small=1.0):
    """Atoms, and the density of each at every voxel in 64 bits, of a Gaussian cut at `multiple` radii."""
    g = torch.Generator().manual_seed(5)
    coords = (torch.randn(N, 3, generator=g) * 3).cuda()
    types = torch.randint(T, (N,), generator=g).float().cuda()
    radii = ((torch.rand(N, generator=g) + 1.2) * small).cuda()
    ax = torch.arange(P, device="cuda", dtype=torch.float64) * 0.5 - (P - 1) * 0.25
    x = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    d = ((x[None] - coords.double()[:, None]) ** 2).sum(-1).sqrt() / radii.double()[:, None]
    return coords, types, radii, torch.where(d <= multiple, torch.exp(-2 * d * d), 0.0), g


def relevance(multiple, coords, types, radii, density, diff, shift):
    gm = lmg.GridMaker(0.5, (P - 1) * 0.5, False, False, 1.0, -multiple)
    out = torch.empty(N, device="cuda")
    if shift:  # no aligned rows: voxels one at a time
        density, diff = (torch.empty(t.numel() + 1, device="cuda")[1:].view(t.shape).copy_(t) for t in (density, diff))
    gm.backward_relevance((0.0, 0.0, 0.0), coords, types, radii, density, diff, out)
    return out.double()


@pytest.mark.parametrize("shift", [False, True])
def test_gaussian_part(shift):
    """A term has five roundings (two exponentials, their product, that with the gradient, the quotient), each
    2^-24 / sqrt(3) in the mean: 7.7e-8 together.  Two approximate exponentials alone brought 8.5e-8."""
    coords, types, radii, v, g = terms(1.5)
    density, diff = ((torch.rand((T, P, P, P), generator=g) + 0.5).cuda() for _ in range(2))
    got = relevance(1.5, coords, types, radii, density, diff, shift)
    want = (v * (diff.double() / density.double()).reshape(T, -1)[types.long()]).sum(1)
    assert float((got - want).norm() / want.norm()) < 7.7e-8


@pytest.mark.parametrize("shift", [False, True])
def test_densities_that_are_not_normal_numbers(shift):
    """exp(-2 * 6.8^2) = 7e-41: terms as small are whole multiples of 2^-149, 2e-5 of their value."""
    coords, types, radii, v, g = terms(6.8, 0.25)
    diff = (torch.rand((T, P, P, P), generator=g) + 0.5).cuda()
    got = relevance(6.8, coords, types, radii, torch.full_like(diff, 1e-36), diff, shift)
    want = (v * diff.double().reshape(T, -1)[types.long()]).sum(1) / float(np.float32(1e-36))
    ok = want > 0
    assert bool(ok.any()) and float(((got - want).abs() / want)[ok].max()) < 2e-5


@pytest.mark.parametrize("shift", [False, True])
def test_quotients_by_densities_that_are_not_normal_numbers(shift):
    """The reciprocal of 1e-39 is not a number of 32 bits, the quotients by it are."""
    coords, types, radii, v, g = terms(1.5)
    diff = (torch.rand((T, P, P, P), generator=g) + 0.5).cuda() * 1e-4
    got = relevance(1.5, coords, types, radii, torch.full_like(diff, 1e-39), diff, shift)
    want = (v * diff.double().reshape(T, -1)[types.long()]).sum(1) / float(np.float32(1e-39))
    assert float((got - want).norm() / want.norm()) < 1e-6


SOURCE = r"""
#include "lmg_device.cuh"
#include <math_constants.h>
using namespace lmg;
__device__ unsigned units(float a, float b) {
  if (!(a == a) || !(b == b)) return (a == a) == (b == b) ? 0u : 0xffffffffu;
  long long d = (long long)__float_as_int(a) - __float_as_int(b);
  return (unsigned)(d < 0 ? -d : d);
}
__device__ unsigned draw(unsigned x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; return x ^ x >> 16;
}
// out[0]: cases off by a unit, out[1]: the most units; a thread per case, 2^25 of them
__global__ void sweep(int what, unsigned* out) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned d = 0;
  if (what == 0) {                                     // every significand, both parities of the exponent
    const float x = __int_as_float((127u << 23) + (i & 0xffffffu));
    d = units(root(x), __fsqrt_rn(x));
  } else if (what == 1) {                              // distances over radii
    const float n = __int_as_float(((118u + (draw(i) >> 28)) << 23) + (draw(i) & 0x7fffffu));
    const float r = __int_as_float(((122u + (draw(i + 77u) >> 29)) << 23) + (draw(3u * i + 1u) & 0x7fffffu));
    d = units(divide_by(n, r, 1.f / r), __fdiv_rn(n, r));
  } else {                                             // all positive numbers; the quotient neither tiny nor infinite
    const float n = __int_as_float(draw(i) >> 1), v = __int_as_float(draw(5u * i + 3u) >> 1), q = __fdiv_rn(n, v);
    if (n >= 1e-30f && n < CUDART_INF_F && v < 1e38f && q > 1e-37f && q < 1e38f) d = units(divide_near(n, v), q);
  }
  if (d) { atomicAdd(out, 1u); atomicMax(out + 1, d); }
}
extern "C" int run(int what, unsigned* out) {
  unsigned* p;
  if (cudaMalloc(&p, 8) != cudaSuccess) return 1;
  cudaMemset(p, 0, 8);
  sweep<<<1 << 17, 256>>>(what, p);
  int e = (int)cudaMemcpy(out, p, 8, cudaMemcpyDeviceToHost);
  cudaFree(p);
  return e;
}
"""


@pytest.fixture(scope="module")
def sweeps(tmp_path_factory):
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc) and shutil.which("nvcc") is None:
        pytest.skip("no CUDA compiler")
    d = tmp_path_factory.mktemp("sweeps")
    (d / "s.cu").write_text(SOURCE)
    root = os.path.dirname(os.path.abspath(lmg.__file__))
    subprocess.check_call([nvcc if os.path.exists(nvcc) else "nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                           "-shared", "-Xcompiler", "-fPIC", "-I" + os.path.join(root, "csrc"), str(d / "s.cu"), "-o", str(d / "s.so")])
    return ctypes.CDLL(str(d / "s.so"))


@pytest.mark.parametrize("what", [0, 1, 2])
def test_roots_and_quotients(sweeps, what):
    out = (ctypes.c_uint * 2)()
    assert sweeps.run(what, out) == 0
    assert (out[0], out[1]) == (0, 0)


# four warps an atom, on either side of the lines between the kernels with room and the tight ones
@pytest.mark.parametrize("n", [1, 740, 741, 889, 1037, 1185])
@pytest.mark.parametrize("points", [12, 13])
@pytest.mark.parametrize("binary", [False, True])
def test_relevance_of_some_atoms(n, points, binary):
    from libmolgrid_b200 import synthetic as cases
    from oracle.oracle import CpuOracle
    port = CpuOracle("port")
    gm, og = lmg.GridMaker(0.5, (points - 1) * 0.5, binary), port.gm(0.5, (points - 1) * 0.5, binary)
    coords, types, radii = cases.index_case(n, n, T, 3.0)
    c, t, r = (torch.from_numpy(a).cuda() for a in (coords, types, radii))
    grid, out = torch.empty(gm.grid_dimensions(T), device="cuda"), torch.full((n,), 7.0, device="cuda")
    gm.forward((0.0, 0.0, 0.0), c, t, r, grid)
    diff = torch.randn_like(grid)
    diff[0, 0, 0, 0], grid[0, 1, 1, 1] = float("inf"), 1e-35  # one beyond most cut-offs, one that the short division does not take
    gm.backward_relevance((0.0, 0.0, 0.0), c, t, r, grid, diff, out)
    want = port.backward_relevance(og, (0, 0, 0), coords, types, radii, grid.cpu().numpy(), diff.cpu().numpy())
    fine = np.isfinite(want)
    assert np.array_equal(fine, np.isfinite(out.cpu().numpy()))
    np.testing.assert_allclose(out.cpu().numpy()[fine], want[fine], rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(want[fine]).max())))
