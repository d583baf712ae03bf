// Binary occupancy of index types: every voxel is written once.
#include "lmg_atoms.cuh"
#include "lmg_device.cuh"
#include "lmg_launch.h"

#include <algorithm>

namespace lmg {

// ---------------------------------------------------------------------------------------------
// k_occupancy: a block owns some x planes of one channel of one example.  It looks through the example's
// types, prepares the atoms of its channel that reach its planes (a lane each: fused Transform, footprint,
// threshold), marks the voxels inside their spheres in a bit mask in shared memory (a column of the sphere per
// lane: the run of z that passes the exact test, one or two atomic ORs) and turns the mask into floats.
//
// Bound by the output once enough blocks are at work: 28 x 48^3 is 12.4 MB an example, its mask 387 kB.  Clearing
// the output and then storing ones into it (a warp per atom) took 207 us for 50 examples of 2000 to 4000
// atoms, of which 90 were the clearing; this takes 126 us (floor 95), and 6 more for k_occupancy_full.  What counted on the way: the ends of a
// run from its root, with the exact test only near a voxel (170 -> 141 us), and candidates cut to the
// sphere's own box (141 -> 126 us).
// ---------------------------------------------------------------------------------------------
constexpr int OCC_THREADS = 256;
constexpr int OCC_CHUNK = 2048;            // atoms looked through at a time
constexpr unsigned OCC_WORDS = 10 * 1024;  // most words of mask per block (40 kB: no opt-in needed)

// An atom as occupancy needs it: the part of make_rec that its results depend on.
struct OccAtom {
  float x, y, z, Tbin;
  // lo.x | lo.y << 16 and hi.x | hi.y << 16 of the columns its sphere can reach (and a voxel more on either side),
  // lo.z | hi.z << 16 of the footprint; xy0 == xy1 where nothing is reached
  unsigned xy0, xy1, zz;
};

__device__ __forceinline__ OccAtom make_occ(const EmitArgs& A, int b, int a) {
  const GMParams& gm = A.gm;
  AtomIn I = load_atom(A, b, a);
  atom_move(I);
  OccAtom O;
  O.x = I.x; O.y = I.y; O.z = I.z;
  const float ar = __fmul_rn(I.radius, gm.rscale), densityrad = __fmul_rn(ar, gm.finalm);
  O.Tbin = __fmul_rn(ar, ar);
  const float ox = __fsub_rn(I.cx, gm.half), oy = __fsub_rn(I.cy, gm.half);
  unsigned lox, hix, loy, hiy, loz, hiz;
  bounds_1d(ox, I.x, densityrad, gm.res, gm.dim, lox, hix);
  bounds_1d(oy, I.y, densityrad, gm.res, gm.dim, loy, hiy);
  bounds_1d(__fsub_rn(I.cz, gm.half), I.z, densityrad, gm.res, gm.dim, loz, hiz);
  within(ox, I.x, ar, gm.res, lox, hix);
  within(oy, I.y, ar, gm.res, loy, hiy);
  const bool any = ar > 0.f && hix > lox && hiy > loy && hiz > loz;
  O.xy0 = any ? lox | loy << 16 : 0u;
  O.xy1 = any ? hix | hiy << 16 : 0u;
  O.zz = loz | hiz << 16;
  return O;
}

// Real structures put a third and more of their atoms into two or three channels, and the blocks of a channel last
// as long as its atoms take eight warps.  Channels of more than `most` atoms in an example are marked by this kernel
// and their atoms listed: k_occupancy writes zeros there, and the atoms are stored afterwards (launch_occupancy_listed).
// 50 x 3000 atoms in 28 channels, evenly / a third in one / all in one: 126/213/396 us without, 132/157/181 with.
constexpr int FULL_THREADS = 1024;  // 256: 3 us more
__global__ void __launch_bounds__(FULL_THREADS) k_occupancy_full(EmitArgs A, OccList L, unsigned most) {
  extern __shared__ unsigned count[];
  __shared__ unsigned listed;
  const int tid = threadIdx.x, bl = blockIdx.x, b = A.b0 + bl;
  for (int t = tid; t < A.T; t += FULL_THREADS) count[t] = 0;
  if (tid == 0) listed = 0;
  __syncthreads();
  wait_for_stream();
  let_next_begin();
  const int n = A.n_atoms != nullptr ? min(A.N, A.n_atoms[b]) : A.N;
  const float* types = A.type_index + (size_t)b * A.N;
  bool bad = false;
#pragma unroll 4
  for (int i = tid; i < n; i += FULL_THREADS) {
    const float tc = floorf(types[i]);
    if (tc >= (float)A.T) bad = true;
    else if (tc >= 0.f) atomicAdd(&count[(int)tc], 1u);
  }
  bad = __syncthreads_or(bad && A.check_types) != 0;
  if (tid == 0) put_flag(A, bl, A.nb, bad);
  bool any = false;
  for (int t = tid; t < A.T; t += FULL_THREADS) {
    L.mark[(size_t)bl * A.T + t] = count[t] > most;
    any = any || count[t] > most;
  }
  if (__syncthreads_or(any)) {
    for (int i = tid; i < n; i += FULL_THREADS) {
      const float tc = floorf(types[i]);
      if (tc >= 0.f && tc < (float)A.T && count[(int)tc] > most) L.atom[(size_t)bl * A.N + atomicAdd(&listed, 1u)] = (unsigned)i;
    }
    __syncthreads();
  }
  if (tid == 0) L.n[bl] = listed;
}

// MARKED: k_occupancy_full went before.
template <bool MARKED>
__global__ void __launch_bounds__(OCC_THREADS, 6) k_occupancy(EmitArgs A, float* __restrict__ out, unsigned planes,
                                                              const unsigned char* mark) {
  extern __shared__ unsigned bits[];
  __shared__ unsigned short list[OCC_CHUNK];
  __shared__ unsigned listed;
  const GMParams& gm = A.gm;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int chan = blockIdx.y, bl = blockIdx.z, b = A.b0 + bl;
  const unsigned dim = gm.dim, x0 = blockIdx.x * planes, x1 = min(x0 + planes, dim);
  const unsigned total = (x1 - x0) * dim * dim, words = (total + 31) / 32;
  for (unsigned i = tid; i <= words; i += OCC_THREADS) bits[i] = 0;  // and one word to read beyond the last
  wait_for_stream();
  int n = A.n_atoms != nullptr ? min(A.N, A.n_atoms[b]) : A.N;
  if (MARKED && mark[(size_t)bl * A.T + chan]) n = 0;
  const float* types = A.type_index + (size_t)b * A.N;

  bool bad = false;
  for (int base = 0; base < n; base += OCC_CHUNK) {
    if (tid == 0) listed = 0;
    __syncthreads();
    float ty[OCC_CHUNK / OCC_THREADS];  // requested together
#pragma unroll
    for (int k = 0; k < OCC_CHUNK / OCC_THREADS; k++) {
      const int i = base + k * OCC_THREADS + tid;
      ty[k] = i < n ? types[i] : -1.f;
    }
#pragma unroll
    for (int k = 0; k < OCC_CHUNK / OCC_THREADS; k++) {
      const float tc = floorf(ty[k]);
      bad = bad || (A.check_types && tc >= (float)A.T);
      const bool hit = tc == (float)chan;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (m == 0u) continue;
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(&listed, __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (hit) list[at + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(k * OCC_THREADS + tid);
    }
    __syncthreads();
    // entry e is lane e / warps of warp e % warps in the round of its 32 * warps entries
    for (unsigned e0 = wid; e0 < listed; e0 += OCC_THREADS) {
      const unsigned e = e0 + lane * (OCC_THREADS / 32);
      OccAtom O;
      bool use = e < listed;
      if (use) {
        O = make_occ(A, b, base + list[e]);
        use = lo16(O.xy0) < x1 && lo16(O.xy1) > x0;
      }
      float cx, cy, cz;
      if (A.centers != nullptr) {
        cx = A.centers[b * 3]; cy = A.centers[b * 3 + 1]; cz = A.centers[b * 3 + 2];
      } else {
        cx = A.center_host[0]; cy = A.center_host[1]; cz = A.center_host[2];
      }
      const float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
      const float inv = __fdividef(1.f, gm.res);
      for (unsigned m = __ballot_sync(0xffffffffu, use); m != 0u; m &= m - 1u) {
        const int s = __ffs(m) - 1;
        const float px = __shfl_sync(0xffffffffu, O.x, s), py = __shfl_sync(0xffffffffu, O.y, s),
                    pz = __shfl_sync(0xffffffffu, O.z, s), Tbin = __shfl_sync(0xffffffffu, O.Tbin, s);
        const unsigned bxy = __shfl_sync(0xffffffffu, O.xy0, s), hxy = __shfl_sync(0xffffffffu, O.xy1, s),
                       bz = __shfl_sync(0xffffffffu, O.zz, s);
        const unsigned lx = max(lo16(bxy), x0), ly = hi16(bxy), ny = hi16(hxy) - ly, ncols = (min(lo16(hxy), x1) - lx) * ny;
        const int lz = (int)lo16(bz), hz = (int)hi16(bz) - 1;
        // What the ends of a run of half length h may be off by, in voxels: the roundings of the positions and of the
        // root that gives them, and 1.2e-7 R^2 / h for a sphere of R voxels, because the exact test compares numbers
        // near Tbin, each off by up to 2^-24 of it, whose difference is h^2.  Enough for h > 0.05.
        const float eps = 1e-3f + fmaxf(fabsf(pz), fabsf(oz)) * inv * 4e-6f + Tbin * inv * inv * 3e-6f;
        const float zc = (pz - oz) * inv, inv_ny = __fdividef(1.f, small_float(ny));
        if (!(eps < 0.25f)) {  // ends that may be off by half a voxel: voxel by voxel
          for (unsigned c = lane; c < ncols; c += 32) {
            const unsigned x = lx + c / ny, y = ly + c % ny;
            const float dx = __fsub_rn(voxel_coord(ox, x, gm.res), px), dy = __fsub_rn(voxel_coord(oy, y, gm.res), py);
            const float dxy2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
            for (int z = lz; z <= hz; z++) {
              const float dz = __fsub_rn(voxel_coord(oz, (unsigned)z, gm.res), pz);
              const unsigned p = ((x - x0) * dim + y) * dim + z;
              if (__fadd_rn(dxy2, __fmul_rn(dz, dz)) < Tbin) atomicOr(&bits[p >> 5], 1u << (p & 31));
            }
          }
          continue;
        }
        for (unsigned c = lane; c < ncols; c += 32) {
          const unsigned xi = ncols < 4096u ? (unsigned)((small_float(c) + 0.5f) * inv_ny) : c / ny, x = lx + xi, y = ly + c - xi * ny;
          const float dx = __fsub_rn(voxel_coord(ox, x, gm.res), px), dy = __fsub_rn(voxel_coord(oy, y, gm.res), py);
          const float dxy2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
          if (!(dxy2 < Tbin)) continue;
          auto in = [&](int z) {
            const float dz = __fsub_rn(voxel_coord(oz, (unsigned)z, gm.res), pz);
            return __fadd_rn(dxy2, __fmul_rn(dz, dz)) < Tbin;
          };
          // |dz| grows away from the atom, so the voxels that pass are one run.  The root gives its ends; where
          // one lies near a voxel, the exact test has the last word.  (With R left out of eps, ends are wrong from
          // radii of 60 voxels on.)
          const float h = sqrt_approx(Tbin - dxy2) * inv, e0 = fmaxf(zc - h, -1e6f), e1 = fminf(zc + h, 1e6f);
          const float f0 = ceilf(e0), f1 = floorf(e1);
          int z0 = max(lz, (int)f0), z1 = min(hz, (int)f1);
          const float d0 = f0 - e0, d1 = e1 - f1;  // distances from the next voxel inside
          if (!(fminf(d0, d1) > eps && fmaxf(d0, d1) < 1.f - eps && h > 0.05f)) {
            if (z0 > lz && in(z0 - 1)) z0--;
            while (z0 <= z1 && !in(z0)) z0++;
            if (z1 < hz && z1 >= lz - 1 && in(z1 + 1)) z1++;
            while (z1 >= z0 && !in(z1)) z1--;
          }
          if (z0 > z1) continue;
          const unsigned first = ((x - x0) * dim + y) * dim + z0, last = first + (z1 - z0);
          const unsigned head = 0xffffffffu << (first & 31), tail = 0xffffffffu >> (31 - (last & 31));
          unsigned w = first >> 5;
          const unsigned wl = last >> 5;
          if (w == wl) {
            atomicOr(&bits[w], head & tail);
          } else {
            atomicOr(&bits[w], head);
            while (++w < wl) atomicOr(&bits[w], 0xffffffffu);
            atomicOr(&bits[wl], tail);
          }
        }
      }
    }
    __syncthreads();
  }
  if (!MARKED && chan == 0 && blockIdx.x == 0) {  // one block per example reports types beyond the channels
    bad = __syncthreads_or(bad) != 0;
    if (tid == 0) put_flag(A, bl, A.nb, bad);
  }
  __syncthreads();

  float* o = out + (((size_t)b * A.T + chan) * dim + x0) * dim * dim;
  const unsigned head = min(total, (unsigned)(4 - ((uintptr_t)o >> 2 & 3)) & 3u), quads = (total - head) / 4;
  for (unsigned q = tid; q < quads; q += OCC_THREADS) {
    const unsigned p = head + 4 * q, w = __funnelshift_r(bits[p >> 5], bits[(p >> 5) + 1], p & 31);
    reinterpret_cast<float4*>(o + head)[q] = make_float4(w & 1u ? 1.f : 0.f, w & 2u ? 1.f : 0.f, w & 4u ? 1.f : 0.f, w & 8u ? 1.f : 0.f);
  }
  const unsigned rest = total - head - 4 * quads;  // and what the aligned quads leave at either end
  if (tid < head + rest) {
    const unsigned p = tid < head ? tid : head + 4 * quads + (tid - head);
    o[p] = bits[p >> 5] >> (p & 31) & 1u ? 1.f : 0.f;
  }
}

// Most atoms of a channel that its blocks take: four times a block's share of the pass when six blocks an SM share it
// evenly (a larger share outlasts the others), or as few as cost next to nothing.
static long occupancy_most(const EmitArgs& A) { return std::max(128L, (long)A.nb * A.N / 222); }

// Whether the pass is this kernel's.  A block looks through all of its example's types and marks its atoms
// with eight warps, so it wants a channel per block and a chip full of such blocks, or hardly any atoms (40 atoms, 28
// channels: 5.2 against 5.9 us; 300 atoms: 6.4 against 6.2).  Against clearing and storing, us for types spread
// evenly / a third in one channel / all in one (channels x examples x atoms, 48^3): 28x50x3000 132/157/181 and
// 251/223/165; 28x24x3000 81/93/98 and 128/114/83; 28x16x3000 64/73/75 and 83/73/60; 4x100x3000 149/185/179 and
// 183/185/177; 14x50x2000 87/100/112 and 147/134/99; 14x16x3000 83/75/63 and 46; 2x100x4000 216/376/218 and 212;
// 28x8x3000 50/54/50 and 38; and where no channel can be too full, 1x256x1000 123 and 155; 4x256x300 95/96/109 and
// 161/157/124.
bool occupancy_serves(const EmitArgs& A) {
  const long blocks = (long)A.T * A.nb;
  const bool pays = A.N <= 128 || blocks >= 400 || (blocks >= 222 && A.N <= occupancy_most(A));
  return pays && !A.vec && A.gm.binary && A.gm.dim * A.gm.dim <= OCC_WORDS * 32 && A.T <= 65535 && A.nb <= 65535;
}

cudaError_t launch_occupancy(const EmitArgs& A, float* out, long* launches, cudaStream_t st) {
  const unsigned dim = A.gm.dim, per_plane = dim * dim;
  const long per = (long)A.T * A.nb;
  // whole channels per block for large batches, parts of them while that leaves SMs idle
  unsigned slabs = (unsigned)((500 + per - 1) / per);
  if (slabs > dim) slabs = dim;
  unsigned planes = (dim + slabs - 1) / slabs;
  if ((size_t)planes * per_plane > (size_t)OCC_WORDS * 32) planes = OCC_WORDS * 32 / per_plane;
  const size_t smem = ((size_t)planes * per_plane + 31) / 32 * 4 + 4;
  const dim3 grid((dim + planes - 1) / planes, A.T, A.nb);
  const long most = occupancy_most(A);
  // marks and lists lie where other passes keep their records
  const bool marked = A.N > most + most / 4 && A.T <= 8192 && 4 + 4 * (size_t)A.N + A.T <= A.N * sizeof(Rec);
  *launches += marked ? 3 : 1;
  if (!marked) return launch_early(k_occupancy<false>, grid, OCC_THREADS, smem, st, A, out, planes, (const unsigned char*)nullptr);
  OccList L;
  L.atom = reinterpret_cast<unsigned*>(A.recs);
  L.n = L.atom + (size_t)A.nb * A.N;
  L.mark = reinterpret_cast<unsigned char*>(L.n + A.nb);
  cudaError_t e = launch_early(k_occupancy_full, dim3(A.nb), FULL_THREADS, A.T * sizeof(unsigned), st, A, L, (unsigned)most);
  if (e != cudaSuccess) return e;
  e = launch_early(k_occupancy<true>, grid, OCC_THREADS, smem, st, A, out, planes, (const unsigned char*)L.mark);
  return e != cudaSuccess ? e : launch_occupancy_listed(A, L, out, st);
}

}  // namespace lmg
