// sm_100a kernels for Transform forward/backward on coordinate arrays and for the
// GridInterpolater trilinear resample.
#include <cuda.h>
#include <stdint.h>

#include <algorithm>

#include "lmg_device.cuh"
#include "lmg_launch.h"
#include "lmg_misc.h"

namespace lmg {

// Transform::forward (src/transform.cpp:57-79): Q.transform(x, y, z, center, translate)
__global__ void __launch_bounds__(256) k_transform_forward(Xform X, int n, const float* in, float* out,
                                                           int dotranslate) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float cn[4];
  quat_conj_over_norm(X.q, cn);
  float x = in[3 * i], y = in[3 * i + 1], z = in[3 * i + 2];
  xform_apply(X, cn, x, y, z, dotranslate != 0);
  out[3 * i] = x;
  out[3 * i + 1] = y;
  out[3 * i + 2] = z;
}

// Transform::backward (src/transform.cpp:85-108): untranslate, rotate by the inverse, re-centre
__global__ void __launch_bounds__(256) k_transform_backward(Xform X, int n, const float* in, float* out,
                                                            int dotranslate) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float inv[4], cn[4];
  quat_inverse(X.q, inv);
  quat_conj_over_norm(inv, cn);
  float ux, uy, uz;
  if (dotranslate) {
    ux = __fsub_rn(-X.t[0], X.c[0]); uy = __fsub_rn(-X.t[1], X.c[1]); uz = __fsub_rn(-X.t[2], X.c[2]);
  } else {
    ux = -X.c[0]; uy = -X.c[1]; uz = -X.c[2];
  }
  float r[3];
  quat_rotate(inv, cn, __fadd_rn(in[3 * i], ux), __fadd_rn(in[3 * i + 1], uy), __fadd_rn(in[3 * i + 2], uz), r);
  out[3 * i] = __fadd_rn(r[0], X.c[0]);
  out[3 * i + 1] = __fadd_rn(r[1], X.c[1]);
  out[3 * i + 2] = __fadd_rn(r[2], X.c[2]);
}

cudaError_t launch_transform(const Xform& X, int n, const float* in, float* out, int dotranslate,
                             bool forward, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  int blocks = (n + 255) / 256;
  if (forward)
    k_transform_forward<<<blocks, 256, 0, st>>>(X, n, in, out, dotranslate);
  else
    k_transform_backward<<<blocks, 256, 0, st>>>(X, n, in, out, dotranslate);
  return cudaGetLastError();
}

// Position of output voxel (i,j,k) in input-grid index units (src/grid_interpolater.cpp:31-45).
__device__ __forceinline__ void interp_point(const InterpArgs& I, const InterpFrame& F, unsigned i, unsigned j,
                                             unsigned k, float& gx, float& gy, float& gz) {
  float px = voxel_coord(F.oox, i, I.out_res), py = voxel_coord(F.ooy, j, I.out_res),
        pz = voxel_coord(F.ooz, k, I.out_res);
  float r[3];
  quat_rotate(F.inv, F.cn, __fadd_rn(px, F.ux), __fadd_rn(py, F.uy), __fadd_rn(pz, F.uz), r);
  gx = __fsub_rn(__fadd_rn(r[0], F.cx), F.iox);
  gy = __fsub_rn(__fadd_rn(r[1], F.cy), F.ioy);
  gz = __fsub_rn(__fadd_rn(r[2], F.cz), F.ioz);
  if (I.inv_in_res != 0.f) {  // the quotient by a power of two is the product with its inverse
    gx = __fmul_rn(gx, I.inv_in_res);
    gy = __fmul_rn(gy, I.inv_in_res);
    gz = __fmul_rn(gz, I.inv_in_res);
  } else {
    gx = __fdiv_rn(gx, I.in_res);
    gy = __fdiv_rn(gy, I.in_res);
    gz = __fdiv_rn(gz, I.in_res);
  }
}

// Corner indices and weights of the trilinear blend (src/grid_interpolater.cu:26-58).
struct InterpCell {
  int xl, xh, yl, yh, zl, zh;
  float xd, yd, zd, xm, ym, zm;
};

__device__ __forceinline__ InterpCell interp_cell(float gx, float gy, float gz) {
  InterpCell C;
  C.xl = (int)floorf(gx); C.xh = (int)ceilf(gx);
  C.yl = (int)floorf(gy); C.yh = (int)ceilf(gy);
  C.zl = (int)floorf(gz); C.zh = (int)ceilf(gz);
  // the reference divides by upper - lower, which is one wherever the two differ
  C.xd = C.xh > C.xl ? __fsub_rn(gx, (float)C.xl) : 0.f;
  C.yd = C.yh > C.yl ? __fsub_rn(gy, (float)C.yl) : 0.f;
  C.zd = C.zh > C.zl ? __fsub_rn(gz, (float)C.zl) : 0.f;
  C.xm = __fsub_rn(1.f, C.xd); C.ym = __fsub_rn(1.f, C.yd); C.zm = __fsub_rn(1.f, C.zd);
  return C;
}

// Products and sums of two lerps at a time, each rounded on its own as the reference rounds them.  A packed
// product followed by a packed sum would be contracted; the sum of a product and -0 is the rounded product,
// and `nz` (-0 from the kernel's parameters) keeps the compiler from knowing it.
__device__ __forceinline__ float interp_blend(const InterpCell& C, float nz, float p000, float p001, float p010,
                                              float p011, float p100, float p101, float p110, float p111) {
  const Pair xm = pair(C.xm), xd = pair(C.xd), n = pair(nz);
  const Pair c0 = add2(fma2(pair(p000, p001), xm, n), fma2(pair(p100, p101), xd, n));  // y low: z low, z high
  const Pair c1 = add2(fma2(pair(p010, p011), xm, n), fma2(pair(p110, p111), xd, n));  // y high
  float z0, z1;
  split(add2(fma2(c0, pair(C.ym), n), fma2(c1, pair(C.yd), n)), z0, z1);
  return __fadd_rn(__fmul_rn(z0, C.zm), __fmul_rn(z1, C.zd));
}

// Where a voxel read straight from the input grid finds its corners: a row per (x, y) corner at the lower z,
// the step to the upper z, and which of the eight lie inside the grid (the others read as zero, from
// an address inside it).
struct InterpReads {
  size_t row[4];
  int sz;
  unsigned inside;
  __device__ __forceinline__ InterpReads(const InterpCell& C, int id) {
    const bool xi[2] = {C.xl >= 0 && C.xl < id, C.xh >= 0 && C.xh < id}, yi[2] = {C.yl >= 0 && C.yl < id, C.yh >= 0 && C.yh < id},
               zi[2] = {C.zl >= 0 && C.zl < id, C.zh >= 0 && C.zh < id};
    const int z0 = zi[0] ? C.zl : zi[1] ? C.zh : 0;
    sz = zi[0] && zi[1] ? C.zh - C.zl : 0;
    inside = 0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const bool in = xi[r >> 1] && yi[r & 1];
      row[r] = in ? ((size_t)(r & 2 ? C.xh : C.xl) * id + (r & 1 ? C.yh : C.yl)) * id + z0 : 0;
      inside |= (in && zi[0] ? 1u : 0u) << (2 * r) | (in && zi[1] ? 2u : 0u) << (2 * r);
    }
  }
};

__device__ __forceinline__ float interp_direct(const InterpCell& C, const InterpReads& Q, float nz, const float* g) {
  float p[8];
#pragma unroll
  for (int r = 0; r < 4; r++) {
    p[2 * r] = __ldg(g + Q.row[r]);
    p[2 * r + 1] = __ldg(g + Q.row[r] + Q.sz);
  }
#pragma unroll
  for (int r = 0; r < 8; r++) p[r] = Q.inside >> r & 1u ? p[r] : 0.f;
  return interp_blend(C, nz, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7]);
}

// The channels [c0, c1) of a block: a launch whose voxels alone do not fill the chip shares the channels
// out over blockIdx.z.  The position of a voxel is then computed once per share, which is why the shares
// are no smaller than they have to be (channel_shares).
struct ChannelRange {
  int c0, c1;
  __device__ __forceinline__ explicit ChannelRange(int K, int step = 1) {
    const int per = ((K + gridDim.z - 1) / gridDim.z + step - 1) / step * step;
    c0 = blockIdx.z * per;
    c1 = min(K, c0 + per);
  }
};

// One thread per output voxel (and share of the channels); the inverse transform is computed once and
// reused for every channel (GridInterpolater::forward, src/grid_interpolater.cpp:31-45).  Used when the
// input grid does not meet the alignment rules of the tiled kernel below.
__global__ void __launch_bounds__(256) k_interpolate(InterpArgs I) {
  int bl = blockIdx.y;
  const InterpFrame& F = I.ex[bl];
  unsigned od = I.out_dim;
  // a warp is a brick of 2 x 2 x 8 voxels: under a random rotation its reads of one corner touch 16 lines
  // of the input, those of 32 voxels in a row 26
  const unsigned tid = threadIdx.x, nz = (od + 7) / 8, ny = (od + 7) / 8;
  const unsigned k = blockIdx.x % nz * 8 + (tid & 7), j = blockIdx.x / nz % ny * 8 + (tid >> 5 & 3) * 2 + (tid >> 3 & 1),
                 i = blockIdx.x / (nz * ny) * 4 + (tid >> 7) * 2 + (tid >> 4 & 1);
  if (i >= od || j >= od || k >= od) return;
  float gx, gy, gz;
  interp_point(I, F, i, j, k, gx, gy, gz);
  InterpCell C = interp_cell(gx, gy, gz);
  int id = (int)I.in_dim;
  size_t ichan = (size_t)id * id * id, ochan = (size_t)od * od * od;
  size_t b = (size_t)I.b0 + bl;
  const float* in = I.in + b * I.K * ichan;
  float* out = I.out + b * I.K * ochan + ((size_t)i * od + j) * od + k;
  const ChannelRange R(I.K);
  const InterpReads Q(C, id);
  wait_for_stream();
#pragma unroll 2
  for (int c = R.c0; c < R.c1; c++) __stcs(out + c * ochan, interp_direct(C, Q, I.minus_zero, in + c * ichan));
}

// ---------------------------------------------------------------------------------------------
// Tiled interpolation: a block owns an ITILE^3 tile of output voxels (12^3).  The input voxels that
// tile can touch form a box (the rotated tile's bounding box, z rounded down to a 16-byte
// boundary).  One elected thread of a warp of its own brings that box of channel c into shared memory
// with a single tensor copy (cp.async.bulk.tensor, zero fill outside the grid = the reference's zero
// padding) whose extents are, per axis, one of a few fixed sizes that hold the tile (one tensor map per
// combination).  The staging area of a block is cut into as many slots as boxes of its extents fit (two to
// three on average, one for the few tiles that need the largest box); nine warps blend their voxels of the
// channel from shared memory, each at its own pace between a barrier "box has arrived" and a barrier "done
// with the box" per slot.  The blend arithmetic is that of the direct kernel.  Every wait is bounded; a
// warp whose wait runs out finishes its voxels through the direct reads.
// Bound by the shared-memory pipe (8 loads per voxel and channel at 2.3 lanes per bank) and instruction
// issue.  Measured per 48 examples of 28 x 48^3 with random rotations: 560 us with 432 threads that
// met twice per channel, positions and frames computed by every thread; 548 with the frames from
// the host and a corner per lane; 508 with the box's pitches chosen by bank conflicts and uniform corner
// distances; 497 with six voxels a thread; 472 with the barriers per slot and two lerps per instruction.
// (Tiles of 8^3: 683 in the first of these, 16^3 with one block per SM 644; a copy per x plane 1080.)
// ---------------------------------------------------------------------------------------------
__device__ unsigned g_tma_timeouts = 0;

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// false when the phase did not complete within the limit
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity) {
  for (int it = 0; it < (1 << 20); it++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma_load_box(float* dst, const CUtensorMap* map, uint64_t* bar, int z, int y,
                                             int x, int chan) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(z), "r"(y), "r"(x), "r"(chan), "r"(smem_u32(bar))
      : "memory");
}

constexpr int INT = 288;                 // threads that blend; one more warp stages the boxes
constexpr int IVPT = ITILE * ITILE * ITILE / INT;       // voxels per thread
static_assert(IVPT * INT == ITILE * ITILE * ITILE, "the threads of a block share the tile evenly");
constexpr int IMAXST = 4;            // most boxes in flight or in use per block
constexpr int IRING = 28160;  // floats of staging per block (110 KB: two blocks per SM)
static_assert(IMAXST >= 1 && IRING >= ITILE_BOX && IRING % 32 == 0, "the staging area holds at least one box");
static_assert(ITILE_BX < 1024 && ITILE_BY < 1024 && ITILE_BZ < 1024, "a position in the box is packed into one word");

// What a thread keeps per voxel between the channels: the offset of corner (xl, yl, zl) in the box (until
// the box's pitches are chosen, its position there: x | y << 10 | z << 20) and the three upper weights.
// Where floor == ceil along an axis the upper corner is the lower one; its weight is zero exactly then.
struct InterpVoxel {
  unsigned base;
  float xd, yd, zd;
};

__global__ void __launch_bounds__(INT + 32, 2) k_interpolate_tiled(const __grid_constant__ InterpMaps maps, InterpArgs I) {
  // the staging area is cut into as many slots as boxes of this block's extents fit
  extern __shared__ __align__(128) float ring[];
  __shared__ __align__(8) uint64_t full[IMAXST], empty[IMAXST];
  __shared__ unsigned score[4];
  const int tid = threadIdx.x, bl = blockIdx.y;
  const InterpFrame& F = I.ex[bl];
  const unsigned od = I.out_dim;
  const unsigned nt = (od + ITILE - 1) / ITILE;
  const unsigned tk = blockIdx.x % nt, tj = (blockIdx.x / nt) % nt, ti = blockIdx.x / (nt * nt);

  // bounding box of the tile in input index units, from its eight corner voxels: a corner per lane, the
  // same in every warp
  float lo[3], hi[3];
  {
    const unsigned ci = min(ti * ITILE + ((tid & 4) ? ITILE - 1 : 0), od - 1), cj = min(tj * ITILE + ((tid & 2) ? ITILE - 1 : 0), od - 1),
                   ck = min(tk * ITILE + ((tid & 1) ? ITILE - 1 : 0), od - 1);
    interp_point(I, F, ci, cj, ck, lo[0], lo[1], lo[2]);
    static_assert(INT % 32 == 0, "whole warps");
#pragma unroll
    for (int a = 0; a < 3; a++) {
      hi[a] = lo[a];
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
        hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
      }
    }
  }
  // every voxel of the tile lies in the hull of the corners up to rounding: a margin of 0.01 cells
  bool sane = true;
#pragma unroll
  for (int a = 0; a < 3; a++) sane = sane && lo[a] > -1e6f && hi[a] < 1e6f;  // also false where all are NaN
  int bx0 = 0, by0 = 0, bz0 = 0;
  int BX = ITILE_BX, BY = ITILE_BY, BZ = ITILE_BZ, mapi = 0;  // extents of the staged box
  bool tiled = sane;
  if (sane) {
    bx0 = (int)floorf(lo[0] - 0.01f);
    by0 = (int)floorf(lo[1] - 0.01f);
    int z0 = (int)floorf(lo[2] - 0.01f);
    bz0 = z0 & ~3;  // rounds down for negative values too (two's complement): 16-byte boundary
    int nx = (int)ceilf(hi[0] + 0.01f) - bx0 + 1, ny = (int)ceilf(hi[1] + 0.01f) - by0 + 1,
        nz = (int)ceilf(hi[2] + 0.01f) - bz0 + 1;
    tiled = nx <= ITILE_BX && ny <= ITILE_BY && nz <= ITILE_BZ;
    int ix = nx <= ITILE_XY0 ? 0 : (nx - ITILE_XY0 + ITILE_XYSTEP - 1) / ITILE_XYSTEP;
    int iy = ny <= ITILE_XY0 ? 0 : (ny - ITILE_XY0 + ITILE_XYSTEP - 1) / ITILE_XYSTEP;
    int iz = nz <= ITILE_Z0 ? 0 : (nz - ITILE_Z0 + 3) / 4;
    BX = itile_xy(ix);
    BY = itile_xy(iy);
    BZ = itile_z(iz);
    mapi = (ix * ITILE_NXY + iy) * ITILE_NZ + iz;
  }

  // this thread's voxels
  const int id = (int)I.in_dim;
  const size_t ichan = (size_t)id * id * id, ochan = (size_t)od * od * od;
  const size_t b = (size_t)I.b0 + bl;
  const float* in = I.in + b * I.K * ichan;
  float* outb = I.out + b * I.K * ochan;
  InterpVoxel V[IVPT];
  unsigned livemask = 0;
  bool whole = true;  // no voxel lies on a plane of the input grid
  static_assert(INT % (ITILE * ITILE) == 0, "a thread's voxels differ in the slowest index only");
  // voxel u of this thread: (i0 + u * INT / ITILE^2, j0, k0) within the tile
  const unsigned i0 = ti * ITILE + tid / (ITILE * ITILE), j0 = tj * ITILE + (tid / ITILE) % ITILE,
                 k0 = tk * ITILE + tid % ITILE;
  const size_t ov0 = ((size_t)i0 * od + j0) * od + k0;
  const size_t ovstep = (size_t)(INT / (ITILE * ITILE)) * od * od;
#pragma unroll
  for (int u = 0; u < IVPT; u++) {
    unsigned i = i0 + u * (INT / (ITILE * ITILE));
    bool live = tid < INT && i < od && j0 < od && k0 < od;
    float gx, gy, gz;
    interp_point(I, F, min(i, od - 1), min(j0, od - 1), min(k0, od - 1), gx, gy, gz);
    InterpCell C = interp_cell(gx, gy, gz);
    V[u].base = (unsigned)(C.xl - bx0) | (unsigned)(C.yl - by0) << 10 | (unsigned)(C.zl - bz0) << 20;
    V[u].xd = C.xd; V[u].yd = C.yd; V[u].zd = C.zd;
    // belt and braces: a corner outside the staged box sends the whole block down the direct path
    bool inside = C.xl >= bx0 && C.xh < bx0 + BX && C.yl >= by0 && C.yh < by0 + BY &&
                  C.zl >= bz0 && C.zh < bz0 + BZ;
    if (live && !inside) tiled = false;
    if (live) livemask |= 1u << u;
    if (!live) V[u].base = 0;  // reads the first words of the box, stores nothing
    whole = whole && (!live || (C.xd != 0.f && C.yd != 0.f && C.zd != 0.f));
  }
  tiled = __syncthreads_and(tiled) != 0;
  whole = __syncthreads_and(whole) != 0;

  // The lanes of a warp walk the box along the tile's k axis as the rotation turned it, and the pitches of the
  // box decide how many of them meet in a bank: 2.9 lanes on average with the smallest box, 2.3 with the
  // best of four boxes that are up to four voxels longer in z and two in y.  The warps try them out.
  const ChannelRange R(I.K);
  if (tiled && R.c1 - R.c0 >= 8) {  // fewer channels do not earn the search back
    if (tid < 4) score[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int by = BY + (k & 1 ? ITILE_XYSTEP : 0), bz = BZ + (k & 2 ? 4 : 0);
      const unsigned bank = ((V[0].base & 1023u) * by + (V[0].base >> 10 & 1023u)) * bz + (V[0].base >> 20);
      const unsigned met = __reduce_max_sync(0xffffffffu, __popc(__match_any_sync(0xffffffffu, bank & 31u)));
      if ((tid & 31) == 0 && tid < INT) atomicAdd(&score[k], met);
    }
    __syncthreads();
    int best = 0;
#pragma unroll
    for (int k = 1; k < 4; k++)
      if (score[k] < score[best] && !((k & 1) && BY + ITILE_XYSTEP > ITILE_BY) && !((k & 2) && BZ + 4 > ITILE_BZ)) best = k;
    if (best & 1) {
      BY += ITILE_XYSTEP;
      mapi += ITILE_NZ;
    }
    if (best & 2) {
      BZ += 4;
      mapi += 1;
    }
  }
  const int sy = BZ, sx = BY * BZ;  // steps to the upper corners; one in z
#pragma unroll
  for (int u = 0; u < IVPT; u++)
    V[u].base = (V[u].base & 1023u) * sx + (V[u].base >> 10 & 1023u) * sy + (V[u].base >> 20);

  int c = R.c0;
  wait_for_stream();
  if (tiled) {
    const int slot = (BX * BY * BZ + 31) & ~31;  // floats from box to box: 128-byte boundaries
    const int nst = min(IMAXST, IRING / slot);
    if (tid == 0) {
      for (int s = 0; s < IMAXST; s++) {
        mbar_init(&full[s], 1);
        mbar_init(&empty[s], INT / 32);
      }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tid >= INT) {
      // The staging warp: a box as soon as every warp is done with what its slot held before.
      if (tid == INT) {
        const CUtensorMap* map = &maps.m[mapi];
        const int chan0 = (int)(b * I.K), n = R.c1 - R.c0;
        int s = 0, sent = 0;
        unsigned phase = 0;
        for (; sent < n; sent++) {
          if (sent >= nst && !mbar_wait_bounded(&empty[s], phase ^ 1u)) break;
          mbar_expect_tx(&full[s], (unsigned)(BX * BY * BZ) * (unsigned)sizeof(float));
          tma_load_box(ring + s * slot, map, &full[s], bz0, by0, bx0, chan0 + R.c0 + sent);
          if (++s == nst) {
            s = 0;
            phase ^= 1u;
          }
        }
        // Shared memory is not given up before the copies into it have landed (or had the time of another
        // bounded wait): the last one of each slot.
        for (int k = max(0, sent - nst); k < sent; k++) mbar_wait_bounded(&full[k % nst], (k / nst) & 1u);
      }
      return;
    }
    int s = 0;
    unsigned phase = 0;
    float* oc = outb + c * ochan + ov0;  // this thread's first voxel in channel c
    for (; c < R.c1; c++, oc += ochan) {
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[s], phase))) {
        // a copy did not arrive: this warp finishes through the direct reads
        if ((tid & 31) == 0) atomicAdd(&g_tma_timeouts, 1u);
        break;
      }
      const float* sm = ring + s * slot;
      if (whole) {
        // the corners lie at the same distances for every voxel of the block: four base addresses that
        // differ by uniform numbers, and a word beyond each
        const float *p0 = sm, *p1 = sm + sy, *p2 = sm + sx, *p3 = sm + sx + sy;
#pragma unroll
        for (int u = 0; u < IVPT; u++) {
          const unsigned o = V[u].base;
          InterpCell C;
          C.xd = V[u].xd; C.yd = V[u].yd; C.zd = V[u].zd;
          C.xm = __fsub_rn(1.f, C.xd); C.ym = __fsub_rn(1.f, C.yd); C.zm = __fsub_rn(1.f, C.zd);
          float res = interp_blend(C, I.minus_zero, p0[o], p0[o + 1], p1[o], p1[o + 1], p2[o], p2[o + 1], p3[o], p3[o + 1]);
          if (livemask >> u & 1u) __stcs(oc + u * ovstep, res);
        }
      } else {
#pragma unroll
        for (int u = 0; u < IVPT; u++) {
          const float* p = sm + V[u].base;
          const int vx = V[u].xd != 0.f ? sx : 0, vy = V[u].yd != 0.f ? sy : 0, vz = V[u].zd != 0.f ? 1 : 0;
          InterpCell C;
          C.xd = V[u].xd; C.yd = V[u].yd; C.zd = V[u].zd;
          C.xm = __fsub_rn(1.f, C.xd); C.ym = __fsub_rn(1.f, C.yd); C.zm = __fsub_rn(1.f, C.zd);
          float res = interp_blend(C, I.minus_zero, p[0], p[vz], p[vy], p[vy + vz], p[vx], p[vx + vz], p[vx + vy], p[vx + vy + vz]);
          if (livemask >> u & 1u) __stcs(oc + u * ovstep, res);
        }
      }
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(&empty[s]);
      if (++s == nst) {
        s = 0;
        phase ^= 1u;
      }
    }
  }
  if (c < R.c1) {
#pragma unroll 1
    for (int u = 0; u < IVPT; u++) {
      if (!(livemask >> u & 1u)) continue;
      float gx, gy, gz;
      interp_point(I, F, i0 + u * (INT / (ITILE * ITILE)), j0, k0, gx, gy, gz);
      InterpCell C = interp_cell(gx, gy, gz);
      const InterpReads Q(C, id);
      size_t ov = ov0 + u * ovstep;
      for (int cc = c; cc < R.c1; cc++) __stcs(outb + cc * ochan + ov, interp_direct(C, Q, I.minus_zero, in + cc * ichan));
    }
  }
}

// Shares of the channels for launches of `blocks` blocks without sharing: enough for `want` blocks.
static unsigned channel_shares(unsigned long blocks, int K, unsigned long want) {
  const unsigned long z = blocks == 0 ? 1 : (want + blocks - 1) / blocks;
  const unsigned shares = (unsigned)(z < (unsigned long)K ? z : (unsigned long)K);
  const unsigned per = (K + shares - 1) / shares;
  return (K + per - 1) / per;
}

unsigned interp_tile_count(unsigned out_dim) {
  unsigned nt = (out_dim + ITILE - 1) / ITILE;
  return nt * nt * nt;
}

// Tiles cost a block's start (positions, choice of a box) before the first channel, and the voxels that the last of a row has
// too many.  Of 1064 calls (1 to 40 examples, 1 to 28 channels, 20^3 to 96^3) direct reads are taken where they are no slower but for
// one, by 1.08.  Tiles / direct, us: 48^3 from 48^3, 1 x 4 / 2 x 4 channels 7.8 / 12.3 and 6.3 / 8.5; 41^3 from 48^3, 1 x 4 / 1 x 14 7.6 / 15.2
// and 5.3 / 12.0; 57^3 from 64^3, 1 x 4 15.5 and 13.2; 17^3 from 40^3, 8 x 28 22.9 and 14.4.  Input channels that fit the L1 are read there:
// 24^3 from 24^3, 1 x 14 / 8 x 28 / 16 x 28 5.7 / 21.4 / 36.4 and 4.2 / 18.7 / 38.0.  A single channel is the slower directly, because a
// thread's position serves it alone: 33^3 from 64^3, 40 examples 25.5 and 29.3, 47^3 from 24^3 50.1 and 59.4.  What the line leaves to the
// tiles because calls beside it lose: 3 x 4 channels of 48^3 18.8 and 12.3, 8 x 8 of 40^3 36.1 and 27.1.
bool interp_tiles_pay(unsigned in_dim, unsigned out_dim, int nb, int K) {
  const double tiles = (double)interp_tile_count(out_dim) * nb * K * (ITILE * ITILE * ITILE);
  const double waste = tiles / ((double)out_dim * out_dim * out_dim * nb * K);
  if (K == 1 && waste < 1.35) return tiles > 0.4e6;
  if (in_dim <= 25) return tiles > (K > 2 ? 5e6 : 2.5e6);
  return tiles > (waste < 1.35 ? 1.0e6 * waste : 1.2e6 * waste * waste);
}

cudaError_t launch_interpolate_tiled(const InterpMaps& maps, const InterpArgs& I, int nb, cudaStream_t st) {
  unsigned ntiles = interp_tile_count(I.out_dim);
  if (ntiles == 0 || nb == 0 || I.K == 0) return cudaSuccess;
  dim3 grid(ntiles, nb, channel_shares((unsigned long)ntiles * nb, I.K, 592));
  constexpr size_t smem = (size_t)IRING * sizeof(float);
  if (smem > 48 * 1024) {
    // more than the default dynamic shared memory: opted into once per device
    static bool opted[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !opted[dev]) {
      e = cudaFuncSetAttribute(k_interpolate_tiled, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      if (dev >= 0 && dev < 64) opted[dev] = true;
    }
  }
  return launch_early(k_interpolate_tiled, grid, INT + 32, smem, st, maps, I);
}

cudaError_t read_tma_timeouts(unsigned* count) {
  return cudaMemcpyFromSymbol(count, g_tma_timeouts, sizeof(unsigned));
}

// Adjoint of the interpolation (the reference leaves it as a TODO, include/libmolgrid/
// grid_interpolater.h:179): an input voxel receives the gradient of every output voxel that was blended
// from it, with the forward pass's weights.  A thread owns an INPUT voxel and looks up the output voxels
// whose position falls into the cube of two cells about it - eight on average for equal resolutions - so
// nothing is cleared and nothing is reduced in memory, and the sums have a fixed order.
//
// The map from output to input indices is affine.  First the few output voxels near the voxel's image are
// sifted by that map (a dozen instructions each); for those that pass, the position is computed as the
// forward pass computes it, which decides and gives the weight.  Both lists live in shared memory; the
// channels then read the gradient straight through it, all channels of the block for one entry at a time.
// Scattering the eight products of an output voxel with reductions was bound by these (about one lane per
// clock and SM): 3840 us for 48 x 28 channels of 48^3 with random rotations.
//
// I.in is the gradient with respect to the output (read), I.out the gradient with respect to the input
// (written).
constexpr int IG_X = 4, IG_Y = 8, IG_Z = 8;  // input voxels of a block; a warp is a brick of 2 x 2 x 8
constexpr int IG_THREADS = IG_X * IG_Y * IG_Z;
constexpr int IG_CAP = 16;                   // entries per list; a list that fills up is worked off in between
constexpr int IG_MINB = 3;

// BIG: an output grid of 2^32 voxels or more; offsets are then counted from the plane of the first candidate of a list, whose
// entries, neighbours, span few planes.
template <int CH, bool BIG = false>
__global__ void __launch_bounds__(IG_THREADS, IG_MINB) k_interpolate_gather(InterpArgs I, GatherFrames G) {
  __shared__ uint2 list[IG_CAP][IG_THREADS];  // first the candidates (i << 16 | j, k), then (weight, offset)
  const int tid = threadIdx.x, bl = blockIdx.y;
  const InterpFrame& F = I.ex[bl];
  const GatherFrame& W = G.ex[bl];
  const int id = (int)I.in_dim, od = (int)I.out_dim;
  const unsigned nz = (id + IG_Z - 1) / IG_Z, ny = (id + IG_Y - 1) / IG_Y;
  const int w = tid >> 5, z = blockIdx.x % nz * IG_Z + (tid & 7), y = blockIdx.x / nz % ny * IG_Y + (w & 3) * 2 + (tid >> 3 & 1),
            x = blockIdx.x / (nz * ny) * IG_X + (w >> 2) * 2 + (tid >> 4 & 1);
  const bool live = x < id && y < id && z < id;
  const size_t ichan = (size_t)id * id * id, ochan = (size_t)od * od * od;
  const size_t b = (size_t)I.b0 + bl;
  const int c0 = I.c0 + blockIdx.z * CH, nch = min(CH, I.K - c0);
  const float* gout = I.in + (b * I.K + c0) * ochan;
  float acc[CH];
#pragma unroll
  for (int c = 0; c < CH; c++) acc[c] = 0.f;

  int n = 0;
  auto work_off = [&]() {
    int m = 0;
    const unsigned plane = BIG && n > 0 ? list[0][tid].x >> 16 : 0u;
    for (int e = 0; e < n; e++) {
      const uint2 cand = list[e][tid];
      const unsigned i = cand.x >> 16, j = cand.x & 0xffffu, k = cand.y;
      float gx, gy, gz;
      interp_point(I, F, i, j, k, gx, gy, gz);
      const InterpCell C = interp_cell(gx, gy, gz);
      const float wx = x == C.xl ? C.xm : x == C.xh ? C.xd : 0.f, wy = y == C.yl ? C.ym : y == C.yh ? C.yd : 0.f,
                  wz = z == C.zl ? C.zm : z == C.zh ? C.zd : 0.f;
      const float w = wx * wy * wz;
      if (w != 0.f) list[m++][tid] = make_uint2(__float_as_uint(w), ((i - plane) * od + j) * od + k);
    }
    n = 0;
    wait_for_stream();
    for (int e = 0; e < m; e++) {
      const uint2 t = list[e][tid];
      const float w = __uint_as_float(t.x);
      const float* p = gout + (size_t)plane * od * od + t.y;
#pragma unroll
      for (int c = 0; c < CH; c++)
        if (c < nch) acc[c] = fmaf(w, __ldg(p + c * ochan), acc[c]);
    }
  };

  int lo[3] = {0, 0, 0}, hi[3] = {-1, -1, -1};  // zeros where the map has no use: k_interpolate_scatter adds to them
  float at[3] = {0.f, 0.f, 0.f};                // the voxel's image in output indices
  if (W.sane) {
    const float d[3] = {(float)x - W.g0[0], (float)y - W.g0[1], (float)z - W.g0[2]};
#pragma unroll
    for (int i = 0; i < 3; i++) {
      at[i] = fmaf(W.ai[i][0], d[0], fmaf(W.ai[i][1], d[1], W.ai[i][2] * d[2]));
      const float h = W.reach[i] * (1.f + W.slack);
      // inside [-1, od] before the conversions
      lo[i] = max(0, (int)ceilf(fmaxf(at[i] - h, -1.f)));
      hi[i] = min(od - 1, (int)floorf(fminf(at[i] + h, (float)od)));
    }
  }
  if (live) {
    const float limit = 1.f + W.slack;
    for (int i = lo[0]; i <= hi[0]; i++) {
      for (int j = lo[1]; j <= hi[1]; j++) {
        const float fi = (float)i - at[0], fj = (float)j - at[1], fk = (float)lo[2] - at[2];
        float dx = fmaf(W.a[0][0], fi, fmaf(W.a[0][1], fj, W.a[0][2] * fk)),
              dy = fmaf(W.a[1][0], fi, fmaf(W.a[1][1], fj, W.a[1][2] * fk)),
              dz = fmaf(W.a[2][0], fi, fmaf(W.a[2][1], fj, W.a[2][2] * fk));
        for (int k = lo[2]; k <= hi[2]; k++) {
          if (fmaxf(fmaxf(fabsf(dx), fabsf(dy)), fabsf(dz)) < limit) {
            list[n++][tid] = make_uint2((unsigned)i << 16 | (unsigned)j, (unsigned)k);
            if (n == IG_CAP) work_off();
          }
          dx += W.a[0][2];
          dy += W.a[1][2];
          dz += W.a[2][2];
        }
      }
    }
    work_off();
    float* gin = I.out + (b * I.K + c0) * ichan + ((size_t)x * id + y) * id + z;
#pragma unroll
    for (int c = 0; c < CH; c++)
      if (c < nch) gin[c * ichan] = acc[c];
  }
}

// The same for output grids about as fine as the input grid or coarser, whose voxels are few enough to be looked up
// once for a whole block: the block sifts the output voxels near its tile by the affine map, computes the position of
// each that passes once (not once for each of the eight input voxels that it was blended from), and sorts them by the
// cell of the input grid that they lie in.  An input voxel then reads the eight cells about it, whose entries are
// exactly its own, in a fixed order: by cell, then by output voxel.  The gradient is brought into shared memory for
// IC_CH channels at a time, in the order of the output, where neighbouring voxels share lines: a request costs a
// clock for each line that it touches, which bounded the reads through the lists (about ten lines each).  48 x 28
// channels of 48^3 with random rotations: 1876 -> 1072 us; 14 channels of 49^3 from 41^3: 35.8 -> 22.8 us (the lookup
// alone, with the reads left as they were: 1652 and 36.6).
constexpr int IC_X = IG_X + 1, IC_Y = IG_Y + 1, IC_Z = IG_Z + 1;  // cells of a tile, with those below its first voxels
constexpr int IC_CELLS = IC_X * IC_Y * IC_Z, IC_SCAN = (IC_CELLS + 1 + 31) / 32;
constexpr int IC_CAP = 790;  // output voxels of a block: what fits for equal resolutions, and five blocks an SM
constexpr int IC_CH = 8, IC_MINB = 5;

// BIG: an output grid of 2^32 voxels or more; offsets are then counted from the block's first plane.
// OUTSIDE: blocks without output voxels skip the rounds over the channels.  64^3 from 16^3 of the same resolution, 48 x 14
// channels, 330 -> 254 us, 48^3 from 48^3 616 -> 588; from outputs twice as coarse, which leave few such blocks, 234 -> 242, so
// these go without.
template <bool BIG, bool OUTSIDE>
__global__ void __launch_bounds__(IG_THREADS, IC_MINB) k_interpolate_cells(InterpArgs I, GatherFrames G) {
  // entries as they were found (weights of the upper corners, offset in a channel), then gradients by place
  __shared__ float4 val[2][IC_CAP];
  __shared__ float4 sorted[IC_CAP];           // entries by cell
  __shared__ unsigned cand[IC_CAP];           // position in the box of candidates, then cell and rank, then place and offset
  __shared__ unsigned short order[IC_CAP];    // what stands at a place
  __shared__ unsigned start[32 * IC_SCAN];    // first place of a cell
  __shared__ unsigned count;
  float4* const entry = val[0];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, bl = blockIdx.y;
  const InterpFrame& F = I.ex[bl];
  const GatherFrame& W = G.ex[bl];
  const int id = (int)I.in_dim, od = (int)I.out_dim;
  const unsigned nz = (id + IG_Z - 1) / IG_Z, ny = (id + IG_Y - 1) / IG_Y;
  const int z0 = blockIdx.x % nz * IG_Z, y0 = blockIdx.x / nz % ny * IG_Y, x0 = blockIdx.x / (nz * ny) * IG_X;

  for (int c = tid; c < 32 * IC_SCAN; c += IG_THREADS) start[c] = 0;
  if (tid == 0) count = 0;
  __syncthreads();
  int found = 0, plane = 0;
  if (W.sane) {
    const float h[3] = {0.5f * IC_X + W.slack, 0.5f * IC_Y + W.slack, 0.5f * IC_Z + W.slack};
    const float d[3] = {(float)x0 - 1.f + 0.5f * IC_X - W.g0[0], (float)y0 - 1.f + 0.5f * IC_Y - W.g0[1],
                        (float)z0 - 1.f + 0.5f * IC_Z - W.g0[2]};
    float at[3];  // the middle of the cells in output indices
    int lo[3], n[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      at[i] = fmaf(W.ai[i][0], d[0], fmaf(W.ai[i][1], d[1], W.ai[i][2] * d[2]));
      const float e = fmaf(fabsf(W.ai[i][0]), h[0], fmaf(fabsf(W.ai[i][1]), h[1], fabsf(W.ai[i][2]) * h[2])) + W.slack;
      lo[i] = max(0, (int)ceilf(fmaxf(at[i] - e, -1.f)));  // inside [-1, od] before the conversions
      n[i] = max(0, min(od - 1, (int)floorf(fminf(at[i] + e, (float)od))) - lo[i] + 1);
    }
    if (BIG) plane = lo[0];
    const int njk = n[1] * n[2], all = n[0] * njk;
    const float inv_njk = __fdividef(1.f, (float)njk), inv_nk = __fdividef(1.f, (float)n[2]);
    for (int c0 = 0; c0 < all; c0 += IG_THREADS) {
      const int c = c0 + tid, ci = (int)(((float)c + 0.5f) * inv_njk), r = c - ci * njk, cj = (int)(((float)r + 0.5f) * inv_nk),
                ck = r - cj * n[2];
      const float fi = (float)(lo[0] + ci) - at[0], fj = (float)(lo[1] + cj) - at[1], fk = (float)(lo[2] + ck) - at[2];
      const float dx = fmaf(W.a[0][0], fi, fmaf(W.a[0][1], fj, W.a[0][2] * fk)),
                  dy = fmaf(W.a[1][0], fi, fmaf(W.a[1][1], fj, W.a[1][2] * fk)),
                  dz = fmaf(W.a[2][0], fi, fmaf(W.a[2][1], fj, W.a[2][2] * fk));
      const bool in = c < all && fabsf(dx) < h[0] && fabsf(dy) < h[1] && fabsf(dz) < h[2];
      const unsigned m = __ballot_sync(0xffffffffu, in);
      unsigned at0 = 0;
      if (lane == 0 && m != 0u) at0 = atomicAdd(&count, __popc(m));
      at0 = __shfl_sync(0xffffffffu, at0, 0) + __popc(m & ((1u << lane) - 1u));
      if (in && at0 < IC_CAP) cand[at0] = (unsigned)(ci | cj << 10 | ck << 20);
    }
    __syncthreads();
    found = min((int)count, IC_CAP);
    for (int e = tid; e < found; e += IG_THREADS) {
      const unsigned c = cand[e], i = lo[0] + (c & 1023u), j = lo[1] + (c >> 10 & 1023u), k = lo[2] + (c >> 20);
      float gx, gy, gz;
      interp_point(I, F, i, j, k, gx, gy, gz);
      const InterpCell C = interp_cell(gx, gy, gz);
      const int cx = C.xl - x0 + 1, cy = C.yl - y0 + 1, cz = C.zl - z0 + 1;
      unsigned key = 0xffffffffu;
      if (cx >= 0 && cx < IC_X && cy >= 0 && cy < IC_Y && cz >= 0 && cz < IC_Z) {
        const unsigned cell = (cx * IC_Y + cy) * IC_Z + cz;
        key = cell | atomicAdd(&start[cell], 1u) << 16;
        entry[e] = make_float4(C.xd, C.yd, C.zd, __uint_as_float(((i - plane) * od + j) * od + k));
      }
      cand[e] = key;
    }
    __syncthreads();
    if (w == 0) {  // counts to first places
      unsigned sum = 0;
#pragma unroll
      for (int c = 0; c < IC_SCAN; c++) sum += start[lane * IC_SCAN + c];
      unsigned before = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += t;
      }
      before -= sum;
#pragma unroll
      for (int c = 0; c < IC_SCAN; c++) {
        const unsigned t = start[lane * IC_SCAN + c];
        start[lane * IC_SCAN + c] = before;
        before += t;
      }
    }
    __syncthreads();
    for (int e = tid; e < found; e += IG_THREADS) {
      const unsigned key = cand[e];
      if (key != 0xffffffffu) order[start[key & 0xffffu] + (key >> 16)] = (unsigned short)e;
    }
    __syncthreads();
    // a cell's entries by output voxel: as their places came from an atomic counter, their order is any
    for (int c = tid; c < IC_CELLS; c += IG_THREADS) {
      const int s = (int)start[c], t = (int)start[c + 1];
      for (int p = s; p < t; p++) {
        const unsigned short v = order[p];
        const unsigned key = __float_as_uint(entry[v].w);
        int q = p;
        for (; q > s && __float_as_uint(entry[order[q - 1]].w) > key; q--) order[q] = order[q - 1];
        order[q] = v;
      }
      for (int p = s; p < t; p++) {
        sorted[p] = entry[order[p]];
        cand[order[p]] = (unsigned)p;
      }
    }
    __syncthreads();
  }

  const int z = tid & 7, y = (w & 3) * 2 + (tid >> 3 & 1), x = (w >> 2) * 2 + (tid >> 4 & 1);  // in the tile
  const bool live = x0 + x < id && y0 + y < id && z0 + z < id;
  const size_t ichan = (size_t)id * id * id, ochan = (size_t)od * od * od;
  const size_t b = (size_t)I.b0 + bl;
  const ChannelRange R(I.K, IC_CH);
  float* gin = I.out + b * I.K * ichan + ((size_t)(x0 + x) * id + y0 + y) * id + z0 + z;
  wait_for_stream();
  if (OUTSIDE && found == 0) {
    if (live)
      for (int c = R.c0; c < R.c1; c++) gin[c * ichan] = 0.f;
    return;
  }
  for (int c0 = R.c0; c0 < R.c1; c0 += IC_CH) {
    const float* gout = I.in + (b * I.K + c0) * ochan + (size_t)plane * od * od;
    const int nch = min(IC_CH, R.c1 - c0);
    for (int e = tid; e < found; e += IG_THREADS) {
      const unsigned p = cand[e];
      if (p == 0xffffffffu) continue;
      const unsigned at0 = __float_as_uint(sorted[p].w);
      float v[IC_CH];
#pragma unroll
      for (int c = 0; c < IC_CH; c++) v[c] = c < nch ? __ldg(gout + c * ochan + at0) : 0.f;
      val[0][p] = make_float4(v[0], v[1], v[2], v[3]);
      val[1][p] = make_float4(v[4], v[5], v[6], v[7]);
    }
    __syncthreads();
    if (live) {
      float acc[IC_CH];
#pragma unroll
      for (int c = 0; c < IC_CH; c++) acc[c] = 0.f;
      unsigned p = 0, mid = 0, end = 0;
      for (int r = -1;;) {
        while (p == end && ++r < 4) {  // the two cells about an edge of the voxel's cube along z: they follow one another
          const int cell = ((x + (r >> 1)) * IC_Y + y + (r & 1)) * IC_Z + z;
          p = start[cell];
          mid = start[cell + 1];
          end = start[cell + 2];
        }
        if (r == 4) break;
        const float4 E = sorted[p], va = val[0][p], vb = val[1][p];
        // the voxel is the upper corner of the cell below it, the lower corner of its own
        const float wx = r >> 1 ? __fsub_rn(1.f, E.x) : E.x, wy = r & 1 ? __fsub_rn(1.f, E.y) : E.y,
                    wz = p >= mid ? __fsub_rn(1.f, E.z) : E.z;
        const float wt = wx * wy * wz;
        p++;
        if (wt == 0.f) continue;
        acc[0] = fmaf(wt, va.x, acc[0]); acc[1] = fmaf(wt, va.y, acc[1]);
        acc[2] = fmaf(wt, va.z, acc[2]); acc[3] = fmaf(wt, va.w, acc[3]);
        acc[4] = fmaf(wt, vb.x, acc[4]); acc[5] = fmaf(wt, vb.y, acc[5]);
        acc[6] = fmaf(wt, vb.z, acc[6]); acc[7] = fmaf(wt, vb.w, acc[7]);
      }
#pragma unroll
      for (int c = 0; c < IC_CH; c++)
        if (c < nch) gin[(c0 + c) * ichan] = acc[c];
    }
    __syncthreads();  // the next channels' gradients take the place of these
  }
}

// The adjoint for the examples of `which`, whose maps have no use (a quaternion of length zero, an infinite or
// enormous transform): every output voxel adds to the input voxels it was blended from, as far as there are any.  (A search of
// all output voxels by every input voxel: 48^6 positions for two grids of 48^3.)
__global__ void __launch_bounds__(256) k_interpolate_scatter(InterpArgs I, unsigned long long which) {
  wait_for_stream();
  const int bl = blockIdx.y, id = (int)I.in_dim;
  if (!(which >> bl & 1ull)) return;
  const InterpFrame& F = I.ex[bl];
  const size_t od = I.out_dim, v = (size_t)blockIdx.x * blockDim.x + threadIdx.x, ichan = (size_t)id * id * id, ochan = od * od * od;
  if (v >= ochan) return;
  float gx, gy, gz;
  interp_point(I, F, (unsigned)(v / (od * od)), (unsigned)(v / od % od), (unsigned)(v % od), gx, gy, gz);
  const InterpCell C = interp_cell(gx, gy, gz);
  const size_t b = (size_t)I.b0 + bl;
  const float* gout = I.in + b * I.K * ochan + v;
  float* gin = I.out + b * I.K * ichan;
  const int xs[2] = {C.xl, C.xh}, ys[2] = {C.yl, C.yh}, zs[2] = {C.zl, C.zh};
  const float wx[2] = {C.xm, C.xd}, wy[2] = {C.ym, C.yd}, wz[2] = {C.zm, C.zd};
  for (int k = 0; k < 8; k++) {
    const int x = xs[k >> 2], y = ys[k >> 1 & 1], z = zs[k & 1];
    const float w = wx[k >> 2] * wy[k >> 1 & 1] * wz[k & 1];
    if (w == 0.f || x < 0 || x >= id || y < 0 || y >= id || z < 0 || z >= id) continue;
    float* p = gin + ((size_t)x * id + y) * id + z;
    for (int c = 0; c < I.K; c++) atomicAdd(p + c * ichan, w * __ldg(gout + c * ochan));
  }
}

// The examples of one pass, which all take the same kernel.
static cudaError_t interpolate_backward_run(const InterpArgs& I, const GatherFrames& W, int nb, bool cells, cudaStream_t st) {
  const unsigned id = I.in_dim, tiles = ((id + IG_X - 1) / IG_X) * ((id + IG_Y - 1) / IG_Y) * ((id + IG_Z - 1) / IG_Z);
  const bool big = (unsigned long long)I.out_dim * I.out_dim * I.out_dim >> 32 != 0;
  if (cells) {
    // shares of the channels as long as the blocks fit the chip at a time
    const unsigned long room = 148ul * IC_MINB / ((unsigned long)tiles * nb), groups = ((unsigned long)I.K + IC_CH - 1) / IC_CH;
    return launch_early(big ? k_interpolate_cells<true, true> : I.out_res < 1.5f * I.in_res ? k_interpolate_cells<false, true> : k_interpolate_cells<false, false>, dim3(tiles, nb, (unsigned)std::max(1ul, std::min(room, groups))), IG_THREADS, 0, st, I, W);
  }
  // More channels per block mean fewer searches for the same voxel, fewer channels more blocks.
  const unsigned long shares = channel_shares((unsigned long)tiles * nb, I.K, 592);
  const int per = (I.K + (int)shares - 1) / (int)shares;
  const int ch = big ? 8 : per > 16 ? 32 : per > 8 ? 16 : 8;
  InterpArgs J = I;
  cudaError_t e = cudaSuccess;
  for (int left = (I.K + ch - 1) / ch; left > 0 && e == cudaSuccess; left -= 65535, J.c0 += 65535 * ch)
    e = launch_early(big ? k_interpolate_gather<8, true> : ch == 32 ? k_interpolate_gather<32> : ch == 16 ? k_interpolate_gather<16> : k_interpolate_gather<8>,
                     dim3(tiles, nb, left < 65535 ? left : 65535), IG_THREADS, 0, st, J, W);
  return e;
}

cudaError_t launch_interpolate_backward(const InterpArgs& I, const GatherFrames& W, int nb, cudaStream_t st) {
  if (I.in_dim == 0 || nb == 0 || I.K == 0) return cudaSuccess;
  // Each output voxel has a cube of its own, f cells wide and turned, so that no more of them lie in a box of cells than
  // volumes of such cubes fit in the box widened by their half diagonal on each side: resolutions that are equal, with
  // centres up to some 2600 cells away, outputs up to 0.28 % finer about the origin, and coarser ones.  Finer ones would
  // need more room than five blocks an SM have.
  const double f = (double)I.out_res / I.in_res;
  // Much coarser outputs leave a block few voxels to look up, in rounds of eight channels, where the search takes up to 32
  // together.  96^3 of 0.25 A, cells / search: from 0.5 A 4 / 24 / 28 / 40 channels 27 / 59 / 72 / 93 and 35 / 67 / 67 / 117 us, from 0.7 A
  // 4 / 28 channels 25 / 60 and 22 / 52, from 1 A 22 / 54 and 19 / 42; one wave of blocks, 28 x 48^3 from outputs twice as coarse
  // 11.7 and 15.0.
  const unsigned long tiles = (unsigned long)((I.in_dim + IG_X - 1) / IG_X) * ((I.in_dim + IG_Y - 1) / IG_Y) * ((I.in_dim + IG_Z - 1) / IG_Z);
  const bool few = f >= 2.5 || (f >= 1.75 && (I.K + 7) / 8 % 4 == 0 && tiles > 148 * IC_MINB);
  auto fits = [&](int i) {
    if (few) return false;
    const double more = 2.0 * W.ex[i].slack + 1.7321 * f;
    return 1.005 * (IC_X + more) * (IC_Y + more) * (IC_Z + more) < IC_CAP * f * f * f;
  };
  // Every example is judged by itself: the kernels sum in different orders, and its gradient is not to depend on the
  // others of its call.  Neighbours that agree share a launch (nothing is looked up for maps without use, which agree with
  // any): one for nearly all calls.
  unsigned long long which = 0;
  static_assert(INTERP_MAX_EX <= 64, "a bit per example");
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < nb && e == cudaSuccess;) {
    const int first = i;
    int cells = -1;
    for (; i < nb; i++) {
      if (W.ex[i].sane == 0) which |= 1ull << i;
      else if (cells < 0) cells = fits(i);
      else if (cells != (int)fits(i)) break;
    }
    if (first == 0 && i == nb) {
      e = interpolate_backward_run(I, W, nb, cells != 0, st);
    } else {
      InterpArgs J = I;
      GatherFrames V;
      J.b0 += first;
      std::copy(I.ex + first, I.ex + i, J.ex);
      std::copy(W.ex + first, W.ex + i, V.ex);
      e = interpolate_backward_run(J, V, i - first, cells != 0, st);
    }
  }
  if (which == 0 || e != cudaSuccess || I.out_dim == 0) return e;
  const size_t voxels = (size_t)I.out_dim * I.out_dim * I.out_dim;
  return launch_early(k_interpolate_scatter, dim3((unsigned)((voxels + 255) / 256), nb), 256, 0, st, I, which);
}

cudaError_t launch_interpolate(const InterpArgs& I, int nb, cudaStream_t st) {
  if (I.out_dim == 0 || nb == 0 || I.K == 0) return cudaSuccess;
  const unsigned od = I.out_dim, nblk = ((od + 3) / 4) * ((od + 7) / 8) * ((od + 7) / 8);
  dim3 grid(nblk, nb, channel_shares((unsigned long)nblk * nb, I.K, 1184));
  return launch_early(k_interpolate, grid, 256, 0, st, I);
}

}  // namespace lmg
