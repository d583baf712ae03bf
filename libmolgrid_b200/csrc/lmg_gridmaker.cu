// sm_100a kernels for GridMaker forward / backward / backward_gradients / backward_relevance.
//
// An atom is prepared once - fused Transform, exact footprint bounds and distance thresholds -> 64-byte atom record -
// by a thread of k_emit in front of the pass, or, in small passes of index types, by the warps that sweep it
// (k_forward_self, k_backward_quads_self); binary grids of index types have kernels of their own (lmg_occupancy.cu).
//
// Default forward: the output is zero-filled, then one warp per atom (per (atom, channel) with vector
// types) compacts the columns of the atom's footprint that lie inside the cut-off circle and adds
// the density into the grid with red.global.add (k_forward_quads*, k_forward_scatter).
// Backward passes: one warp per atom reads the grid gradient under the footprint and reduces with
// shuffles, so no global atomics are needed (k_backward_quads*, k_backward_warp).
#include "lmg_atoms.cuh"
#include "lmg_device.cuh"
#include "lmg_launch.h"

#include <algorithm>
#include <type_traits>

namespace lmg {

// ---------------------------------------------------------------------------------------------
// emit
// ---------------------------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_chan_params(EmitArgs A) {
  wait_for_stream();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= A.nb * A.T) return;
  int b = A.b0 + i / A.T, t = i % A.T;
  ChanParam cp;
  make_chan_param(A.gm, A.radii[(size_t)b * A.T + t], cp);
  A.chanp[i] = cp;
}

// One thread per atom slot of the pass.
__global__ void __launch_bounds__(256) k_emit(EmitArgs A) {
  wait_for_stream();
  let_next_begin();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool bad = false;
  if (i < A.nb * A.N) {
    int bl = i / A.N, a = i - bl * A.N;
    Rec r;
    bad = make_rec(A, A.b0 + bl, a, r);
    A.recs[i] = r;
  }
  bad = __syncthreads_or(bad) != 0;
  if (threadIdx.x == 0) put_flag(A, blockIdx.x, gridDim.x, bad);
}

// ---------------------------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------------------------

struct ItemParams {
  float x, y, z;
  float inv_ar2, inv_ar, Tg, Tcut, Tbin, w, ar;
  unsigned lox, hix, loy, hiy, loz, hiz;
  int chan;
  bool valid;
};

// The constants of an index-typed atom from its record.
__device__ __forceinline__ ItemParams item_of(const Rec& r) {
  ItemParams P;
  P.valid = ((r.c.w >> 16) & REC_VALID) != 0;
  P.x = r.a.x; P.y = r.a.y; P.z = r.a.z;
  P.chan = (int)(r.c.w & 0xffffu);
  P.w = 1.f;
  P.inv_ar2 = r.b.y; P.Tg = r.b.z; P.inv_ar = r.b.w; P.Tcut = r.d.x; P.Tbin = r.d.y; P.ar = r.d.z;
  P.lox = lo16(r.c.x); P.loy = hi16(r.c.x); P.hix = lo16(r.c.y); P.hiy = hi16(r.c.y);
  P.loz = lo16(r.c.z); P.hiz = hi16(r.c.z);
  return P;
}

// Loads the constants of work item `item` (an atom, or an (atom, channel) pair with VEC).
template <bool VEC>
__device__ __forceinline__ ItemParams load_item(const BwdArgs& G, int bl, int b, int item,
                                                float ox, float oy, float oz) {
  ItemParams P;
  int ai = VEC ? item / G.T : item;
  const Rec* rp = G.recs + (size_t)bl * G.N + ai;
  float4 ra = rp->a, rb = rp->b, rd = rp->d;
  uint4 rc = rp->c;
  P.valid = ((rc.w >> 16) & REC_VALID) != 0;
  P.x = ra.x; P.y = ra.y; P.z = ra.z;
  P.chan = VEC ? item - ai * G.T : (int)(rc.w & 0xffffu);
  P.w = 1.f;
  if (VEC) P.w = G.type_vector[((size_t)b * G.N + ai) * G.T + P.chan];
  if (VEC && G.gm.rti) {
    ChanParam cp = G.chanp[(size_t)bl * G.T + P.chan];
    P.inv_ar2 = cp.p.x; P.Tg = cp.p.y; P.inv_ar = cp.p.z; P.Tcut = cp.p.w; P.Tbin = cp.q.x;
    P.ar = cp.q.y;
    bounds_1d(ox, P.x, cp.q.z, G.gm.res, G.gm.dim, P.lox, P.hix);
    bounds_1d(oy, P.y, cp.q.z, G.gm.res, G.gm.dim, P.loy, P.hiy);
    bounds_1d(oz, P.z, cp.q.z, G.gm.res, G.gm.dim, P.loz, P.hiz);
    P.valid = P.valid && cp.q.y > 0.f;
  } else {
    P.inv_ar2 = rb.y; P.Tg = rb.z; P.inv_ar = rb.w; P.Tcut = rd.x; P.Tbin = rd.y; P.ar = rd.z;
    P.lox = lo16(rc.x); P.loy = hi16(rc.x); P.hix = lo16(rc.y); P.hiy = hi16(rc.y);
    P.loz = lo16(rc.z); P.hiz = hi16(rc.z);
  }
  return P;
}

// What a sweep multiplies to exp(-2 d^2 / ar^2), from the squared distances in the plane and along z.  Relevance (MODE 2)
// wants it to the last place: the exponent by an exact quotient and the exponential of full precision, both once per
// column or z position.  Against 64 bits, 2-norm over 400 atoms: 1.6e-7 where approximate factors, as elsewhere, give
// 2.1e-7, 6.0e-8 and 8.5e-8 for a Gaussian cut at 1.5 radii; 50 x 3000 atoms on 28x48^3: 468 and 445 us (an
// exponential per voxel: 705).
template <int MODE>
__device__ __forceinline__ float gauss_factor(float d2, const ItemParams& P, float kexp) {
  return MODE == 2 ? expf(-2.f * divide_by(d2, __fmul_rn(P.ar, P.ar), P.inv_ar2)) : ex2_approx(d2 * kexp);
}

// Backward and scatter-forward kernels: one warp per work item.  The warp first compacts the
// columns (x,y) of the item's footprint that lie within the cut-off circle, then sweeps eight
// columns at a time with four lanes along z each, and finally reduces with shuffles.  All lanes
// work on the same atom, so footprints of different size do not idle each other.
//
// Everything that depends on z alone (dz, dz^2, the z factor of the Gaussian) is the same for every
// column, so each lane keeps it in registers for its (up to) four z positions of the current chunk
// of 16 voxels; everything that depends on (x,y) alone is computed once per column at compaction
// time and parked in shared memory.  The inner step is then  rsq = dxy2 + dz2[k]  (the reference's
// own association, src/grid_maker.cu:82-92), one compare, and the density arithmetic.  The Gaussian
// is evaluated as exp(-2 dxy2/ar^2) * exp(-2 dz2/ar^2): one ex2 per column instead of one per voxel.
// One warp per block in the backward kernels: the kernel waits on its loads of the grid gradient,
// and a block of several warps keeps its registers until its slowest atom is done.
constexpr int BWD2_WARPS = 1;    // warps (work items) per block, backward kernels
constexpr int SCAT_WARPS = 4;   // the same for the scatter kernels
// One warp per block for the quad forward kernels whose work items differ a lot in size (an atom's
// footprint grows with the cube of its radius): a block of several warps keeps its registers and
// its slot until its slowest item is done.  Measured per batch of 50: index-typed forward 0.266 ->
// 0.258 ms, one-hot vector forward 0.322 -> 0.286 ms; the binary and the weighted-channel kernels
// are faster with four and keep SCAT_WARPS.
constexpr int QS_WARPS = 1;
constexpr int SELF_SPLIT = 1200;   // most of them that four warps each take
constexpr int SELF_ATOMS = 8192;   // most atom slots of a backward pass without k_emit
// Gradients on loose rows, by quads / by records and single voxels, whose lines cross at different counts: 2600 and 4000
// slots on 14x25^3 of 1 A 4.9 and 6.6, 6.1 and 7.7 us; on 8x65^3 of 0.375 A 19.6 and 20.3, 24.5 and 26.6; on 22x41^3 of
// 0.5 A 10.8 and 10.3, 13.6 and 13.2; 4x97^3 of 0.25 A 47.6 and 41.6, 62.1 and 58.8.
constexpr int LOOSE_SELF_ATOMS = 4096;
constexpr int FWD_SELF_ATOMS = 32768;  // the same for the forward pass (densities)
constexpr int REL_SELF_ATOMS = 2560;                // ... and for relevance, whose kernel is the heaviest
constexpr int BWD2_COLS = 256;  // compacted columns held per warp at a time
constexpr int ZSTEPS = 4;       // z positions per lane and chunk; a chunk covers 4*ZSTEPS voxels

template <int CAP_>
struct ColBufT {
  static constexpr unsigned CAP = CAP_;
  // x*dim + y and (gx-ax)^2 + (gy-ay)^2: one load brings both (soft types at 28x96^3, forward and both backward
  // passes: 8.72 -> 8.67 ms; index types unchanged)
  uint2 col[CAP_];
  __device__ __forceinline__ void put(unsigned slot, unsigned row, float dxy2) { col[slot] = make_uint2(row, __float_as_uint(dxy2)); }
  __device__ __forceinline__ float get(unsigned i, unsigned& row) const {
    const uint2 c = col[i];
    row = c.x;
    return __uint_as_float(c.y);
  }
};
template <int CAP_>
struct ColBufDT {
  static constexpr unsigned CAP = CAP_;
  unsigned row[CAP_];
  float dxy2[CAP_];
  float dx[CAP_];  // gx-ax
  float dy[CAP_];  // gy-ay
  __device__ __forceinline__ void put(unsigned slot, unsigned r, float d) { row[slot] = r; dxy2[slot] = d; }
  __device__ __forceinline__ float get(unsigned i, unsigned& r) const { r = row[i]; return dxy2[i]; }
};
typedef ColBufT<BWD2_COLS> ColBuf;
typedef ColBufDT<BWD2_COLS> ColBufD;

// Walk over the columns (x, y) of an item's footprint, a candidate per lane and 32 further on per round.
// Within a stretch the coordinates are carried along as floats (whole numbers, exact) and the row as an
// integer, so a round has no division and no conversion: those run on the special-function pipe, which
// the sweeps need for themselves (occupancy: 34 % of the pipe before).  Between stretches - most
// footprints are one - only the position is kept.  Of `parts` warps that share an item each walks its
// share of whole rounds.
struct Columns {
  unsigned next, end;

  __device__ __forceinline__ Columns(const ItemParams& P, unsigned part = 0, unsigned parts = 1) {
    next = 0;
    end = (P.hix - P.lox) * (P.hiy - P.loy);
    if (parts > 1) {
      const unsigned rounds = (end + 31) / 32, per = (rounds + parts - 1) / parts * 32;
      next = part * per;
      end = min(end, next + per);
    }
  }
  __device__ __forceinline__ bool more() const { return next < end; }

  // Appends the columns whose squared distance in the xy plane is <= Tcull to the buffer until it is
  // (nearly) full or the walk is over; returns how many it holds.
  template <bool WITH_D, class BUF>
  __device__ __forceinline__ unsigned compact(BUF& buf, const ItemParams& P, float Tcull, float ox, float oy, float res,
                                              unsigned dim, int lane) {
    const unsigned ny = P.hiy - P.loy;
    const float nyf = small_float(ny), inv_ny = __fdividef(1.f, nyf);
    unsigned c = next + lane;
    // small quotients through the reciprocal: off by less than the half that is added
    const unsigned xi = next != 0 ? c / ny : (unsigned)((small_float(c) + 0.5f) * inv_ny), yi = c - xi * ny;
    const unsigned q = (unsigned)(32.5f * inv_ny), r = 32u - q * ny;
    float xf = small_float(P.lox + xi), yf = small_float(P.loy + yi);
    const float yend = small_float(P.hiy), qf = small_float(q), rf = small_float(r);
    unsigned row = (P.lox + xi) * dim + P.loy + yi;
    unsigned nkept = 0;
    do {
      const float dx = __fsub_rn(__fadd_rn(ox, __fmul_rn(xf, res)), P.x), dy = __fsub_rn(__fadd_rn(oy, __fmul_rn(yf, res)), P.y);
      const float dxy2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
      const bool keep = c < end && dxy2 <= Tcull;
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const unsigned slot = nkept + __popc(m & ((1u << lane) - 1u));
        buf.put(slot, row, dxy2);
        if constexpr (WITH_D) {
          buf.dx[slot] = dx;
          buf.dy[slot] = dy;
        }
      }
      nkept += __popc(m);
      next += 32;
      c += 32;
      yf += rf;
      xf += qf;
      row += q * dim + r;
      if (yf >= yend) {
        yf -= nyf;
        xf += 1.f;
        row += dim - ny;
      }
    } while (next < end && nkept + 32 <= BUF::CAP);
    return nkept;
  }
};

// MODE 0: atom gradient (index types)          -> atom_gradients[b][a][3]
// MODE 1: atom + type gradient (vector types)  -> partial[b][a][t][3], type_gradients[b][a][t]
// MODE 2: relevance (index types)              -> relevance[b][a]
// MODE 3: backward_gradients' atom term        -> partial[b][a][t][3]  (src/grid_maker.cpp:636-662)
template <int MODE, bool BINARY>
__global__ void __launch_bounds__(BWD2_WARPS * 32) k_backward_warp(BwdArgs G) {
  wait_for_stream();
  constexpr bool VEC = MODE == 1 || MODE == 3;
  __shared__ ColBufD bufs[BWD2_WARPS];
  const GMParams& gm = G.gm;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int items_per_ex = VEC ? G.N * G.T : G.N;
  int item = blockIdx.x * BWD2_WARPS + wid;
  int bl = blockIdx.y;
  int b = G.b0 + bl;
  if (item >= items_per_ex) return;
  if (MODE == 3 || (MODE == 1 && G.type_gradients == nullptr)) {
    // an (atom, channel) pair without weight contributes nothing: leave before any other load
    int ea = item / G.T;
    if (G.type_vector[((size_t)b * G.N + ea) * G.T + (item - ea * G.T)] == 0.f) return;
  }
  ColBufD& buf = bufs[wid];

  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  ItemParams P = load_item<VEC>(G, bl, b, item, ox, oy, oz);

  size_t dim = gm.dim;
  size_t chan_off = ((size_t)b * G.T + P.chan) * dim * dim * dim;
  const float* diff = G.diff + chan_off;
  const float* dens = MODE == 2 ? G.density + chan_off : nullptr;

  float agx = 0.f, agy = 0.f, agz = 0.f, tg = 0.f;
  bool want_ag = MODE == 0 || ((MODE == 1 || MODE == 3) && P.w != 0.f);
  float Tcull = (MODE == 0 || MODE == 3) ? P.Tcut : fmaxf(P.Tcut, BINARY ? P.Tbin : -1.f);
  float inx = 0.f, iny = 0.f, inz = 0.f, intg = 0.f;  // MODE 3: incoming gradients of this item
  if (MODE == 3) {
    size_t gi = (size_t)b * G.N + item / G.T;
    inx = G.ag_in[gi * 3]; iny = G.ag_in[gi * 3 + 1]; inz = G.ag_in[gi * 3 + 2];
    intg = G.tg_in[gi * G.T + P.chan];
    if (!want_ag) P.valid = false;  // zero-weight channels contribute nothing (src/grid_maker.cpp:573)
  }
  const float kexp = P.inv_ar2 * NEG2_LOG2E;
  const float k4 = 4.f * P.inv_ar2, kD = -gm.D * P.inv_ar2, kE = -gm.E * P.inv_ar;  // sign of -(s*dv) folded in
  const bool has_tail = gm.ta != 0.f || gm.tb != 0.f;
  const float kDn = has_tail ? -0.25f * gm.D : 0.f, kEn = has_tail ? -0.25f * gm.E * P.ar : 0.f;  // in units of k4

  if (P.valid) {
    int grp = lane >> 2, sub = lane & 3;
    for (Columns cols(P); cols.more();) {
      const unsigned nkept = cols.compact<true>(buf, P, Tcull, ox, oy, gm.res, gm.dim, lane);
      __syncwarp();
      for (unsigned zc = P.loz; zc < P.hiz; zc += 4 * ZSTEPS) {
        // this lane's z positions of the chunk; positions past the footprint get NaN, which fails
        // every comparison below
        unsigned z0 = zc + sub;
        float dzt[ZSTEPS], dz2t[ZSTEPS], ezt[ZSTEPS];
#pragma unroll
        for (int k = 0; k < ZSTEPS; k++) {
          unsigned zz = z0 + 4 * k;
          float dz = __fsub_rn(voxel_coord(oz, zz, gm.res), P.z);
          dzt[k] = dz;
          dz2t[k] = zz < P.hiz ? __fmul_rn(dz, dz) : CUDART_NAN_F;
          ezt[k] = gauss_factor<MODE>(dz2t[k], P, kexp);
        }
        for (unsigned i = grp; i < nkept; i += 8) {
          float dxy2 = buf.dxy2[i], dx = buf.dx[i], dy = buf.dy[i];
          size_t rowoff = (size_t)buf.row[i] * dim + z0;
          const float* row = diff + rowoff;
          float exy = gauss_factor<MODE>(dxy2, P, kexp);
          // the loads of the four z steps are issued together before any is used.  (Fetching one
          // column ahead was measured slower: the extra registers cost more occupancy than the
          // deeper queue of loads gains.)
          float rsqv[ZSTEPS], dvv[ZSTEPS];
          bool okv[ZSTEPS];
#pragma unroll
          for (int k = 0; k < ZSTEPS; k++) {
            rsqv[k] = __fadd_rn(dxy2, dz2t[k]);
            okv[k] = rsqv[k] <= Tcull;
            dvv[k] = okv[k] ? __ldg(row + 4 * k) : 0.f;
          }
          float fsum = 0.f;  // sum over the column of -(d density / d dist) / dist * dv
          if constexpr (MODE == 0) {
            // Without branches: the tail's factor in units of 4 / ar^2 is at most one where it is taken, zero beyond the
            // cut-off and for a NaN distance.  Waits on its loads at half of the issue rate: 17 x 700 / 1500 / 4000 slots on 22x41^3 26.0 / 41.0 /
            // 98.1 us with a branch per voxel, 22.7 / 35.4 / 82.9 like this; against 64 bits 2.3e-7 and 1.7e-7, because
            // the factor's constant is exact in these units.
#pragma unroll
            for (int k = 0; k < ZSTEPS; k++) {
              const float t = fma_sat(kEn, rsqrt_approx(rsqv[k]), kDn);
              const float f = (rsqv[k] <= P.Tg ? exy * ezt[k] : t) * dvv[k];
              fsum += f;
              agz = fmaf(f, dzt[k], agz);
            }
          }
#pragma unroll
          for (int k = 0; k < (MODE == 0 ? 0 : ZSTEPS); k++) {
            if (!okv[k]) continue;
            float dz = dzt[k], rsq = rsqv[k], dv = dvv[k];
            float g = exy * ezt[k];  // exp(-2 rsq / ar^2)
            if (MODE == 3) {
              // second derivatives H_ab = alpha*delta_a*delta_b + [a==b]*beta of the density
              // (src/grid_maker.cu:812-878); delta = atom - grid point
              float alpha, beta;
              if (rsq <= P.Tg) {
                alpha = 16.f * g * P.inv_ar2 * P.inv_ar2;
                beta = -4.f * g * P.inv_ar2;
              } else {
                float id = rsqrt_approx(rsq);
                float S = fmaf(gm.D * P.inv_ar, rsq * id, gm.E);
                beta = S * id * P.inv_ar;
                alpha = fmaf(gm.D * P.inv_ar2, id * id, -beta * id * id);
              }
              float dot = fmaf(dx, inx, fmaf(dy, iny, dz * inz));
              float wa = P.w * alpha * dot;
              float wb = P.w * beta;
              float tt = alpha * intg;
              float bt = beta * intg;
              agx = fmaf(dv, fmaf(wa, dx, fmaf(wb, inx, fmaf(tt, dx * dx, bt))), agx);
              agy = fmaf(dv, fmaf(wa, dy, fmaf(wb, iny, fmaf(tt, dy * dy, bt))), agy);
              agz = fmaf(dv, fmaf(wa, dz, fmaf(wb, inz, fmaf(tt, dz * dz, bt))), agz);
            } else if (MODE != 2) {
              if (want_ag && rsq <= P.Tcut) {
                // -(d density / d dist) / dist * dv, src/grid_maker.cu:881-919; rsq == 0 contributes
                // nothing because dx = dy = dz = 0 there
                float s = rsq <= P.Tg ? k4 * g : fmaf(kE, rsqrt_approx(rsq), kD);
                float f = s * dv;
                fsum += f;
                agz = fmaf(f, dz, agz);
              }
            }
            if (MODE == 1 || MODE == 2) {
              float v;
              if (BINARY) {
                v = rsq < P.Tbin ? 1.f : 0.f;
              } else if (MODE == 2) {
                v = rsq <= P.Tg ? g : tail_quotient(rsq, P.ar, P.inv_ar, gm.A, gm.B, gm.C);
                v = rsq <= P.Tcut ? v : 0.f;
              } else {
                float sq = sqrt_approx(rsq * P.inv_ar2);
                float q = fmaxf(fmaf(fmaf(gm.A, sq, gm.B), sq, gm.C), 0.f);
                v = rsq <= P.Tg ? g : q;
                v = rsq <= P.Tcut ? v : 0.f;
              }
              if (MODE == 1) {
                tg = fmaf(v, dv, tg);
              } else if (v > 0.f) {
                float de = __ldg(dens + rowoff + 4 * k);
                if (de > 0.f) tg += divide_near(__fmul_rn(dv, v), de);
              }
            }
          }  // k
          if (MODE == 0 || MODE == 1) {
            agx = fmaf(fsum, dx, agx);
            agy = fmaf(fsum, dy, agy);
          }
        }
      }
      __syncwarp();
    }
  }
  if (MODE == 0) {
    // k4 is infinite for radii below 1.1e-19, within whose reach there is hardly a voxel: nothing times it is nothing
    agx = agx != 0.f ? agx * k4 : 0.f;
    agy = agy != 0.f ? agy * k4 : 0.f;
    agz = agz != 0.f ? agz * k4 : 0.f;
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    if (MODE != 2) {
      agx += __shfl_xor_sync(0xffffffffu, agx, o);
      agy += __shfl_xor_sync(0xffffffffu, agy, o);
      agz += __shfl_xor_sync(0xffffffffu, agz, o);
    }
    if (MODE == 1 || MODE == 2) tg += __shfl_xor_sync(0xffffffffu, tg, o);
  }
  if (lane == 0) {
    size_t ai = (size_t)b * G.N + (VEC ? item / G.T : item);
    if (MODE == 0) {
      G.atom_gradients[ai * 3] = agx;
      G.atom_gradients[ai * 3 + 1] = agy;
      G.atom_gradients[ai * 3 + 2] = agz;
    } else if (MODE == 1 || MODE == 3) {
      size_t pi = (size_t)bl * G.N * G.T + item;
      G.partial[pi * 3] = agx;
      G.partial[pi * 3 + 1] = agy;
      G.partial[pi * 3 + 2] = agz;
      if (MODE == 1 && G.type_gradients != nullptr) G.type_gradients[ai * G.T + P.chan] = tg;
    } else {
      G.relevance[ai] = tg;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// forward by scatter: the grid is zero-filled first, then one warp per atom (or per (atom, channel)
// pair with vector types) sweeps the atom's footprint exactly as the backward kernel does and adds
// its density into the grid with fire-and-forget reductions (red.global.add.f32), which resolve in
// L2.  No lists, no per-region work: the cost is proportional to the atoms' footprints.
// ---------------------------------------------------------------------------------------------
template <bool BINARY, bool PRECISE, bool VEC>  // not <true, *, false>: k_forward_binary
__global__ void __launch_bounds__(SCAT_WARPS * 32) k_forward_scatter(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBuf bufs[SCAT_WARPS];
  const GMParams& gm = G.gm;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int items_per_ex = VEC ? G.N * G.T : G.N;
  int item = blockIdx.x * SCAT_WARPS + wid;
  int bl = blockIdx.y;
  int b = G.b0 + bl;
  if (item >= items_per_ex) return;
  if (VEC) {
    // an (atom, channel) pair without weight contributes nothing: leave before any other load
    int ea = item / G.T;
    if (G.type_vector[((size_t)b * G.N + ea) * G.T + (item - ea * G.T)] == 0.f) return;
  }
  ColBuf& buf = bufs[wid];

  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  ItemParams P = load_item<VEC>(G, bl, b, item, ox, oy, oz);
  if (!P.valid || (VEC && P.w == 0.f)) return;  // zero weights add nothing (src/grid_maker.cpp:229)

  size_t dim = gm.dim;
  float* out = G.out_grid + ((size_t)b * G.T + P.chan) * dim * dim * dim;
  const float Tcull = BINARY ? P.Tbin : P.Tcut;
  const float kexp = P.inv_ar2 * NEG2_LOG2E;

  int grp = lane >> 2, sub = lane & 3;
  for (Columns cols(P); cols.more();) {
    const unsigned nkept = cols.compact<false>(buf, P, Tcull, ox, oy, gm.res, gm.dim, lane);
    __syncwarp();
    for (unsigned zc = P.loz; zc < P.hiz; zc += 4 * ZSTEPS) {
      unsigned z0 = zc + sub;
      float dz2t[ZSTEPS], ezt[ZSTEPS];
#pragma unroll
      for (int k = 0; k < ZSTEPS; k++) {
        unsigned zz = z0 + 4 * k;
        float dz = __fsub_rn(voxel_coord(oz, zz, gm.res), P.z);
        dz2t[k] = zz < P.hiz ? __fmul_rn(dz, dz) : CUDART_NAN_F;
        ezt[k] = (BINARY || PRECISE) ? 0.f : ex2_approx(dz2t[k] * kexp);
      }
      for (unsigned i = grp; i < nkept; i += 8) {
        unsigned cell;
        float dxy2 = buf.get(i, cell);
        float* row = out + (size_t)cell * dim + z0;
        float exy = (BINARY || PRECISE) ? 0.f : ex2_approx(dxy2 * kexp);
#pragma unroll
        for (int k = 0; k < ZSTEPS; k++) {
          float rsq = __fadd_rn(dxy2, dz2t[k]);
          if (BINARY) {
            if (rsq < P.Tbin) atomicAdd(row + 4 * k, P.w);  // type vectors: weights add up
          } else {
            if (!(rsq <= P.Tcut)) continue;
            float v;
            if (PRECISE) {
              v = density_precise(rsq, P.ar, P.Tg, P.Tcut, gm.A, gm.B, gm.C);
            } else {
              float sq = sqrt_approx(rsq * P.inv_ar2);
              float q = fmaxf(fmaf(fmaf(gm.A, sq, gm.B), sq, gm.C), 0.f);
              v = rsq <= P.Tg ? exy * ezt[k] : q;
            }
            if (VEC) v *= P.w;
            if (v != 0.f) atomicAdd(row + 4 * k, v);
          }
        }
      }
    }
    __syncwarp();
  }
}

// Grid term of backward_gradients by scatter (src/grid_maker.cpp:618-634): per (atom, channel) with
// non-zero weight, every voxel within the cut-off receives
//   density * type_gradient  -  w * ((d density/d dist)/dist) * (delta . atom_gradient),
// delta = grid point - atom.  The output is zero-filled before the launch.
__global__ void __launch_bounds__(SCAT_WARPS * 32) k_gradgrad_scatter(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBufD bufs[SCAT_WARPS];
  const GMParams& gm = G.gm;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int item = blockIdx.x * SCAT_WARPS + wid;
  int bl = blockIdx.y;
  int b = G.b0 + bl;
  if (item >= G.N * G.T) return;
  // an (atom, channel) pair without weight contributes nothing: leave before any other load
  if (G.type_vector[((size_t)b * G.N + item / G.T) * G.T + item % G.T] == 0.f) return;
  ColBufD& buf = bufs[wid];

  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  ItemParams P = load_item<true>(G, bl, b, item, ox, oy, oz);
  if (!P.valid || P.w == 0.f) return;

  size_t dim = gm.dim;
  float* out = G.out_grid + ((size_t)b * G.T + P.chan) * dim * dim * dim;
  size_t gi = (size_t)b * G.N + item / G.T;
  const float inx = G.ag_in[gi * 3], iny = G.ag_in[gi * 3 + 1], inz = G.ag_in[gi * 3 + 2];
  const float intg = G.tg_in[gi * G.T + P.chan];
  const float kexp = P.inv_ar2 * NEG2_LOG2E;
  // -w * (d density/d dist)/dist: Gaussian 4 w g / ar^2; tail -w (D/ar^2 + E/(ar dist))
  const float k4 = 4.f * P.inv_ar2 * P.w, kD = -gm.D * P.inv_ar2 * P.w, kE = -gm.E * P.inv_ar * P.w;

  int grp = lane >> 2, sub = lane & 3;
  for (Columns cols(P); cols.more();) {
    const unsigned nkept = cols.compact<true>(buf, P, P.Tcut, ox, oy, gm.res, gm.dim, lane);
    __syncwarp();
    for (unsigned zc = P.loz; zc < P.hiz; zc += 4 * ZSTEPS) {
      unsigned z0 = zc + sub;
      float dzt[ZSTEPS], dz2t[ZSTEPS], ezt[ZSTEPS];
#pragma unroll
      for (int k = 0; k < ZSTEPS; k++) {
        unsigned zz = z0 + 4 * k;
        float dz = __fsub_rn(voxel_coord(oz, zz, gm.res), P.z);
        dzt[k] = dz * inz;
        dz2t[k] = zz < P.hiz ? __fmul_rn(dz, dz) : CUDART_NAN_F;
        ezt[k] = ex2_approx(dz2t[k] * kexp);
      }
      for (unsigned i = grp; i < nkept; i += 8) {
        float dxy2 = buf.dxy2[i];
        float dotxy = fmaf(buf.dx[i], inx, buf.dy[i] * iny);
        float* row = out + (size_t)buf.row[i] * dim + z0;
        float exy = ex2_approx(dxy2 * kexp);
#pragma unroll
        for (int k = 0; k < ZSTEPS; k++) {
          float rsq = __fadd_rn(dxy2, dz2t[k]);
          if (!(rsq <= P.Tcut)) continue;
          float g = exy * ezt[k];
          float sq = sqrt_approx(rsq * P.inv_ar2);
          float q = fmaxf(fmaf(fmaf(gm.A, sq, gm.B), sq, gm.C), 0.f);
          bool gauss = rsq <= P.Tg;
          float val = gauss ? g : q;
          float s = gauss ? k4 * g : fmaf(kE, rsqrt_approx(rsq), kD);
          float dot = rsq > 0.f ? dotxy + dzt[k] : 0.f;
          float gval = fmaf(val, intg, s * dot);
          if (gval != 0.f) atomicAdd(row + 4 * k, gval);
        }
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------
// Quad kernels: the same work items, for grids whose rows are 16-byte aligned (dim % 4 == 0 and an
// aligned base).  Here a lane owns a whole column (x,y) and walks it in aligned quads of four z
// voxels: the forward adds a quad with one red.global.add.v4.f32, the backward reads it with one
// 16-byte load, so a warp has 32 columns x 4 quads in flight per round trip to memory instead of
// 8 columns x 4 voxels.  What depends on z alone sits in a small shared table per warp (one pass
// covers 32 z positions from the aligned start of the footprint).  This lane-per-column layout
// serves the backward passes of index types and of (atom, channel) items, the atom gradients alone of
// type vectors and their densities in the reference's order of operations, which spend their time
// issuing instructions and amortise the per-column terms over the quads of a column; the other forward
// passes and the type gradients by atom are bound by the lines that they touch and use the (column,
// z-quad) layout of qlane_sweep instead.
// ---------------------------------------------------------------------------------------------
constexpr int QPASS = 8;  // quads per pass

struct __align__(16) ZTabs {
  float4 dz2[QPASS];  // (gz-az)^2 (relevance: negated), NaN outside [loz, hiz)
  float4 ez[QPASS];   // exp(-2 dz2 / ar^2)
  float4 dz[QPASS];   // gz-az
  float lo[QPASS];    // smallest dz2 of the quad (NaN when no z of it lies in the footprint)
};

template <int MODE = 0>
__device__ __forceinline__ void fill_ztabs(ZTabs& zt, unsigned zc, const ItemParams& P, float oz, float res,
                                           float kexp, int lane) {
  unsigned zz = zc + lane;
  float dz = __fsub_rn(voxel_coord(oz, zz, res), P.z);
  bool in = zz >= P.loz && zz < P.hiz;
  float d2 = in ? __fmul_rn(dz, dz) : CUDART_NAN_F;
  reinterpret_cast<float*>(zt.dz2)[lane] = MODE == 2 ? -d2 : d2;  // relevance wants it negated
  reinterpret_cast<float*>(zt.ez)[lane] = gauss_factor<MODE>(d2, P, kexp);
  reinterpret_cast<float*>(zt.dz)[lane] = dz;
  float lo = fminf(d2, __shfl_xor_sync(0xffffffffu, d2, 1));  // fminf skips the NaN entries
  lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, 2));
  if ((lane & 3) == 0) zt.lo[lane >> 2] = lo;
}

// Rows of any alignment (a side that is no multiple of four, on an aligned tensor).  A column starts 0 to 3 floats
// beyond a 16-byte boundary; its quads are the aligned ones of memory all the same, and reach up to three voxels
// into the rows beside it, where they add zero or are not looked at.  What depends on z is tabulated once for each
// of the four shifts.  Against lanes of one voxel, 17 x 700 atoms on 22x41^3: forward
// 44.9 -> 39.3 us; 300 atoms on 28x41^3, forward and gradients in launches of their own: 25.9 -> 11.4.
__device__ __forceinline__ unsigned quad_shift(unsigned chan_low, unsigned row, unsigned dim, unsigned zc) {
  return (chan_low + row * dim + zc) & 3u;
}

struct __align__(16) LooseForward {
  float4 dz2[QPASS], ez[QPASS];
  float lo[QPASS], pad[8];  // 80 words: two shifts' quads lie in different banks
};
struct __align__(16) LooseBackward {
  float4 dz2[QPASS], ez[QPASS], dz[QPASS];
  float lo[QPASS], pad[8];  // 112 words
};
typedef LooseBackward LooseZTabs[4];

// squared distances times `scale`
template <bool SCALED, int MODE = 0, class TAB>
__device__ __forceinline__ void fill_loose(TAB (&f)[4], unsigned zc, const ItemParams& P, float oz, float res, float kexp,
                                           float scale, int lane) {
#pragma unroll
  for (int t = 0; t < 4; t++) {
    const unsigned zz = zc - t + lane;
    const bool in = zz >= P.loz && zz < P.hiz;  // not the places before zero either, which voxel_coord() does not take
    const float dz = in ? __fsub_rn(voxel_coord(oz, zz, res), P.z) : 0.f;
    float d2 = in ? __fmul_rn(dz, dz) : CUDART_NAN_F;
    if (SCALED) d2 *= scale;
    reinterpret_cast<float*>(f[t].dz2)[lane] = MODE == 2 ? -d2 : d2;
    reinterpret_cast<float*>(f[t].ez)[lane] = gauss_factor<MODE>(d2, P, kexp);
    if constexpr (std::is_same<TAB, LooseBackward>::value) reinterpret_cast<float*>(f[t].dz)[lane] = dz;
    float lo = fminf(d2, __shfl_xor_sync(0xffffffffu, d2, 1));
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, 2));
    if ((lane & 3) == 0) f[t].lo[lane >> 2] = lo;
  }
}

// quads along z that a footprint spans with the widest shift
__device__ __forceinline__ unsigned loose_span(const ItemParams& P) { return (P.hiz - P.loz + 6) >> 2; }

// where the pass's examples end, counted from an example's channel
__device__ __forceinline__ long floats_left(const BwdArgs& G, size_t chan_off, size_t dim) {
  return (long)((size_t)(G.b0 + G.nb) * G.T * dim * dim * dim - chan_off);
}

__device__ __forceinline__ void red_add_v4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
               : "memory");
}

// Sweep over the compacted columns of a footprint with the lanes laid out as (column, z-quad): ZQ
// lanes along z hold one aligned quad each, 32/ZQ columns per step (ZQ need not divide 32: with 3, 5
// or 6 quads two lanes idle, which costs less than a quad lane without voxels for every column).  A lane's z terms live in
// registers for the whole item, and the lanes of a column touch neighbouring 16-byte pieces of one
// line, so a warp's reduction reaches 32/ZQ rows instead of 32 (the scatter kernels are bound by the
// number of distinct lines their reductions touch).  `quad(i, dxy2, exy, d2v, ev, dzv, off)` is called
// by every lane whose quad can hold a voxel of the item: i = column slot, off = row*dim + z of the quad.
template <int ZQ, bool SCALED, class BUF, class QuadFn>
__device__ __forceinline__ void qlane_sweep(const ItemParams& P, const BUF& buf, unsigned nkept, size_t dim,
                                            float oz, float res, float kexp, float Tcull, float scale, int lane,
                                            QuadFn quad) {
  constexpr int CPI = 32 / ZQ;
  const int zq = lane % ZQ, cl = lane / ZQ;
  for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * ZQ) {
    float d2v[4], ev[4], dzv[4];
    float lo = CUDART_INF_F;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      unsigned zz = zc + 4 * zq + j;
      dzv[j] = __fsub_rn(voxel_coord(oz, zz, res), P.z);
      bool in = zz >= P.loz && zz < P.hiz;
      d2v[j] = in ? __fmul_rn(dzv[j], dzv[j]) : CUDART_NAN_F;
      if (SCALED) d2v[j] *= scale;
      ev[j] = ex2_approx(d2v[j] * kexp);
      lo = fminf(lo, d2v[j]);  // fminf skips the NaN entries
    }
    const size_t zoff = zc + 4 * zq;
    for (unsigned i = 32 % ZQ == 0 || cl < CPI ? cl : nkept; i < nkept; i += CPI) {
      unsigned row;
      float dxy2 = buf.get(i, row);
      if (SCALED) dxy2 *= scale;
      if (!(__fadd_rn(dxy2, lo) <= Tcull)) continue;  // also false for NaN: no z in range
      quad(i, dxy2, ex2_approx(dxy2 * kexp), d2v, ev, dzv, (size_t)row * dim + zoff);
    }
  }
}

// The sweep with as many lanes along z as the footprint spans aligned quads.  Measured: dense type
// vectors at 96^3 (spans of 6) 2.16 -> 1.97 ms per 4 examples; the index-typed benchmark (spans of
// 3 to 5) unchanged at 0.259 ms per 50.
// SCALED: squared distances are handed to `quad` (and compared with Tcull) in units of the squared
// atom radius, `scale` = 1 / ar^2 and `kexp` = -2 log2(e): one multiplication per column instead of
// one per voxel for callers that want rsq / ar^2 (density only: the binary test keeps rsq itself).
// The sweep on rows of any alignment; off may be up to three floats before the row.  (The lanes along z as a
// variable instead of a template argument: 39.3 -> 41.4 us at the size above.)
template <int ZQ, bool SCALED, class BUF, class QuadFn>
__device__ __forceinline__ void loose_sweep(const BUF& buf, unsigned nkept, unsigned dim, unsigned chan_low,
                                            const LooseForward (&tabs)[4], unsigned zc, float kexp, float Tcull, float scale,
                                            int lane, QuadFn quad) {
  constexpr int CPI = 32 / ZQ;
  const int zq = lane % ZQ, cl = lane / ZQ;
  for (unsigned c0 = 0; c0 < nkept; c0 += CPI) {
    const unsigned i = c0 + cl;
    if (cl >= CPI || i >= nkept) continue;
    unsigned row;
    float dxy2 = buf.get(i, row);
    if (SCALED) dxy2 *= scale;
    const unsigned t = quad_shift(chan_low, row, dim, zc);
    if (!(__fadd_rn(dxy2, tabs[t].lo[zq]) <= Tcull)) continue;
    const float4 d2 = tabs[t].dz2[zq], e = tabs[t].ez[zq];
    const float d2v[4] = {d2.x, d2.y, d2.z, d2.w}, ev[4] = {e.x, e.y, e.z, e.w};
    quad(i, dxy2, ex2_approx(dxy2 * kexp), d2v, ev, d2v, (long)((size_t)row * dim + zc + 4 * zq) - (long)t);
  }
}
template <bool SCALED, class BUF, class QuadFn>
__device__ __forceinline__ void loose_sweep_span(const ItemParams& P, const BUF& buf, unsigned nkept, unsigned dim,
                                                 unsigned chan_low, LooseForward (&tabs)[4], float oz, float res, float kexp,
                                                 float Tcull, float scale, int lane, QuadFn quad) {
  const unsigned span = loose_span(P);
  for (unsigned zc = P.loz; zc < P.hiz + 3; zc += 4 * QPASS) {
    fill_loose<SCALED>(tabs, zc, P, oz, res, kexp, scale, lane);
    __syncwarp();
    if (span <= 2) loose_sweep<2, SCALED>(buf, nkept, dim, chan_low, tabs, zc, kexp, Tcull, scale, lane, quad);
    else if (span == 3) loose_sweep<3, SCALED>(buf, nkept, dim, chan_low, tabs, zc, kexp, Tcull, scale, lane, quad);
    else if (span == 4) loose_sweep<4, SCALED>(buf, nkept, dim, chan_low, tabs, zc, kexp, Tcull, scale, lane, quad);
    else if (span == 5) loose_sweep<5, SCALED>(buf, nkept, dim, chan_low, tabs, zc, kexp, Tcull, scale, lane, quad);
    else loose_sweep<8, SCALED>(buf, nkept, dim, chan_low, tabs, zc, kexp, Tcull, scale, lane, quad);
    __syncwarp();
  }
}

template <bool SCALED, class BUF, class QuadFn>
__device__ __forceinline__ void qlane_sweep_span_t(unsigned span, const ItemParams& P, const BUF& buf, unsigned nkept,
                                                   size_t dim, float oz, float res, float kexp, float Tcull,
                                                   float scale, int lane, QuadFn quad) {
  if (span <= 2) qlane_sweep<2, SCALED>(P, buf, nkept, dim, oz, res, kexp, Tcull, scale, lane, quad);
  else if (span == 3) qlane_sweep<3, SCALED>(P, buf, nkept, dim, oz, res, kexp, Tcull, scale, lane, quad);
  else if (span == 4) qlane_sweep<4, SCALED>(P, buf, nkept, dim, oz, res, kexp, Tcull, scale, lane, quad);
  else if (span == 5) qlane_sweep<5, SCALED>(P, buf, nkept, dim, oz, res, kexp, Tcull, scale, lane, quad);
  else if (span == 6) qlane_sweep<6, SCALED>(P, buf, nkept, dim, oz, res, kexp, Tcull, scale, lane, quad);
  else qlane_sweep<8, SCALED>(P, buf, nkept, dim, oz, res, kexp, Tcull, scale, lane, quad);
}
template <class BUF, class QuadFn>
__device__ __forceinline__ void qlane_sweep_span(unsigned span, const ItemParams& P, const BUF& buf, unsigned nkept,
                                                 size_t dim, float oz, float res, float kexp, float Tcull, int lane,
                                                 QuadFn quad) {
  qlane_sweep_span_t<false>(span, P, buf, nkept, dim, oz, res, kexp, Tcull, 1.f, lane, quad);
}

// The same with the lanes along z as a variable: one copy of a large `quad` instead of six.  Atoms of one launch differ in
// their spans, and several copies of such a loop do not fit the instruction cache (k_backward_quads_atom).
template <class BUF, class QuadFn>
__device__ __forceinline__ void qlane_sweep_any(unsigned span, const ItemParams& P, const BUF& buf, unsigned nkept,
                                                size_t dim, float oz, float res, float kexp, float Tcull, int lane,
                                                QuadFn quad) {
  const unsigned nq = span <= 2 ? 2u : span <= 6 ? span : 8u, cpi = 32u / nq, cl = lane / nq, zq = lane - cl * nq;
  for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * nq) {
    float d2v[4], ev[4], dzv[4];
    float lo = CUDART_INF_F;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const unsigned zz = zc + 4 * zq + j;
      dzv[j] = __fsub_rn(voxel_coord(oz, zz, res), P.z);
      d2v[j] = zz >= P.loz && zz < P.hiz ? __fmul_rn(dzv[j], dzv[j]) : CUDART_NAN_F;
      ev[j] = ex2_approx(d2v[j] * kexp);
      lo = fminf(lo, d2v[j]);  // fminf skips the NaN entries
    }
    const size_t zoff = zc + 4 * zq;
#pragma unroll 1
    for (unsigned i = cl < cpi ? cl : nkept; i < nkept; i += cpi) {
      unsigned row;
      const float dxy2 = buf.get(i, row);
      if (!(__fadd_rn(dxy2, lo) <= Tcull)) continue;  // also false for NaN: no z in range
      quad(i, dxy2, ex2_approx(dxy2 * kexp), d2v, ev, dzv, (size_t)row * dim + zoff);
    }
  }
}

// number of aligned quads between the first and the last z of a footprint
__device__ __forceinline__ unsigned quad_span(const ItemParams& P) { return (P.hiz - (P.loz & ~3u) + 3) >> 2; }

// The sweep of one work item of the forward pass on aligned quads, whose constants are in P.  Of
// `parts` warps that share an item, this one takes the `part`-th share of its columns.
// LATE: the grid is zero only once wait_for_stream() returns, which is called when the first columns are at hand (zeros
// and sums of 300 atoms in 28x48^3: 5.8 us waiting before the columns, 5.6 like this).
// PACKED: the tail clamped after packed multiply-adds, which is the faster form on loose rows but where four warps share an
// atom and registers are short.  14 channels of 41^3, 1300 / 5000 atoms 9.0 / 14.4 us with the clamp in the multiply-add,
// 8.8 / 13.9 packed, 65^3 17.9 / 27.4 and 17.1 / 26.2; 1000 atoms by four warps 7.0 and 8.4.
template <bool VEC, bool LOOSE, bool LATE = false, bool PACKED = LOOSE>
__device__ __forceinline__ void forward_quads_core(const BwdArgs& G, const ItemParams& P, int b, float ox, float oy,
                                                   float oz, ColBuf& buf, LooseForward (&tabs)[4], int lane,
                                                   unsigned part = 0, unsigned parts = 1) {
  const GMParams& gm = G.gm;
  size_t dim = gm.dim;
  const size_t chan_off = ((size_t)b * G.T + P.chan) * dim * dim * dim;
  float* out = G.out_grid + chan_off;
  const long whole = LOOSE ? floats_left(G, chan_off, dim) - 4 : 0;  // the last place of a quad
  auto add = [&](auto off, const float (&v)[4]) {
    if (!LOOSE || (long)off <= whole) {
      red_add_v4(out + off, v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++)
        if ((long)off + j < whole + 4) atomicAdd(out + off + j, v[j]);
    }
  };
  const float kexp = P.inv_ar2 * NEG2_LOG2E;
  const float ta = gm.ta, tb = gm.tb, ntb = -tb;

  for (Columns cols(P, part, parts); cols.more();) {
    const unsigned nkept = cols.compact<false>(buf, P, P.Tcut, ox, oy, gm.res, gm.dim, lane);
    if (LATE) wait_for_stream();
    __syncwarp();
    // With a tail the density is continuous in the distance, and the squared distances may be taken
    // in units of ar^2 (s = rsq / ar^2: one multiplication per column and z position instead of one per
    // voxel; the Gaussian part ends at s = G^2, the tail clamps to zero at the cut-off).  Without a
    // tail (negative gaussian_radius_multiple) the density jumps at the cut-off, and the comparison
    // stays the reference's own, rsq against the threshold.
    const bool tail = ta != 0.f || ntb != 0.f;
    if (tail) {
      const float sg = P.Tg * P.inv_ar2, scut = P.Tcut * P.inv_ar2;
      auto quad = [&](unsigned, float dxy2, float exy, const float (&d2v)[4], const float (&ev)[4],
                      const float (&)[4], auto off) {
        float v[4];
        const Pair xy = pair(dxy2);
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          float s0, s1;
          split(add2(xy, pair(d2v[j], d2v[j + 1])), s0, s1);
          if constexpr (PACKED) {
            float g0, g1, t0, t1;
            split(mul2(pair(exy), pair(ev[j], ev[j + 1])), g0, g1);
            split(fma2(pair(ta), pair(sqrt_approx(s0), sqrt_approx(s1)), pair(ntb)), t0, t1);
            const Pair tq = pair(fminf(t0, 0.f), fminf(t1, 0.f));  // zero beyond the cut-off and for a NaN
            split(mul2(tq, tq), t0, t1);
            v[j] = s0 <= sg ? g0 : t0;
            v[j + 1] = s1 <= sg ? g1 : t1;
          } else {
            // the tail's root, tb - ta * distance: at most one where the tail is taken, zero beyond the cut-off and for a
            // NaN.  Clamps and packed products instead: soft types at 28x96^3 1735 us, like this 1650; 50 x 3000 atoms
            // on 28x48^3 168 and 164.
            const float t0 = fma_sat(-ta, sqrt_approx(s0), tb), t1 = fma_sat(-ta, sqrt_approx(s1), tb);
            v[j] = s0 <= sg ? exy * ev[j] : t0 * t0;
            v[j + 1] = s1 <= sg ? exy * ev[j + 1] : t1 * t1;
          }
          if (VEC) {
            v[j] *= P.w;
            v[j + 1] *= P.w;
          }
        }
        add(off, v);
      };
      if constexpr (LOOSE)
        loose_sweep_span<true>(P, buf, nkept, gm.dim, (unsigned)chan_off, tabs, oz, gm.res, NEG2_LOG2E, scut, P.inv_ar2, lane, quad);
      else
        qlane_sweep_span_t<true>(quad_span(P), P, buf, nkept, dim, oz, gm.res, NEG2_LOG2E, scut, P.inv_ar2, lane, quad);
    } else {
      auto quad = [&](unsigned, float dxy2, float exy, const float (&d2v)[4], const float (&ev)[4],
                      const float (&)[4], auto off) {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          float rsq = __fadd_rn(dxy2, d2v[j]);
          // tail (ta*dr - tb)^2 clamped to zero beyond the cut-off; a NaN rsq gives zero too
          float tq = fminf(fmaf(ta, sqrt_approx(rsq * P.inv_ar2), ntb), 0.f);
          float val = rsq <= P.Tg ? exy * ev[j] : tq * tq;
          v[j] = VEC ? val * P.w : val;
        }
        add(off, v);
      };
      if constexpr (LOOSE)
        loose_sweep_span<false>(P, buf, nkept, gm.dim, (unsigned)chan_off, tabs, oz, gm.res, kexp, P.Tcut, 1.f, lane, quad);
      else
        qlane_sweep_span(quad_span(P), P, buf, nkept, dim, oz, gm.res, kexp, P.Tcut, lane, quad);
    }
    __syncwarp();
  }
}

// One work item (an atom, or an (atom, channel) pair with VEC) of the forward pass on aligned quads.
template <bool VEC, bool LOOSE>
__device__ __forceinline__ void forward_quads_item(const BwdArgs& G, int item, int bl, ColBuf& buf,
                                                   LooseForward (&tabs)[4], int lane) {
  const GMParams& gm = G.gm;
  int b = G.b0 + bl;
  if (VEC) {
    // an (atom, channel) pair without weight contributes nothing: leave before any other load
    int ea = item / G.T;
    if (G.type_vector[((size_t)b * G.N + ea) * G.T + (item - ea * G.T)] == 0.f) return;
  }

  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  ItemParams P = load_item<VEC>(G, bl, b, item, ox, oy, oz);
  if (!P.valid || (VEC && P.w == 0.f)) return;  // zero weights add nothing (src/grid_maker.cpp:229)
  forward_quads_core<VEC, LOOSE>(G, P, b, ox, oy, oz, buf, tabs, lane);
}

template <bool VEC, bool LOOSE>
__global__ void __launch_bounds__(QS_WARPS * 32) k_forward_quads(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBuf bufs[QS_WARPS];
  __shared__ LooseForward tabs[QS_WARPS][4];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int item = blockIdx.x * QS_WARPS + wid;
  if (item >= (VEC ? G.N * G.T : G.N)) return;
  forward_quads_item<VEC, LOOSE>(G, item, blockIdx.y, bufs[wid], tabs[wid], lane);
}

// Occupancy of index types: every writer stores the same 1.0, so nothing is reduced and any alignment
// will do.  A sphere of one radius lies in a third of the columns of the density's footprint (1.5 radii):
// the candidates are cut down to it, and the z steps to its height.  The lanes are eight columns of four.
template <int STEPS>
__device__ __forceinline__ void occupancy_sweep(const ItemParams& P, const ColBuf& buf, unsigned nkept, unsigned zlo,
                                                unsigned zhi, float oz, const GMParams& gm, float* out, int lane) {
  const int grp = lane >> 2, sub = lane & 3;
  for (unsigned zc = zlo; zc < zhi; zc += 4 * STEPS) {
    const unsigned z0 = zc + sub;
    float dz2[STEPS];
#pragma unroll
    for (int k = 0; k < STEPS; k++) {
      const unsigned zz = z0 + 4 * k;
      const float dz = __fsub_rn(voxel_coord(oz, zz, gm.res), P.z);
      dz2[k] = zz < zhi ? __fmul_rn(dz, dz) : CUDART_NAN_F;
    }
    for (unsigned i = grp; i < nkept; i += 8) {
      unsigned cell;
      const float dxy2 = buf.get(i, cell);
      float* row = out + (size_t)cell * gm.dim + z0;
#pragma unroll
      for (int k = 0; k < STEPS; k++)
        if (__fadd_rn(dxy2, dz2[k]) < P.Tbin) row[4 * k] = 1.f;
    }
  }
}

__device__ __forceinline__ void forward_binary_core(const BwdArgs& G, ItemParams P, int b, float ox, float oy, float oz,
                                                    ColBuf& buf, int lane, unsigned part = 0, unsigned parts = 1) {
  const GMParams& gm = G.gm;
  const size_t dim = gm.dim;
  float* out = G.out_grid + ((size_t)b * G.T + P.chan) * dim * dim * dim;
  within(ox, P.x, P.ar, gm.res, P.lox, P.hix);
  within(oy, P.y, P.ar, gm.res, P.loy, P.hiy);
  within(oz, P.z, P.ar, gm.res, P.loz, P.hiz);
  if (P.hix <= P.lox || P.hiy <= P.loy || P.hiz <= P.loz) return;
  for (Columns cols(P, part, parts); cols.more();) {
    const unsigned nkept = cols.compact<false>(buf, P, P.Tbin, ox, oy, gm.res, gm.dim, lane);
    __syncwarp();
    const unsigned nz = P.hiz - P.loz;
    if (nz <= 8) occupancy_sweep<2>(P, buf, nkept, P.loz, P.hiz, oz, gm, out, lane);
    else if (nz <= 12) occupancy_sweep<3>(P, buf, nkept, P.loz, P.hiz, oz, gm, out, lane);
    else occupancy_sweep<4>(P, buf, nkept, P.loz, P.hiz, oz, gm, out, lane);
    __syncwarp();
  }
}

constexpr int BIN_WARPS = 4;
__global__ void __launch_bounds__(BIN_WARPS * 32) k_forward_binary(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBuf bufs[BIN_WARPS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, item = blockIdx.x * BIN_WARPS + wid;
  if (item >= G.N) return;
  const int bl = blockIdx.y, b = G.b0 + bl;
  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  const float ox = __fsub_rn(cx, G.gm.half), oy = __fsub_rn(cy, G.gm.half), oz = __fsub_rn(cz, G.gm.half);
  const ItemParams P = load_item<false>(G, bl, b, item, ox, oy, oz);
  if (P.valid) forward_binary_core(G, P, b, ox, oy, oz, bufs[wid], lane);
}

// The listed atoms of a pass of k_occupancy, whose output is zero in their channels: a warp prepares 32 atoms, one a
// lane, and stores their ones together (each atom prepared by the whole warp: 150 x 4000 atoms in one channel 482 us,
// like this 298).
__global__ void __launch_bounds__(BIN_WARPS * 32) k_occupancy_listed(EmitArgs A, BwdArgs G, OccList L) {
  wait_for_stream();
  __shared__ ColBuf bufs[BIN_WARPS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, bl = blockIdx.y, b = A.b0 + bl;
  const unsigned n = L.n[bl], warps = gridDim.x * BIN_WARPS;
  float cx, cy, cz;
  if (A.centers != nullptr) {
    cx = A.centers[b * 3]; cy = A.centers[b * 3 + 1]; cz = A.centers[b * 3 + 2];
  } else {
    cx = A.center_host[0]; cy = A.center_host[1]; cz = A.center_host[2];
  }
  const float ox = __fsub_rn(cx, A.gm.half), oy = __fsub_rn(cy, A.gm.half), oz = __fsub_rn(cz, A.gm.half);
  for (unsigned i0 = blockIdx.x * BIN_WARPS + wid; i0 < n; i0 += 32 * warps) {
    Rec own = empty_rec();
    if (i0 + lane * warps < n) make_rec(A, b, (int)L.atom[(size_t)bl * A.N + i0 + lane * warps], own);
    for (unsigned m = __ballot_sync(0xffffffffu, own.c.w >> 16 & REC_VALID); m != 0u; m &= m - 1u) {
      const int k = __ffs(m) - 1;
      Rec r = empty_rec();
      r.a.x = __shfl_sync(0xffffffffu, own.a.x, k);
      r.a.y = __shfl_sync(0xffffffffu, own.a.y, k);
      r.a.z = __shfl_sync(0xffffffffu, own.a.z, k);
      r.c.x = __shfl_sync(0xffffffffu, own.c.x, k);
      r.c.y = __shfl_sync(0xffffffffu, own.c.y, k);
      r.c.z = __shfl_sync(0xffffffffu, own.c.z, k);
      r.c.w = __shfl_sync(0xffffffffu, own.c.w, k);
      r.d.y = __shfl_sync(0xffffffffu, own.d.y, k);
      r.d.z = __shfl_sync(0xffffffffu, own.d.z, k);
      forward_binary_core(G, item_of(r), b, ox, oy, oz, bufs[wid], lane);
      __syncwarp();
    }
  }
}

// Index types without k_emit: every warp prepares its atom itself, and WARPS warps share an atom's columns
// while the atoms alone would leave most of the chip idle.  With the zero fill, 300 atoms into 28x48^3:
// 11.6 -> 7.3 us; 64 x 1000 atoms: 234.9 -> 229.7 us; 50 x 3000: 264 -> 285 us, so densities of more than
// FWD_SELF_ATOMS slots keep k_emit.  Occupancy, whose sweeps are a third as long, gains at every size
// (50 x 3000: 250 -> 228 us).
template <bool BINARY, int WARPS, bool ZEROED_BEFORE, bool LOOSE>
__global__ void __launch_bounds__(32 * WARPS) k_forward_self(EmitArgs A, BwdArgs G) {
  __shared__ ColBuf bufs[WARPS];
  __shared__ LooseForward tabs[WARPS][4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, a = blockIdx.x, bl = blockIdx.y, b = A.b0 + bl;
  Rec r;
  float ox, oy, oz;
  const bool bad = make_rec_warp(A, b, a, lane, r, ox, oy, oz);
  const ItemParams P = item_of(r);
  if (BINARY) {
    if (ZEROED_BEFORE) wait_for_stream();  // the output is zero
    if (P.valid) forward_binary_core(G, P, b, ox, oy, oz, bufs[w], lane, w, WARPS);
  } else {
    if (P.valid) forward_quads_core<false, LOOSE, ZEROED_BEFORE, LOOSE && WARPS == 1>(G, P, b, ox, oy, oz, bufs[w], tabs[w], lane, w, WARPS);
    if (ZEROED_BEFORE) wait_for_stream();  // nothing to add: not done before the zeros are, either
  }
  if (threadIdx.x == 0) put_flag(A, bl * A.N + a, A.nb * A.N, bad);
}

// Vector types whose radii differ by channel: one warp takes a group of NZ_GROUP consecutive channels
// of an atom and runs the (atom, channel) item of every channel of the group in which the atom
// carries weight - no work item, and no block, per channel without weight (27 of 28 with one-hot
// types), and still several warps per atom when every channel is weighted.
constexpr int NZ_GROUP = 8;
__host__ __device__ inline int nz_groups(int T) { return (T + NZ_GROUP - 1) / NZ_GROUP; }

#define LMG_FOR_EACH_WEIGHTED_CHANNEL(G, b, unit, lane, atom, t)                                        \
  if (int atom = (unit) % (G).N; true)                                                                  \
    if (int t0_ = ((unit) / (G).N) * NZ_GROUP; true)                                                    \
      for (unsigned m_ = __ballot_sync(                                                                 \
               0xffffffffu, (lane) < NZ_GROUP && t0_ + (lane) < (G).T &&                                \
                                (G).type_vector[((size_t)(b) * (G).N + atom) * (G).T + t0_ + (lane)] != 0.f); \
           m_ != 0u; m_ &= m_ - 1u)                                                                     \
        if (int t = t0_ + __ffs(m_) - 1; true)

__global__ void __launch_bounds__(SCAT_WARPS * 32) k_forward_quads_nz(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBuf bufs[SCAT_WARPS];
  __shared__ LooseForward tabs[SCAT_WARPS][4];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int unit = blockIdx.x * SCAT_WARPS + wid;
  if (unit >= G.N * nz_groups(G.T)) return;
  int b = G.b0 + blockIdx.y;
  LMG_FOR_EACH_WEIGHTED_CHANNEL(G, b, unit, lane, atom, t) {
    forward_quads_item<true, false>(G, atom * G.T + t, blockIdx.y, bufs[wid], tabs[wid], lane);
    __syncwarp();
  }
}

// The backward passes (modes as in k_backward_warp) on aligned quads.
struct BwdSums {
  float agx, agy, agz, tg;  // reduced over the warp: every lane holds the totals
};

// The quad at the end of the grids, of which `n` floats are left.
__device__ __forceinline__ float4 last_quad(const float* p, long n) {
  return make_float4(n > 0 ? __ldg(p) : 0.f, n > 1 ? __ldg(p + 1) : 0.f, n > 2 ? __ldg(p + 2) : 0.f, n > 3 ? __ldg(p + 3) : 0.f);
}

// The sweep of one work item whose constants are in P: sums over the item's footprint, reduced
// over the warp.  Of `parts` warps that share an item, this one takes the `part`-th share of its columns.
template <int MODE, bool BINARY, class BUF, class TABS>
__device__ __forceinline__ BwdSums backward_quads_core(const BwdArgs& G, const ItemParams& P, int b,
                                                       float ox, float oy, float oz, BUF& buf, TABS& zt,
                                                       int lane, unsigned part = 0, unsigned parts = 1) {
  constexpr bool LOOSE = !std::is_same<TABS, ZTabs>::value;
  const GMParams& gm = G.gm;
  size_t dim = gm.dim;
  size_t chan_off = ((size_t)b * G.T + P.chan) * dim * dim * dim;
  const float* diff = G.diff + chan_off;
  const float* dens = MODE == 2 ? G.density + chan_off : nullptr;
  float agx = 0.f, agy = 0.f, agz = 0.f, tg = 0.f;
  const bool want_ag = MODE == 0 || (MODE == 1 && P.w != 0.f);
  const float Tcull = MODE == 0 ? P.Tcut : fmaxf(P.Tcut, BINARY ? P.Tbin : -1.f);
  const float kexp = P.inv_ar2 * NEG2_LOG2E;
  // The gradient's radial factor beyond the Gaussian part is kE/d + kD: positive inside the cut-off,
  // zero at it (the tail polynomial has a double root there) and negative beyond, so a clamp at zero
  // stands in for the comparison with the cut-off.  Items that want no atom gradient (zero weight)
  // and grid makers without a tail (ta == tb == 0) get zero factors.
  const bool tail = gm.ta != 0.f || gm.tb != 0.f;
  const float k4 = want_ag ? 4.f * P.inv_ar2 : 0.f;
  const float kD = (want_ag && tail) ? -gm.D * P.inv_ar2 : 0.f, kE = (want_ag && tail) ? -gm.E * P.inv_ar : 0.f;
  const float ta = gm.ta, ntb = -gm.tb;
  Pair az2 = pair(0.f), tg2 = pair(0.f);  // agz and tg of even and odd voxels

  // one quad of a column
  auto voxels = [&](float dxy2, float exy, float exy4, const float (&d2v)[4], const float (&ev)[4], const float (&dzv)[4],
                    const float (&dvv)[4], const float (&dev)[4], Pair& fs2) {
    if (MODE == 0 || MODE == 1) {
      // -(d density / d dist) / dist * dv, src/grid_maker.cu:881-919, two voxels at a time; rsq == 0
      // contributes nothing because dx = dy = dz = 0 there, a NaN rsq (z outside the footprint)
      // takes the tail, which the clamp makes zero
      const Pair xy = pair(dxy2), e4 = pair(exy4), kE2 = pair(kE), kD2 = pair(kD);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        float r0, r1, g0, g1, t0, t1;
        const Pair r = add2(xy, pair(d2v[j], d2v[j + 1])), e2 = pair(ev[j], ev[j + 1]);
        split(r, r0, r1);
        split(mul2(e4, e2), g0, g1);
        // a neighbouring row's values, whatever they are, are not looked at
        const float v0_ = !LOOSE || r0 <= Tcull ? dvv[j] : 0.f, v1_ = !LOOSE || r1 <= Tcull ? dvv[j + 1] : 0.f;
        const Pair id = pair(rsqrt_approx(r0), rsqrt_approx(r1)), d2 = pair(v0_, v1_);
        split(fma2(kE2, id, kD2), t0, t1);
        const Pair f = mul2(pair(r0 <= P.Tg ? g0 : fmaxf(t0, 0.f), r1 <= P.Tg ? g1 : fmaxf(t1, 0.f)), d2);
        fs2 = add2(fs2, f);
        az2 = fma2(f, pair(dzv[j], dzv[j + 1]), az2);
        if (MODE == 1) {
          float v0, v1;
          if (BINARY) {
            v0 = r0 < P.Tbin ? 1.f : 0.f;
            v1 = r1 < P.Tbin ? 1.f : 0.f;
          } else {
            // the distance in radii from the reciprocal root that the gradient needs
            float q0, q1;
            split(fma2(pair(ta), mul2(mul2(r, id), pair(P.inv_ar)), pair(ntb)), q0, q1);
            const Pair tq = pair(fminf(q0, 0.f), fminf(q1, 0.f));  // zero beyond the cut-off and for a NaN
            split(mul2(tq, tq), q0, q1);
            split(mul2(pair(exy), e2), g0, g1);
            v0 = r0 <= P.Tg ? g0 : q0;
            v1 = r1 <= P.Tg ? g1 : q1;
          }
          tg2 = fma2(pair(v0, v1), d2, tg2);
        }
      }
    }
    if constexpr (MODE == 2 && BINARY) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float t = divide_near(dvv[j], dev[j]);
        if (__fsub_rn(dxy2, d2v[j]) < P.Tbin && dev[j] > 0.f) tg += t;
      }
    } else if constexpr (MODE == 2) {
      // density * dv / total density, two voxels at a time with the roundings of tail_quotient() and divide_near(): the
      // negated numbers of these where that saves a negation.  Divisors and quotients that the short division cannot take go
      // through the long one afterwards; such a quotient is no number, and neither is the sum then.  The kernel is bound by
      // issue, and this is most of it: 434 -> 388 us for 50 x 3000 atoms on 28x48^3, the same bits.
      float v[4], c[4];
      bool in[4], odd = false;
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        // the squared distance, its root and the root over the radius, all three negated
        const Pair r = add2(pair(-dxy2), pair(d2v[j], d2v[j + 1]));
        float r0, r1, t0, t1, g0, g1;
        split(r, r0, r1);
        r0 = -r0;
        r1 = -r1;
        const Pair y = pair(rsqrt_approx(r0), rsqrt_approx(r1)), s = mul2(r, y);
        const Pair dist = fma2(fma2(s, s, r), mul2(pair(0.5f), y), s);
        const Pair ir = pair(P.inv_ar), q = mul2(dist, ir), dr = fma2(fma2(q, pair(-P.ar), dist), ir, q);
        const Pair nz = pair(copysignf(0.f, -gm.res));  // see interp_blend(): keeps the products' own roundings
        const Pair t = add2(fma2(add2(fma2(pair(gm.A), dr, nz), pair(-gm.B)), dr, nz), pair(gm.C));
        split(t, t0, t1);
        split(mul2(pair(exy), pair(ev[j], ev[j + 1])), g0, g1);
        v[j] = r0 <= P.Tg ? g0 : fmaxf(t0, 0.f);
        v[j + 1] = r1 <= P.Tg ? g1 : fmaxf(t1, 0.f);
        in[j] = r0 <= P.Tcut && v[j] > 0.f && dev[j] > 0.f;  // false for a NaN
        in[j + 1] = r1 <= P.Tcut && v[j + 1] > 0.f && dev[j + 1] > 0.f;
        const Pair n = mul2(pair(dvv[j], dvv[j + 1]), pair(v[j], v[j + 1])), d = pair(dev[j], dev[j + 1]);
        const Pair rd = pair(rcp_approx(-dev[j]), rcp_approx(-dev[j + 1])), share = mul2(n, rd);  // and the quotient
        split(fma2(fma2(share, d, n), rd, share), c[j], c[j + 1]);
        odd = odd || (in[j] && dev[j] < 1e-30f) || (in[j + 1] && dev[j + 1] < 1e-30f);
      }
      float sum = tg;
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (in[j]) sum -= c[j];
      if (odd || sum != sum) {
        sum = tg;
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (in[j]) sum += divide_near(__fmul_rn(dvv[j], v[j]), dev[j]);
      }
      tg = sum;
    }
  };

  if (P.valid) {
    for (Columns cols(P, part, parts); cols.more();) {
      const unsigned nkept = cols.compact<true>(buf, P, Tcull, ox, oy, gm.res, gm.dim, lane);
      if constexpr (LOOSE) {
        // The lanes are (column, z quad), the quads of COLS columns requested at a time: a lane per column, as below,
        // would read four different tables at a time (17 x 700 atoms on 22x41^3, relevance: 90 against 60 us).
        constexpr int COLS = MODE == 2 ? 2 : 4;
        const unsigned nz = min(loose_span(P), (unsigned)QPASS), cpi = 32u / nz, cl = lane / nz, zq = lane - cl * nz;
        const long whole = floats_left(G, chan_off, dim) - 4;  // the last place of a quad
        for (unsigned zc = P.loz; zc < P.hiz + 3; zc += 4 * QPASS) {
          __syncwarp();
          fill_loose<false, MODE>(zt, zc, P, oz, gm.res, kexp, 1.f, lane);
          __syncwarp();
          for (unsigned c0 = 0; c0 < nkept; c0 += COLS * cpi) {
            float dxy2[COLS];
            unsigned t[COLS];
            float4 dv[COLS], de[COLS];
            bool in[COLS];
#pragma unroll
            for (int u = 0; u < COLS; u++) {
              const unsigned i = c0 + u * cpi + cl;
              const bool have = cl < cpi && i < nkept;
              const unsigned cell = have ? buf.row[i] : 0u;
              dxy2[u] = have ? buf.dxy2[i] : CUDART_NAN_F;
              t[u] = quad_shift((unsigned)chan_off, cell, gm.dim, zc);
              in[u] = __fadd_rn(dxy2[u], zt[t[u]].lo[zq]) <= Tcull;  // false for a NaN
              dv[u] = de[u] = make_float4(0.f, 0.f, 0.f, 0.f);
              const long off = (long)((size_t)cell * dim + zc + 4 * zq) - (long)t[u];
              if (in[u]) {
                dv[u] = off <= whole ? __ldg(reinterpret_cast<const float4*>(diff + off)) : last_quad(diff + off, whole + 4 - off);
                if (MODE == 2)
                  de[u] = off <= whole ? __ldg(reinterpret_cast<const float4*>(dens + off)) : last_quad(dens + off, whole + 4 - off);
              }
            }
#pragma unroll
            for (int u = 0; u < COLS; u++) {
              if (!in[u]) continue;
              const float4 d2 = zt[t[u]].dz2[zq], e = zt[t[u]].ez[zq], dz = zt[t[u]].dz[zq];
              const float d2v[4] = {d2.x, d2.y, d2.z, d2.w}, ev[4] = {e.x, e.y, e.z, e.w}, dzv[4] = {dz.x, dz.y, dz.z, dz.w};
              const float dvv[4] = {dv[u].x, dv[u].y, dv[u].z, dv[u].w}, dev[4] = {de[u].x, de[u].y, de[u].z, de[u].w};
              const float exy = gauss_factor<MODE>(dxy2[u], P, kexp);
              Pair fs2 = pair(0.f);
              voxels(dxy2[u], exy, k4 * exy, d2v, ev, dzv, dvv, dev, fs2);
              if (MODE != 2) {
                float f0, f1;
                split(fs2, f0, f1);
                const unsigned i = c0 + u * cpi + cl;
                agx = fmaf(f0 + f1, buf.dx[i], agx);
                agy = fmaf(f0 + f1, buf.dy[i], agy);
              }
            }
          }
        }
      } else for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * QPASS) {
        __syncwarp();
        fill_ztabs<MODE>(zt, zc, P, oz, gm.res, kexp, lane);
        __syncwarp();
        unsigned nq = min((unsigned)QPASS, (P.hiz - zc + 3) >> 2);
        for (unsigned c0 = 0; c0 < nkept; c0 += 32) {
          unsigned i = c0 + lane;
          bool have = i < nkept;
          float dxy2 = have ? buf.dxy2[i] : CUDART_NAN_F;
          float dx = have ? buf.dx[i] : 0.f, dy = have ? buf.dy[i] : 0.f;
          size_t rowoff = (size_t)(have ? buf.row[i] : 0u) * dim + zc;
          const float4* row = reinterpret_cast<const float4*>(diff + rowoff);
          float exy = gauss_factor<MODE>(dxy2, P, kexp);
          float exy4 = k4 * exy;
          Pair fs2 = pair(0.f);  // sum over the column of -(d density / d dist) / dist * dv, even and odd voxels
          for (unsigned q0 = 0; q0 < nq; q0 += 4) {
            // up to four quads of the column are requested together, then used.  The vote: 50 x 3000 atoms on 28x48^3,
            // gradients 219 -> 215 us, relevance 417 -> 395; soft types at 28x96^3 2551 -> 2457.
            float4 dv[4];
            bool live[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
              dv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
              // no load where no voxel of the quad can lie inside the cut-off (false for a NaN too)
              live[u] = q0 + u < nq && __fadd_rn(dxy2, zt.lo[q0 + u]) <= Tcull;
              if (live[u]) dv[u] = __ldg(row + q0 + u);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
              if (__any_sync(0xffffffffu, live[u])) {  // a quarter of them are in no lane's reach
                float4 d2 = zt.dz2[q0 + u], e = zt.ez[q0 + u], dz = zt.dz[q0 + u];
                float d2v[4] = {d2.x, d2.y, d2.z, d2.w}, ev[4] = {e.x, e.y, e.z, e.w};
                float dzv[4] = {dz.x, dz.y, dz.z, dz.w}, dvv[4] = {dv[u].x, dv[u].y, dv[u].z, dv[u].w};
                float dev[4] = {0.f, 0.f, 0.f, 0.f};
                if (MODE == 2) {
                  // the density is only needed where this quad can hold a voxel of the atom
                  if (live[u]) {
                    float4 de = __ldg(reinterpret_cast<const float4*>(dens + rowoff) + q0 + u);
                    dev[0] = de.x; dev[1] = de.y; dev[2] = de.z; dev[3] = de.w;
                  }
                }
                voxels(dxy2, exy, exy4, d2v, ev, dzv, dvv, dev, fs2);
              }
            }
          }
          if (MODE != 2) {
            float f0, f1;
            split(fs2, f0, f1);
            agx = fmaf(f0 + f1, dx, agx);
            agy = fmaf(f0 + f1, dy, agy);
          }
        }
      }
      __syncwarp();
    }
  }
  if (MODE != 2) {
    float z0, z1;
    split(az2, z0, z1);
    agz = z0 + z1;
    if (MODE == 1) {
      split(tg2, z0, z1);
      tg = z0 + z1;
    }
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    if (MODE != 2) {
      agx += __shfl_xor_sync(0xffffffffu, agx, o);
      agy += __shfl_xor_sync(0xffffffffu, agy, o);
      agz += __shfl_xor_sync(0xffffffffu, agz, o);
    }
    if (MODE == 1 || MODE == 2) tg += __shfl_xor_sync(0xffffffffu, tg, o);
  }
  BwdSums R;
  R.agx = agx; R.agy = agy; R.agz = agz; R.tg = tg;
  return R;
}

// One work item (an atom, or an (atom, channel) pair for the vector modes) from its record in the
// workspace.
template <int MODE, bool BINARY, class TABS>
__device__ __forceinline__ void backward_quads_item(const BwdArgs& G, int item, int bl, ColBufD& buf, TABS& zt,
                                                    int lane) {
  constexpr bool VEC = MODE == 1;
  const GMParams& gm = G.gm;
  int b = G.b0 + bl;
  if (MODE == 1 && G.type_gradients == nullptr) {
    // an (atom, channel) pair without weight contributes nothing: leave before any other load
    int ea = item / G.T;
    if (G.type_vector[((size_t)b * G.N + ea) * G.T + (item - ea * G.T)] == 0.f) return;
  }

  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  ItemParams P = load_item<VEC>(G, bl, b, item, ox, oy, oz);
  BwdSums R = backward_quads_core<MODE, BINARY, ColBufD, TABS>(G, P, b, ox, oy, oz, buf, zt, lane);
  float agx = R.agx, agy = R.agy, agz = R.agz, tg = R.tg;
  if (lane == 0) {
    size_t ai = (size_t)b * G.N + (VEC ? item / G.T : item);
    if (MODE == 0) {
      G.atom_gradients[ai * 3] = agx;
      G.atom_gradients[ai * 3 + 1] = agy;
      G.atom_gradients[ai * 3 + 2] = agz;
    } else if (MODE == 1) {
      size_t pi = (size_t)bl * G.N * G.T + item;
      G.partial[pi * 3] = agx;
      G.partial[pi * 3 + 1] = agy;
      G.partial[pi * 3 + 2] = agz;
      if (G.type_gradients != nullptr) G.type_gradients[ai * G.T + P.chan] = tg;
    } else {
      G.relevance[ai] = tg;
    }
  }
}

// 64 registers: the most of the blocks of one warp that an SM takes.  MODE 1 waits on the L1 (89 % of its throughput: a lane per column touches 32 lines a load): 64 registers and
// 32 resident warps instead of 72 and 28, 2.67 -> 2.58 ms at 28x96^3 (4 x 3000 atoms, 28 channels).
template <int MODE, bool BINARY, class TABS>
__global__ void __launch_bounds__(BWD2_WARPS * 32, 32) k_backward_quads(BwdArgs G) {
  wait_for_stream();
  constexpr bool VEC = MODE == 1;
  __shared__ ColBufD bufs[BWD2_WARPS];
  __shared__ TABS ztabs[BWD2_WARPS];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int item = blockIdx.x * BWD2_WARPS + wid;
  if (item >= (VEC ? G.N * G.T : G.N)) return;
  backward_quads_item<MODE, BINARY, TABS>(G, item, blockIdx.y, bufs[wid], ztabs[wid], lane);
}

// Atom gradients (MODE 0) and relevance (MODE 2) of index types for inputs of at most SELF_ATOMS slots:
// every warp prepares its atom itself, so the pass is one launch, and WARPS warps share an atom's
// columns, because so few atoms leave most of the chip idle and the pass lasts as long as one atom.
// Larger inputs notice that every warp repeats the preparation (with 200 000 slots 0.230-0.316 ms
// against 0.225 ms for k_emit and the kernel above).
//
// Relevance by four warps an atom takes 80 to 94 registers, five or six blocks an SM.  The `tight` variant, of which six to
// eight fit (loose rows need larger tables), is for the counts that are one wave with it and two without: 800 / 1000 atoms on
// 14x24^3 of 1 A 6.3 / 6.6 us with room and 4.8 / 5.0 tight, occupancy of 1000 6.5 and 4.7; one wave or two either way, 600
// atoms 4.1 and 4.3, 1200 on 14x41^3 14.9 and 15.2.  Examples with counts of their own: the slots behind them leave at once
// and are taken for a quarter (16 x 26 to 53 atoms in 848 slots on 31x48^3 8.1 and 8.7).
constexpr long SELF_ROOMY = 5 * 148;
constexpr int self_blocks(bool binary, bool loose, bool tight) { return !tight ? 0 : loose ? (binary ? 7 : 6) : binary ? 8 : 7; }
template <int MODE, bool BINARY, int WARPS, class TABS, bool TIGHT = false>
__global__ void __launch_bounds__(32 * WARPS, self_blocks(BINARY, !std::is_same<TABS, ZTabs>::value, TIGHT))
    k_backward_quads_self(EmitArgs A, BwdArgs G) {
  __shared__ ColBufD bufs[WARPS];
  __shared__ TABS zts[WARPS];
  __shared__ float4 sums[WARPS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, a = blockIdx.x, bl = blockIdx.y, b = A.b0 + bl;
  wait_for_stream();
  Rec r;
  float ox, oy, oz;
  const bool bad = make_rec_warp(A, b, a, lane, r, ox, oy, oz);
  if (threadIdx.x == 0) put_flag(A, bl * A.N + a, A.nb * A.N, bad);
  ItemParams P = item_of(r);
  BwdSums R = backward_quads_core<MODE, BINARY, ColBufD, TABS>(G, P, b, ox, oy, oz, bufs[w], zts[w], lane, w, WARPS);
  if (WARPS > 1) {
    if (lane == 0) sums[w] = make_float4(R.agx, R.agy, R.agz, R.tg);
    __syncthreads();
    if (w != 0) return;
    R.agx = R.agy = R.agz = R.tg = 0.f;
#pragma unroll
    for (int k = 0; k < WARPS; k++) {
      R.agx += sums[k].x; R.agy += sums[k].y; R.agz += sums[k].z; R.tg += sums[k].w;
    }
  }
  const size_t ai = (size_t)b * A.N + a;
  if (MODE == 0) {
    if (lane < 3) G.atom_gradients[ai * 3 + lane] = lane == 0 ? R.agx : lane == 1 ? R.agy : R.agz;
  } else if (lane == 0) {
    G.relevance[ai] = R.tg;
  }
}

// The (atom, channel) items of the weighted channels of one atom, by one warp: modes that need
// nothing from channels without weight (MODE 1 when no type gradients are wanted).
template <int MODE, bool BINARY>
__global__ void __launch_bounds__(BWD2_WARPS * 32) k_backward_quads_nz(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBufD bufs[BWD2_WARPS];
  __shared__ ZTabs ztabs[BWD2_WARPS];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int unit = blockIdx.x * BWD2_WARPS + wid;
  if (unit >= G.N * nz_groups(G.T)) return;
  int b = G.b0 + blockIdx.y;
  LMG_FOR_EACH_WEIGHTED_CHANNEL(G, b, unit, lane, atom, t) {
    backward_quads_item<MODE, BINARY, ZTabs>(G, atom * G.T + t, blockIdx.y, bufs[wid], ztabs[wid], lane);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------
// backward_gradients on aligned quads: the grid term and the atom term in one sweep of the footprint, which
// share the distance, the Gaussian and its two derivatives.  With s = -(d density / d dist) / dist and the
// second derivatives H_ab = alpha delta_a delta_b - [a == b] s of the density (src/grid_maker.cu:812-878;
// delta = grid point - atom up to a sign that cancels):
//   Gaussian  g = exp(-2 d^2 / ar^2):   s = 4 g / ar^2,    alpha = 4 s / ar^2
//   tail      (D and E of the reference): s = kE / d + kD,   alpha = kE / d^3,   kE = -E / ar, kD = -D / ar^2
// the grid receives  density * type_gradient + w * s * (delta . atom_gradient)  (src/grid_maker.cpp:618-634),
// the atom needs, per column, the sums of diff * alpha * {1, dz, dz^2} and of diff * s (:636-662).
// Bound by instruction issue: 28x96^3 at 0.25 A, 4 x 3000 atoms of 28 weighted channels each: 6.70 ms as
// two sweeps with scalar arithmetic, 4.17 ms as one (issue 68 %, L1 75 %), 4.25 with values outside the cut-off left out.
// ---------------------------------------------------------------------------------------------
constexpr int SO_WARPS = 1;
// Two lanes share a column, each taking every other quad: a load or reduction of a warp touches 16 lines
// instead of 32 (4.54 -> 4.17 ms; the sweeps without reductions lose more to their column terms).
constexpr int SO_ZL = 2;
constexpr int SO_MINB = 16, SO_ATOM_MINB = 26;  // resident blocks: 114 and 72 registers

struct SecondConst {
  Pair k4, c4, kE, kD, ta, ntb, inv_ar, inv_ar2;
  __device__ __forceinline__ SecondConst(const GMParams& gm, const ItemParams& P) {
    const bool tail = gm.ta != 0.f || gm.tb != 0.f;
    k4 = c4 = pair(4.f * P.inv_ar2);
    kE = pair(tail ? -gm.E * P.inv_ar : 0.f);
    kD = pair(tail ? -gm.D * P.inv_ar2 : 0.f);
    ta = pair(gm.ta);
    ntb = pair(-gm.tb);
    inv_ar = pair(P.inv_ar);
    inv_ar2 = pair(P.inv_ar2);
  }
};

// density, s and alpha at two voxels; all zero beyond the cut-off and for a NaN distance (z outside the
// footprint), which `in0` and `in1` tell for products with values that need not be finite.  OWN_ROOT: the density
// from a root of its own and s in one rounding, instead of both from the reciprocal root and the product that alpha
// needs.  With radii by atom the grid term is else 6 % further from 64 bits than it was as a sweep of its own (1.85e-7,
// 1.75e-7 like this); with radii by type it is as near either way, and 2 % of the time less without.
template <bool OWN_ROOT>
__device__ __forceinline__ void second_factors(const SecondConst& K, const ItemParams& P, Pair rsq, Pair g, Pair& val, Pair& s,
                                               Pair& alpha, bool& in0, bool& in1) {
  float r0, r1, a0, a1, b0, b1;
  split(rsq, r0, r1);
  const bool gauss0 = r0 <= P.Tg, gauss1 = r1 <= P.Tg;
  in0 = r0 <= P.Tcut;
  in1 = r1 <= P.Tcut;
  const Pair id = pair(rsqrt_approx(r0), rsqrt_approx(r1));
  float g0, g1;
  split(g, g0, g1);
  Pair dr;
  if (OWN_ROOT) {
    split(mul2(rsq, K.inv_ar2), a0, a1);
    dr = pair(sqrt_approx(a0), sqrt_approx(a1));
  } else {
    dr = mul2(mul2(rsq, id), K.inv_ar);
  }
  split(fma2(K.ta, dr, K.ntb), a0, a1);
  const Pair tq = pair(fminf(a0, 0.f), fminf(a1, 0.f));
  split(mul2(tq, tq), a0, a1);
  val = pair(gauss0 ? g0 : a0, gauss1 ? g1 : a1);
  const Pair sg = mul2(K.k4, g), kid = mul2(K.kE, id);
  split(sg, g0, g1);
  split(OWN_ROOT ? fma2(K.kE, id, K.kD) : add2(kid, K.kD), a0, a1);
  s = pair(gauss0 ? g0 : fmaxf(a0, 0.f), gauss1 ? g1 : fmaxf(a1, 0.f));
  split(mul2(K.c4, sg), g0, g1);
  split(mul2(kid, mul2(id, id)), b0, b1);
  alpha = pair(gauss0 ? g0 : in0 ? b0 : 0.f, gauss1 ? g1 : in1 ? b1 : 0.f);
}

// The values at two voxels, zero where `in0`, `in1` are false.
__device__ __forceinline__ Pair only(Pair v, bool in0, bool in1) {
  float a, b;
  split(v, a, b);
  return pair(in0 ? a : 0.f, in1 ? b : 0.f);
}
// s * (delta . atom_gradient) at two voxels for an atom gradient that is not finite: nothing beyond the cut-off
// nor on the atom itself.
__device__ __forceinline__ Pair only_off_atom(Pair sd, Pair rsq, bool in0, bool in1) {
  float r0, r1;
  split(rsq, r0, r1);
  return only(sd, in0 && r0 > 0.f, in1 && r1 > 0.f);
}
__device__ __forceinline__ bool finite3(float x, float y, float z) {
  return fabsf(x) < CUDART_INF_F && fabsf(y) < CUDART_INF_F && fabsf(z) < CUDART_INF_F;
}

// What the atom term keeps over an item's voxels: sums over pairs of voxels of one column, then over columns.
struct SecondColumn {
  Pair a0, a1, a2;  // diff * alpha * {1, dz, dz^2}
};

__device__ __forceinline__ void second_quads_item(const BwdArgs& G, int item, int bl, ColBufD& buf, ZTabs& zt, int lane) {
  const GMParams& gm = G.gm;
  const int b = G.b0 + bl;
  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  const float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  const ItemParams P = load_item<true>(G, bl, b, item, ox, oy, oz);
  float agx = 0.f, agy = 0.f, agz = 0.f;
  if (P.valid) {
    const size_t dim = gm.dim, chan = ((size_t)b * G.T + P.chan) * dim * dim * dim, gi = (size_t)b * G.N + item / G.T;
    const float inx = G.ag_in[gi * 3], iny = G.ag_in[gi * 3 + 1], inz = G.ag_in[gi * 3 + 2];
    const float intg = G.tg_in[gi * G.T + P.chan];
    const float kexp = P.inv_ar2 * NEG2_LOG2E;
    const SecondConst K(gm, P);
    const Pair winz = pair(P.w * inz), tg2 = pair(intg);
    const bool odd = !finite3(P.w * inx, P.w * iny, P.w * inz) || !finite3(intg, 0.f, 0.f);  // the same for every lane
    Pair sb = pair(0.f);  // sum of diff * s
    auto sweep = [&](auto odd) {
      for (Columns cols(P); cols.more();) {
        const unsigned nkept = cols.compact<true>(buf, P, P.Tcut, ox, oy, gm.res, gm.dim, lane);
        for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * QPASS) {
          __syncwarp();
          fill_ztabs(zt, zc, P, oz, gm.res, kexp, lane);
          __syncwarp();
          const unsigned nq = min((unsigned)QPASS, (P.hiz - zc + 3) >> 2);
          for (unsigned c0 = 0; c0 < nkept; c0 += 32 / SO_ZL) {
            const unsigned i = c0 + lane / SO_ZL;
            const bool have = i < nkept;
            const float dxy2 = have ? buf.dxy2[i] : CUDART_NAN_F, dx = have ? buf.dx[i] : 0.f, dy = have ? buf.dy[i] : 0.f;
            const size_t off = chan + (size_t)(have ? buf.row[i] : 0u) * dim + zc;
            const float4* row = reinterpret_cast<const float4*>(G.diff + off);
            float* out = G.out_grid + off;
            const Pair xy = pair(dxy2), exy = pair(ex2_approx(dxy2 * kexp));
            const float dotxy = fmaf(dx, inx, dy * iny);
            const Pair wdot = pair(P.w * dotxy);
            SecondColumn C = {pair(0.f), pair(0.f), pair(0.f)};
            for (unsigned q0 = lane % SO_ZL; q0 < nq; q0 += 4 * SO_ZL) {
              float4 dv[4];
              unsigned live = 0;
#pragma unroll
              for (int u = 0; u < 4; u++) {
                dv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (q0 + SO_ZL * u < nq && __fadd_rn(dxy2, zt.lo[q0 + SO_ZL * u]) <= P.Tcut) {
                  live |= 1u << u;
                  dv[u] = __ldg(row + q0 + SO_ZL * u);
                }
              }
#pragma unroll
              for (int u = 0; u < 4; u++) {
                if (!(live >> u & 1u)) continue;
                const float4 d2 = zt.dz2[q0 + SO_ZL * u], e = zt.ez[q0 + SO_ZL * u], dz = zt.dz[q0 + SO_ZL * u];
                const Pair d2p[2] = {pair(d2.x, d2.y), pair(d2.z, d2.w)}, ep[2] = {pair(e.x, e.y), pair(e.z, e.w)},
                           dzp[2] = {pair(dz.x, dz.y), pair(dz.z, dz.w)};
                Pair dvp[2] = {pair(dv[u].x, dv[u].y), pair(dv[u].z, dv[u].w)};
                float v[4];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                  Pair val, s, alpha;
                  bool in0, in1;
                  const Pair rsq = add2(xy, d2p[j]);
                  second_factors<false>(K, P, rsq, mul2(exy, ep[j]), val, s, alpha, in0, in1);
                  Pair sd = mul2(s, fma2(dzp[j], winz, wdot));
                  if constexpr (odd.value) sd = only_off_atom(sd, rsq, in0, in1);
                  Pair out2 = fma2(val, tg2, sd);
                  if constexpr (odd.value) out2 = only(out2, in0, in1);
                  split(out2, v[2 * j], v[2 * j + 1]);
                  dvp[j] = only(dvp[j], in0, in1);  // a neighbour's value may be anything
                  const Pair t0 = mul2(dvp[j], alpha), t1 = mul2(t0, dzp[j]);
                  C.a0 = add2(C.a0, t0);
                  C.a1 = add2(C.a1, t1);
                  C.a2 = fma2(t1, dzp[j], C.a2);
                  sb = fma2(dvp[j], s, sb);
                }
                red_add_v4(out + 4 * (q0 + SO_ZL * u), v[0], v[1], v[2], v[3]);
              }
            }
            // sum over the column of diff * (w*alpha*dot*delta_c + intg*alpha*delta_c^2), dot = dotxy + dz*inz
            float a0, a1, a2, t;
            split(C.a0, a0, t); a0 += t;
            split(C.a1, a1, t); a1 += t;
            split(C.a2, a2, t); a2 += t;
            const float wd = P.w * fmaf(dotxy, a0, inz * a1);
            agx = fmaf(dx, fmaf(intg * dx, a0, wd), agx);
            agy = fmaf(dy, fmaf(intg * dy, a0, wd), agy);
            agz += fmaf(P.w, fmaf(dotxy, a1, inz * a2), intg * a2);
          }
        }
        __syncwarp();
      }
    };
    if (odd) sweep(std::true_type());
    else sweep(std::false_type());
    // the isotropic part: -diff * s * (w*in_c + intg), the same factor for every voxel of the item
    float s0, s1;
    split(sb, s0, s1);
    s0 = -(s0 + s1);
    agx = fmaf(s0, fmaf(P.w, inx, intg), agx);
    agy = fmaf(s0, fmaf(P.w, iny, intg), agy);
    agz = fmaf(s0, fmaf(P.w, inz, intg), agz);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    agx += __shfl_xor_sync(0xffffffffu, agx, o);
    agy += __shfl_xor_sync(0xffffffffu, agy, o);
    agz += __shfl_xor_sync(0xffffffffu, agz, o);
  }
  if (lane < 3) G.partial[((size_t)bl * G.N * G.T + item) * 3 + lane] = lane == 0 ? agx : lane == 1 ? agy : agz;
}

__global__ void __launch_bounds__(SO_WARPS * 32, SO_MINB) k_second_quads_nz(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBufD bufs[SO_WARPS];
  __shared__ ZTabs ztabs[SO_WARPS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, unit = blockIdx.x * SO_WARPS + wid;
  if (unit >= G.N * nz_groups(G.T)) return;
  const int b = G.b0 + blockIdx.y;
  LMG_FOR_EACH_WEIGHTED_CHANNEL(G, b, unit, lane, atom, t) {
    second_quads_item(G, atom * G.T + t, blockIdx.y, bufs[wid], ztabs[wid], lane);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------
// Vector types with per-atom radii (the layout of the autograd bindings): the footprint and the
// density of an atom are the same for every channel, so one warp owns the ATOM, evaluates each voxel
// once and loops over the channels inside - the reuse the reference's kernel makes too
// (src/grid_maker.cu:322-325).  With one-hot type vectors this is the index-typed cost instead of
// one work item per (atom, channel).  Channels are handled in rounds of VA_CH.
// ---------------------------------------------------------------------------------------------
constexpr int VA_CH = 32;  // channels per round
// Rounds with at most this many weighted channels sweep once per channel, but for densities in the reference's order of
// operations.  Three: 50 x 3000 atoms on 28x48^3 511 us together and 482 one by one, 8 x 1000 on 28x24^3 of 1 A 14.1 and 15.8.
// Occupancy with one / two: 8 x 1000 atoms on 28x48^3 30.0 / 33.2 us together, 26.9 / 31.4 one by one.
constexpr int VA_SPARSE = 2;
// Densities in the reference's order of operations cost most of the sweep, and a lane per column branches less among them than
// lanes along z do.  One / 5 / 8 / 28 weighted channels at `grm` 3: 8 x 1000 atoms on 28x48^3 300 / 421 / 598 / 1835 us like that, 467 /
// 526 / 540 / 1300 along z; 2 x 300 on 28x96^3 of 0.25 A 1040 / 1190 / 1291 / 2793 and 1594 / 1713 / 1698 / 2199; 40 atoms on 28x48^3
// 144 / 153 / 149 / 257 and 208 / 206 / 202 / 277.
constexpr int VA_COLUMNS = 6, VA_COLUMNS_FEW = 12;  // most channels for that, and for passes of few atoms
constexpr long VA_FEW = 1200;

template <bool BINARY, bool PRECISE>
__global__ void __launch_bounds__(QS_WARPS * 32, 32) k_forward_quads_atom(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBuf bufs[QS_WARPS];
  __shared__ ZTabs ztabs[PRECISE ? QS_WARPS : 1];
  __shared__ int nz_t[QS_WARPS][VA_CH];
  __shared__ float nz_w[QS_WARPS][VA_CH];
  const GMParams& gm = G.gm;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int item = blockIdx.x * QS_WARPS + wid;
  int bl = blockIdx.y;
  int b = G.b0 + bl;
  if (item >= G.N) return;
  ColBuf& buf = bufs[wid];

  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  ItemParams P = load_item<false>(G, bl, b, item, ox, oy, oz);
  if (!P.valid) return;

  size_t dim = gm.dim;
  const size_t chan_stride = dim * dim * dim;
  float* outb = G.out_grid + (size_t)b * G.T * chan_stride;
  const float* wrow = G.type_vector + ((size_t)b * G.N + item) * G.T;
  const float Tcull = BINARY ? P.Tbin : P.Tcut;
  const float kexp = P.inv_ar2 * NEG2_LOG2E;
  const float ta = gm.ta, ntb = -gm.tb;

  for (int tb = 0; tb < G.T; tb += VA_CH) {
    // channels of this round that carry weight (zero weights add nothing, src/grid_maker.cpp:229)
    int t = tb + lane;
    float w = t < G.T ? wrow[t] : 0.f;
    unsigned m = __ballot_sync(0xffffffffu, w != 0.f);
    int nnz = __popc(m);
    if (nnz == 0) continue;
    __syncwarp();
    if (w != 0.f) {
      int slot = __popc(m & ((1u << lane) - 1u));
      nz_t[wid][slot] = t;
      nz_w[wid][slot] = w;
    }
    __syncwarp();
    for (Columns cols(P); cols.more();) {
      const unsigned nkept = cols.compact<false>(buf, P, Tcull, ox, oy, gm.res, gm.dim, lane);
      if (PRECISE && nnz <= ((long)G.N * G.nb <= VA_FEW ? VA_COLUMNS_FEW : VA_COLUMNS)) {
        ZTabs& zt = ztabs[wid];
        for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * QPASS) {
          __syncwarp();
          fill_ztabs(zt, zc, P, oz, gm.res, kexp, lane);
          __syncwarp();
          const unsigned nq = min((unsigned)QPASS, (P.hiz - zc + 3) >> 2);
          for (unsigned c0 = 0; c0 < nkept; c0 += 32) {
            const unsigned i = c0 + lane;
            unsigned cell = 0;
            const float dxy2 = i < nkept ? buf.get(i, cell) : CUDART_NAN_F;
            float* row = outb + (size_t)cell * dim + zc;
            for (unsigned q = 0; q < nq; q++) {
              const float4 d2 = zt.dz2[q];
              const float d2v[4] = {d2.x, d2.y, d2.z, d2.w};
              float v[4];
#pragma unroll
              for (int j = 0; j < 4; j++)
                v[j] = density_precise(__fadd_rn(dxy2, d2v[j]), P.ar, P.Tg, P.Tcut, gm.A, gm.B, gm.C);
              if ((__float_as_uint(v[0]) | __float_as_uint(v[1]) | __float_as_uint(v[2]) | __float_as_uint(v[3])) == 0u) continue;
              for (int k = 0; k < nnz; k++) {
                const float wk = nz_w[wid][k];
                red_add_v4(row + (size_t)nz_t[wid][k] * chan_stride + 4 * q, v[0] * wk, v[1] * wk, v[2] * wk, v[3] * wk);
              }
            }
          }
        }
        __syncwarp();
        continue;
      }
      if (!PRECISE && nnz <= VA_SPARSE) {
        // few weighted channels (one-hot types): one sweep per channel in the lane layout of the
        // index-typed forward, whose reductions touch a quarter of the rows
        __syncwarp();
        for (int k = 0; k < nnz; k++) {
          float* out = outb + (size_t)nz_t[wid][k] * chan_stride;
          const float wk = nz_w[wid][k];
          auto quad = [&](unsigned, float dxy2, float exy, const float (&d2v)[4], const float (&ev)[4],
                          const float (&)[4], size_t off) {
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
              float rsq = __fadd_rn(dxy2, d2v[j]);
              float tq = fma_sat(-ta, sqrt_approx(rsq * P.inv_ar2), -ntb);
              v[j] = BINARY ? (rsq < P.Tbin ? wk : 0.f) : (rsq <= P.Tg ? exy * ev[j] : tq * tq) * wk;
            }
            red_add_v4(out + off, v[0], v[1], v[2], v[3]);
          };
          qlane_sweep_span(quad_span(P), P, buf, nkept, dim, oz, gm.res, kexp, Tcull, lane, quad);
        }
        __syncwarp();
        continue;
      }
      // Many weighted channels: densities once, then a reduction for each.  The reductions bound this, by the lines that
      // they touch: 50 x 3000 atoms on 28x48^3 with 28 / 10 / 5 / 4 weighted channels 4361 / 1782 / 966 / 818 us with a
      // lane per column, 2964 / 1167 / 628 / 531 like this.
      auto quad = [&](unsigned, float dxy2, float exy, const float (&d2v)[4], const float (&ev)[4], const float (&)[4],
                      size_t off) {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          float rsq = __fadd_rn(dxy2, d2v[j]);
          if (BINARY) {
            v[j] = rsq < P.Tbin ? 1.f : 0.f;
          } else if (PRECISE) {
            v[j] = density_precise(rsq, P.ar, P.Tg, P.Tcut, gm.A, gm.B, gm.C);
          } else {
            float tq = fma_sat(-ta, sqrt_approx(rsq * P.inv_ar2), -ntb);
            v[j] = rsq <= P.Tg ? exy * ev[j] : tq * tq;
          }
        }
        const unsigned any = __float_as_uint(v[0]) | __float_as_uint(v[1]) | __float_as_uint(v[2]) | __float_as_uint(v[3]);
        if (any == 0u) return;
        float* to = outb + off;
        for (int k = 0; k < nnz; k++) {
          const float wk = nz_w[wid][k];
          red_add_v4(to + (size_t)nz_t[wid][k] * chan_stride, v[0] * wk, v[1] * wk, v[2] * wk, v[3] * wk);
        }
      };
      __syncwarp();
      qlane_sweep_span(quad_span(P), P, buf, nkept, dim, oz, gm.res, kexp, Tcull, lane, quad);
      __syncwarp();
    }
  }
}

// Backward for the same layout: atom gradient = sum over voxels of s * delta * (sum_t w_t diff_t),
// type gradient of EVERY channel = sum over voxels of density * diff_t (src/grid_maker.cpp:508-517).
// A lane keeps the type gradients of a round's CH channels in registers; their quads are requested together.  The kernel
// waits on those loads (they come from L2: every channel is read under every footprint), so what counts is how many are in
// flight per SM: registers per warp against loads per warp.  Measured per batch of 50 (28 channels, one-hot types):
// rounds of 16 with 4 loads together 2.79 ms, 8 / 8 2.08 ms, 14 / 7 1.82 ms, 14 / 14 1.70 ms,
// 16 / 16 2.17 ms, 28 / 14 2.05 ms; blocks of
// several warps, or atoms sorted by cell (for L1 reuse between neighbours) change nothing or lose.
// Few channels get shorter rounds, without loads and sums for channels that there are not (16 x 1000 atoms on 48^3, one /
// all weighted): 4 channels 100 / 107 us in rounds of 14, 60 / 56 in rounds of 4; 7 channels 102 / 110 and 73 / 74 in
// rounds of 7.
constexpr int VA_BCH = 14;
static_assert(VA_BCH <= 32, "a lane per channel of a round reads the weights");
constexpr int VA_WARPS = BWD2_WARPS;
// What else counts is the size of the loop.  A round's loop over quads comes in two forms (DENSE below); with a copy of
// each for every span of quads, atoms that take different ones turn each other's out of the instruction cache.
// 50 x 3000 atoms on 28x48^3, one / 2 / 5 / 28 weighted channels an atom: copies, 80 registers and 22 blocks an SM
// 1667 / 3233 / 3364 / 1898 us (an atom's channels of one round are then DENSE, of the other not), copies and 96
// registers 1741 / 1778 / 2943 / 2222; one copy of each form and 96 registers 1681 / 1630 / 1656 / 1739, with 80 registers
// 1684 / 1780 / 1846 / 2054, with 128 2447 / 2521 / 2402 / 2451.
constexpr int VA_MINB = 20;

// per-warp shared state of the kernel below
struct VaShared {
  ColBufD buf;
  float w[VA_BCH];   // weights of the round's channels
  int nz_t[VA_BCH];  // the weighted ones: channel (relative to the round) and weight
  float nz_w[VA_BCH];
};

// A quad of the gradient, zero where there is none.  In order: the loads of a round are issued one after the other before
// any is used.  Placed by the compiler, some waited for others: 2430 us with one weighted channel instead of 1681.
__device__ __forceinline__ float4 load_quad(const float4* p, bool there) {
  float4 v;
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.u32 q, %5, 0;\n\t"
      "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
      "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
      "@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w)
      : "l"(p), "r"((unsigned)there));
  return v;
}

// One round of k_backward_quads_atom: channels [tb, tb + nch) under the whole footprint of the atom.
// Lanes as (column, z-quad): the lanes of a column read neighbouring 16-byte pieces of one line in
// every channel, a quarter of the lines a lane-per-column load touches.  The sum over weighted
// channels that the atom gradient needs is taken inside the channel loop when several channels of the
// round carry weight (DENSE), and from a re-read of the one that does otherwise (one-hot types: one
// extra load per quad in one round, nothing in the others).
template <bool BINARY, bool DENSE, int CH>
__device__ __forceinline__ void va_round(const BwdArgs& G, const ItemParams& P, VaShared& sh, const float* diffb,
                                         int tb, int nch, int nnz, float ox, float oy, float oz,
                                         float (&tgacc)[CH], float& agx, float& agy, float& agz, int lane) {
  const GMParams& gm = G.gm;
  const size_t dim = gm.dim;
  const size_t cs4 = dim * dim * dim / 4;  // channel stride in quads
  const float Tcull = fmaxf(P.Tcut, BINARY ? P.Tbin : -1.f);
  const float kexp = P.inv_ar2 * NEG2_LOG2E;
  const bool tail = gm.ta != 0.f || gm.tb != 0.f;  // without a tail nothing lies beyond the Gaussian part
  const float k4 = 4.f * P.inv_ar2, kD = tail ? -gm.D * P.inv_ar2 : 0.f, kE = tail ? -gm.E * P.inv_ar : 0.f;
  const float ta = gm.ta, ntb = -gm.tb;
  const unsigned span = quad_span(P);
  ColBufD& buf = sh.buf;
  for (Columns cols(P); cols.more();) {
    const unsigned nkept = cols.compact<true>(buf, P, Tcull, ox, oy, gm.res, gm.dim, lane);
    __syncwarp();
    auto quad = [&](unsigned i, float dxy2, float exy, const float (&d2v)[4], const float (&ev)[4],
                    const float (&dzv)[4], size_t off) {
      float v[4], dsum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float rsq = __fadd_rn(dxy2, d2v[j]);
        if (BINARY) {
          v[j] = rsq < P.Tbin ? 1.f : 0.f;
        } else {
          float tq = fma_sat(-ta, sqrt_approx(rsq * P.inv_ar2), -ntb);
          v[j] = rsq <= P.Tg ? exy * ev[j] : tq * tq;  // tq is zero beyond the cut-off and for a NaN rsq
        }
      }
      const float4* qp = reinterpret_cast<const float4*>(diffb + off) + (size_t)tb * cs4;
      // the channels requested together, then used
      float4 dv[CH];
#pragma unroll
      for (int u = 0; u < CH; u++) {
        dv[u] = load_quad(qp, u < nch);
        qp += cs4;
      }
#pragma unroll
      for (int u = 0; u < CH; u++) {
        tgacc[u] = fmaf(v[0], dv[u].x, fmaf(v[1], dv[u].y, fmaf(v[2], dv[u].z, fmaf(v[3], dv[u].w, tgacc[u]))));
        if (DENSE) {
          const float wk = sh.w[u];
          dsum[0] = fmaf(wk, dv[u].x, dsum[0]);
          dsum[1] = fmaf(wk, dv[u].y, dsum[1]);
          dsum[2] = fmaf(wk, dv[u].z, dsum[2]);
          dsum[3] = fmaf(wk, dv[u].w, dsum[3]);
        }
      }
      if (!DENSE) {
        if (nnz == 0) return;  // the same for every lane
        const float4 d = __ldg(reinterpret_cast<const float4*>(diffb + off) + (size_t)(tb + sh.nz_t[0]) * cs4);
        const float wk = sh.nz_w[0];
        dsum[0] = wk * d.x;
        dsum[1] = wk * d.y;
        dsum[2] = wk * d.z;
        dsum[3] = wk * d.w;
      } else {
        // What stands in a channel without weight is not the atom's: where it was no number, zero times it is none
        // either, and the sum is taken again.
        const float whole = (dsum[0] + dsum[1]) + (dsum[2] + dsum[3]);
        if (whole != whole) {
#pragma unroll
          for (int j = 0; j < 4; j++) dsum[j] = 0.f;
#pragma unroll 1
          for (int k = 0; k < nnz; k++) {
            const float4 d = __ldg(reinterpret_cast<const float4*>(diffb + off) + (size_t)(tb + sh.nz_t[k]) * cs4);
            const float wk = sh.nz_w[k];
            dsum[0] = fmaf(wk, d.x, dsum[0]);
            dsum[1] = fmaf(wk, d.y, dsum[1]);
            dsum[2] = fmaf(wk, d.z, dsum[2]);
            dsum[3] = fmaf(wk, d.w, dsum[3]);
          }
        }
      }
      float fsum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float rsq = __fadd_rn(dxy2, d2v[j]);
        // kE/d + kD is zero at the cut-off and negative beyond it: the clamp stands in for the comparison
        float s1 = rsq <= P.Tg ? k4 * (exy * ev[j]) : fmaxf(fmaf(kE, rsqrt_approx(rsq), kD), 0.f);
        float f = s1 * dsum[j];
        fsum += f;
        agz = fmaf(f, dzv[j], agz);
      }
      agx = fmaf(fsum, buf.dx[i], agx);
      agy = fmaf(fsum, buf.dy[i], agy);
    };
    qlane_sweep_any(span, P, buf, nkept, dim, oz, gm.res, kexp, Tcull, lane, quad);
    __syncwarp();
  }
}

template <bool BINARY, int CH>
__global__ void __launch_bounds__(VA_WARPS * 32, VA_MINB) k_backward_quads_atom(BwdArgs G) {
  wait_for_stream();
  __shared__ VaShared shs[VA_WARPS];
  const GMParams& gm = G.gm;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int item = blockIdx.x * VA_WARPS + wid;
  int bl = blockIdx.y;
  int b = G.b0 + bl;
  if (item >= G.N) return;
  VaShared& sh = shs[wid];

  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  ItemParams P = load_item<false>(G, bl, b, item, ox, oy, oz);

  const size_t chan_stride = (size_t)gm.dim * gm.dim * gm.dim;
  const float* diffb = G.diff + (size_t)b * G.T * chan_stride;
  const size_t ai = (size_t)b * G.N + item;
  const float* wrow = G.type_vector + ai * G.T;
  float agx = 0.f, agy = 0.f, agz = 0.f;

  for (int tb = 0; tb < G.T; tb += CH) {
    const int nch = min(CH, G.T - tb);
    float tgacc[CH];
#pragma unroll
    for (int c = 0; c < CH; c++) tgacc[c] = 0.f;
    if (P.valid) {
      // the round's weights, and the list of the channels that carry one
      __syncwarp();
      float w = lane < nch ? wrow[tb + lane] : 0.f;
      unsigned m = __ballot_sync(0xffffffffu, w != 0.f);
      if (lane < CH) sh.w[lane] = w;
      if (w != 0.f) {
        int k = __popc(m & ((1u << lane) - 1u));
        sh.nz_t[k] = lane;
        sh.nz_w[k] = w;
      }
      __syncwarp();
      int nnz = __popc(m);
      if ((m & (m - 1u)) != 0u) va_round<BINARY, true, CH>(G, P, sh, diffb, tb, nch, nnz, ox, oy, oz, tgacc, agx, agy, agz, lane);
      else va_round<BINARY, false, CH>(G, P, sh, diffb, tb, nch, nnz, ox, oy, oz, tgacc, agx, agy, agz, lane);
    }
    // type gradients of this round
#pragma unroll
    for (int c = 0; c < CH; c++) {
      float x = tgacc[c];
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane == 0 && c < nch) G.type_gradients[ai * G.T + tb + c] = x;
    }
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    agx += __shfl_xor_sync(0xffffffffu, agx, o);
    agy += __shfl_xor_sync(0xffffffffu, agy, o);
    agz += __shfl_xor_sync(0xffffffffu, agz, o);
  }
  if (lane == 0) {
    G.atom_gradients[ai * 3] = agx;
    G.atom_gradients[ai * 3 + 1] = agy;
    G.atom_gradients[ai * 3 + 2] = agz;
  }
}

// ---------------------------------------------------------------------------------------------
// The same for many atoms a grid: every channel is read under every footprint, and above the L1 takes a clock for each line
// that a request touches, 85 columns in each of 28 channels.  A copy of the gradient with the channels of a voxel next to
// each other makes that one line a voxel, and what bounds the sums are the loads from the L2 (83 kB an atom, 11.8 TB/s; L1 69 %
// with 8 % hits, issue 47 %).  50 x 3000 atoms on 28x48^3, one / all weighted, 1690 / 1730 us without a copy and 1171 / 1661 like this.
// Blocks of one warp: eight atoms a block, neighbours by Morton's curve, meet too few lines of each other's in the L1 (hits 22 to
// 35 %, with the order and without) for what the wait for the slowest costs: 1590 us where blocks of one warp had 1225.  In the build
// of that time, quads of a column and voxels of a lane requested together, blocks an SM: 4 / 4 / 20 1226 us, 2 / 4 / 20 1301, 4 / 4 / 24
// 1297 to 1505 (the L1 gets what shared memory leaves), 4 / 6 / 20 1267; with the atoms of many weighted channels beside, 1271; with a
// single channel's values weighted afterwards 1171.
// ---------------------------------------------------------------------------------------------
constexpr int CL_VOXELS = 128, CL_PITCH = CL_VOXELS + 1;

// Channels [0, T) of the voxels to rows of TQ quads a voxel, filled up with zeros, and a row of zeros behind the last.  A
// block of TQ warps turns 128 voxels: a warp reads four channels, a thread writes one quad of channels of every 32nd voxel.
// Bound by memory: 4 examples of 28x48^3 17 us, 6.2 TB/s.
template <int TQ>
__global__ void __launch_bounds__(32 * TQ) k_channel_last(const float* diff, float4* copy, unsigned voxels, int T) {
  __shared__ float tile[4 * TQ * CL_PITCH];
  wait_for_stream();
  let_next_begin();
  const unsigned v0 = blockIdx.x * CL_VOXELS, lane = threadIdx.x & 31, c0 = threadIdx.x >> 5 << 2, n = min((unsigned)CL_VOXELS, voxels - v0);
  const float* src = diff + (size_t)blockIdx.y * T * voxels + (size_t)c0 * voxels + v0 + lane;
  float d[4][4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
#pragma unroll
    for (int k = 0; k < 4; k++) d[c][k] = c0 + c < T && lane + 32 * k < n ? __ldcs(src + 32 * k) : 0.f;
    src += voxels;
  }
  float* to = tile + c0 * CL_PITCH + lane;
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int k = 0; k < 4; k++) to[c * CL_PITCH + 32 * k] = d[c][k];
  __syncthreads();
  const unsigned v = threadIdx.x / TQ, q = threadIdx.x % TQ;
  const float* p = tile + 4 * q * CL_PITCH + v;
  float4* dst = copy + ((size_t)blockIdx.y * (voxels + 1) + v0) * TQ + threadIdx.x;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (v + 32 * k < n) dst[32 * k * TQ] = make_float4(p[32 * k], p[CL_PITCH + 32 * k], p[2 * CL_PITCH + 32 * k], p[3 * CL_PITCH + 32 * k]);
  if (v0 + n == voxels && threadIdx.x < TQ) copy[((size_t)blockIdx.y * (voxels + 1) + voxels) * TQ + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
}

constexpr int TG_MINB = 20;       // blocks of one warp an SM
constexpr int TG_COLS = 128;
constexpr int TG_Q = 4;           // quads of a column that are requested together
constexpr int TG_U = 4;           // voxels of a lane that are requested together

// Eight channels of a voxel in one load.
struct __align__(32) Eight {
  Pair p[4];
};
__device__ __forceinline__ Eight load_eight(const Eight* p) {
  Eight v;
  asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v.p[0].v), "=l"(v.p[1].v), "=l"(v.p[2].v), "=l"(v.p[3].v) : "l"(p) : "memory");
  return v;
}

struct TgArgs {
  BwdArgs G;
  const Eight* copy;  // [examples of the launch][voxels + 1][TO]
  int first;          // first example of the launch, counted in the pass
};

// TO: eights of channels a voxel.  The lanes are (voxel, eight) while voxels are added up, VOXELS at a time.
template <int TO>
struct __align__(16) TgShared {
  static constexpr unsigned VOXELS = 32 / TO, BATCH = TG_U * VOXELS;
  // voxels within reach, filled up to a whole batch: place in the copy and density; for atoms of many weighted channels
  // place, density and its gradient by the atom's position, of one step (128 voxels at most)
  static constexpr unsigned CAP = 128 * TG_Q + BATCH, DENSE_CAP = 128 + BATCH;
  union {
    uint2 list[CAP];
    struct {
      unsigned place[DENSE_CAP];
      float v[DENSE_CAP], slope[3][DENSE_CAP];
    } dense;
    float sums[32][9];
  };
  ColBufT<TG_COLS> cols;
  ZTabs zt;
};

// Sums of the n listed voxels; places up to a whole batch are the copy's row of zeros.  `mine` is the lane's eight of voxel 0.
template <int TO, bool DENSE>
__device__ __forceinline__ void tg_add(TgShared<TO>& sh, unsigned n, const Eight* mine, unsigned zeros, int lane, Pair (&tg)[4],
                                       const Pair (&w)[4], float (&ag)[3]) {
  constexpr unsigned VOXELS = TgShared<TO>::VOXELS, BATCH = TgShared<TO>::BATCH;
  const unsigned whole = (n + BATCH - 1) / BATCH * BATCH, g = min((unsigned)lane / TO, VOXELS - 1u);
  for (unsigned i = n + lane; i < whole; i += 32) {
    if (DENSE) {
      sh.dense.place[i] = zeros;
      sh.dense.v[i] = sh.dense.slope[0][i] = sh.dense.slope[1][i] = sh.dense.slope[2][i] = 0.f;
    } else {
      sh.list[i] = make_uint2(zeros, 0u);
    }
  }
  __syncwarp();
  Pair acc[4] = {pair(0.f), pair(0.f), pair(0.f), pair(0.f)};
  float own[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
  for (unsigned i = g; i < whole; i += BATCH) {
    uint2 e[TG_U];
    Eight d[TG_U];
#pragma unroll
    for (int u = 0; u < TG_U; u++) {
      const unsigned k = i + u * VOXELS;
      e[u] = DENSE ? make_uint2(sh.dense.place[k], __float_as_uint(sh.dense.v[k])) : sh.list[k];
    }
#pragma unroll
    for (int u = 0; u < TG_U; u++) d[u] = load_eight(mine + e[u].x);
    // by batches, then by calls, then for the atom: sums of few terms each
    Pair sum[4];
    float a[3];
#pragma unroll
    for (int u = 0; u < TG_U; u++) {
      const Pair v = pair(__uint_as_float(e[u].y));
#pragma unroll
      for (int c = 0; c < 4; c++) sum[c] = u == 0 ? mul2(v, d[u].p[c]) : fma2(v, d[u].p[c], sum[c]);
      if (DENSE) {
        float x, y;
        split(fma2(w[0], d[u].p[0], fma2(w[1], d[u].p[1], fma2(w[2], d[u].p[2], mul2(w[3], d[u].p[3])))), x, y);
        const unsigned k = i + u * VOXELS;
#pragma unroll
        for (int j = 0; j < 3; j++) a[j] = u == 0 ? sh.dense.slope[j][k] * (x + y) : fmaf(sh.dense.slope[j][k], x + y, a[j]);
      }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) acc[c] = add2(acc[c], sum[c]);
#pragma unroll
    for (int j = 0; j < 3; j++)
      if (DENSE) own[j] += a[j];
  }
#pragma unroll
  for (int c = 0; c < 4; c++) tg[c] = add2(tg[c], acc[c]);
#pragma unroll
  for (int j = 0; j < 3; j++)
    if (DENSE) ag[j] += own[j];
  __syncwarp();
}

// One atom, whose weights `w` are those of a lane's channel.  A lane owns a column, as in backward_quads_core(), and lists the
// voxels of its quads that lie within reach.  The atom gradient takes the values of `channel`, not weighted, where they lie, or
// of all channels (DENSE) from the copy, by the gradients of the density that are listed too.
template <int TO, bool BINARY, bool DENSE>
__device__ __forceinline__ void tg_atom(const TgArgs& A, const ItemParams& P, TgShared<TO>& sh, const float* diffb, const Eight* mine,
                                        float ox, float oy, float oz, float w, int channel, Pair (&tg)[4], float (&ag)[3], int lane) {
  const GMParams& gm = A.G.gm;
  const unsigned dim = gm.dim, voxels = dim * dim * dim;
  const bool aligned = dim % 4 == 0 && (uintptr_t)A.G.diff % 16 == 0;
  const float Tcull = fmaxf(P.Tcut, BINARY ? P.Tbin : -1.f);
  const float kexp = P.inv_ar2 * NEG2_LOG2E;
  const bool tail = gm.ta != 0.f || gm.tb != 0.f;
  const float k4 = 4.f * P.inv_ar2, kD = tail ? -gm.D * P.inv_ar2 : 0.f, kE = tail ? -gm.E * P.inv_ar : 0.f;
  const float inv_dim = 1.f / small_float(dim);
  const float* one = diffb + (size_t)channel * voxels;
  Pair w8[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    w8[c] = pair(0.f);
    if (DENSE) w8[c] = pair(__shfl_sync(0xffffffffu, w, lane % TO * 8 + 2 * c), __shfl_sync(0xffffffffu, w, lane % TO * 8 + 2 * c + 1));
  }
  Pair az = pair(0.f);
  unsigned n = 0;
  for (Columns cols(P); cols.more();) {
    const unsigned nkept = cols.compact<false>(sh.cols, P, Tcull, ox, oy, gm.res, dim, lane);
    for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * QPASS) {
      __syncwarp();
      fill_ztabs(sh.zt, zc, P, oz, gm.res, kexp, lane);
      __syncwarp();
      const unsigned nq = min((unsigned)QPASS, (P.hiz - zc + 3) >> 2);
#pragma unroll 1
      for (unsigned c0 = 0; c0 < nkept; c0 += 32) {
        const unsigned i = c0 + lane;
        unsigned row = 0;
        const float dxy2 = i < nkept ? sh.cols.get(i, row) : CUDART_NAN_F;
        const unsigned voxel = row * dim + zc;
        float dx = 0.f, dy = 0.f;
        auto from_atom = [&] {
          const unsigned x = (unsigned)((small_float(row) + 0.5f) * inv_dim);
          dx = __fsub_rn(voxel_coord(ox, x, gm.res), P.x);
          dy = __fsub_rn(voxel_coord(oy, row - x * dim, gm.res), P.y);
        };
        if (DENSE) from_atom();
        const float exy = ex2_approx(dxy2 * kexp);
        const Pair xy = pair(dxy2);
        Pair fs = pair(0.f);
#pragma unroll 1
        for (unsigned q0 = 0; q0 < nq; q0 += TG_Q) {
          float4 dv[TG_Q];
          bool live[TG_Q];
#pragma unroll
          for (int u = 0; u < TG_Q; u++) {
            live[u] = q0 + u < nq && __fadd_rn(dxy2, sh.zt.lo[q0 + u]) <= Tcull;  // false for a NaN
            if (DENSE) continue;
            dv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            const float* p = one + voxel + 4 * (q0 + u);
            if (aligned) {
              if (live[u]) dv[u] = __ldg(reinterpret_cast<const float4*>(p));
            } else if (live[u]) {
              const unsigned z = zc + 4 * (q0 + u);
              if (z >= P.loz && z < P.hiz) dv[u].x = __ldg(p);
              if (z + 1 >= P.loz && z + 1 < P.hiz) dv[u].y = __ldg(p + 1);
              if (z + 2 >= P.loz && z + 2 < P.hiz) dv[u].z = __ldg(p + 2);
              if (z + 3 >= P.loz && z + 3 < P.hiz) dv[u].w = __ldg(p + 3);
            }
          }
#pragma unroll
          for (int u = 0; u < TG_Q; u++) {
            if (!__any_sync(0xffffffffu, live[u])) continue;
            const float4 d2 = sh.zt.dz2[q0 + u], e = sh.zt.ez[q0 + u], dz = sh.zt.dz[q0 + u];
            const Pair d2p[2] = {pair(d2.x, d2.y), pair(d2.z, d2.w)}, ep[2] = {pair(e.x, e.y), pair(e.z, e.w)},
                       dzp[2] = {pair(dz.x, dz.y), pair(dz.z, dz.w)};
            float v[4], s[4];
            bool listed[4];
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
              float r0, r1, a0, a1, b0, b1;
              const Pair r = add2(xy, d2p[j / 2]), gauss = mul2(pair(exy), ep[j / 2]);
              split(r, r0, r1);
              const Pair id = pair(rsqrt_approx(r0), rsqrt_approx(r1));
              split(fma2(pair(kE), id, pair(kD)), a0, a1);  // zero at the cut-off and negative beyond it
              split(mul2(pair(k4), gauss), b0, b1);
              const bool g0 = r0 <= P.Tg, g1 = r1 <= P.Tg, in0 = r0 <= Tcull, in1 = r1 <= Tcull;
              s[j] = g0 ? b0 : fmaxf(a0, 0.f);
              s[j + 1] = g1 ? b1 : fmaxf(a1, 0.f);
              listed[j] = BINARY && !DENSE ? r0 < P.Tbin : in0;
              listed[j + 1] = BINARY && !DENSE ? r1 < P.Tbin : in1;
              if (BINARY) {
                v[j] = r0 < P.Tbin ? 1.f : 0.f;
                v[j + 1] = r1 < P.Tbin ? 1.f : 0.f;
              } else {
                // from a root of its own: through the reciprocal one of the gradient it is 5 to 14 % further from 64 bits
                split(mul2(r, pair(P.inv_ar2)), a0, a1);
                a0 = fma_sat(-gm.ta, sqrt_approx(a0), gm.tb);
                a1 = fma_sat(-gm.ta, sqrt_approx(a1), gm.tb);
                split(gauss, b0, b1);
                v[j] = g0 ? b0 : a0 * a0;
                v[j + 1] = g1 ? b1 : a1 * a1;
              }
              if (!DENSE) {
                float x0, x1;
                split(mul2(pair(s[j], s[j + 1]), j == 0 ? pair(dv[u].x, dv[u].y) : pair(dv[u].z, dv[u].w)), x0, x1);
                const Pair f = pair(in0 ? x0 : 0.f, in1 ? x1 : 0.f);  // a neighbour's value may be anything
                fs = add2(fs, f);
                az = fma2(f, dzp[j / 2], az);
              }
            }
            unsigned place = (voxel + 4 * (q0 + u)) * TO;
            const float dzv[4] = {dz.x, dz.y, dz.z, dz.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const unsigned them = __ballot_sync(0xffffffffu, listed[j]), at = n + __popc(them & ((1u << lane) - 1u));
              if (DENSE) {
                if (listed[j]) {
                  sh.dense.place[at] = place;
                  sh.dense.v[at] = v[j];
                  sh.dense.slope[0][at] = s[j] * dx;
                  sh.dense.slope[1][at] = s[j] * dy;
                  sh.dense.slope[2][at] = s[j] * dzv[j];
                }
              } else if (listed[j]) {
                sh.list[at] = make_uint2(place, __float_as_uint(v[j]));
              }
              n += __popc(them);
              place += TO;
            }
            if (DENSE) {
              tg_add<TO, DENSE>(sh, n, mine, voxels * TO, lane, tg, w8, ag);
              n = 0;
            }
          }
          if (!DENSE && n != 0) {
            tg_add<TO, DENSE>(sh, n, mine, voxels * TO, lane, tg, w8, ag);
            n = 0;
          }
        }
        if (!DENSE) {
          float f0, f1;
          split(fs, f0, f1);
          from_atom();
          ag[0] = fmaf(f0 + f1, dx, ag[0]);
          ag[1] = fmaf(f0 + f1, dy, ag[1]);
        }
      }
    }
    __syncwarp();
  }
  if (!DENSE) {
    float z0, z1;
    split(az, z0, z1);
    ag[2] += z0 + z1;
  } else if (lane / TO >= (int)TgShared<TO>::VOXELS) {
    ag[0] = ag[1] = ag[2] = 0.f;  // a lane too many for whole voxels
  }
}

// Sum by pairs, then pairs of pairs: as near to 64 bits as lanes that add up by shuffles.
template <int N>
__device__ __forceinline__ float tree_sum(float (&v)[N]) {
#pragma unroll
  for (int step = 1; step < N; step *= 2)
#pragma unroll
    for (int k = 0; k + step < N; k += 2 * step) v[k] += v[k + step];
  return v[0];
}

// Whether a sum over voxels of weight * slope * value has to be taken of slope * value alone and weighted afterwards: an
// infinite weight is no number where slope or value is zero, and a huge one makes the products overflow before the sum does.
__device__ __forceinline__ bool weigh_afterwards(float w, float inv_ar2) {
  return w != 0.f && !(fabsf(w) * fmaxf(1.f, 4.f * inv_ar2) < 1e30f);
}

template <int TO, bool BINARY>
__global__ void __launch_bounds__(32, TG_MINB) k_type_gradients(TgArgs A) {
  wait_for_stream();
  __shared__ TgShared<TO> sh;
  const BwdArgs& G = A.G;
  const GMParams& gm = G.gm;
  const int lane = threadIdx.x, item = blockIdx.x, bl = A.first + blockIdx.y, b = G.b0 + bl;
  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  const float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  const ItemParams P = load_item<false>(G, bl, b, item, ox, oy, oz);
  const size_t voxels = (size_t)gm.dim * gm.dim * gm.dim, ai = (size_t)b * G.N + item;
  const float* diffb = G.diff + (size_t)b * G.T * voxels;
  const Eight* mine = A.copy + blockIdx.y * (voxels + 1) * TO + lane % TO;
  const float w = lane < G.T ? G.type_vector[ai * G.T + lane] : 0.f;
  const unsigned m = __ballot_sync(0xffffffffu, w != 0.f);
  Pair tg[4];
  float ag[3] = {0.f, 0.f, 0.f}, sum = 0.f;
  unsigned left = m;
  tg[0] = tg[1] = tg[2] = tg[3] = pair(0.f);
  for (bool dense = (m & (m - 1u)) != 0u; P.valid; dense = false) {
    tg[0] = tg[1] = tg[2] = tg[3] = pair(0.f);
    ag[0] = ag[1] = ag[2] = 0.f;
    if (dense) tg_atom<TO, BINARY, true>(A, P, sh, diffb, mine, ox, oy, oz, w, 0, tg, ag, lane);
    else tg_atom<TO, BINARY, false>(A, P, sh, diffb, mine, ox, oy, oz, 0.f, left != 0u ? __ffs(left) - 1 : 0, tg, ag, lane);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
#pragma unroll
      for (int c = 0; c < 3; c++) ag[c] += __shfl_xor_sync(0xffffffffu, ag[c], o);
    }
    if (dense) {
      // What stands in a channel without weight is not the atom's: where it was no number, zero times it is none either.  An
      // infinite weight is none where slope or value is zero, and a huge one overflows before the sum does.  Then the weighted
      // channels are summed one by one and weighted afterwards, as a single one is.
      if (fabsf((ag[0] + ag[1]) + ag[2]) < CUDART_INF_F && !__any_sync(0xffffffffu, fabsf(w) == CUDART_INF_F)) break;
      continue;
    }
    if (left != 0u) {
      sum = fmaf(lane == 0 ? ag[0] : lane == 1 ? ag[1] : ag[2], __shfl_sync(0xffffffffu, w, __ffs(left) - 1), sum);
      left &= left - 1u;
      if (left != 0u) continue;
    }
#pragma unroll
    for (int c = 0; c < 3; c++) ag[c] = __shfl_sync(0xffffffffu, sum, c);
    break;
  }
#pragma unroll
  for (int c = 0; c < 4; c++) split(tg[c], sh.sums[lane][2 * c], sh.sums[lane][2 * c + 1]);
  __syncwarp();
  if (lane < G.T) {
    float part[TgShared<TO>::VOXELS];
#pragma unroll
    for (unsigned g = 0; g < TgShared<TO>::VOXELS; g++) part[g] = sh.sums[g * TO + (lane >> 3)][lane & 7];
    G.type_gradients[ai * G.T + lane] = tree_sum(part);
  }
  if (lane < 3) G.atom_gradients[ai * 3 + lane] = lane == 0 ? ag[0] : lane == 1 ? ag[1] : ag[2];
}

// The same without type gradients (the caller passed none: types that are inputs, not parameters):
// only the channels that carry weight are read.
__global__ void __launch_bounds__(BWD2_WARPS * 32) k_backward_quads_atom_ag(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBufD bufs[BWD2_WARPS];
  __shared__ ZTabs ztabs[BWD2_WARPS];
  __shared__ int nz_t[BWD2_WARPS][VA_CH];
  __shared__ float nz_w[BWD2_WARPS][VA_CH];
  const GMParams& gm = G.gm;
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int item = blockIdx.x * BWD2_WARPS + wid;
  int bl = blockIdx.y;
  int b = G.b0 + bl;
  if (item >= G.N) return;
  ColBufD& buf = bufs[wid];
  ZTabs& zt = ztabs[wid];

  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  ItemParams P = load_item<false>(G, bl, b, item, ox, oy, oz);

  size_t dim = gm.dim;
  const size_t chan_stride = dim * dim * dim;
  const float* diffb = G.diff + (size_t)b * G.T * chan_stride;
  const size_t ai = (size_t)b * G.N + item;
  const float* wrow = G.type_vector + ai * G.T;
  const float kexp = P.inv_ar2 * NEG2_LOG2E;
  const float k4 = 4.f * P.inv_ar2, kD = -gm.D * P.inv_ar2, kE = -gm.E * P.inv_ar;
  float agx = 0.f, agy = 0.f, agz = 0.f;

  for (int tb = 0; P.valid && tb < G.T; tb += VA_CH) {
    int t = tb + lane;
    float w = t < G.T ? wrow[t] : 0.f;
    unsigned m = __ballot_sync(0xffffffffu, w != 0.f);
    int nnz = __popc(m);
    if (nnz == 0) continue;
    __syncwarp();
    if (w != 0.f) {
      int slot = __popc(m & ((1u << lane) - 1u));
      nz_t[wid][slot] = t;
      nz_w[wid][slot] = w;
    }
    __syncwarp();
    for (Columns cols(P); cols.more();) {
      const unsigned nkept = cols.compact<true>(buf, P, P.Tcut, ox, oy, gm.res, gm.dim, lane);
      for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * QPASS) {
        __syncwarp();
        fill_ztabs(zt, zc, P, oz, gm.res, kexp, lane);
        __syncwarp();
        unsigned nq = min((unsigned)QPASS, (P.hiz - zc + 3) >> 2);
        for (unsigned c0 = 0; c0 < nkept; c0 += 32) {
          unsigned i = c0 + lane;
          bool have = i < nkept;
          float dxy2 = have ? buf.dxy2[i] : CUDART_NAN_F;
          float dx = have ? buf.dx[i] : 0.f, dy = have ? buf.dy[i] : 0.f;
          const float4* row = reinterpret_cast<const float4*>(diffb + (size_t)(have ? buf.row[i] : 0u) * dim + zc);
          float exy4 = k4 * ex2_approx(dxy2 * kexp);
          float fsum = 0.f;
          for (unsigned q = 0; q < nq; q++) {
            float4 d2 = zt.dz2[q], e = zt.ez[q], dz = zt.dz[q];
            float lo = zt.lo[q];
            bool live = __fadd_rn(dxy2, lo) <= P.Tcut;
            float4 ds = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int k = 0; k < nnz; k++) {
              if (live) {
                float wk = nz_w[wid][k];
                float4 dv = __ldg(row + q + (size_t)nz_t[wid][k] * (chan_stride / 4));
                ds.x = fmaf(wk, dv.x, ds.x); ds.y = fmaf(wk, dv.y, ds.y);
                ds.z = fmaf(wk, dv.z, ds.z); ds.w = fmaf(wk, dv.w, ds.w);
              }
            }
            float d2v[4] = {d2.x, d2.y, d2.z, d2.w}, ev[4] = {e.x, e.y, e.z, e.w};
            float dzv[4] = {dz.x, dz.y, dz.z, dz.w}, dsv[4] = {ds.x, ds.y, ds.z, ds.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
              float rsq = __fadd_rn(dxy2, d2v[j]);
              float sg = rsq <= P.Tg ? exy4 * ev[j] : fmaf(kE, rsqrt_approx(rsq), kD);
              float f = rsq <= P.Tcut ? sg * dsv[j] : 0.f;
              fsum += f;
              agz = fmaf(f, dzv[j], agz);
            }
          }
          agx = fmaf(fsum, dx, agx);
          agy = fmaf(fsum, dy, agy);
        }
      }
      __syncwarp();
    }
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    agx += __shfl_xor_sync(0xffffffffu, agx, o);
    agy += __shfl_xor_sync(0xffffffffu, agy, o);
    agz += __shfl_xor_sync(0xffffffffu, agz, o);
  }
  if (lane == 0) {
    G.atom_gradients[ai * 3] = agx;
    G.atom_gradients[ai * 3 + 1] = agy;
    G.atom_gradients[ai * 3 + 2] = agz;
  }
}

// backward_gradients for the same layout (vector types, per-atom radii), one warp per atom, both terms in
// one sweep as above.  Only channels in which the atom carries weight take part (src/grid_maker.cpp:573); the
// voxel-dependent factors are shared by them.  Grid term of channel t: density * tgrad_t + w_t * s * (delta .
// agrad); atom term: (alpha (delta.agrad) delta_a - s agrad_a) S1 + (alpha delta_a^2 - s) S2 with
// S1 = sum_t w_t diff_t and S2 = sum_t tgrad_t diff_t.
__global__ void __launch_bounds__(SO_WARPS * 32, SO_ATOM_MINB) k_second_quads_atom(BwdArgs G) {
  wait_for_stream();
  __shared__ ColBufD bufs[SO_WARPS];
  __shared__ ZTabs ztabs[SO_WARPS];
  __shared__ int nz_t[SO_WARPS][VA_CH];
  __shared__ float2 nz_wg[SO_WARPS][VA_CH];  // weight and incoming type gradient
  const GMParams& gm = G.gm;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, item = blockIdx.x * SO_WARPS + wid;
  const int bl = blockIdx.y, b = G.b0 + bl;
  if (item >= G.N) return;
  ColBufD& buf = bufs[wid];
  ZTabs& zt = ztabs[wid];

  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  const float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  const ItemParams P = load_item<false>(G, bl, b, item, ox, oy, oz);

  const size_t dim = gm.dim, cs = dim * dim * dim, base = (size_t)b * G.T * cs, ai = (size_t)b * G.N + item;
  const float* wrow = G.type_vector + ai * G.T;
  const float* grow = G.tg_in + ai * G.T;
  const float inx = G.ag_in[ai * 3], iny = G.ag_in[ai * 3 + 1], inz = G.ag_in[ai * 3 + 2];
  const bool odd = !finite3(inx, iny, inz);  // the same for every lane
  const float kexp = P.inv_ar2 * NEG2_LOG2E;
  const SecondConst K(gm, P);
  float agx = 0.f, agy = 0.f, agz = 0.f;

  for (int tb = 0; P.valid && tb < G.T; tb += VA_CH) {
    const int t = tb + lane;
    const float w = t < G.T ? wrow[t] : 0.f;
    const unsigned m = __ballot_sync(0xffffffffu, w != 0.f);
    const int nnz = __popc(m);
    if (nnz == 0) continue;
    __syncwarp();
    if (w != 0.f) {
      const int slot = __popc(m & ((1u << lane) - 1u));
      nz_t[wid][slot] = t;
      nz_wg[wid][slot] = make_float2(w, grow[t]);
    }
    __syncwarp();
    Pair sb1 = pair(0.f), sb2 = pair(0.f);  // sums of s * S1 and s * S2
    auto sweep = [&](auto odd) {
      for (Columns cols(P); cols.more();) {
        const unsigned nkept = cols.compact<true>(buf, P, P.Tcut, ox, oy, gm.res, gm.dim, lane);
        for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * QPASS) {
          __syncwarp();
          fill_ztabs(zt, zc, P, oz, gm.res, kexp, lane);
          __syncwarp();
          const unsigned nq = min((unsigned)QPASS, (P.hiz - zc + 3) >> 2);
          for (unsigned c0 = 0; c0 < nkept; c0 += 32) {
            const unsigned i = c0 + lane;
            const bool have = i < nkept;
            const float dxy2 = have ? buf.dxy2[i] : CUDART_NAN_F, dx = have ? buf.dx[i] : 0.f, dy = have ? buf.dy[i] : 0.f;
            const size_t off = base + (size_t)(have ? buf.row[i] : 0u) * dim + zc;
            const Pair xy = pair(dxy2), exy = pair(ex2_approx(dxy2 * kexp));
            const float dotxy = fmaf(dx, inx, dy * iny);
            // sums over the column: alpha * S2 * {1, dz^2}, alpha * (delta . agrad) * S1 * {1, dz}
            Pair p0 = pair(0.f), p2 = pair(0.f), u0 = pair(0.f), u1 = pair(0.f);
            for (unsigned q = 0; q < nq; q++) {
              if (!(__fadd_rn(dxy2, zt.lo[q]) <= P.Tcut)) continue;
              const float4 d2 = zt.dz2[q], e = zt.ez[q], dz = zt.dz[q];
              const Pair d2p[2] = {pair(d2.x, d2.y), pair(d2.z, d2.w)}, ep[2] = {pair(e.x, e.y), pair(e.z, e.w)},
                         dzp[2] = {pair(dz.x, dz.y), pair(dz.z, dz.w)};
              Pair val[2], s[2], sd[2], alpha[2], dot[2], s1[2], s2[2];
              bool in[4];
#pragma unroll
              for (int j = 0; j < 2; j++) {
                const Pair rsq = add2(xy, d2p[j]);
                second_factors<true>(K, P, rsq, mul2(exy, ep[j]), val[j], s[j], alpha[j], in[2 * j], in[2 * j + 1]);
                dot[j] = fma2(dzp[j], pair(inz), pair(dotxy));
                sd[j] = mul2(s[j], dot[j]);
                if constexpr (odd.value) {
                  sd[j] = only_off_atom(sd[j], rsq, in[2 * j], in[2 * j + 1]);
                  dot[j] = only(dot[j], in[2 * j], in[2 * j + 1]);
                }
                s1[j] = s2[j] = pair(0.f);
              }
              const float* src = G.diff + off + 4 * q;
              float* dst = G.out_grid + off + 4 * q;
              for (int k = 0; k < nnz; k++) {
                const float2 wg = nz_wg[wid][k];
                const size_t co = (size_t)nz_t[wid][k] * cs;
                const float4 dv = __ldg(reinterpret_cast<const float4*>(src + co));
                const Pair dvp[2] = {pair(dv.x, dv.y), pair(dv.z, dv.w)}, wk = pair(wg.x), gk = pair(wg.y);
                float v[4];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                  s1[j] = fma2(wk, dvp[j], s1[j]);
                  s2[j] = fma2(gk, dvp[j], s2[j]);
                  split(fma2(val[j], gk, mul2(sd[j], wk)), v[2 * j], v[2 * j + 1]);
                }
                red_add_v4(dst + co, v[0], v[1], v[2], v[3]);
              }
#pragma unroll
              for (int j = 0; j < 2; j++) {
                s1[j] = only(s1[j], in[2 * j], in[2 * j + 1]);  // a neighbour's values may be anything
                s2[j] = only(s2[j], in[2 * j], in[2 * j + 1]);
                const Pair a2 = mul2(alpha[j], s2[j]), a1 = mul2(mul2(alpha[j], dot[j]), s1[j]);
                p0 = add2(p0, a2);
                p2 = fma2(a2, mul2(dzp[j], dzp[j]), p2);
                u0 = add2(u0, a1);
                u1 = fma2(a1, dzp[j], u1);
                sb1 = fma2(s[j], s1[j], sb1);
                sb2 = fma2(s[j], s2[j], sb2);
              }
            }
            float a, b0, c, d, t0;
            split(p0, a, t0); a += t0;
            split(p2, b0, t0); b0 += t0;
            split(u0, c, t0); c += t0;
            split(u1, d, t0); d += t0;
            agx = fmaf(dx, fmaf(a, dx, c), agx);
            agy = fmaf(dy, fmaf(a, dy, c), agy);
            agz += b0 + d;
          }
        }
        __syncwarp();
      }
    };
    if (odd) sweep(std::true_type());
    else sweep(std::false_type());
    float x0, x1, y0, y1;
    split(sb1, x0, x1);
    split(sb2, y0, y1);
    x0 += x1;
    y0 += y1;
    agx -= fmaf(x0, inx, y0);
    agy -= fmaf(x0, iny, y0);
    agz -= fmaf(x0, inz, y0);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    agx += __shfl_xor_sync(0xffffffffu, agx, o);
    agy += __shfl_xor_sync(0xffffffffu, agy, o);
    agz += __shfl_xor_sync(0xffffffffu, agz, o);
  }
  if (lane < 3) G.atom_gradients[ai * 3 + lane] = lane == 0 ? agx : lane == 1 ? agy : agz;
}

// ---------------------------------------------------------------------------------------------
// Type vectors whose radii differ by channel, all channels wanted: the footprints of an atom's channels lie in each other, so
// a warp takes up to RT_CH channels of an ATOM, and what depends on the place alone - column, squared distance, its roots,
// the address - is computed once for all of them.  A warp lists the quads that the largest sphere reaches and takes 32 at a
// time, whose lines are mostly neighbours; a channel whose sphere reaches none of these is skipped.
// Bound by issue.  Item by item the L1 bounded it (95 %: a lane per column touches 32 lines a load): soft types, 28 channels, 4 x
// 3000 atoms on 96^3 of 0.25 A 2469 us, 4 x 1500 on 48^3 of 0.5 A 283, 8 x 1000 with 20 channels on 40^3 of 0.75 A 173; like this
// 2045, 188 and 85, of which sums of few terms (RT_STEPS) take 1 to 2 %.  On the way: lanes as (column, z-quad) of the whole
// footprint 3338 / 255 / 109, the list 2271 / 196 / 88; quads in three shells by distance 2202 / 195 / 95; the tails of all
// channels apart 2514 / 221 / 105; channels by radius, blocks of an atom's warps 2870 / 250 / 110, of one warp 2267 / 209 / 94;
// blocks of one warp, channels as they come 2185 / 194 / 86, then no test of a weight for each.  A channel much smaller than the
// largest is listed with it all the same: see channels_together() for what that costs.  Tried against it: a vote for four channels
// together before their loads 10 % slower with all channels weighted; sweeps of their own for channels of half the radius and less
// 3 (0.25 A) to 20 % (24^3 of 1 A) slower where there are none.
// ---------------------------------------------------------------------------------------------
constexpr int RT_CH = 16, RT_WARPS = 4;  // channels a warp, most warps an atom
constexpr int RT_MINB = 20;              // blocks of one warp an SM: 96 registers (16 / 24: 2395 / 2313 us instead of 2267)
constexpr int RT_COLS = 128;
constexpr int RT_LOADS = 4;              // channels that are requested together
constexpr unsigned RT_STEPS = 8;         // groups of 32 quads whose atom gradients are summed by themselves

struct __align__(16) RtChannel {
  float kexp, Tg, Tcut, inv_ar;
  float k4, kE, kD, w;
};
struct __align__(16) RtShared {
  RtChannel ch[RT_CH];
  union {
    ColBufDT<RT_COLS> cols;
    float sums[RT_CH][33];
  };
  ZTabs zt;
  float4 ez[RT_CH][QPASS];                // exp(-2 dz2 / ar^2) for each channel
  float atom[5][32];                      // a lane's sums for the atom gradient: x, y, z of even and odd voxels; or as k_second_channels has them
  unsigned short list[RT_COLS * QPASS];   // quads within reach: column | quad << 8
};

// Lists the quads of the nkept columns whose nearest voxel lies within Tcut; returns how many.
__device__ __forceinline__ unsigned list_quads(unsigned short* list, const ColBufDT<RT_COLS>& cols, const ZTabs& zt, unsigned nkept,
                                               unsigned nq, float Tcut, int lane) {
  unsigned n = 0;
  for (unsigned c0 = 0; c0 < nkept; c0 += 32) {
    const unsigned i = c0 + lane;
    const float dxy2 = i < nkept ? cols.dxy2[i] : CUDART_NAN_F;
    unsigned mask = 0;
#pragma unroll
    for (unsigned q = 0; q < QPASS; q++)
      if (q < nq && __fadd_rn(dxy2, zt.lo[q]) <= Tcut) mask |= 1u << q;  // false for a NaN
    unsigned upto = __popc(mask);
    const unsigned own = upto;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += x;
    }
    for (unsigned at = n + upto - own; mask != 0u; mask &= mask - 1u) list[at++] = (unsigned short)(i | (__ffs(mask) - 1) << 8);
    n += __shfl_sync(0xffffffffu, upto, 31);
  }
  return n;
}

// A channel whose sphere is smaller than a voxel reaches the voxel nearest to the atom at most, and not even that where its
// own footprint leaves it out: beside a coordinate a radius of 1e-7 times it is nothing, and the footprint is empty.
// The footprint that it shares with larger channels does not tell.
__device__ __forceinline__ bool reaches_nothing(const GMParams& gm, float densityrad, const ItemParams& P, float ox, float oy, float oz) {
  if (!(densityrad < 0.5f * gm.res && densityrad > 0.f)) return false;
  auto along = [&](float origin, float at) {
    unsigned lo, hi;
    bounds_1d(origin, at, densityrad, gm.res, gm.dim, lo, hi);
    const float nearest = rintf(__fdiv_rn(__fsub_rn(at, origin), gm.res));
    return nearest >= (float)lo && nearest < (float)hi;
  };
  return !(along(ox, P.x) && along(oy, P.y) && along(oz, P.z));
}

__global__ void __launch_bounds__(32, RT_MINB) k_backward_channels(BwdArgs G, int per, int warps) {
  wait_for_stream();
  __shared__ RtShared sh;
  const GMParams& gm = G.gm;
  const int lane = threadIdx.x, item = blockIdx.x / warps, wid = blockIdx.x - item * warps, bl = blockIdx.y, b = G.b0 + bl;
  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  const float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  const ItemParams P = item_of(G.recs[(size_t)bl * G.N + item]);  // of the largest radius
  const size_t dim = gm.dim, cs4 = dim * dim * dim / 4, ai = (size_t)b * G.N + item;
  const int t0 = wid * per, nch = min(per, G.T - t0);
  const ChanParam* params = G.chanp + (size_t)bl * G.T;
  if (lane < RT_CH) {
    RtChannel c = {0.f, -1.f, -1.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (lane < nch) {
      const ChanParam cp = params[t0 + lane];
      const float4 p = cp.p;
      c.kexp = p.x * NEG2_LOG2E; c.Tg = p.y; c.inv_ar = p.z;
      c.Tcut = reaches_nothing(gm, cp.q.z, P, ox, oy, oz) ? -1.f : p.w;
      c.k4 = 4.f * p.x; c.kE = -gm.E * p.z; c.kD = -gm.D * p.x;
      c.w = G.type_vector[ai * G.T + t0 + lane];
    }
    sh.ch[lane] = c;
  }
  __syncwarp();
  const float4* diff = reinterpret_cast<const float4*>(G.diff) + ((size_t)b * G.T + t0) * cs4;
  float tg[RT_CH], agx, agy, agz;
  // SKIP: channels without weight stay out of the atom gradient
  auto sweep = [&](auto skip) {
    constexpr bool SKIP = decltype(skip)::value;
#pragma unroll
    for (int c = 0; c < RT_CH; c++) tg[c] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; c++) sh.atom[c][lane] = 0.f;
    agx = agy = 0.f;
    Pair az = pair(0.f);
    auto put_by = [&] {
      float z0, z1;
      split(az, z0, z1);
      sh.atom[0][lane] += agx;
      sh.atom[1][lane] += agy;
      sh.atom[2][lane] += z0;
      sh.atom[3][lane] += z1;
      agx = agy = 0.f;
      az = pair(0.f);
    };
    for (Columns cols(P); cols.more();) {
      const unsigned nkept = cols.compact<true>(sh.cols, P, P.Tcut, ox, oy, gm.res, gm.dim, lane);
      for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * QPASS) {
        __syncwarp();
        fill_ztabs(sh.zt, zc, P, oz, gm.res, 0.f, lane);
        __syncwarp();
        for (int c = 0; c < nch; c++) reinterpret_cast<float*>(sh.ez[c])[lane] = ex2_approx(reinterpret_cast<const float*>(sh.zt.dz2)[lane] * sh.ch[c].kexp);
        const unsigned n = list_quads(sh.list, sh.cols, sh.zt, nkept, min((unsigned)QPASS, (P.hiz - zc + 3) >> 2), P.Tcut, lane);
        __syncwarp();
#pragma unroll 1
        for (unsigned e0 = 0; e0 < n; e0 += 32) {
          const unsigned e = sh.list[min(e0 + lane, n - 1u)], i = e & 255u, zq = e >> 8;
          const float dxy2 = sh.cols.dxy2[i], near = e0 + lane < n ? __fadd_rn(dxy2, sh.zt.lo[zq]) : CUDART_NAN_F;
          const float4* from = diff + (((size_t)sh.cols.row[i] * dim + zc) / 4 + zq);
          const float4 d2 = sh.zt.dz2[zq];
          const float d2v[4] = {d2.x, d2.y, d2.z, d2.w};
          float r[4], root[4], id[4];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            r[j] = __fadd_rn(dxy2, d2v[j]);
            // the root to the last place (root(), from the reciprocal root at hand): shared by the channels it costs little, and
            // the type gradients are 3 to 17 % nearer to 64 bits than with the approximate one
            id[j] = rsqrt_approx(r[j]);
            const float x = __fmul_rn(r[j], id[j]);
            root[j] = fmaf(fmaf(-x, x, r[j]), 0.5f * id[j], x);
          }
          Pair f[2] = {pair(0.f), pair(0.f)};
#pragma unroll
          for (int q = 0; q < RT_CH; q += RT_LOADS) {
            if (q >= nch) break;
            float4 dv[RT_LOADS];
            bool live[RT_LOADS];
#pragma unroll
            for (int u = 0; u < RT_LOADS; u++) {
              live[u] = near <= sh.ch[q + u].Tcut;  // false for a NaN, and for a channel that there is not
              dv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (live[u]) dv[u] = __ldg(from);
              from += cs4;
            }
#pragma unroll
            for (int u = 0; u < RT_LOADS; u++) {
              if (!__any_sync(0xffffffffu, live[u])) continue;
              const RtChannel& C = sh.ch[q + u];
              const Pair dvp[2] = {pair(dv[u].x, dv[u].y), pair(dv[u].z, dv[u].w)};
              const float4 e = sh.ez[q + u][zq];
              const Pair exy = pair(ex2_approx(dxy2 * C.kexp)), ep[2] = {pair(e.x, e.y), pair(e.z, e.w)};
              Pair sum = pair(0.f);
#pragma unroll
              for (int j = 0; j < 2; j++) {
                float e0, e1, x0, x1, a0, a1, b0, b1;
                split(mul2(exy, ep[j]), e0, e1);
                const bool g0 = r[2 * j] <= C.Tg, g1 = r[2 * j + 1] <= C.Tg;
                split(mul2(pair(root[2 * j], root[2 * j + 1]), pair(C.inv_ar)), x0, x1);
                x0 = fma_sat(-gm.ta, x0, gm.tb);
                x1 = fma_sat(-gm.ta, x1, gm.tb);
                const Pair v = pair(g0 ? e0 : x0 * x0, g1 ? e1 : x1 * x1);
                sum = j == 0 ? mul2(v, dvp[0]) : fma2(v, dvp[1], sum);
                split(fma2(pair(C.kE), pair(id[2 * j], id[2 * j + 1]), pair(C.kD)), a0, a1);  // negative beyond the cut-off
                split(mul2(pair(C.k4), pair(e0, e1)), b0, b1);
                if (!SKIP || C.w != 0.f)  // the same for every lane
                  f[j] = fma2(mul2(pair(g0 ? b0 : fmaxf(a0, 0.f), g1 ? b1 : fmaxf(a1, 0.f)), pair(C.w)), dvp[j], f[j]);
              }
              float sum0, sum1;
              split(sum, sum0, sum1);
              tg[q + u] += sum0 + sum1;
            }
          }
          float f0, f1;
          split(add2(f[0], f[1]), f0, f1);
          agx = fmaf(f0 + f1, sh.cols.dx[i], agx);
          agy = fmaf(f0 + f1, sh.cols.dy[i], agy);
          const float4 dz = sh.zt.dz[zq];
          az = fma2(f[0], pair(dz.x, dz.y), fma2(f[1], pair(dz.z, dz.w), az));
          if ((e0 & 32 * (RT_STEPS - 1)) == 32 * (RT_STEPS - 1)) put_by();  // sums of few terms each
        }
      }
      __syncwarp();
    }
    put_by();
    agx = sh.atom[0][lane];
    agy = sh.atom[1][lane];
    agz = sh.atom[2][lane] + sh.atom[3][lane];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      agx += __shfl_xor_sync(0xffffffffu, agx, o);
      agy += __shfl_xor_sync(0xffffffffu, agy, o);
      agz += __shfl_xor_sync(0xffffffffu, agz, o);
    }
  };
  agx = agy = agz = 0.f;
#pragma unroll
  for (int c = 0; c < RT_CH; c++) tg[c] = 0.f;
  if (P.valid && __any_sync(0xffffffffu, sh.ch[lane & (RT_CH - 1)].Tcut >= 0.f)) {
    // What stands in a channel without weight is not the atom's: where it was no number, zero times it is none either, and
    // the sums are taken again.  Most without weight: left out at once.  28 channels of 96^3, 4 x 3000 atoms, all / one
    // weighted: a test in any case 2185 / 1904 us, none 2075 / 2063.
    const RtChannel& own = sh.ch[lane & (RT_CH - 1)];
    const unsigned weighted = __ballot_sync(0xffffffffu, lane < nch && own.w != 0.f);
    const bool apart = __any_sync(0xffffffffu, weigh_afterwards(own.w, 0.25f * own.k4));
    bool again = apart || 2 * __popc(weighted) < nch;
    if (!again) {
      sweep(std::false_type());
      const float whole = (agx + agy) + agz;
      again = __popc(weighted) < nch && whole != whole;
    }
    if (again) {
      float sum = 0.f;  // of an axis a lane, channel by channel
      unsigned left = apart ? weighted : 1u;
      do {
        __syncwarp();
        if (apart && lane < nch) sh.ch[lane].w = lane == __ffs(left) - 1 ? 1.f : 0.f;
        __syncwarp();
        sweep(std::true_type());
        if (apart) sum = fmaf(lane == 0 ? agx : lane == 1 ? agy : agz, G.type_vector[ai * G.T + t0 + __ffs(left) - 1], sum);
        left &= left - 1u;
      } while (left != 0u);
      if (apart) {
        agx = __shfl_sync(0xffffffffu, sum, 0);
        agy = __shfl_sync(0xffffffffu, sum, 1);
        agz = __shfl_sync(0xffffffffu, sum, 2);
      }
    }
  }
  // of several warps an atom, k_sum_parts adds up the parts
  float* to = warps == 1 ? G.atom_gradients + ai * 3 : G.partial + (((size_t)bl * G.N + item) * warps + wid) * 3;
  if (lane < 3) to[lane] = lane == 0 ? agx : lane == 1 ? agy : agz;
#pragma unroll
  for (int c = 0; c < RT_CH; c++) sh.sums[c][lane] = tg[c];
  __syncwarp();
  static_assert(RT_CH == 16, "two lanes a channel");
  float part[16];
#pragma unroll
  for (int k = 0; k < 16; k++) part[k] = sh.sums[lane & 15][(lane & 16) + k];
  float sum = tree_sum(part);
  sum += __shfl_xor_sync(0xffffffffu, sum, 16);
  if (lane < nch) G.type_gradients[ai * G.T + t0 + lane] = sum;
}

// backward_gradients for the same layout (see k_second_quads_nz for the terms): the sums over an atom's channels that its
// term needs, with the weights w and the incoming type gradients t, are taken voxel by voxel - of w alpha diff and t alpha diff for
// the products of distances, of w s diff and t s diff for the rest.  Only channels that carry weight take part.
// Bound by issue at few warps: 20 blocks an SM spill and gain nothing (soft types, 4 x 1500 atoms on 28x48^3 of 0.5 A: item by item
// 542 us, like this 353, with 20 some 10 more).
constexpr int RS_MINB = 16;
constexpr int RS_LOADS = 2;
__global__ void __launch_bounds__(32, RS_MINB) k_second_channels(BwdArgs G, int per, int warps) {
  wait_for_stream();
  __shared__ RtShared sh;
  __shared__ float tgrad[RT_CH];
  __shared__ size_t offset[RT_CH];  // of the weighted channels, from the first of the warp's
  const GMParams& gm = G.gm;
  const int lane = threadIdx.x, item = blockIdx.x / warps, wid = blockIdx.x - item * warps, bl = blockIdx.y, b = G.b0 + bl;
  float cx, cy, cz;
  if (G.centers != nullptr) {
    cx = G.centers[b * 3]; cy = G.centers[b * 3 + 1]; cz = G.centers[b * 3 + 2];
  } else {
    cx = G.center_host[0]; cy = G.center_host[1]; cz = G.center_host[2];
  }
  const float ox = __fsub_rn(cx, gm.half), oy = __fsub_rn(cy, gm.half), oz = __fsub_rn(cz, gm.half);
  ItemParams P = item_of(G.recs[(size_t)bl * G.N + item]);
  const size_t dim = gm.dim, cs = dim * dim * dim, ai = (size_t)b * G.N + item;
  const int t0 = wid * per, nch = min(per, G.T - t0);
  const float inx = G.ag_in[ai * 3], iny = G.ag_in[ai * 3 + 1], inz = G.ag_in[ai * 3 + 2];
  bool strange = false;
  float cut = -1.f;
  const float weight = lane < nch ? G.type_vector[ai * G.T + t0 + lane] : 0.f;
  const unsigned weighted = __ballot_sync(0xffffffffu, weight != 0.f);
  const int count = __popc(weighted);
  if (lane < RT_CH) {
    sh.ch[lane].Tcut = -1.f;
    offset[lane] = 0;
  }
  __syncwarp();
  if (weight != 0.f) {
    const ChanParam cp = G.chanp[(size_t)bl * G.T + t0 + lane];
    const float4 p = cp.p;
    RtChannel c;
    c.kexp = p.x * NEG2_LOG2E; c.Tg = p.y; c.inv_ar = p.z;
    c.Tcut = cut = reaches_nothing(gm, cp.q.z, P, ox, oy, oz) ? -1.f : p.w;
    c.k4 = 4.f * p.x; c.kE = -gm.E * p.z; c.kD = -gm.D * p.x;
    c.w = weight;
    const float t = G.tg_in[ai * G.T + t0 + lane];
    strange = !finite3(weight * inx, weight * iny, weight * inz) || !finite3(t, 0.f, 0.f);
    const int slot = __popc(weighted & ((1u << lane) - 1u));
    sh.ch[slot] = c;
    tgrad[slot] = t;
    offset[slot] = lane * cs;
  }
  const bool odd = __any_sync(0xffffffffu, strange);
  // the footprint of the largest of the weighted channels, which the others lie in
  float most = cut;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
  P.valid = P.valid && most >= 0.f;
  if (P.valid) {
    const ChanParam big = G.chanp[(size_t)bl * G.T + t0 + __ffs(__ballot_sync(0xffffffffu, cut == most)) - 1];
    P.Tcut = big.p.w;
    bounds_1d(ox, P.x, big.q.z, gm.res, gm.dim, P.lox, P.hix);
    bounds_1d(oy, P.y, big.q.z, gm.res, gm.dim, P.loy, P.hiy);
    bounds_1d(oz, P.z, big.q.z, gm.res, gm.dim, P.loz, P.hiz);
    P.valid = P.hix > P.lox && P.hiy > P.loy && P.hiz > P.loz;
  }
  __syncwarp();
  float agx = 0.f, agy = 0.f, agz = 0.f;
  // a lane's sums: of the products of distances by axis, of w s diff and t s diff
  Pair sb1 = pair(0.f), sb2 = pair(0.f);
#pragma unroll
  for (int c = 0; c < 5; c++) sh.atom[c][lane] = 0.f;
  auto put_by = [&] {
    sh.atom[0][lane] += agx;
    sh.atom[1][lane] += agy;
    sh.atom[2][lane] += agz;
    float x0, x1, y0, y1;
    split(sb1, x0, x1);
    split(sb2, y0, y1);
    sh.atom[3][lane] += x0 + x1;
    sh.atom[4][lane] += y0 + y1;
    agx = agy = agz = 0.f;
    sb1 = sb2 = pair(0.f);
  };
  const size_t first = ((size_t)b * G.T + t0) * cs;
  auto sweep = [&](auto odd) {
    for (Columns cols(P); cols.more();) {
      const unsigned nkept = cols.compact<true>(sh.cols, P, P.Tcut, ox, oy, gm.res, gm.dim, lane);
      for (unsigned zc = P.loz & ~3u; zc < P.hiz; zc += 4 * QPASS) {
        __syncwarp();
        fill_ztabs(sh.zt, zc, P, oz, gm.res, 0.f, lane);
        __syncwarp();
        for (int c = 0; c < count; c++) reinterpret_cast<float*>(sh.ez[c])[lane] = ex2_approx(reinterpret_cast<const float*>(sh.zt.dz2)[lane] * sh.ch[c].kexp);
        const unsigned n = list_quads(sh.list, sh.cols, sh.zt, nkept, min((unsigned)QPASS, (P.hiz - zc + 3) >> 2), P.Tcut, lane);
        __syncwarp();
#pragma unroll 1
        for (unsigned e0 = 0; e0 < n; e0 += 32) {
          const unsigned e = sh.list[min(e0 + lane, n - 1u)], i = e & 255u, zq = e >> 8;
          const float dxy2 = sh.cols.dxy2[i], dx = sh.cols.dx[i], dy = sh.cols.dy[i];
          const float near = e0 + lane < n ? __fadd_rn(dxy2, sh.zt.lo[zq]) : CUDART_NAN_F;
          const size_t off = first + (size_t)sh.cols.row[i] * dim + zc + 4 * zq;
          const float* from = G.diff + off;
          float* to = G.out_grid + off;
          const float4 d2 = sh.zt.dz2[zq], dz = sh.zt.dz[zq];
          const Pair r[2] = {add2(pair(dxy2), pair(d2.x, d2.y)), add2(pair(dxy2), pair(d2.z, d2.w))}, dzp[2] = {pair(dz.x, dz.y), pair(dz.z, dz.w)};
          const float dotxy = fmaf(dx, inx, dy * iny);
          float rv[4];
          Pair id[2], id2[2], dist[2], dot[2], a1[2], a2[2], b1 = pair(0.f), b2 = pair(0.f);
#pragma unroll
          for (int j = 0; j < 2; j++) {
            split(r[j], rv[2 * j], rv[2 * j + 1]);
            id[j] = pair(rsqrt_approx(rv[2 * j]), rsqrt_approx(rv[2 * j + 1]));
            id2[j] = mul2(id[j], id[j]);
            dist[j] = mul2(r[j], id[j]);
            dot[j] = fma2(dzp[j], pair(inz), pair(dotxy));
            a1[j] = a2[j] = pair(0.f);
          }
#pragma unroll 1
          for (int q = 0; q < count; q += RS_LOADS) {
            float4 dv[RS_LOADS];
            bool live[RS_LOADS];
#pragma unroll
            for (int u = 0; u < RS_LOADS; u++) {
              live[u] = near <= sh.ch[q + u].Tcut;  // false for a NaN, and for a channel that there is not
              dv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (live[u]) dv[u] = __ldg(reinterpret_cast<const float4*>(from + offset[q + u]));
            }
#pragma unroll
            for (int u = 0; u < RS_LOADS; u++) {
              if (!__any_sync(0xffffffffu, live[u])) continue;
              const RtChannel& C = sh.ch[q + u];
              const float4 e = sh.ez[q + u][zq];
              const Pair exy = pair(ex2_approx(dxy2 * C.kexp)), ep[2] = {pair(e.x, e.y), pair(e.z, e.w)}, w = pair(C.w), t = pair(tgrad[q + u]);
              float v[4];
#pragma unroll
              for (int j = 0; j < 2; j++) {
                float g0, g1, x0, x1, y0, y1;
                const bool gauss0 = rv[2 * j] <= C.Tg, gauss1 = rv[2 * j + 1] <= C.Tg, in0 = rv[2 * j] <= C.Tcut, in1 = rv[2 * j + 1] <= C.Tcut;
                const Pair g = mul2(exy, ep[j]), kid = mul2(pair(C.kE), id[j]), sg = mul2(pair(C.k4), g);
                split(mul2(dist[j], pair(C.inv_ar)), x0, x1);
                x0 = fma_sat(-gm.ta, x0, gm.tb);
                x1 = fma_sat(-gm.ta, x1, gm.tb);
                split(g, g0, g1);
                const Pair val = pair(gauss0 ? g0 : x0 * x0, gauss1 ? g1 : x1 * x1);
                split(sg, g0, g1);
                split(add2(kid, pair(C.kD)), x0, x1);
                const Pair sl = pair(gauss0 ? g0 : fmaxf(x0, 0.f), gauss1 ? g1 : fmaxf(x1, 0.f));
                split(mul2(pair(C.k4), sg), g0, g1);
                split(mul2(kid, id2[j]), y0, y1);
                const Pair alpha = pair(gauss0 ? g0 : in0 ? y0 : 0.f, gauss1 ? g1 : in1 ? y1 : 0.f);
                Pair sd = mul2(sl, mul2(dot[j], w));
                if constexpr (odd.value) sd = only_off_atom(sd, r[j], in0, in1);
                Pair out2 = fma2(val, t, sd);
                if constexpr (odd.value) out2 = only(out2, in0, in1);
                split(out2, v[2 * j], v[2 * j + 1]);
                // a neighbour's value may be anything
                const Pair d = only(j == 0 ? pair(dv[u].x, dv[u].y) : pair(dv[u].z, dv[u].w), in0, in1);
                const Pair da = mul2(d, alpha), ds = mul2(d, sl);
                a1[j] = fma2(w, da, a1[j]);
                a2[j] = fma2(t, da, a2[j]);
                b1 = fma2(w, ds, b1);
                b2 = fma2(t, ds, b2);
              }
              if (live[u]) red_add_v4(to + offset[q + u], v[0], v[1], v[2], v[3]);
            }
          }
          float x0, x1, y0, y1, z0, z1;
          sb1 = add2(sb1, b1);
          sb2 = add2(sb2, b2);
          const Pair p[2] = {mul2(a1[0], dot[0]), mul2(a1[1], dot[1])};
          split(add2(p[0], p[1]), x0, x1);
          split(add2(a2[0], a2[1]), y0, y1);
          split(fma2(dzp[0], fma2(a2[0], dzp[0], p[0]), mul2(dzp[1], fma2(a2[1], dzp[1], p[1]))), z0, z1);
          agx = fmaf(dx, fmaf(y0 + y1, dx, x0 + x1), agx);
          agy = fmaf(dy, fmaf(y0 + y1, dy, x0 + x1), agy);
          agz += z0 + z1;
          if ((e0 & 32 * (RT_STEPS - 1)) == 32 * (RT_STEPS - 1)) put_by();  // sums of few terms each
        }
      }
      __syncwarp();
    }
  };
  if (P.valid) {
    if (odd) sweep(std::true_type());
    else sweep(std::false_type());
    put_by();
    const float s1 = sh.atom[3][lane], s2 = sh.atom[4][lane];
    agx = sh.atom[0][lane] - fmaf(s1, inx, s2);
    agy = sh.atom[1][lane] - fmaf(s1, iny, s2);
    agz = sh.atom[2][lane] - fmaf(s1, inz, s2);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    agx += __shfl_xor_sync(0xffffffffu, agx, o);
    agy += __shfl_xor_sync(0xffffffffu, agy, o);
    agz += __shfl_xor_sync(0xffffffffu, agz, o);
  }
  float* parts = warps == 1 ? G.atom_gradients + ai * 3 : G.partial + (((size_t)bl * G.N + item) * warps + wid) * 3;
  if (lane < 3) parts[lane] = lane == 0 ? agx : lane == 1 ? agy : agz;
}

__global__ void __launch_bounds__(256) k_sum_parts(BwdArgs G, int warps) {
  wait_for_stream();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= G.nb * G.N * 3) return;
  const int a = i / 3, axis = i - a * 3;
  float sum = 0.f;
  for (int w = 0; w < warps; w++) sum += G.partial[((size_t)a * warps + w) * 3 + axis];
  G.atom_gradients[(size_t)G.b0 * G.N * 3 + i] = sum;
}

// atom_gradients[a] = sum over channels in ascending order of partial[a][t] * w[a][t] for w != 0
// (src/grid_maker.cpp:508-515)
__global__ void __launch_bounds__(256) k_reduce_types(BwdArgs G) {
  wait_for_stream();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= G.nb * G.N) return;
  int bl = i / G.N, a = i - bl * G.N;
  int b = G.b0 + bl;
  const float* w = G.type_vector + ((size_t)b * G.N + a) * G.T;
  const float* p = G.partial + (size_t)i * G.T * 3;
  float gx = 0.f, gy = 0.f, gz = 0.f;
  for (int t = 0; t < G.T; t++) {
    float wt = w[t];
    if (wt != 0.f) {
      if (G.plain_reduce) wt = 1.f;  // backward_gradients: the weight is already inside the partial
      gx = __fadd_rn(gx, __fmul_rn(p[t * 3], wt));
      gy = __fadd_rn(gy, __fmul_rn(p[t * 3 + 1], wt));
      gz = __fadd_rn(gz, __fmul_rn(p[t * 3 + 2], wt));
    }
  }
  size_t ai = (size_t)b * G.N + a;
  G.atom_gradients[ai * 3] = gx;
  G.atom_gradients[ai * 3 + 1] = gy;
  G.atom_gradients[ai * 3 + 2] = gz;
}

// ---------------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------------

cudaError_t launch_emit(const EmitArgs& A, cudaStream_t st) {
  if (A.gm.rti && A.vec) {
    int n = A.nb * A.T;
    const cudaError_t e = launch_early(k_chan_params, dim3((n + 255) / 256), 256, 0, st, A);
    if (e != cudaSuccess) return e;
  }
  int n = A.nb * A.N;
  return launch_early(k_emit, dim3((n + 255) / 256), 256, 0, st, A);
}

// tensors that quads are taken from: on 16-byte boundaries
static bool quads_of(const BwdArgs& G, const void* p, const void* q = nullptr) {
  return G.quads && (uintptr_t)p % 16 == 0 && (uintptr_t)q % 16 == 0;
}
static bool loose_rows(const BwdArgs& G) { return G.gm.dim % 4 != 0; }  // else every row is on one as well

bool backward_self_serves(const EmitArgs& A, const BwdArgs& G, int mode) {
  const long most = mode == 2 ? REL_SELF_ATOMS : loose_rows(G) ? LOOSE_SELF_ATOMS : SELF_ATOMS;
  return (mode == 0 || mode == 2) && !A.vec && (long)A.nb * A.N <= most &&
         quads_of(G, G.diff, mode == 2 ? G.density : nullptr);
}

// Densities of many atoms a grid, whose sums outlast the zeros, have records of k_emit earlier on loose rows, whose tables make a
// warp's own preparation the longer one: us without and with, all slots atoms, 8 x 2500 / 8 x 4000 atoms on 14x33^3 36.0 / 52.5 and
// 34.8 / 48.8, on 22x41^3 41.6 / 58.5 and 39.7 / 54.0, on 14x25^3 of 1 A 19.2 / 28.2 and 18.0 / 24.5; 4 x 4000 15.9 and 15.5, 3 x 4000
// 12.8 and 13.2.  An atom beside the grid leaves at once without (8 x 2500 atoms, 7 of 8 of them there: 20.5 / 25.9 / 14.1 and 21.0 / 25.5 /
// 16.2), as an empty slot does: calls with counts have them on fine grids, where half of 8 x 3000 slots pay (27.1 / 32.7 / 16.1 and 26.8 /
// 31.4 / 18.0 with half of them atoms, 34.4 / 40.0 / 18.6 and 33.1 / 38.0 / 18.9 with three quarters).  Aligned rows gain nothing
// (8 x 2500 / 8 x 4000 atoms on 28x48^3 43.0 / 54.5 and 44.8 / 53.1, on 14x24^3 of 1 A 16.0 / 23.5 and 16.6 / 22.8).
bool forward_self_serves(const EmitArgs& A, const BwdArgs& G) {
  const long slots = (long)A.nb * A.N;
  if (A.vec || slots > FWD_SELF_ATOMS) return false;
  if (A.gm.binary) return true;
  const double voxels = (double)A.T * A.gm.dim * A.gm.dim * A.gm.dim;
  if (loose_rows(G) && slots >= (A.n_atoms == nullptr ? 20000 : 24000) && (A.n_atoms == nullptr || A.gm.res <= 0.6f) && voxels <= 1500.0 * A.N)
    return false;
  return !G.precise && quads_of(G, G.out_grid);
}

template <bool BINARY, int WARPS, bool LOOSE>
static cudaError_t forward_self(const EmitArgs& A, const BwdArgs& G, bool early, cudaStream_t st) {
  const dim3 grid(A.N, A.nb);
  if (early) return launch_early(k_forward_self<BINARY, WARPS, true, LOOSE>, grid, 32 * WARPS, 0, st, A, G);
  k_forward_self<BINARY, WARPS, false, LOOSE><<<grid, 32 * WARPS, 0, st>>>(A, G);
  return cudaGetLastError();
}

template <int WARPS>
static cudaError_t forward_self(const EmitArgs& A, const BwdArgs& G, bool early, cudaStream_t st) {
  if (A.gm.binary) return forward_self<true, WARPS, false>(A, G, early, st);
  return loose_rows(G) ? forward_self<false, WARPS, true>(A, G, early, st) : forward_self<false, WARPS, false>(A, G, early, st);
}

// `early`: the launch before this one is launch_zero() of this call's output
cudaError_t launch_forward_self(const EmitArgs& A, const BwdArgs& G, bool early, cudaStream_t st) {
  if (A.N == 0 || A.nb == 0) return cudaSuccess;
  return (long)A.nb * A.N <= SELF_SPLIT ? forward_self<4>(A, G, early, st) : forward_self<1>(A, G, early, st);
}

cudaError_t launch_occupancy_listed(const EmitArgs& A, const OccList& L, float* out, cudaStream_t st) {
  BwdArgs G = {};
  G.gm = A.gm;
  G.T = A.T;
  G.out_grid = out;
  // what the chip holds at a time, and a few per example at least: how many atoms there are is not known here
  const unsigned blocks = std::min((unsigned)(A.N + BIN_WARPS - 1) / BIN_WARPS, std::max(8u, (16 * 148 + (unsigned)A.nb - 1) / A.nb));
  return launch_early(k_occupancy_listed, dim3(blocks, A.nb), BIN_WARPS * 32, 0, st, A, G, L);
}

// Bound by its stores.  Two of 16 bytes a thread: with more per thread small outputs take longer (12.4 MB: 7 us of zeros and
// reductions instead of 5.5).
constexpr int ZERO_THREADS = 256, ZERO_QUADS = 2;
// BESIDE: runs beside the kernel before it, which began once all earlier work was done.
template <bool BESIDE>
__global__ void __launch_bounds__(ZERO_THREADS) k_zero(float4* p, size_t n) {
  if (!BESIDE) wait_for_stream();
  let_next_begin();  // earlier work is done: the next kernel may read what this one does not write
  const size_t i0 = (size_t)blockIdx.x * (ZERO_THREADS * ZERO_QUADS) + threadIdx.x;
#pragma unroll
  for (int k = 0; k < ZERO_QUADS; k++)
    if (i0 + ZERO_THREADS * k < n / 4) p[i0 + ZERO_THREADS * k] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (blockIdx.x == 0 && threadIdx.x < n % 4) reinterpret_cast<float*>(p)[n - 1 - threadIdx.x] = 0.f;
  if (BESIDE) wait_for_stream();  // this kernel is not done before the one before it
}

cudaError_t launch_zero(float* p, size_t n, bool beside, cudaStream_t st) {
  const size_t per = (size_t)ZERO_THREADS * ZERO_QUADS;
  const dim3 grid((unsigned)(n / 4 / per + 1));
  return launch_early(beside ? k_zero<true> : k_zero<false>, grid, ZERO_THREADS, 0, st, reinterpret_cast<float4*>(p), n);
}

template <int WARPS, class TABS>
static cudaError_t backward_self(const EmitArgs& A, const BwdArgs& G, int mode, cudaStream_t st) {
  const dim3 grid(A.N, A.nb);
  if (mode == 0) return launch_early(k_backward_quads_self<0, false, WARPS, TABS>, grid, 32 * WARPS, 0, st, A, G);
  if constexpr (WARPS > 1) {
    const long slots = (long)A.nb * A.N, atoms = A.n_atoms != nullptr ? slots * 3 / 4 : slots;
    if (atoms > SELF_ROOMY && atoms <= 148 * self_blocks(A.gm.binary != 0, !std::is_same<TABS, ZTabs>::value, true))
      return launch_early(A.gm.binary ? k_backward_quads_self<2, true, WARPS, TABS, true> : k_backward_quads_self<2, false, WARPS, TABS, true>,
                          grid, 32 * WARPS, 0, st, A, G);
  }
  if (A.gm.binary) return launch_early(k_backward_quads_self<2, true, WARPS, TABS>, grid, 32 * WARPS, 0, st, A, G);
  return launch_early(k_backward_quads_self<2, false, WARPS, TABS>, grid, 32 * WARPS, 0, st, A, G);
}

template <int WARPS>
static cudaError_t backward_self(const EmitArgs& A, const BwdArgs& G, int mode, cudaStream_t st) {
  return loose_rows(G) ? backward_self<WARPS, LooseZTabs>(A, G, mode, st) : backward_self<WARPS, ZTabs>(A, G, mode, st);
}

cudaError_t launch_backward_self(const EmitArgs& A, const BwdArgs& G, int mode, cudaStream_t st) {
  if (A.N == 0 || A.nb == 0) return cudaSuccess;
  // up to one atom's warps per scheduler and a bit: shared columns, beyond that a warp per atom
  return (long)A.nb * A.N <= SELF_SPLIT ? backward_self<4>(A, G, mode, st) : backward_self<1>(A, G, mode, st);
}

// `quads`: rows of diff (and of the density, for relevance) start on 16-byte boundaries
template <int MODE, bool BINARY>
static cudaError_t backward_items(const BwdArgs& G, bool quads, dim3 grid, cudaStream_t st) {
  if (!quads) return launch_early(k_backward_warp<MODE, BINARY>, grid, BWD2_WARPS * 32, 0, st, G);
  return launch_early(k_backward_quads<MODE, BINARY, ZTabs>, grid, BWD2_WARPS * 32, 0, st, G);
}

template <bool BINARY>
static cudaError_t backward_quads_atom(const BwdArgs& G, dim3 grid, cudaStream_t st) {
  return launch_early(G.T <= 4 ? k_backward_quads_atom<BINARY, 4> : G.T <= 7 ? k_backward_quads_atom<BINARY, 7>
                                                                             : k_backward_quads_atom<BINARY, VA_BCH>,
                      grid, VA_WARPS * 32, 0, st, G);
}

// Enough atoms a grid pay for the copy, which costs the same for any of them, and enough (atom, channel) pairs in all fill the
// chip.  What counts is atoms that reach the grid; known here are slots: those of a call without counts may lie beside the grid,
// of one with counts be empty, and the kernels without a copy are quick with both.
// Loose rows have their pairs one by one otherwise, an empty slot's too: us without / with a copy, one weighted channel, all slots
// atoms: 14 channels of 41^3 of 0.5 A, 40 x 1500 / 8 x 400 / 1 x 1500 atoms 1530 / 99 / 52 and 366 / 44 / 26.  With a copy over
// without, for all slots atoms / 7 of 8 atoms beside the grid / 1 slot of 10 an atom, 14 channels of 41^3 by slots a voxel: 0.003,
// 8 x 207 0.67 / 1.15 / 1.61, 40 x 207 0.56 / 0.82 / 1.20; 0.005, 8 x 345 0.48 / 0.86 / 1.29; 0.008, 8 x 551 0.42 / 0.63 / 0.98; of one
// example on 57^3 0.008 (21e3 pairs) 0.63 / 1.15 / 1.97, 0.012 (31e3) 0.47 / 0.91 / 1.43, 0.02 (52e3) 0.39 / 0.67 / 0.91.
// Aligned rows have rounds of 14 channels, and up to 24 are about as fast without the copy (40 x 3000 atoms, 20 channels of 48^3 of 0.5
// A, one / 3 / all weighted 1086 / 1151 / 1197 and 950 / 1183 / 1183 us, a fifth of the slots atoms 336 and 407).  More channels, one / 3 /
// all weighted: 28, 50 x 3000 atoms 1541 / 1585 / 1573 and 1120 / 1541 / 1541, half / a fifth of the slots atoms 865 / 454 and 825 / 604
// with one, 885 / 463 and 1000 / 705 with all; of 24^3 of 1 A, 8 x 2000 atoms 56 / 24 and 37 / 21 with all slots / a twentieth atoms; 32,
// 8 x 400 on 48^3 103 / 105 / 105 and 95 / 111 / 111.  Still the slower way: 28 channels, 50 x 3000 atoms 7 of 8 beside the grid 466 and 591,
// all of 0.5 to 0.9 A 442 and 467.  (Which examples are copied, decided on the GPU by their atoms' footprints, cost 5 % of full calls.)
bool type_copies_serve(const GMParams& gm, int nb, int N, int T, bool aligned, bool counted) {
  if (gm.rti || T > 32 || gm.dim == 0 || type_copy_bytes(gm, T) > TYPE_COPY_MOST) return false;
  const double side = (double)gm.dim * gm.res, dense = N / (side * side * side), pairs = (double)nb * N * T;
  const double slots = N / ((double)gm.dim * gm.dim * gm.dim);  // a voxel
  if (!aligned) {
    if (T < 8 || dense < 0.011 || pairs < 16000) return false;
    if (counted) return nb >= 4 ? slots >= 0.005 : slots >= 0.012 && pairs >= 30000;
    return slots >= 0.003 && (nb >= 4 || slots >= 0.02 || pairs >= 30000);
  }
  if (counted && T <= 28 && slots < 0.1) return false;
  return T > 24 && dense >= (T > 28 ? 0.05 : 0.12) && pairs >= 300e3 * gm.res * gm.res * gm.res;
}

template <int TO>
static cudaError_t type_gradients(const TgArgs& A, unsigned voxels, float* copy, int n, cudaStream_t st) {
  const BwdArgs& G = A.G;
  const cudaError_t e = launch_early(k_channel_last<2 * TO>, dim3((voxels + CL_VOXELS - 1) / CL_VOXELS, n), 64 * TO, 0, st,
                                     G.diff + (size_t)(G.b0 + A.first) * G.T * voxels, reinterpret_cast<float4*>(copy), voxels, G.T);
  if (e != cudaSuccess) return e;
  return launch_early(G.gm.binary ? k_type_gradients<TO, true> : k_type_gradients<TO, false>, dim3(G.N, n), 32, 0, st, A);
}

cudaError_t launch_type_gradients(const BwdArgs& G, float* copy, int per_copy, long* launches, cudaStream_t st) {
  if (G.N == 0 || G.nb == 0) return cudaSuccess;
  TgArgs A;
  A.G = G;
  A.copy = reinterpret_cast<const Eight*>(copy);
  const unsigned voxels = G.gm.dim * G.gm.dim * G.gm.dim;
  cudaError_t e = cudaSuccess;
  for (A.first = 0; e == cudaSuccess && A.first < G.nb; A.first += per_copy, *launches += 2) {
    const int n = std::min(per_copy, G.nb - A.first);
    e = G.T <= 8 ? type_gradients<1>(A, voxels, copy, n, st) : G.T <= 16 ? type_gradients<2>(A, voxels, copy, n, st)
        : G.T <= 24 ? type_gradients<3>(A, voxels, copy, n, st) : type_gradients<4>(A, voxels, copy, n, st);
  }
  return e;
}

// Warps that share an atom's places among its channels serve coarse grids at any count, finer ones where there is work enough
// for warps that last 4 to 16 times as long: us item by item / together, soft types, 28 channels, 8 x 1500 / 1 x 200 / 1 x 16 atoms on
// 24^3 of 1 A 279 / 17.8 / 11.9 and 88 / 10.5 / 9.5, on 40^3 of 0.75 A 352 / 19.7 / 12.5 and 157 / 13.7 / 12.3, on 48^3 of 0.5 A 551 /
// 24.7 / 14.6 and 360 / 23.6 / 21.1, 4 channels there 86 / 11.5 / 10.4 and 73 / 14.4 / 13.9; on 96^3 of 0.25 A 4 x 3000 / 8 x 400 / 1 x 1500
// 2473 / 691 / 328 and 2075 / 855 / 446, which have most of their spheres' quads in the tail and in full columns.  (By the rule, with
// sums of few terms: 279 / 17.7 and 86 / 11.6, 351 / 19.6 and 146 / 14.5, 552 and 345, 85 and 70, 2469 and 2045.)
// Radii are not known here.  Still slower together: one radius of 4 A among channels of 0.8 to 1.2 (28 channels, 4 x 3000 atoms on
// 96^3 1660 and 5500, 4 x 1500 on 48^3 246 and 454, 4 channels there 177 and 249, but 8 x 1500 on 24^3 279 and 181); three quarters
// of the radii zero on 96^3 783 and 930; 7 of 8 atoms beside that grid 568 and 702.
static bool channels_together(const BwdArgs& G) {
  if (G.T < 4 || G.T > RT_CH * RT_WARPS || G.gm.binary) return false;
  if (G.gm.ta == 0.f && G.gm.tb == 0.f) return false;  // a Gaussian without a tail is cut by each channel's own footprint too
  const double pairs = (double)G.N * G.first_nb * G.T;
  return G.gm.res >= 0.7f ? pairs >= 600 : G.gm.res >= 0.4f ? pairs >= 12000 : G.gm.res >= 0.2f && G.T > 8 && pairs >= 300e3;
}

static cudaError_t channels_together_launch(void (*kernel)(BwdArgs, int, int), const BwdArgs& G, long enough, long* launches, cudaStream_t st) {
  // as few warps an atom as its channels need, more while the atoms alone leave the chip idle
  const long atoms = (long)G.N * G.first_nb;
  const int most = std::min(RT_WARPS, (G.T + 3) / 4), warps = std::max((G.T + RT_CH - 1) / RT_CH, (int)std::min((long)most, enough / atoms));
  const cudaError_t e = launch_early(kernel, dim3(G.N * warps, G.nb), 32, 0, st, G, (G.T + warps - 1) / warps, warps);
  ++*launches;
  if (e != cudaSuccess || warps == 1) return e;
  ++*launches;
  return launch_early(k_sum_parts, dim3((G.nb * G.N * 3 + 255) / 256), 256, 0, st, G, warps);
}

// Loose rows: relevance, which reads two tensors and divides, gains at every size (17 x 700 atoms on 22x41^3:
// 72.5 -> 59.8 us; 50 x 3000 on 28x41^3: 525 -> 501).  Gradients with records do not (22.7 us by single voxels, 28.7
// by quads), nor do type vectors (4 x 1000 atoms, 28 channels of 41^3: 212 and 251 us).
cudaError_t launch_backward(const BwdArgs& G, int mode, long* launches, cudaStream_t st) {
  long items = (long)G.N * (mode == 1 ? G.T : 1);
  if (items == 0 || G.nb == 0) return cudaSuccess;
  dim3 grid((unsigned)((items + BWD2_WARPS - 1) / BWD2_WARPS), G.nb);
  const bool bin = G.gm.binary != 0, any = quads_of(G, G.diff, mode == 2 ? G.density : nullptr), loose = any && loose_rows(G);
  const bool quads = any && !loose;
  if (quads && mode == 1 && G.gm.rti && G.type_gradients != nullptr && channels_together(G))
    return channels_together_launch(k_backward_channels, G, 8000, launches, st);
  ++*launches;
  if (mode == 0) return backward_items<0, false>(G, quads, grid, st);
  if (mode == 2) {
    if (loose)
      return bin ? launch_early(k_backward_quads<2, true, LooseZTabs>, grid, BWD2_WARPS * 32, 0, st, G)
                 : launch_early(k_backward_quads<2, false, LooseZTabs>, grid, BWD2_WARPS * 32, 0, st, G);
    return bin ? backward_items<2, true>(G, quads, grid, st) : backward_items<2, false>(G, quads, grid, st);
  }
  if (quads && !G.gm.rti) {
    // per-atom radii: one work item per atom writes both gradients, no reduction over channels after it
    dim3 ga((unsigned)((G.N + BWD2_WARPS - 1) / BWD2_WARPS), G.nb);
    dim3 gv((unsigned)((G.N + VA_WARPS - 1) / VA_WARPS), G.nb);
    if (G.type_gradients == nullptr) return launch_early(k_backward_quads_atom_ag, ga, BWD2_WARPS * 32, 0, st, G);
    return bin ? backward_quads_atom<true>(G, gv, st) : backward_quads_atom<false>(G, gv, st);
  }
  cudaError_t e;
  if (quads && G.type_gradients == nullptr) {
    // radii by channel, no type gradients wanted: only the weighted channels of each atom
    dim3 ga((unsigned)(((long)G.N * nz_groups(G.T) + BWD2_WARPS - 1) / BWD2_WARPS), G.nb);
    e = bin ? launch_early(k_backward_quads_nz<1, true>, ga, BWD2_WARPS * 32, 0, st, G)
            : launch_early(k_backward_quads_nz<1, false>, ga, BWD2_WARPS * 32, 0, st, G);
  } else {
    e = bin ? backward_items<1, true>(G, quads, grid, st) : backward_items<1, false>(G, quads, grid, st);
  }
  if (e != cudaSuccess) return e;
  ++*launches;
  const int n = G.nb * G.N;
  return launch_early(k_reduce_types, dim3((n + 255) / 256), 256, 0, st, G);
}

cudaError_t launch_second_order(const BwdArgs& G, long* launches, cudaStream_t st) {
  const long items = (long)G.N * G.T;
  if (items == 0 || G.nb == 0) return cudaSuccess;
  const bool quads = G.quads && G.gm.dim % 4 == 0 && (uintptr_t)G.out_grid % 16 == 0 && (uintptr_t)G.diff % 16 == 0;
  if (quads && !G.gm.rti) {
    ++*launches;
    return launch_early(k_second_quads_atom, dim3((G.N + SO_WARPS - 1) / SO_WARPS, G.nb), SO_WARPS * 32, 0, st, G);
  }
  // Item by item only the weighted channels have warps, so one of many (as one-hot types have) gains less: us item by item /
  // together, 28 channels, soft / one-hot types, 8 x 1500 atoms on 24^3 of 1 A 447 / 61 and 163 / 50, 4 x 1500 on 48^3 of 0.5 A 542 / 73 and
  // 353 / 71, but 8 channels there, 8 x 1500 atoms one-hot 69 and 80, and 28 of 96^3 of 0.25 A, 4 x 3000 atoms 4241 / 356 and 4177 / 456.
  if (quads && (G.gm.res >= 0.7f || (G.gm.res >= 0.4f && G.T >= 24)) && channels_together(G))
    return channels_together_launch(k_second_channels, G, 3000, launches, st);
  *launches += quads ? 1 : 2;
  cudaError_t e;
  if (quads) {
    const long units = (long)G.N * nz_groups(G.T);
    e = launch_early(k_second_quads_nz, dim3((unsigned)((units + SO_WARPS - 1) / SO_WARPS), G.nb), SO_WARPS * 32, 0, st, G);
  } else {
    e = launch_early(k_gradgrad_scatter, dim3((unsigned)((items + SCAT_WARPS - 1) / SCAT_WARPS), G.nb), SCAT_WARPS * 32, 0, st, G);
    if (e == cudaSuccess)
      e = launch_early(k_backward_warp<3, false>, dim3((unsigned)((items + BWD2_WARPS - 1) / BWD2_WARPS), G.nb), BWD2_WARPS * 32, 0, st, G);
  }
  if (e != cudaSuccess) return e;
  ++*launches;
  const int n = G.nb * G.N;
  return launch_early(k_reduce_types, dim3((n + 255) / 256), 256, 0, st, G);
}

cudaError_t launch_forward_scatter(const BwdArgs& G, bool vec, cudaStream_t st) {
  long items = (long)G.N * (vec ? G.T : 1);
  if (items == 0 || G.nb == 0) return cudaSuccess;
  dim3 grid((unsigned)((items + SCAT_WARPS - 1) / SCAT_WARPS), G.nb);
  bool bin = G.gm.binary != 0;
  const bool quads = quads_of(G, G.out_grid), loose = loose_rows(G);
  if (vec && !G.gm.rti && quads && !loose) {
    // per-atom radii: one work item per atom, channels inside
    dim3 ga((unsigned)((G.N + QS_WARPS - 1) / QS_WARPS), G.nb);
    if (bin) return launch_early(k_forward_quads_atom<true, false>, ga, QS_WARPS * 32, 0, st, G);
    if (G.precise) return launch_early(k_forward_quads_atom<false, true>, ga, QS_WARPS * 32, 0, st, G);
    return launch_early(k_forward_quads_atom<false, false>, ga, QS_WARPS * 32, 0, st, G);
  }
  if (quads && !bin && !G.precise && !(vec && loose)) {  // soft types on loose rows: 157 us by single voxels, 209 by quads
    if (vec) {
      // radii by channel: one warp per atom runs the items of its weighted channels
      dim3 ga((unsigned)(((long)G.N * nz_groups(G.T) + SCAT_WARPS - 1) / SCAT_WARPS), G.nb);
      return launch_early(k_forward_quads_nz, ga, SCAT_WARPS * 32, 0, st, G);
    }
    dim3 gq((unsigned)((items + QS_WARPS - 1) / QS_WARPS), G.nb);
    return loose ? launch_early(k_forward_quads<false, true>, gq, QS_WARPS * 32, 0, st, G)
                 : launch_early(k_forward_quads<false, false>, gq, QS_WARPS * 32, 0, st, G);
  }
  if (vec) {
    if (bin) return launch_early(k_forward_scatter<true, false, true>, grid, SCAT_WARPS * 32, 0, st, G);
    if (G.precise) return launch_early(k_forward_scatter<false, true, true>, grid, SCAT_WARPS * 32, 0, st, G);
    return launch_early(k_forward_scatter<false, false, true>, grid, SCAT_WARPS * 32, 0, st, G);
  }
  if (bin) return launch_early(k_forward_binary, dim3((G.N + BIN_WARPS - 1) / BIN_WARPS, G.nb), BIN_WARPS * 32, 0, st, G);
  if (G.precise) return launch_early(k_forward_scatter<false, true, false>, grid, SCAT_WARPS * 32, 0, st, G);
  return launch_early(k_forward_scatter<false, false, false>, grid, SCAT_WARPS * 32, 0, st, G);
}
}  // namespace lmg
