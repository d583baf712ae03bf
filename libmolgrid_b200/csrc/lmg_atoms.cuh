// Preparation of one atom: fused Transform, footprint, thresholds -> Rec.
#pragma once
#include "lmg_device.cuh"
#include "lmg_launch.h"

namespace lmg {

// Type-indexed radii: constants of channel t of example b.
__device__ __forceinline__ void make_chan_param(const GMParams& gm, float radius, ChanParam& cp) {
  float ar = __fmul_rn(radius, gm.rscale);
  float densityrad = __fmul_rn(ar, gm.finalm);
  float Tcut = sqrt_threshold(densityrad);
  float Tg = sqrt_threshold(__fmul_rn(ar, gm.G));
  float Tbin = __fmul_rn(ar, ar);
  bool ok = ar > 0.f;
  float inv_ar = ok ? 1.f / ar : 0.f;
  float inv_ar2 = ok ? 1.f / Tbin : 0.f;
  if (!ok) { Tcut = -1.f; Tg = -1.f; Tbin = -1.f; }
  cp.p = make_float4(inv_ar2, Tg, inv_ar, Tcut);
  cp.q = make_float4(Tbin, ar, densityrad, fmaxf(Tcut, gm.binary ? Tbin : -1.f));
}

// What an atom slot is made from.  Everything is requested before anything is looked at: a slot's
// loads cost one round trip to memory instead of one per question (counted? typed? where?).
struct AtomIn {
  float type, x, y, z, radius, cx, cy, cz;
  Xform X;
  bool counted, moved;
};

__device__ __forceinline__ AtomIn load_atom(const EmitArgs& A, int b, int a) {
  AtomIn I;
  const size_t i = (size_t)b * A.N + a;
  const int n = A.n_atoms != nullptr ? A.n_atoms[b] : A.N;
  I.type = A.vec ? 0.f : A.type_index[i];
  I.x = A.coords[3 * i]; I.y = A.coords[3 * i + 1]; I.z = A.coords[3 * i + 2];
  I.radius = A.gm.rti ? 0.f : A.radii[i];
  I.moved = A.transforms != nullptr || A.has_xform_host;
  if (I.moved) I.X = A.transforms != nullptr ? A.transforms[b] : A.xform_host;
  if (A.centers != nullptr) {
    I.cx = A.centers[b * 3]; I.cy = A.centers[b * 3 + 1]; I.cz = A.centers[b * 3 + 2];
  } else {
    I.cx = A.center_host[0]; I.cy = A.center_host[1]; I.cz = A.center_host[2];
  }
  I.counted = a < n;
  return I;
}

// The channel of an atom, -1 if it has none; `bad` if its type index lies beyond the channels.
__device__ __forceinline__ int atom_channel(const EmitArgs& A, const AtomIn& I, bool& bad) {
  bad = false;
  if (!I.counted) return -1;
  if (A.vec) return 0;
  // forward takes floor (src/grid_maker.cpp:171), the backward passes round (:456, :698)
  const float tc = A.round_types ? roundf(I.type) : floorf(I.type);
  if (!(tc >= 0.f)) return -1;
  if (tc >= (float)A.T) {
    bad = A.check_types != 0;
    return -1;
  }
  return (int)tc;
}

__device__ __forceinline__ void atom_move(AtomIn& I) {
  if (!I.moved) return;
  float cn[4];
  quat_conj_over_norm(I.X.q, cn);
  xform_apply(I.X, cn, I.x, I.y, I.z, true);
}

__device__ __forceinline__ Rec empty_rec() {
  Rec r;
  r.a = make_float4(0.f, 0.f, 0.f, -1.f);
  r.b = make_float4(0.f, 0.f, -1.f, 0.f);
  r.c = make_uint4(0u, 0u, 0u, 0u);
  r.d = make_float4(-1.f, -1.f, 0.f, 0.f);
  return r;
}

__device__ __forceinline__ Rec full_rec(const AtomIn& I, const ChanParam& cp, int chan, unsigned lox, unsigned hix,
                                        unsigned loy, unsigned hiy, unsigned loz, unsigned hiz) {
  if (!(cp.q.y > 0.f && hix > lox && hiy > loy && hiz > loz)) return empty_rec();
  Rec r;
  r.a = make_float4(I.x, I.y, I.z, cp.q.w);
  r.b = make_float4(1.f, cp.p.x, cp.p.y, cp.p.z);
  r.c = make_uint4(lox | (loy << 16), hix | (hiy << 16), loz | (hiz << 16), (unsigned)chan | (REC_VALID << 16));
  r.d = make_float4(cp.p.w, cp.q.x, cp.q.y, cp.q.z);
  return r;
}

// The record of atom slot `a` of example `b`; true if its type index lies beyond the channels.
__device__ __forceinline__ bool make_rec(const EmitArgs& A, int b, int a, Rec& r) {
  const GMParams& gm = A.gm;
  AtomIn I = load_atom(A, b, a);
  bool bad;
  const int chan = atom_channel(A, I, bad);
  if (chan < 0) {
    r = empty_rec();
    return bad;
  }
  atom_move(I);
  if (gm.rti) {
    // footprint for binning = the largest channel radius of this example
    I.radius = -CUDART_INF_F;
    for (int t = 0; t < A.T; t++) I.radius = fmaxf(I.radius, A.radii[(size_t)b * A.T + t]);
  }
  ChanParam cp;
  make_chan_param(gm, I.radius, cp);
  // binary occupancy extends to ar, which exceeds densityrad only when final_radius_multiple < 1;
  // the reference still clips it to the densityrad footprint, and so do the bounds below
  unsigned lox, hix, loy, hiy, loz, hiz;
  bounds_1d(__fsub_rn(I.cx, gm.half), I.x, cp.q.z, gm.res, gm.dim, lox, hix);
  bounds_1d(__fsub_rn(I.cy, gm.half), I.y, cp.q.z, gm.res, gm.dim, loy, hiy);
  bounds_1d(__fsub_rn(I.cz, gm.half), I.z, cp.q.z, gm.res, gm.dim, loz, hiz);
  r = full_rec(I, cp, chan, lox, hix, loy, hiy, loz, hiz);
  return false;
}

// The same record (index types) computed by a warp that has the atom to itself: the two thresholds and
// the three axes, the long chains of the preparation, go to different lanes.
__device__ __forceinline__ bool make_rec_warp(const EmitArgs& A, int b, int a, int lane, Rec& r, float& ox, float& oy,
                                              float& oz) {
  const GMParams& gm = A.gm;
  AtomIn I = load_atom(A, b, a);
  ox = __fsub_rn(I.cx, gm.half); oy = __fsub_rn(I.cy, gm.half); oz = __fsub_rn(I.cz, gm.half);
  bool bad;
  const int chan = atom_channel(A, I, bad);
  if (chan < 0) {
    r = empty_rec();
    return bad;
  }
  atom_move(I);
  ChanParam cp;
  const float ar = __fmul_rn(I.radius, gm.rscale), densityrad = __fmul_rn(ar, gm.finalm);
  const float T = sqrt_threshold(lane & 1 ? densityrad : __fmul_rn(ar, gm.G));
  const int axis = lane % 3;
  unsigned lo, hi;
  bounds_1d(axis == 0 ? ox : axis == 1 ? oy : oz, axis == 0 ? I.x : axis == 1 ? I.y : I.z, densityrad, gm.res, gm.dim, lo, hi);
  const bool ok = ar > 0.f;
  float Tg = __shfl_sync(0xffffffffu, T, 0), Tcut = __shfl_sync(0xffffffffu, T, 1), Tbin = __fmul_rn(ar, ar);
  const float inv_ar = ok ? 1.f / ar : 0.f, inv_ar2 = ok ? 1.f / Tbin : 0.f;
  if (!ok) { Tcut = -1.f; Tg = -1.f; Tbin = -1.f; }
  cp.p = make_float4(inv_ar2, Tg, inv_ar, Tcut);
  cp.q = make_float4(Tbin, ar, densityrad, fmaxf(Tcut, gm.binary ? Tbin : -1.f));
  const unsigned lh = lo | hi << 16;  // both fit 16 bits
  const unsigned lx = __shfl_sync(0xffffffffu, lh, 0), ly = __shfl_sync(0xffffffffu, lh, 1), lz = __shfl_sync(0xffffffffu, lh, 2);
  r = full_rec(I, cp, chan, lo16(lx), hi16(lx), lo16(ly), hi16(ly), lo16(lz), hi16(lz));
  return false;
}

// The flag of block (or warp) i of the kernel that prepares the atoms, and the header that
// lmg_check_status finds it by.  Called by one thread of each.
__device__ __forceinline__ void put_flag(const EmitArgs& A, unsigned i, unsigned count, bool bad) {
  unsigned char* f = reinterpret_cast<unsigned char*>(A.ws + A.flags) + i;
  if (bad) *f = 1;
  else if (!A.later_pass) *f = 0;
  if (i == 0 && !A.later_pass) {
    StatusHeader h;
    h.magic = STATUS_MAGIC;
    h.offset = A.flags;
    h.count = count;
    h.code = A.round_types ? 2 : 1;
    *reinterpret_cast<StatusHeader*>(A.ws) = h;
  }
}

// [lo, hi) cut down to the voxels less than `ar` from the atom along an axis, with an allowance for roundings
__device__ __forceinline__ void within(float origin, float at, float ar, float res, unsigned& lo, unsigned& hi) {
  const float inv = __fdividef(1.f, res), c = (at - origin) * inv, r = ar * inv + 0.01f + (fabsf(at) + fabsf(origin)) * inv * 2e-6f;
  const float l = ceilf(c - r), h = floorf(c + r) + 1.f;
  if (l > (float)lo) lo = l < 65535.f ? (unsigned)l : 65535u;
  if (h < (float)hi) hi = h > 0.f ? (unsigned)h : 0u;
}

}  // namespace lmg
