// Argument blocks passed by value to the gridding kernels, and their host-side launchers.
#pragma once
#include <cuda_runtime.h>

#include "lmg_device.cuh"

namespace lmg {

// Launch that may begin while the kernel before it on the stream drains: what it does before wait_for_stream()
// overlaps with that kernel, the rest finds all earlier work done.  Every kernel launched this way calls
// wait_for_stream() before it touches memory that others write, so that a kernel's end still means the end of all
// before it.  Zeros, then sums, of 300 atoms in 28x48^3: 6.85 -> 5.45 us; 40 atoms in 14x24^3: 3.8 -> 3.0 us; records,
// zeros and sums of 50 x 3000 atoms: 254 -> 248 us.
template <class... P, class... Q>
inline cudaError_t launch_early(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, Q... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &attr;
  c.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&c, kernel, args...);
  if (e != cudaSuccess) cudaGetLastError();  // it is in `e`: not to be found again by a later launch
  return e;
}
#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_stream() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// lets the next launch_early() kernel of the stream begin
__device__ __forceinline__ void let_next_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

// A pass covers examples [b0, b0+nb) of the caller's batch; scratch arrays are indexed by the
// example's position in the pass (bl = b - b0), caller arrays by b.
// Front of the workspace: where the pass left its flags (one byte per block or warp that prepared
// atoms: 1 = it met a type index >= T) and what such an atom means for the call.  Every call writes
// its flags and this header anew, so nothing has to be cleared before it.
constexpr unsigned long long STATUS_MAGIC = 0x6c6d675f737461ull;  // tells a header from a fresh buffer's contents
struct StatusHeader {
  unsigned long long magic;
  unsigned long long offset;  // bytes from the start of the workspace
  unsigned count;
  int code;                   // 1: out of range, 2: invalid argument
};

struct EmitArgs {
  GMParams gm;
  int b0, nb, N, T;
  int vec;          // type vectors (1) or type indices (0)
  int round_types;  // 1: round the type index (backward passes), 0: floor (forward)
  int check_types;  // report type >= T through the status word
  const int* n_atoms;
  const float* coords;
  const float* type_index;
  const float* type_vector;
  const float* radii;
  const float* centers;
  float center_host[3];
  const Xform* transforms;
  Xform xform_host;
  int has_xform_host;
  // scratch
  Rec* recs;          // [nb][N]
  ChanParam* chanp;   // [nb][T], type-indexed radii only
  char* ws;                   // workspace: StatusHeader in front
  unsigned long long flags;   // offset of the flags in it
  int later_pass;             // flags of earlier passes of the same call are kept
};

struct BwdArgs {
  GMParams gm;
  int b0, nb, N, T;
  int first_nb;  // examples of the call's first and largest pass, by which the kernels of all its passes are chosen
  const float* type_vector;
  const float* centers;
  float center_host[3];
  const Rec* recs;
  const ChanParam* chanp;
  const float* diff;
  const float* density;
  float* atom_gradients;
  float* type_gradients;
  float* relevance;
  float* partial;  // [nb][N][T][3] scratch, vector types
  // backward_gradients (mode 3): incoming gradients, and a reduction without the weight factor
  const float* ag_in;  // [B][N][3]
  const float* tg_in;  // [B][N][T]
  int plain_reduce;
  float* out_grid;     // forward by scatter: [B][T][D][D][D], zero-filled before the launch
  int precise;
  int quads;           // rows are walked in aligned quads of four voxels when the grid allows it
};

// zeroes n floats (16-byte aligned); the next kernel may begin meanwhile.  `beside`: while the
// kernel before it, whose results the zeros do not touch, is still at work
cudaError_t launch_zero(float* p, size_t n, bool beside, cudaStream_t st);
cudaError_t launch_emit(const EmitArgs& A, cudaStream_t st);
// counts its launches, as does the next
cudaError_t launch_backward(const BwdArgs& G, int mode, long* launches, cudaStream_t st);
// both terms of backward_gradients: out_grid (zero-filled before) and atom_gradients
cudaError_t launch_second_order(const BwdArgs& G, long* launches, cudaStream_t st);
// occupancy of index types that writes every voxel once, but for channels that hold many atoms (lmg_occupancy.cu);
// counts its launches
bool occupancy_serves(const EmitArgs& A);
cudaError_t launch_occupancy(const EmitArgs& A, float* out, long* launches, cudaStream_t st);
// the atoms of those channels, listed by example, into a grid that is zero there (lmg_gridmaker.cu)
struct OccList {
  unsigned* atom;       // [nb][N]
  unsigned* n;          // [nb]
  unsigned char* mark;  // [nb][T]
};
cudaError_t launch_occupancy_listed(const EmitArgs& A, const OccList& L, float* out, cudaStream_t st);
// the forward pass of index types without k_emit: every warp prepares its own atom (density on a 16-byte
// aligned tensor, or occupancy; the output is zero-filled before)
bool forward_self_serves(const EmitArgs& A, const BwdArgs& G);
cudaError_t launch_forward_self(const EmitArgs& A, const BwdArgs& G, bool early, cudaStream_t st);
// the same for the backward passes (modes 0 and 2, aligned tensors)
bool backward_self_serves(const EmitArgs& A, const BwdArgs& G, int mode);
cudaError_t launch_backward_self(const EmitArgs& A, const BwdArgs& G, int mode, cudaStream_t st);
// type and atom gradients of type vectors from copies of the grid gradient with the channels of a voxel next to each
// other: `per_copy` examples at a time into `copy`
constexpr size_t TYPE_COPY_MOST = (size_t)256 << 20;   // largest copy of one example
// of the examples that are copied together, if more than one: 50 x 3000 atoms on 28x48^3 in copies of 64 / 128 / 256 MB 1478 /
// 1354 / 1276 us (each launch ends with its slowest atoms; two copies that take turns do not help)
constexpr size_t TYPE_COPIES = (size_t)256 << 20;
inline size_t type_copy_bytes(const GMParams& gm, int T) { return ((size_t)gm.dim * gm.dim * gm.dim + 1) * ((T + 7) / 8) * 32; }
// `counted`: not all slots are atoms
bool type_copies_serve(const GMParams& gm, int nb, int N, int T, bool aligned, bool counted);
cudaError_t launch_type_gradients(const BwdArgs& G, float* copy, int per_copy, long* launches, cudaStream_t st);
cudaError_t launch_forward_scatter(const BwdArgs& G, bool vec, cudaStream_t st);

}  // namespace lmg

// Host-side helpers shared by the entry points (defined with the C ABI).
struct lmg_gridmaker;
struct lmg_atoms;
struct lmg_transform;
namespace lmg {
GMParams to_params(const lmg_gridmaker* g);
Xform to_xform(const lmg_transform* t);
// input side of a pass: settings, sizes, the caller's arrays, per-example or single transform
void fill_emit(EmitArgs& E, const lmg_gridmaker* g, const lmg_atoms* a);
cudaError_t clear_status(void* ws, cudaStream_t st);
cudaError_t read_status(const void* ws, int* code, cudaStream_t st);
int quads_setting();  // current value of the aligned-quad kernel switch
}  // namespace lmg
