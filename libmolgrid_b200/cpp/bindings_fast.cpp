// The common case of the gridding calls - every array a contiguous float32 CUDA tensor on the current
// device - from Python arguments to the C ABI in a few hundred nanoseconds: tensors are read through
// torch's C++ interface and no Python code runs.  Each function takes
//     (settings address, args, kwargs or None, workspaces or None)
// and returns None when it does not serve the call (other kinds of arrays, objects, wrong shapes): the
// caller then takes the general route, which also raises what there is to raise.  With `workspaces`
// (a dict (stream << 6 | device) -> uint8 tensor) the call runs on torch's current stream in that
// stream's tensor, which is held for the length of the call and returned; without, on the default stream in this thread's buffer, and True is returned.
#include <torch/csrc/autograd/python_variable.h>
#include <c10/cuda/CUDAStream.h>

#include <cstdint>

#include "bindings_fast.h"
#include "libmolgrid/common.h"

namespace lmgpy {

// Tensors that have no memory of their own (of vmap and other transforms, fake and nested ones) throw at
// one of these questions or answer with a null address: not ours.
bool torch_view(PyObject* o, TorchView& v) try {
  if (!THPVariable_Check(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (t.is_nested()) return false;
  const at::ScalarType st = t.scalar_type();
  v.dtype = st == at::kFloat ? 'f' : st == at::kDouble ? 'd' : st == at::kInt ? 'i' : '?';
  v.ndim = (int)t.dim();
  if (v.ndim > 8 || t.layout() != at::kStrided) return false;
  for (int i = 0; i < v.ndim; i++) v.shape[i] = (size_t)t.size(i);
  v.contiguous = t.is_contiguous();
  v.device = t.is_cuda() ? (int)t.get_device() : t.is_cpu() ? -1 : -2;
  if (v.device == -2) return false;
  v.ptr = t.numel() ? t.data_ptr() : nullptr;
  return v.ptr != nullptr || t.numel() == 0;
} catch (const std::exception&) {
  return false;
}

cudaStream_t torch_stream(int device) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

namespace {

// A tensor argument of the fast route.
struct Arr : TorchView {
  float* f() const { return static_cast<float*>(ptr); }
};

// The interpreter is others' while this lives.
struct Released {
  PyThreadState* state = PyEval_SaveThread();
  ~Released() { PyEval_RestoreThread(state); }
};

struct Call {
  lmg_gridmaker* g;
  PyObject* const* item;  // positional arguments
  Py_ssize_t n;
  PyObject *transforms = nullptr, *n_atoms = nullptr, *type_gradients = nullptr;
  bool want_tg = true;
  bool gradient_words = false;  // keywords of the backward pass alone
  PyObject* workspaces;
  int device = -1;
};

bool take(PyObject* o, int device, char dtype, int ndim, Arr& a) {
  return torch_view(o, a) && a.dtype == dtype && a.device == device && a.contiguous && (ndim < 0 || a.ndim == ndim);
}

bool number(PyObject* o, float* f) {
  if (PyFloat_CheckExact(o)) *f = (float)PyFloat_AS_DOUBLE(o);
  else if (PyLong_CheckExact(o)) *f = (float)PyLong_AsDouble(o);
  else return false;
  if (PyErr_Occurred() == nullptr) return true;
  PyErr_Clear();  // a whole number beyond a double: the general route says so
  return false;
}

// settings, arguments and keywords; false: not for the fast route
bool open(PyObject* const* a, Py_ssize_t nargs, Call& c) {
  if (nargs != 4 || !PyLong_Check(a[0]) || !PyTuple_CheckExact(a[1])) return false;
  c.g = reinterpret_cast<lmg_gridmaker*>(PyLong_AsVoidPtr(a[0]));
  c.item = &PyTuple_GET_ITEM(a[1], 0);
  c.n = PyTuple_GET_SIZE(a[1]);
  c.workspaces = a[3];
  if (a[2] != Py_None) {
    PyObject *k, *v;
    Py_ssize_t at = 0;
    while (PyDict_Next(a[2], &at, &k, &v)) {
      if (PyUnicode_CompareWithASCIIString(k, "transforms") == 0) c.transforms = v == Py_None ? nullptr : v;
      else if (PyUnicode_CompareWithASCIIString(k, "n_atoms") == 0) c.n_atoms = v == Py_None ? nullptr : v;
      else if (PyUnicode_CompareWithASCIIString(k, "type_gradients") == 0) {
        if (c.n > 6) return false;  // given twice
        c.type_gradients = v == Py_None ? nullptr : v;
        c.gradient_words = true;
      } else if (PyUnicode_CompareWithASCIIString(k, "want_type_gradients") == 0) {
        const int yes = PyObject_IsTrue(v);
        if (yes < 0) PyErr_Clear();
        if (yes < 0) return false;
        c.want_tg = yes != 0;
        c.gradient_words = true;
      } else {
        return false;
      }
    }
  }
  return cudaGetDevice(&c.device) == cudaSuccess;
}

// center, coords, types, radii (the first four arguments) and the keywords
bool atoms(Call& c, lmg_atoms& A, bool& vec, size_t& nr) {
  Arr co, ty, ra, x;
  if (!take(c.item[1], c.device, 'f', -1, co) || (co.ndim != 2 && co.ndim != 3)) return false;
  const int batched = co.ndim == 3;
  if (!take(c.item[2], c.device, 'f', -1, ty) || !take(c.item[3], c.device, 'f', 1 + batched, ra)) return false;
  vec = ty.ndim == 2 + batched;
  if (!vec && ty.ndim != 1 + batched) return false;
  const size_t B = batched ? co.shape[0] : 1, N = co.shape[batched];
  if (co.shape[1 + batched] != 3 || ty.shape[batched] != N) return false;
  if (batched && (ty.shape[0] != B || ra.shape[0] != B)) return false;
  if (B == 0 || N == 0 || B > 0x7fffffff || N > 0x7fffffff) return false;
  A = {};
  A.batch = (int)B;
  A.max_atoms = (int)N;
  A.coords = co.f();
  A.radii = ra.f();
  nr = ra.shape[batched];
  if (vec) {
    A.type_vector = ty.f();
    A.ntypes = (int)ty.shape[1 + batched];
  } else {
    A.type_index = ty.f();
  }
  PyObject* ce = c.item[0];
  if (batched && torch_view(ce, x)) {
    if (!take(ce, c.device, 'f', 2, x) || x.shape[0] != B || x.shape[1] != 3) return false;
    A.centers = x.f();
  } else {
    // one centre for a batch: a call of the Python layer, on its stream
    if (batched && c.workspaces == Py_None) return false;
    if (!(PyTuple_CheckExact(ce) || PyList_CheckExact(ce)) || PySequence_Fast_GET_SIZE(ce) != 3) return false;
    for (int i = 0; i < 3; i++)
      if (!number(PySequence_Fast_GET_ITEM(ce, i), &A.center_host[i])) return false;
  }
  if (c.transforms != nullptr) {
    if (!batched || !take(c.transforms, c.device, 'f', 2, x) || x.shape[0] != B || x.shape[1] != 10) return false;
    A.transforms = reinterpret_cast<const lmg_transform*>(x.ptr);
  }
  if (c.n_atoms != nullptr) {
    if (!batched || !take(c.n_atoms, c.device, 'i', 1, x) || x.shape[0] != B) return false;
    A.n_atoms = static_cast<const int*>(x.ptr);
  }
  return true;
}

// a grid argument of this call's batch: [B][T][D][D][D] or [T][D][D][D]
bool grid(const Call& c, PyObject* o, const lmg_atoms& A, bool batched, Arr& x, size_t& T) {
  if (!take(o, c.device, 'f', 4 + batched, x)) return false;
  if (batched && x.shape[0] != (size_t)A.batch) return false;
  for (int i = 1; i <= 3; i++)
    if (x.shape[i + batched] != c.g->dim) return false;
  T = x.shape[batched];
  return T > 0 && T <= 65535;
}

bool per_atom(const Call& c, PyObject* o, const lmg_atoms& A, bool batched, size_t last, Arr& x) {
  if (!take(o, c.device, 'f', (last ? 2 : 1) + batched, x)) return false;
  return (!batched || x.shape[0] == (size_t)A.batch) && x.shape[batched] == (size_t)A.max_atoms &&
         (last == 0 || x.shape[1 + batched] == last);
}

// where the call runs, `ret` a new reference; false leaves it to the general route (no workspace of that size yet, or
// a call that is being captured).  The compiled module's own buffers may hold no more than `least`.
bool place(const Call& c, size_t bytes, size_t least, void** ws, size_t* ws_bytes, cudaStream_t* st, PyObject** ret) {
  if (c.workspaces == Py_None) {
    try {
      *ws = libmolgrid::detail::workspace_or_less(bytes, least);
    } catch (std::exception&) {
      return false;
    }
    *ws_bytes = bytes;
    *st = nullptr;
    *ret = Py_NewRef(Py_True);
    return true;
  }
  if (c.device >= 64) return false;
  *st = torch_stream(c.device);
  cudaStreamCaptureStatus capture;
  if (cudaStreamIsCapturing(*st, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) return false;
  PyObject* key = PyLong_FromUnsignedLongLong((unsigned long long)reinterpret_cast<uintptr_t>(*st) << 6 | (unsigned)c.device);
  PyObject* w = key ? PyDict_GetItem(c.workspaces, key) : nullptr;
  Py_XDECREF(key);
  if (w == nullptr || !THPVariable_Check(w)) return false;
  const at::Tensor& t = THPVariable_Unpack(w);
  if ((size_t)t.numel() < bytes) return false;
  *ws = t.data_ptr();
  *ws_bytes = (size_t)t.numel();
  *ret = Py_NewRef(w);
  return true;
}

// takes over the reference
PyObject* finish(int rc, PyObject* ret) {
  if (rc == LMG_OK) return ret;
  Py_DECREF(ret);
  PyErr_SetString(rc == LMG_ERR_OUT_OF_RANGE ? PyExc_IndexError : rc == LMG_ERR_INVALID_ARGUMENT ? PyExc_ValueError : PyExc_RuntimeError,
                  lmg_last_error());
  return nullptr;
}

bool radii_fit(const Call& c, bool vec, size_t nr, size_t N, size_t T) {
  return nr == (vec && c.g->radii_type_indexed ? T : N);
}

PyObject* fast_forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  Call c;
  lmg_atoms A;
  bool vec;
  size_t nr, T, wb;
  Arr out;
  void* ws;
  cudaStream_t st;
  PyObject* ret;
  if (!open(a, nargs, c) || c.n != 5 || c.gradient_words || !atoms(c, A, vec, nr)) Py_RETURN_NONE;
  const bool batched = THPVariable_Unpack(c.item[1]).dim() == 3;
  if (!grid(c, c.item[4], A, batched, out, T) || (vec && (size_t)A.ntypes != T)) Py_RETURN_NONE;
  A.ntypes = (int)T;
  if (!radii_fit(c, vec, nr, A.max_atoms, T)) Py_RETURN_NONE;
  const size_t bytes = lmg_workspace_bytes(c.g, LMG_OP_FORWARD, A.batch, A.max_atoms, A.ntypes, vec);
  if (!place(c, bytes, bytes, &ws, &wb, &st, &ret)) Py_RETURN_NONE;
  return finish([&] {
    Released r;
    return lmg_forward(c.g, &A, out.f(), ws, wb, st);
  }(), ret);
}

PyObject* fast_backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  Call c;
  lmg_atoms A;
  bool vec;
  size_t nr, T, wb;
  Arr diff, ag, tg;
  tg.ptr = nullptr;
  void* ws;
  cudaStream_t st;
  PyObject* ret;
  if (!open(a, nargs, c) || c.n < 6 || c.n > 7 || !atoms(c, A, vec, nr)) Py_RETURN_NONE;
  PyObject* tgo = c.n == 7 && c.item[6] != Py_None ? c.item[6] : c.type_gradients;
  const bool batched = THPVariable_Unpack(c.item[1]).dim() == 3;
  if (!grid(c, c.item[4], A, batched, diff, T) || (vec && (size_t)A.ntypes != T)) Py_RETURN_NONE;
  A.ntypes = (int)T;
  if (!per_atom(c, c.item[5], A, batched, 3, ag) || !radii_fit(c, vec, nr, A.max_atoms, T)) Py_RETURN_NONE;
  if (vec && c.want_tg) {
    if (tgo == nullptr || !per_atom(c, tgo, A, batched, T, tg)) Py_RETURN_NONE;
  } else if (!vec && (tgo != nullptr || c.g->radii_type_indexed)) {
    Py_RETURN_NONE;
  }
  const size_t least = lmg_workspace_bytes(c.g, LMG_OP_BACKWARD, A.batch, A.max_atoms, A.ntypes, vec);
  const int op = A.n_atoms != nullptr ? LMG_OP_BACKWARD_TYPES_COUNTED : LMG_OP_BACKWARD_TYPES;
  const size_t bytes = tg.ptr != nullptr ? lmg_workspace_bytes(c.g, op, A.batch, A.max_atoms, A.ntypes, vec) : least;
  if (!place(c, bytes, least, &ws, &wb, &st, &ret)) Py_RETURN_NONE;
  return finish([&] {
    Released r;
    return lmg_backward(c.g, &A, diff.f(), ag.f(), tg.f(), ws, wb, st);
  }(), ret);
}

PyObject* fast_relevance(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  Call c;
  lmg_atoms A;
  bool vec;
  size_t nr, T, T2, wb;
  Arr de, diff, rel;
  void* ws;
  cudaStream_t st;
  PyObject* ret;
  if (!open(a, nargs, c) || c.n != 7 || c.gradient_words || !atoms(c, A, vec, nr) || vec || c.g->radii_type_indexed) Py_RETURN_NONE;
  const bool batched = THPVariable_Unpack(c.item[1]).dim() == 3;
  if (!grid(c, c.item[4], A, batched, de, T) || !grid(c, c.item[5], A, batched, diff, T2) || T != T2) Py_RETURN_NONE;
  A.ntypes = (int)T;
  if (!per_atom(c, c.item[6], A, batched, 0, rel) || nr != (size_t)A.max_atoms) Py_RETURN_NONE;
  const size_t bytes = lmg_workspace_bytes(c.g, LMG_OP_BACKWARD_RELEVANCE, A.batch, A.max_atoms, A.ntypes, 0);
  if (!place(c, bytes, bytes, &ws, &wb, &st, &ret)) Py_RETURN_NONE;
  return finish([&] {
    Released r;
    return lmg_backward_relevance(c.g, &A, de.f(), diff.f(), rel.f(), ws, wb, st);
  }(), ret);
}

PyObject* fast_gradients(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  Call c;
  lmg_atoms A;
  bool vec;
  size_t nr, T, T2, wb;
  Arr diff, ag, tg, dd, add, tdd;
  void* ws;
  cudaStream_t st;
  PyObject* ret;
  if (!open(a, nargs, c) || c.n != 10 || c.gradient_words || !atoms(c, A, vec, nr) || !vec) Py_RETURN_NONE;
  const bool batched = THPVariable_Unpack(c.item[1]).dim() == 3;
  if (batched && c.workspaces == Py_None) Py_RETURN_NONE;
  if (!grid(c, c.item[4], A, batched, diff, T) || !grid(c, c.item[7], A, batched, dd, T2) || T != T2 || (size_t)A.ntypes != T)
    Py_RETURN_NONE;
  if (!per_atom(c, c.item[5], A, batched, 3, ag) || !per_atom(c, c.item[6], A, batched, T, tg) ||
      !per_atom(c, c.item[8], A, batched, 3, add) || !per_atom(c, c.item[9], A, batched, T, tdd) ||
      !radii_fit(c, vec, nr, A.max_atoms, T))
    Py_RETURN_NONE;
  const size_t bytes = lmg_workspace_bytes(c.g, LMG_OP_BACKWARD_GRADIENTS, A.batch, A.max_atoms, A.ntypes, 1);
  if (!place(c, bytes, bytes, &ws, &wb, &st, &ret)) Py_RETURN_NONE;
  return finish([&] {
    Released r;
    return lmg_backward_gradients(c.g, &A, diff.f(), ag.f(), tg.f(), dd.f(), add.f(), tdd.f(), ws, wb, st);
  }(), ret);
}

// A float attribute (any Python or numpy number) of an object; false with an exception set.
bool number_of(PyObject* o, PyObject* name, float* f) {
  PyObject* v = PyObject_GetAttr(o, name);
  if (v == nullptr) return false;
  *f = (float)PyFloat_AsDouble(v);
  Py_DECREF(v);
  return !(*f == -1.f && PyErr_Occurred());
}

// (list of Transform objects of the Python layer, address of as many lmg_transform, address of as many
// rotation centres): their numbers in one go instead of a ctypes object each
PyObject* pack_transforms(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  static PyObject *Q = PyUnicode_InternFromString("Q"), *center = PyUnicode_InternFromString("center"),
                  *translate = PyUnicode_InternFromString("translate");
  static PyObject* part[4] = {PyUnicode_InternFromString("a"), PyUnicode_InternFromString("b"), PyUnicode_InternFromString("c"),
                              PyUnicode_InternFromString("d")};
  static PyObject* xyz[3] = {PyUnicode_InternFromString("x"), PyUnicode_InternFromString("y"), PyUnicode_InternFromString("z")};
  if (nargs != 3 || !PyList_Check(a[0])) {
    PyErr_SetString(PyExc_TypeError, "a list and two addresses are needed");
    return nullptr;
  }
  lmg_transform* t = static_cast<lmg_transform*>(PyLong_AsVoidPtr(a[1]));
  float* ce = static_cast<float*>(PyLong_AsVoidPtr(a[2]));
  if (PyErr_Occurred()) return nullptr;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(a[0]); i++) {
    PyObject* o = PyList_GET_ITEM(a[0], i);
    PyObject *q = PyObject_GetAttr(o, Q), *c = q ? PyObject_GetAttr(o, center) : nullptr, *r = c ? PyObject_GetAttr(o, translate) : nullptr;
    bool ok = r != nullptr;
    for (int k = 0; ok && k < 4; k++) ok = number_of(q, part[k], &t[i].q[k]);
    for (int k = 0; ok && k < 3; k++) ok = number_of(c, xyz[k], &t[i].center[k]) && number_of(r, xyz[k], &t[i].translate[k]);
    for (int k = 0; ok && k < 3; k++) ce[3 * i + k] = t[i].center[k];
    Py_XDECREF(q);
    Py_XDECREF(c);
    Py_XDECREF(r);
    if (!ok) return nullptr;
  }
  Py_RETURN_NONE;
}

// No C++ exception crosses into the interpreter, whose frames know none.
typedef PyObject* (*Fast)(PyObject*, PyObject* const*, Py_ssize_t);
template <Fast F>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  try {
    return F(self, a, n);
  } catch (const std::exception& e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}
template <Fast F>
PyCFunction entry() { return (PyCFunction)(void (*)(void))guarded<F>; }

PyMethodDef methods[] = {
    {"_pack_transforms", entry<pack_transforms>(), METH_FASTCALL, nullptr},
    {"_fast_forward", entry<fast_forward>(), METH_FASTCALL, nullptr},
    {"_fast_backward", entry<fast_backward>(), METH_FASTCALL, nullptr},
    {"_fast_relevance", entry<fast_relevance>(), METH_FASTCALL, nullptr},
    {"_fast_gradients", entry<fast_gradients>(), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

}  // namespace

int add_fast_calls(PyObject* module) { return PyModule_AddFunctions(module, methods); }

}  // namespace lmgpy
