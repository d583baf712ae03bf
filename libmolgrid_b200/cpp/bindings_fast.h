// What the rest of the compiled module uses of torch's C++ interface, without its headers.
#ifndef LMGB200_BINDINGS_FAST_H_
#define LMGB200_BINDINGS_FAST_H_
#include <Python.h>
#include <cuda_runtime.h>

#include <cstddef>

namespace lmgpy {

struct TorchView {
  void* ptr;
  size_t shape[8];
  int ndim;
  int device;       // -1: host
  char dtype;       // f, d, i (int32) or ?
  bool contiguous;
};

// false: not a (dense host or CUDA) torch tensor
bool torch_view(PyObject* o, TorchView& v);
cudaStream_t torch_stream(int device);
int add_fast_calls(PyObject* module);

}  // namespace lmgpy
#endif
