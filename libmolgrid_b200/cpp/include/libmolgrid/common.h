// Shared helpers of the C++ host layer: error translation between the C ABI's status codes and the
// exception types libmolgrid's users catch, and small RAII wrappers for device staging.
#ifndef LMGB200_COMMON_H_
#define LMGB200_COMMON_H_

#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <cstddef>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "lmg_b200.h"

#ifdef __CUDACC__
#define CUDA_CALLABLE_MEMBER __host__ __device__
#else
#define CUDA_CALLABLE_MEMBER
#endif

// Same contract as the reference macro of this name (include/libmolgrid/common.h:41-47):
// a failing CUDA runtime call becomes std::runtime_error.
#define LMG_CUDA_CHECK(call)                                                               \
  do {                                                                                     \
    cudaError_t lmg_err_ = (call);                                                         \
    if (lmg_err_ != cudaSuccess)                                                           \
      throw std::runtime_error(std::string("CUDA Error: ") + cudaGetErrorString(lmg_err_)); \
  } while (0)

namespace libmolgrid {

inline std::string itoa(long long v) { return std::to_string(v); }

namespace detail {

// status code of the C ABI -> the exception the reference throws in the same situation
inline void check(int rc) {
  if (rc == LMG_OK) return;
  std::string msg = lmg_last_error();
  if (rc == LMG_ERR_OUT_OF_RANGE) throw std::out_of_range(msg);
  if (rc == LMG_ERR_INVALID_ARGUMENT) throw std::invalid_argument(msg);
  throw std::runtime_error(msg);
}

// Scratch memory handed to the C ABI: one buffer per host thread, device and stream (calls on one
// stream follow one another), grown on demand.  The eight used last are kept.
struct WorkspaceSlot {
  void* p = nullptr;
  size_t cap = 0;
  int device = -1;
  cudaStream_t stream = nullptr;
};
struct Workspaces {
  std::vector<WorkspaceSlot> slots;  // the one used last in front
  // A thread that ends gives its buffers back, also while another one captures a graph, which forbids such calls
  // unless they are declared to have nothing to do with it.
  ~Workspaces() {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (slots.empty() || cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return;
    for (WorkspaceSlot& s : slots)
      if (s.p) cudaFree(s.p);
    cudaThreadExchangeStreamCaptureMode(&mode);
  }
};
inline std::vector<WorkspaceSlot>& workspaces() {
  thread_local Workspaces w;
  return w.slots;
}
inline const WorkspaceSlot* last_workspace() { return workspaces().empty() ? nullptr : &workspaces().front(); }

// The buffer of the calling thread, its device and the stream, as large as it is.
inline WorkspaceSlot& workspace_slot(cudaStream_t stream) {
  std::vector<WorkspaceSlot>& w = workspaces();
  int dev = 0;
  LMG_CUDA_CHECK(cudaGetDevice(&dev));
  size_t i = 0;
  while (i < w.size() && !(w[i].device == dev && w[i].stream == stream)) i++;
  if (i == w.size()) {
    if (i >= 8) {
      cudaFree(w.back().p);  // waits for the work that uses it
      w.pop_back();
      i--;
    }
    WorkspaceSlot n;
    n.device = dev;
    n.stream = stream;
    w.push_back(n);
  }
  if (i != 0) std::swap(w[0], w[i]);
  return w[0];
}

inline void* workspace(size_t bytes, cudaStream_t stream = nullptr) {
  WorkspaceSlot& s = workspace_slot(stream);
  if (bytes > s.cap) {
    if (s.p) cudaFree(s.p);
    s.p = nullptr;
    s.cap = 0;
    LMG_CUDA_CHECK(cudaMalloc(&s.p, bytes));
    s.cap = bytes;
  }
  return s.p;
}

// The same with `least` bytes at least where there is no room for `bytes`, which is then set to what there is.
inline void* workspace_or_less(size_t& bytes, size_t least, cudaStream_t stream = nullptr) {
  WorkspaceSlot& s = workspace_slot(stream);
  if (bytes <= s.cap || least >= bytes) return workspace(bytes, stream);
  void* p = nullptr;
  if (cudaMalloc(&p, bytes) == cudaSuccess) {
    if (s.p) cudaFree(s.p);  // waits for the work that uses it
    s.p = p;
    s.cap = bytes;
  } else {
    cudaGetLastError();  // not to be found by a later check
    bytes = std::max(least, s.cap);
  }
  return workspace(bytes, stream);
}

// Device copy of a host array for the duration of one call (host-grid overloads compute on the
// GPU as well: there is no CPU implementation of the path in this library).
template <typename T>
class Staged {
 public:
  Staged(T* host, size_t n, bool copy_in, bool copy_out) : host_(host), n_(n), out_(copy_out) {
    if (n_ == 0) return;
    LMG_CUDA_CHECK(cudaMalloc(&dev_, n_ * sizeof(T)));
    if (copy_in) LMG_CUDA_CHECK(cudaMemcpy(dev_, host_, n_ * sizeof(T), cudaMemcpyHostToDevice));
  }
  Staged(const Staged&) = delete;
  Staged& operator=(const Staged&) = delete;
  ~Staged() {
    if (dev_) cudaFree(dev_);
  }
  T* get() const { return dev_; }
  void finish() {
    if (out_ && n_) LMG_CUDA_CHECK(cudaMemcpy(host_, dev_, n_ * sizeof(T), cudaMemcpyDeviceToHost));
  }

 private:
  T* host_;
  T* dev_ = nullptr;
  size_t n_;
  bool out_;
};

// Pinned host memory (and, for whole batches, device memory of the same size) through which host
// arrays travel to the GPU without stopping the calling thread.  A slot belongs to one call at a
// time; it is written again only after the copy out of it, and its device side only after the
// kernels that read it, as its two events tell.  At most `slots` of them per device are kept, and a
// slot above 64 MB gives its memory back as soon as its call is over.
class Staging {
 public:
  struct Slot {
    int device = -1;
    char* host = nullptr;
    char* dev = nullptr;
    size_t cap = 0;
    bool busy = false, used = false;
    unsigned long long turn = 0;
    cudaEvent_t copied = nullptr, done = nullptr;
  };

  Staging(int slots, bool device_side) : max_(slots), device_side_(device_side) {}

  // a slot of at least `bytes` on the current device, exclusively the caller's until release()
  Slot* acquire(size_t bytes) {
    int dev = 0;
    LMG_CUDA_CHECK(cudaGetDevice(&dev));
    Slot* s = nullptr;
    {
      std::unique_lock<std::mutex> lock(mutex_);
      for (;;) {
        int mine = 0;
        for (Slot* k : slots_) {
          if (k->device != dev) continue;
          mine++;
          // in turn, so that the slot taken is the one whose work was issued first
          if (!k->busy && (s == nullptr || k->turn < s->turn)) s = k;
        }
        if (mine < max_) {
          s = new Slot();
          s->device = dev;
          slots_.push_back(s);
        }
        if (s != nullptr) break;
        freed_.wait(lock);
      }
      s->busy = true;
      s->turn = ++turns_;
    }
    try {
      if (s->copied == nullptr) {
        LMG_CUDA_CHECK(cudaEventCreateWithFlags(&s->copied, cudaEventDisableTiming));
        LMG_CUDA_CHECK(cudaEventCreateWithFlags(&s->done, cudaEventDisableTiming));
      }
      if (s->used) LMG_CUDA_CHECK(cudaEventSynchronize(s->copied));
      if (s->cap < bytes) {
        drop(s);
        size_t cap = bytes + bytes / 2;
        LMG_CUDA_CHECK(cudaMallocHost(&s->host, cap));
        if (device_side_) LMG_CUDA_CHECK(cudaMalloc(&s->dev, cap));
        s->cap = cap;
      }
    } catch (...) {
      give(s);
      throw;
    }
    return s;
  }

  // the caller has recorded the slot's events behind its work
  void release(Slot* s) {
    s->used = true;
    if (s->cap > ((size_t)64 << 20)) drop(s);
    give(s);
  }
  // the caller failed before it issued anything
  void abandon(Slot* s) { give(s); }

  // the stream on which batches travel beside the kernels of the batch before them
  cudaStream_t copy_stream() {
    int dev = 0;
    LMG_CUDA_CHECK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mutex_);
    if ((int)streams_.size() <= dev) streams_.resize(dev + 1, nullptr);
    if (streams_[dev] == nullptr) LMG_CUDA_CHECK(cudaStreamCreateWithFlags(&streams_[dev], cudaStreamNonBlocking));
    return streams_[dev];
  }

 private:
  void drop(Slot* s) {
    if (s->used) {
      cudaEventSynchronize(s->copied);
      if (device_side_) cudaEventSynchronize(s->done);
    }
    if (s->host) cudaFreeHost(s->host);
    if (s->dev) cudaFree(s->dev);
    s->host = s->dev = nullptr;
    s->cap = 0;
    s->used = false;
  }
  void give(Slot* s) {
    {
      std::lock_guard<std::mutex> lock(mutex_);
      s->busy = false;
    }
    freed_.notify_one();
  }

  int max_;
  bool device_side_;
  std::mutex mutex_;
  std::condition_variable freed_;
  std::vector<Slot*> slots_;
  std::vector<cudaStream_t> streams_;
  unsigned long long turns_ = 0;
};

inline Staging& batch_staging() {
  static Staging* s = new Staging(3, true);  // lives as long as the process, like the CUDA context
  return *s;
}
inline Staging& small_staging() {
  static Staging* s = new Staging(8, false);
  return *s;
}

}  // namespace detail
}  // namespace libmolgrid

#endif
