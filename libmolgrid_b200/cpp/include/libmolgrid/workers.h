// A few threads that share the host half of a batch (decoding records, laying atoms out for the GPU).
#ifndef LMGB200_WORKERS_H_
#define LMGB200_WORKERS_H_

#include <unistd.h>

#include <atomic>
#include <condition_variable>
#include <exception>
#include <functional>
#include <mutex>
#include <thread>

namespace libmolgrid {
namespace detail {

class Workers {
 public:
  // fn(0) .. fn(n-1), in any order, on the calling thread and the pool's; returns when all are done and
  // rethrows the first exception.  One caller at a time has the pool; another one meanwhile does its
  // work alone.
  static void run(size_t n, const std::function<void(size_t)>& fn) {
    Workers* w = n > 1 ? instance() : nullptr;
    if (w == nullptr || !w->call_.try_lock()) {
      for (size_t i = 0; i < n; i++) fn(i);
      return;
    }
    std::lock_guard<std::mutex> call(w->call_, std::adopt_lock);
    w->error_ = nullptr;
    {
      std::lock_guard<std::mutex> lock(w->mutex_);
      w->fn_ = &fn;
      w->n_ = n;
      w->next_.store(0);
      w->inside_ = w->size_;
      w->round_++;
    }
    w->wake_.notify_all();
    w->work();
    {
      std::unique_lock<std::mutex> lock(w->mutex_);
      w->finished_.wait(lock, [w] { return w->inside_ == 0; });
      w->fn_ = nullptr;
    }
    if (w->error_) std::rethrow_exception(w->error_);
  }

 private:
  explicit Workers(int size) : size_(size), pid_(getpid()) {
    for (int i = 0; i < size; i++) std::thread([this] { loop(); }).detach();
  }

  // null on a machine without spare cores; made again in a forked child, which has none of the threads
  static Workers* instance() {
    static std::mutex m;
    static Workers* w = nullptr;  // lives as long as the process: its threads sleep on it
    std::lock_guard<std::mutex> lock(m);
    const int cores = (int)std::thread::hardware_concurrency();
    if (cores < 3) return nullptr;
    if (w == nullptr || w->pid_ != getpid()) w = new Workers(std::min(4, cores / 2 - 1 > 0 ? cores / 2 - 1 : 1));
    return w;
  }

  void work() {
    for (size_t i; (i = next_.fetch_add(1)) < n_;) {
      try {
        (*fn_)(i);
      } catch (...) {
        std::lock_guard<std::mutex> lock(mutex_);
        if (!error_) error_ = std::current_exception();
      }
    }
  }

  void loop() {
    unsigned long long seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> lock(mutex_);
        wake_.wait(lock, [&] { return round_ != seen; });
        seen = round_;
      }
      work();
      std::lock_guard<std::mutex> lock(mutex_);
      if (--inside_ == 0) finished_.notify_one();
    }
  }

  const int size_;
  const pid_t pid_;
  std::mutex call_, mutex_;
  std::condition_variable wake_, finished_;
  const std::function<void(size_t)>* fn_ = nullptr;
  size_t n_ = 0;
  std::atomic<size_t> next_{0};
  int inside_ = 0;
  unsigned long long round_ = 0;
  std::exception_ptr error_;
};

}  // namespace detail
}  // namespace libmolgrid
#endif
