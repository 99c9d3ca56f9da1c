// Host side of the operator face: the interpreter's float buffers <-> native 8-bit (or wider) storage in pinned staging
// memory, converted by a small pool of threads while the previous piece is on the link or in the kernels.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <atomic>
#include <condition_variable>
#include <deque>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "devbuf.h"
#include "host_convert.h"
#include "internal.h"

namespace b200q {

// One conversion of at most a few hundred KB; `left` counts the unfinished tasks of its piece.
struct HostTask {
  const void* src;
  void* dst;
  size_t n;
  int dt;       // < 0: float -> bytes, else q -> float of this storage type
  std::atomic<int>* left;
  bool past_cache;
  void run() const {
    if (dt < 0) host_f32_to_bytes(static_cast<const float*>(src), static_cast<uint8_t*>(dst), n);
    else host_q_to_f32(src, dt, static_cast<float*>(dst), n, past_cache);
    left->fetch_sub(1, std::memory_order_release);
  }
};

// Worker threads for a process that may run on `cpus` processors, one of `local_ranks` processes like it on the machine (as the
// launcher says; null or nonsense: one), with a control group's quota (cpu.max: "<us> <period us>", "max ...", null: none).
int host_workers(int cpus, const char* local_ranks, const char* cpu_max);

// What the handles that stage host buffers share: worker threads (started by the first call that is large enough for
// them), pinned memory and stream sets that a destroyed handle gave back (pinning pages and creating streams takes
// milliseconds).  Made by the first such handle, torn down with the last one; at most CACHE_BYTES of pinned memory and
// CACHE_SETS stream sets wait for the next handle meanwhile.  Several threads may use it at the same time; a submitter
// helps with whatever task is first in the queue while it waits for its own.
class HostPool {
 public:
  struct Pinned {
    uint8_t* p = nullptr;
    size_t cap = 0;
  };
  struct Streams {
    int device = -1;                                    // the device they were made on
    cudaStream_t s[3] = {nullptr, nullptr, nullptr};    // copy in, compute, copy out
    std::vector<cudaEvent_t> ev;
  };
  static std::shared_ptr<HostPool> get();
  ~HostPool();
  void submit(const HostTask* tasks, size_t n);
  bool help();  // runs one queued task on the calling thread; false if the queue is empty
  int take(size_t bytes, Pinned* out);
  void give(Pinned b);
  int take(Streams* out);
  void give(const Streams& st);

 private:
  static constexpr size_t CACHE_BYTES = 64u << 20, CACHE_SETS = 8;
  HostPool() = default;
  void start();
  void loop();
  std::mutex m_;
  std::condition_variable cv_;
  std::deque<HostTask> q_;
  std::atomic<int> queued_{0};
  bool stop_ = false, started_ = false;
  std::vector<std::thread> threads_;
  std::mutex cache_m_;
  std::vector<Pinned> cache_;
  size_t cached_ = 0;
  std::vector<Streams> sets_;
};

// The staging memory, streams and events of one handle.
class HostStage {
 public:
  ~HostStage();
  // units (images or matrix rows) of x_per values in / y_per values of type out_dt (out_size bytes) out.  For every
  // piece of units launch(first, count, x_dev, y_dev, status_dev, stream) enqueues the kernels.  status_dev is an int
  // that is zero before the call and comes back with the results in *status.  Synchronous; everything the caller
  // queued on the default stream is finished before the first kernel.
  // (refers to the caller's function object: making it asks for no memory)
  class Launch {
   public:
    template <typename F>
    Launch(const F& f) : object_(&f), call_([](const void* o, int64_t first, int64_t n, const uint8_t* x, void* y, int* st, cudaStream_t s) -> int {
      return (*static_cast<const F*>(o))(first, n, x, y, st, s);
    }) {}
    int operator()(int64_t first, int64_t n, const uint8_t* x, void* y, int* st, cudaStream_t s) const { return call_(object_, first, n, x, y, st, s); }

   private:
    const void* object_;
    int (*call_)(const void*, int64_t, int64_t, const uint8_t*, void*, int*, cudaStream_t);
  };
  int run(const float* x, float* y, int64_t units, size_t x_per, size_t y_per, int out_dt, size_t out_size, int* status, const Launch& launch);

 private:
  int run_checked(const float* x, float* y, int64_t units, size_t x_per, size_t y_per, int out_dt, size_t out_size, int* status, const Launch& launch);
  int grow(HostPool::Pinned* b, size_t bytes);
  int run_pieces(const float* x, float* y, int64_t units, int64_t per, size_t x_per, size_t y_per, int out_dt, size_t out_size, int* status,
                 const Launch& launch);
  void convert(const void* src, void* dst, size_t n, int dt, size_t out_size, bool alone);   // of a call of one piece
  std::shared_ptr<HostPool> pool_;
  HostPool::Pinned in_, out_;
  HostPool::Streams streams_;
  DevBuf x_dev_, y_dev_;      // y_dev_ ends with the status word, so that one copy brings both
  size_t status_at_ = ~size_t(0);
};

}  // namespace b200q
