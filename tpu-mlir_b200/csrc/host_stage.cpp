// Conversions and the piece pipeline of the operator face (host_stage.h).
//
// What bounds an operator-face call is moving the interpreter's floats: 4 bytes per value in host memory, and the link.
// Copying the floats themselves costs one thread's page-by-page staging copy (about 10 GB/s from pageable memory) and
// four bytes per value on the link.  Here the values are narrowed to their storage type by all cores on the way into
// pinned memory (one read of the floats, the only pass over them), a quarter of the bytes crosses the link, and the
// results are widened the same way; pieces keep the cores, both link directions and the kernels busy at once.
// tpu.Conv2D int8 n8 c256 56x56 -> 256, 3x3 (25.7 MB of pageable floats each way, 16 cores): 3.86 ms with the floats
// copied, 0.47 ms this way.
#include "host_stage.h"

#include <sched.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <exception>

namespace b200q {
namespace {

constexpr size_t TASK_VALUES = 64 * 1024;        // 256 KB of floats: small against a core's share, large against a wake-up
constexpr size_t PIECE_VALUES = 512 * 1024;      // values per piece (the larger of its input and output)
constexpr int MAX_SLOTS = 4;                     // pieces in flight: bounds the pinned memory of a handle
constexpr size_t INLINE_VALUES = 96 * 1024;      // up to here the calling thread converts alone: a wake-up costs as much
// Results of a call from this size on are written past the caches.  Smaller ones stay in them for the host operator that reads
// them next (one core, 64 K values: 4.6 us written and 4.4 us read, past the caches 17 and 15; 1 M: 146 and 108, 190 and 246); from
// 4 M values, 16 MB, on the write itself is as fast past the caches (587 and 555 us) and leaves the call's input there.
constexpr size_t PAST_CACHE_VALUES = 4u << 20;

}  // namespace

int host_workers(int cpus, const char* local_ranks, const char* cpu_max) {
  long long quota = 0, period = 0;
  if (cpu_max && sscanf(cpu_max, "%lld %lld", &quota, &period) == 2 && quota > 0 && period > 0) {
    const long long granted = (quota + period - 1) / period;
    if (granted < cpus) cpus = (int)granted;
  }
  const int ranks = local_ranks ? atoi(local_ranks) : 1;
  if (ranks > 1) cpus /= ranks;
  const int workers = cpus - 1;                   // the calling thread is one more
  return workers < 0 ? 0 : (workers < 15 ? workers : 15);   // memory bandwidth is used up well before 16 cores
}

// ---------------------------------------------------------------------------------------------- HostPool
std::shared_ptr<HostPool> HostPool::get() {
  static std::mutex m;
  static std::weak_ptr<HostPool> current;
  std::lock_guard<std::mutex> lock(m);
  std::shared_ptr<HostPool> p = current.lock();
  if (!p) {
    p.reset(new HostPool());
    current = p;
  }
  return p;
}

void HostPool::start() {
  started_ = true;
  cpu_set_t set;
  CPU_ZERO(&set);
  int cpus = 1;
  if (sched_getaffinity(0, sizeof(set), &set) == 0) cpus = CPU_COUNT(&set);
  char cpu_max[64] = "max";
  if (FILE* f = fopen("/sys/fs/cgroup/cpu.max", "r")) {
    if (!fgets(cpu_max, sizeof(cpu_max), f)) cpu_max[0] = 0;
    fclose(f);
  }
  const int workers = host_workers(cpus, getenv("LOCAL_WORLD_SIZE"), cpu_max);
  try {
    for (int i = 0; i < workers; ++i) threads_.emplace_back([this] { loop(); });
  } catch (const std::exception&) {   // no more threads to be had: a submitter helps with its own tasks anyway
  }
}

HostPool::~HostPool() {
  {
    std::lock_guard<std::mutex> lock(m_);
    stop_ = true;
  }
  cv_.notify_all();
  for (auto& t : threads_) t.join();
  for (auto& b : cache_) cudaFreeHost(b.p);
  for (auto& st : sets_) {
    for (auto& e : st.ev) cudaEventDestroy(e);
    for (auto& x : st.s)
      if (x) cudaStreamDestroy(x);
  }
}

void HostPool::submit(const HostTask* tasks, size_t n) {
  bool queued = false;
  {
    std::lock_guard<std::mutex> lock(m_);
    if (!started_) start();
    try {
      q_.insert(q_.end(), tasks, tasks + n);
      queued = true;
    } catch (const std::exception&) {   // (inserting at the end has no effect then)
    }
    queued_.store((int)q_.size(), std::memory_order_relaxed);
  }
  if (!queued) {
    for (size_t i = 0; i < n; ++i) tasks[i].run();
    return;
  }
  if (n == 1) cv_.notify_one();
  else cv_.notify_all();
}

bool HostPool::help() {
  if (queued_.load(std::memory_order_relaxed) == 0) return false;
  HostTask t;
  {
    std::lock_guard<std::mutex> lock(m_);
    if (q_.empty()) return false;
    t = q_.front();
    q_.pop_front();
    queued_.store((int)q_.size(), std::memory_order_relaxed);
  }
  t.run();
  return true;
}

void HostPool::loop() {
  while (true) {
    // a short look at the queue before sleeping: the next piece's tasks usually follow within microseconds
    bool ran = false;
    for (int spin = 0; spin < 2000 && !ran; ++spin) {
      ran = help();
      if (!ran) host_pause();
    }
    if (ran) continue;
    std::unique_lock<std::mutex> lock(m_);
    cv_.wait(lock, [this] { return stop_ || !q_.empty(); });
    if (stop_) return;
  }
}

int HostPool::take(size_t bytes, Pinned* out) {
  const size_t want = (bytes + 65535) & ~size_t(65535);
  {
    std::lock_guard<std::mutex> lock(cache_m_);
    size_t best = cache_.size();
    for (size_t i = 0; i < cache_.size(); ++i)
      if (cache_[i].cap >= want && (best == cache_.size() || cache_[i].cap < cache_[best].cap)) best = i;
    if (best < cache_.size()) {
      *out = cache_[best];
      cached_ -= out->cap;
      cache_.erase(cache_.begin() + (long)best);
      return B200Q_OK;
    }
  }
  void* p = nullptr;
  const cudaError_t e = cudaHostAlloc(&p, want, cudaHostAllocPortable);
  if (e != cudaSuccess) return cuda_error(e, "cudaHostAlloc", __FILE__, __LINE__);
  out->p = static_cast<uint8_t*>(p);
  out->cap = want;
  return B200Q_OK;
}

void HostPool::give(Pinned b) {
  if (!b.p) return;
  {
    std::lock_guard<std::mutex> lock(cache_m_);
    if (cached_ + b.cap <= CACHE_BYTES) try {
        cache_.push_back(b);
        cached_ += b.cap;
        return;
      } catch (const std::exception&) {   // given back to the system instead
      }
  }
  cudaFreeHost(b.p);
}

int HostPool::take(Streams* out) {
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(cache_m_);
    for (size_t i = 0; i < sets_.size(); ++i)
      if (sets_[i].device == dev) {
        *out = sets_[i];
        sets_.erase(sets_.begin() + (long)i);
        return B200Q_OK;
      }
  }
  Streams made;
  for (auto& st : made.s) {
    const cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) continue;
    st = nullptr;
    for (auto& x : made.s)
      if (x) cudaStreamDestroy(x);
    return cuda_error(e, "cudaStreamCreateWithFlags", __FILE__, __LINE__);
  }
  made.device = dev;
  *out = made;
  return B200Q_OK;
}

void HostPool::give(const Streams& st) {
  if (st.device < 0) return;
  {
    std::lock_guard<std::mutex> lock(cache_m_);
    if (sets_.size() < CACHE_SETS) try {
        sets_.push_back(st);
        return;
      } catch (const std::exception&) {
      }
  }
  for (auto& e : st.ev) cudaEventDestroy(e);
  for (auto& x : st.s)
    if (x) cudaStreamDestroy(x);
}

// ---------------------------------------------------------------------------------------------- HostStage
HostStage::~HostStage() {   // (run() is synchronous: nothing of this handle is in flight)
  if (!pool_) return;
  pool_->give(in_);
  pool_->give(out_);
  pool_->give(streams_);
}

int HostStage::grow(HostPool::Pinned* b, size_t bytes) {
  if (bytes <= b->cap) return B200Q_OK;
  pool_->give(*b);
  *b = HostPool::Pinned();
  return pool_->take(bytes, b);
}

void HostStage::convert(const void* src, void* dst, size_t n, int dt, size_t out_size, bool alone) {
  const bool past_cache = n >= PAST_CACHE_VALUES;
  if (alone) {
    if (dt < 0) host_f32_to_bytes(static_cast<const float*>(src), static_cast<uint8_t*>(dst), n);
    else host_q_to_f32(src, dt, static_cast<float*>(dst), n, past_cache);
    return;
  }
  const size_t step = TASK_VALUES / 4, ss = dt < 0 ? 4 : out_size, ds = dt < 0 ? 1 : 4;
  std::vector<HostTask> tasks;
  tasks.reserve((n + step - 1) / step);
  std::atomic<int> left{(int)((n + step - 1) / step)};
  for (size_t o = 0; o < n; o += step)
    tasks.push_back(HostTask{static_cast<const uint8_t*>(src) + o * ss, static_cast<uint8_t*>(dst) + o * ds, n - o < step ? n - o : step, dt, &left, past_cache});
  pool_->submit(tasks.data(), tasks.size());
  while (left.load(std::memory_order_acquire) > 0)
    if (!pool_->help()) host_pause();
}

int HostStage::run(const float* x, float* y, int64_t units, size_t x_per, size_t y_per, int out_dt, size_t out_size, int* status,
                   const Launch& launch) {
  try {   // the callers are C entries.  Nothing is in flight where memory is asked for.
    return run_checked(x, y, units, x_per, y_per, out_dt, out_size, status, launch);
  } catch (const std::exception& e) {
    status_at_ = ~size_t(0);
    return set_error(B200Q_ERR_NOMEM, "operator face: %s", e.what());
  }
}

int HostStage::run_checked(const float* x, float* y, int64_t units, size_t x_per, size_t y_per, int out_dt, size_t out_size, int* status,
                           const Launch& launch) {
  if (!pool_) pool_ = HostPool::get();
  const size_t larger = x_per > y_per ? x_per : y_per;
  const size_t x_total = x_per * (size_t)units, y_bytes = y_per * (size_t)units * out_size;
  int64_t per = (int64_t)((PIECE_VALUES + larger - 1) / larger);
  // a result that lies over its input is written when all of the input has been read
  if (reinterpret_cast<uintptr_t>(x) < reinterpret_cast<uintptr_t>(y + y_per * (size_t)units) &&
      reinterpret_cast<uintptr_t>(y) < reinterpret_cast<uintptr_t>(x + x_total))
    per = units;
  if (per > units) per = units;
  const bool single = per == units;
  cudaStream_t s = 0;
  const size_t at = (y_bytes + 15) & ~size_t(15);
  const void* before = y_dev_.p;
  B200Q_TRY(x_dev_.ensure(x_total));
  B200Q_TRY(y_dev_.ensure(at + 16));
  if (at != status_at_ || before != y_dev_.p) {
    CUDA_TRY(cudaMemsetAsync(y_dev_.as<uint8_t>() + at, 0, 16, s));
    status_at_ = at;
  }
  *status = 0;
  int rc;
  if (!single) {
    rc = run_pieces(x, y, units, per, x_per, y_per, out_dt, out_size, status, launch);
  } else {
    // a small call: one stream, no events; what it costs is the launches and the round trip
    const size_t y_total = y_per * (size_t)units;
    B200Q_TRY(grow(&in_, x_total));
    B200Q_TRY(grow(&out_, at + 16));
    const bool alone = x_total + y_total <= INLINE_VALUES;
    convert(x, in_.p, x_total, -1, out_size, alone);
    CUDA_TRY(cudaMemcpyAsync(x_dev_.p, in_.p, x_total, cudaMemcpyHostToDevice, s));
    rc = launch(0, units, x_dev_.as<uint8_t>(), y_dev_.p, reinterpret_cast<int*>(y_dev_.as<uint8_t>() + at), s);
    if (rc == B200Q_OK && cudaMemcpyAsync(out_.p, y_dev_.p, at + 4, cudaMemcpyDeviceToHost, s) != cudaSuccess)
      rc = cuda_error(cudaGetLastError(), "D2H output", __FILE__, __LINE__);
    const cudaError_t e = cudaStreamSynchronize(s);
    if (rc == B200Q_OK && e != cudaSuccess) rc = cuda_error(e, "cudaStreamSynchronize", __FILE__, __LINE__);
    if (rc == B200Q_OK) {
      memcpy(status, out_.p + at, 4);
      convert(out_.p, y, y_total, out_dt, out_size, alone);
    }
  }
  if (rc != B200Q_OK || *status != 0) status_at_ = ~size_t(0);   // cleared before the next call
  return rc;
}

int HostStage::run_pieces(const float* x, float* y, int64_t units, int64_t per, size_t x_per, size_t y_per, int out_dt, size_t out_size,
                          int* status, const Launch& launch) {
  const int pieces = (int)((units + per - 1) / per);
  const int slots = pieces < MAX_SLOTS ? pieces : MAX_SLOTS;
  const size_t xs = ((size_t)per * x_per + 255) & ~size_t(255), ys = ((size_t)per * y_per * out_size + 255) & ~size_t(255);
  int* const status_dev = reinterpret_cast<int*>(y_dev_.as<uint8_t>() + status_at_);
  B200Q_TRY(grow(&in_, xs * slots));
  B200Q_TRY(grow(&out_, ys * slots + 16));
  if (streams_.device < 0) B200Q_TRY(pool_->take(&streams_));
  streams_.ev.reserve(3 * MAX_SLOTS);
  while ((int)streams_.ev.size() < 3 * slots) {
    cudaEvent_t e;
    CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    streams_.ev.push_back(e);
  }
  CUDA_TRY(cudaStreamSynchronize(0));  // whatever the caller queued on the default stream comes first
  cudaStream_t s_in = streams_.s[0], s_cmp = streams_.s[1], s_out = streams_.s[2];
  // events of a slot: input copied, kernels done, output copied
  auto ev = [&](int kind, int slot) { return streams_.ev[(size_t)(kind * slots + slot)]; };
  std::vector<std::atomic<int>> in_left((size_t)pieces), out_left((size_t)pieces);
  auto first = [&](int c) { return (int64_t)c * per; };
  auto count = [&](int c) { return first(c) + per <= units ? per : units - first(c); };
  const bool past_cache = y_per * (size_t)units >= PAST_CACHE_VALUES;
  std::vector<HostTask> tasks;
  tasks.reserve(((size_t)per * (x_per > y_per ? x_per : y_per) + TASK_VALUES - 1) / TASK_VALUES);   // nothing below asks for memory
  auto submit = [&](const void* src, void* dst, size_t n, int dt, std::atomic<int>* left) {
    const size_t ss = dt < 0 ? 4 : out_size, ds = dt < 0 ? 1 : 4;
    tasks.clear();
    left->store((int)((n + TASK_VALUES - 1) / TASK_VALUES), std::memory_order_relaxed);
    for (size_t o = 0; o < n; o += TASK_VALUES)
      tasks.push_back(HostTask{static_cast<const uint8_t*>(src) + o * ss, static_cast<uint8_t*>(dst) + o * ds,
                               n - o < TASK_VALUES ? n - o : TASK_VALUES, dt, left, past_cache});
    pool_->submit(tasks.data(), tasks.size());
  };
  int rc = B200Q_OK;
  auto chk = [&](cudaError_t e, const char* what) {
    if (rc == B200Q_OK && e != cudaSuccess) rc = cuda_error(e, what, __FILE__, __LINE__);
  };
  // pieces whose input conversion was queued / kernels enqueued / output conversion queued / output conversion done
  int submitted = 0, launched = 0, drained = 0, finished = 0;
  while (finished < pieces && rc == B200Q_OK) {
    bool moved = false;
    // inputs: a slot's pinned memory is free once the copy of the piece before it has left
    while (rc == B200Q_OK && submitted < pieces && submitted < launched + slots) {
      const int c = submitted;
      if (c >= slots) {
        const cudaError_t q = cudaEventQuery(ev(0, c % slots));
        if (q == cudaErrorNotReady) break;
        chk(q, "cudaEventQuery");
        if (rc != B200Q_OK) break;
      }
      submit(x + (size_t)first(c) * x_per, in_.p + xs * (size_t)(c % slots), (size_t)count(c) * x_per, -1, &in_left[(size_t)c]);
      ++submitted;
      moved = true;
    }
    // kernels, in order; the output slot must have been widened into the caller's buffer
    if (rc == B200Q_OK && launched < submitted && launched < finished + slots && in_left[(size_t)launched].load(std::memory_order_acquire) == 0) {
      const int c = launched, slot = c % slots;
      const size_t xo = (size_t)first(c) * x_per, xn = (size_t)count(c) * x_per;
      const size_t yo = (size_t)first(c) * y_per * out_size, yn = (size_t)count(c) * y_per * out_size;
      chk(cudaMemcpyAsync(x_dev_.as<uint8_t>() + xo, in_.p + xs * (size_t)slot, xn, cudaMemcpyHostToDevice, s_in), "H2D input");
      chk(cudaEventRecord(ev(0, slot), s_in), "event");
      chk(cudaStreamWaitEvent(s_cmp, ev(0, slot), 0), "event");
      try {
        if (rc == B200Q_OK) rc = launch(first(c), count(c), x_dev_.as<uint8_t>() + xo, y_dev_.as<uint8_t>() + yo, status_dev, s_cmp);
      } catch (const std::exception& e) {   // (pieces are in flight: this function ends by waiting for them)
        rc = set_error(B200Q_ERR_NOMEM, "operator face: %s", e.what());
      }
      chk(cudaEventRecord(ev(1, slot), s_cmp), "event");
      chk(cudaStreamWaitEvent(s_out, ev(1, slot), 0), "event");
      chk(cudaMemcpyAsync(out_.p + ys * (size_t)slot, y_dev_.as<uint8_t>() + yo, yn, cudaMemcpyDeviceToHost, s_out), "D2H output");
      if (c == pieces - 1) chk(cudaMemcpyAsync(out_.p + ys * (size_t)slots, status_dev, 4, cudaMemcpyDeviceToHost, s_out), "D2H status");
      chk(cudaEventRecord(ev(2, slot), s_out), "event");
      ++launched;
      moved = true;
    }
    if (rc == B200Q_OK && drained < launched) {
      const int c = drained;
      const cudaError_t q = cudaEventQuery(ev(2, c % slots));
      if (q == cudaSuccess) {
        submit(out_.p + ys * (size_t)(c % slots), y + (size_t)first(c) * y_per, (size_t)count(c) * y_per, out_dt, &out_left[(size_t)c]);
        ++drained;
        moved = true;
      } else if (q != cudaErrorNotReady) {
        chk(q, "cudaEventQuery");
      }
    }
    while (finished < drained && out_left[(size_t)finished].load(std::memory_order_acquire) == 0) {
      ++finished;
      moved = true;
    }
    if (!moved && !pool_->help()) host_pause();
  }
  if (rc != B200Q_OK) {   // nothing of this call may still touch its buffers when it returns
    for (auto& st : streams_.s) cudaStreamSynchronize(st);
    for (int c = 0; c < submitted; ++c)
      while (in_left[(size_t)c].load(std::memory_order_acquire) > 0)
        if (!pool_->help()) host_pause();
    for (int c = 0; c < drained; ++c)
      while (out_left[(size_t)c].load(std::memory_order_acquire) > 0)
        if (!pool_->help()) host_pause();
    return rc;
  }
  memcpy(status, out_.p + ys * (size_t)slots, 4);
  return B200Q_OK;
}

}  // namespace b200q
