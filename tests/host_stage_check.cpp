// The operator face's host side (csrc/host_stage.cpp, csrc/host_convert.cpp) on host memory, without a device: the CUDA calls it
// makes are the fakes below, which work at once and can be told to fail.  usage: host_stage_check <check>
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <errno.h>
#include <math.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <new>
#include <utility>
#include <vector>

#include "held_array.h"
#include "host_stage.h"

using namespace b200q;

#define CHECK(x)                                                       \
  do {                                                                 \
    if (!(x)) {                                                        \
      fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #x);          \
      exit(1);                                                         \
    }                                                                  \
  } while (0)

// ------------------------------------------------------------------------------------------------ fakes
namespace fake {
int streams_made, streams_ended, events_made, events_ended, memory_made, memory_ended, threads_made;
int fail_stream = -1, fail_copy = -1;   // which call fails (counted from 0), -1: none
int threads_allowed = 1 << 30;
bool null_stream_used;
int copies;
std::mutex m;
}  // namespace fake

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { std::lock_guard<std::mutex> l(fake::m); ++fake::memory_made; *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::lock_guard<std::mutex> l(fake::m); ++fake::memory_ended; free(p); return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { std::lock_guard<std::mutex> l(fake::m); ++fake::memory_made; *p = malloc(n); memset(*p, 0xee, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::lock_guard<std::mutex> l(fake::m); ++fake::memory_ended; free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  std::lock_guard<std::mutex> l(fake::m);
  if (fake::fail_stream >= 0 && fake::fail_stream-- == 0) return cudaErrorMemoryAllocation;
  ++fake::streams_made;
  *s = reinterpret_cast<cudaStream_t>(malloc(1));
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { std::lock_guard<std::mutex> l(fake::m); ++fake::streams_ended; free(s); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { std::lock_guard<std::mutex> l(fake::m); ++fake::events_made; *e = reinterpret_cast<cudaEvent_t>(malloc(1)); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::lock_guard<std::mutex> l(fake::m); ++fake::events_ended; free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  std::lock_guard<std::mutex> l(fake::m);
  ++fake::copies;
  if (st == nullptr) fake::null_stream_used = true;
  if (fake::fail_copy >= 0 && fake::fail_copy-- == 0) return cudaErrorUnknown;
  memcpy(d, s, n);
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaErrorUnknown; }
// (the program's own definition comes before the C library's for the C++ runtime too)
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg) {
  typedef int (*create_t)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static create_t real = reinterpret_cast<create_t>(dlsym(RTLD_NEXT, "pthread_create"));
  if (fake::threads_made >= fake::threads_allowed) return EAGAIN;
  ++fake::threads_made;
  return real(t, a, f, arg);
}
}

// the n-th request for memory from now on fails, once
static std::atomic<int> new_fails{-1};
void* operator new(size_t n) {
  if (new_fails.load() >= 0 && new_fails.fetch_sub(1) == 0) throw std::bad_alloc();
  if (void* p = malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

namespace b200q {
int set_error(int code, const char*, ...) { return code; }
int cuda_error(cudaError_t e, const char*, const char*, int) { return e == cudaErrorMemoryAllocation ? B200Q_ERR_NOMEM : B200Q_ERR_CUDA; }
}  // namespace b200q

// ------------------------------------------------------------------------------------------------ checks
// rows of K bytes -> N values: out[n] = x[n % K] + n (as the storage type)
static int run_rows(HostStage& stage, const float* x, float* y, int64_t rows, int K, int N, int dt) {
  const size_t size = dt == B200Q_DT_I32 ? 4 : (dt == B200Q_DT_I16 || dt == B200Q_DT_U16 ? 2 : 1);
  int status = 77;
  const int rc = stage.run(x, y, rows, (size_t)K, (size_t)N, dt, size, &status, [&](int64_t, int64_t cnt, const uint8_t* xb, void* yb, int* st, cudaStream_t) {
    CHECK(*st == 0);
    for (int64_t r = 0; r < cnt; ++r)
      for (int n = 0; n < N; ++n) {
        const int v = (int8_t)xb[r * K + n % K] + n % 50;
        if (size == 4) static_cast<int32_t*>(yb)[r * N + n] = v;
        else if (size == 2) static_cast<int16_t*>(yb)[r * N + n] = (int16_t)v;
        else static_cast<int8_t*>(yb)[r * N + n] = (int8_t)v;
      }
    return B200Q_OK;
  });
  if (rc == B200Q_OK) CHECK(status == 0);
  return rc;
}

static void check_rows(HostStage& stage, int64_t rows, int K, int N, int dt, int expect = B200Q_OK) {
  std::vector<float> x((size_t)rows * K), y((size_t)rows * N, 1e9f);
  for (size_t i = 0; i < x.size(); ++i) x[i] = (float)((int)(i * 7 % 61) - 30);
  CHECK(run_rows(stage, x.data(), y.data(), rows, K, N, dt) == expect);
  if (expect != B200Q_OK) return;
  for (int64_t r = 0; r < rows; ++r)
    for (int n = 0; n < N; ++n) CHECK(y[(size_t)(r * N + n)] == x[(size_t)(r * K + n % K)] + (float)(n % 50));
}

static void check_shapes() {
  HostStage stage;
  for (int dt : {B200Q_DT_I8, B200Q_DT_I16, B200Q_DT_I32}) {
    check_rows(stage, 3, 17, 5, dt);                    // by the calling thread
    check_rows(stage, 300, 999, 77, dt);                // one piece, by the pool
    check_rows(stage, 5000, 777, 33, dt);               // more pieces than slots, odd rows
    check_rows(stage, 700, 33, 1001, dt);
    check_rows(stage, 1, 700000, 9, dt);                // one unit larger than a piece
  }
}

static int checks_pieces() {
  {
    std::vector<std::thread> t;
    for (int i = 0; i < 3; ++i) t.emplace_back(check_shapes);
    check_shapes();
    for (auto& x : t) x.join();
  }
  CHECK(fake::streams_made > 0 && fake::streams_made == fake::streams_ended && fake::events_made == fake::events_ended && fake::memory_made == fake::memory_ended);
  return 0;
}

// Threads that cannot be had are done without: the calling thread does their work.
static int checks_threads(int allowed) {
  fake::threads_allowed = allowed;
  check_shapes();
  CHECK(fake::threads_made <= allowed);
  return 0;
}

static int checks_conversions() {
  std::vector<float> f;
  for (int i = -300; i < 300; ++i) f.push_back((float)i);
  for (size_t n : {size_t(0), size_t(1), size_t(31), size_t(32), size_t(33), f.size() - 3}) {
    for (size_t o : {0, 1, 3}) {
      std::vector<uint8_t> y(n + 8, 0xa5);
      host_f32_to_bytes(f.data() + o, y.data() + o, n);
      for (size_t i = 0; i < n; ++i) CHECK(y[i + o] == (uint8_t)((int)f[i + o] & 0xff));
      CHECK(y[n + o] == 0xa5);
    }
  }
  // fractions, values no int32 holds, infinities, NaN: what the device's conversion gives (-1 stands for 0x7fffffff's low byte)
  const std::vector<std::pair<float, int>> odd = {{-0.9f, 0}, {1.9f, 1}, {-1.5f, -1}, {2147483520.f, 0x80}, {2147483648.f, -1}, {3e9f, -1}, {INFINITY, -1},
                                                  {-2147483648.f, 0}, {-3e9f, 0}, {-INFINITY, 0}, {NAN, 0}, {300.f, 44}, {-129.f, 127}};
  std::vector<float> of;
  for (int r = 0; r < 5; ++r)
    for (auto& v : odd) of.push_back(v.first);
  std::vector<uint8_t> ob(of.size());
  host_f32_to_bytes(of.data(), ob.data(), of.size());
  for (size_t i = 0; i < of.size(); ++i) CHECK(ob[i] == (uint8_t)odd[i % odd.size()].second);
  for (int dt : {B200Q_DT_I8, B200Q_DT_U8, B200Q_DT_I16, B200Q_DT_U16, B200Q_DT_I32}) {
    for (size_t n : {0, 1, 31, 32, 33, 257}) {
      std::vector<int32_t> raw(n + 8);
      for (size_t i = 0; i < raw.size(); ++i) raw[i] = (int32_t)(i * 2654435761u);
      for (size_t o : {0, 1, 5}) {
        std::vector<float> y(n + 8, -7.5f);
        host_q_to_f32(raw.data(), dt, y.data() + o, n, (n & 1) != 0 && o != 1);
        for (size_t i = 0; i < n; ++i) {
          const float want = dt == B200Q_DT_I8    ? (float)reinterpret_cast<int8_t*>(raw.data())[i]
                             : dt == B200Q_DT_U8  ? (float)reinterpret_cast<uint8_t*>(raw.data())[i]
                             : dt == B200Q_DT_I16 ? (float)reinterpret_cast<int16_t*>(raw.data())[i]
                             : dt == B200Q_DT_U16 ? (float)reinterpret_cast<uint16_t*>(raw.data())[i]
                                                  : (float)raw[i];
          CHECK(y[i + o] == want);
        }
        CHECK(y[n + o] == -7.5f);
      }
    }
  }
  host_pause();
  return 0;
}

// Every request for host memory of a call fails once: the call works, or says so and the next one works.
static int checks_memory() {
  std::vector<float> x(1500 * 999, 3.f), y(1500 * 77, 0.f);
  int refused = 0, passed = 0;
  for (int n = 0; n < 120; ++n) {
    HostStage stage;
    new_fails.store(n);
    const int rc = run_rows(stage, x.data(), y.data(), 1500, 999, 77, B200Q_DT_I8);
    const bool met = new_fails.exchange(-1) < 0;
    CHECK(rc == B200Q_OK || rc == B200Q_ERR_NOMEM);
    ++(rc == B200Q_OK ? passed : refused);
    check_rows(stage, 1500, 999, 77, B200Q_DT_I8);
    if (!met) break;   // more than the call asks for
  }
  CHECK(refused > 3 && passed > 3);
  return 0;
}

// A stream that cannot be made: the call fails, nothing half-made is kept, and the next call has three streams again.
static int checks_streams() {
  for (int n = 0; n < 3; ++n) {
    HostStage stage, other;
    fake::fail_stream = n;
    check_rows(stage, 1500, 999, 77, B200Q_DT_I8, B200Q_ERR_NOMEM);
    CHECK(fake::streams_made == fake::streams_ended);
    fake::null_stream_used = false;
    check_rows(stage, 1500, 999, 77, B200Q_DT_I8);
    check_rows(other, 1500, 999, 77, B200Q_DT_I8);
    CHECK(!fake::null_stream_used);
  }
  return 0;
}

// A copy that fails, early or late: the call says so and the next one is right.
static int checks_copies() {
  HostStage stage;
  fake::copies = 0;
  check_rows(stage, 1500, 999, 77, B200Q_DT_I8);
  const int copies = fake::copies;
  for (int n = 0; n < copies; ++n) {
    fake::fail_copy = n;
    check_rows(stage, 1500, 999, 77, B200Q_DT_I8, B200Q_ERR_CUDA);
    fake::fail_copy = -1;
    check_rows(stage, 1500, 999, 77, B200Q_DT_I8);
  }
  return 0;
}

// A result that is written over its own input (rows grow in place, or shrink).
static int checks_overlap() {
  const int64_t rows = 4000;
  for (int N : {999, 501, 333}) {
    const int K = N == 333 ? 999 : 500;
    for (int64_t shift : {int64_t(0), int64_t(12345)}) {   // of the result within the buffer
      HostStage stage;
      std::vector<float> buf((size_t)rows * 1000 + 20000), want((size_t)rows * N);
      for (size_t i = 0; i < buf.size(); ++i) buf[i] = (float)((int)(i * 7 % 61) - 30);
      for (int64_t r = 0; r < rows; ++r)
        for (int n = 0; n < N; ++n) want[(size_t)(r * N + n)] = buf[(size_t)(r * K + n % K)] + (float)(n % 50);
      CHECK(run_rows(stage, buf.data(), buf.data() + shift, rows, K, N, B200Q_DT_I8) == B200Q_OK);
      CHECK(!memcmp(buf.data() + shift, want.data(), want.size() * 4));
    }
  }
  return 0;
}

// An upload that fails: the next call does not take the old contents, or half of the new, for what is on the device.
static int checks_held_arrays() {
  HeldArray mult, shift;
  const std::vector<int32_t> m1 = {1, 2, 3}, s1 = {4, 5, 6}, m2 = {7, 8, 9}, s2 = {9, 9, 9};
  auto both = [&](const std::vector<int32_t>& m, const std::vector<int32_t>& s) {
    const int rc = mult.put(m, nullptr);
    return rc != B200Q_OK ? rc : shift.put(s, nullptr);
  };
  auto holds = [&](const std::vector<int32_t>& m, const std::vector<int32_t>& s) {
    return !memcmp(mult.get(), m.data(), m.size() * 4) && !memcmp(shift.get(), s.data(), s.size() * 4);
  };
  CHECK(both(m1, s1) == B200Q_OK && holds(m1, s1));
  fake::copies = 0;
  CHECK(both(m1, s1) == B200Q_OK && fake::copies == 0);
  for (int n = 0; n < 2; ++n) {
    fake::fail_copy = n;
    CHECK(both(m2, s2) == B200Q_ERR_CUDA);
    fake::fail_copy = -1;
    CHECK(both(m1, s1) == B200Q_OK && holds(m1, s1));
  }
  CHECK(both(m2, s1) == B200Q_OK && holds(m2, s1));
  CHECK(both({1}, {2, 3, 4, 5}) == B200Q_OK && holds({1}, {2, 3, 4, 5}));
  return 0;
}

static int checks_workers() {
  CHECK(host_workers(16, nullptr, nullptr) == 15 && host_workers(200, nullptr, "max 100000") == 15 && host_workers(8, "", "") == 7);
  CHECK(host_workers(1, nullptr, nullptr) == 0 && host_workers(0, nullptr, nullptr) == 0);
  CHECK(host_workers(128, "8", nullptr) == 15 && host_workers(64, "8", nullptr) == 7 && host_workers(4, "8", nullptr) == 0 && host_workers(16, "x", nullptr) == 15);
  CHECK(host_workers(64, nullptr, "400000 100000") == 3 && host_workers(64, nullptr, "50000 100000") == 0 && host_workers(2, nullptr, "900000 100000") == 1);
  CHECK(host_workers(64, "2", "800000 100000") == 3);
  return 0;
}

int main(int argc, char** argv) {
  const char* what = argc > 1 ? argv[1] : "";
  if (!strcmp(what, "conversions")) return checks_conversions();
  if (!strcmp(what, "pieces")) return checks_pieces();
  if (!strcmp(what, "no threads")) return checks_threads(0);
  if (!strcmp(what, "streams")) return checks_streams();
  if (!strcmp(what, "copies")) return checks_copies();
  if (!strcmp(what, "overlap")) return checks_overlap();
  if (!strcmp(what, "held arrays")) return checks_held_arrays();
  if (!strcmp(what, "workers")) return checks_workers();
  if (!strcmp(what, "out of memory")) return checks_memory();
  if (!strcmp(what, "two threads")) return checks_threads(2);
  fprintf(stderr, "unknown check '%s'\n", what);
  return 2;
}
