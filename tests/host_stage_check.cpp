// The operator face's host side (csrc/host_stage.cpp, csrc/host_convert.cpp) on host memory, without a device: the CUDA calls it
// makes are the fakes below, which work at once and can be told to fail.  usage: host_stage_check <check>
#include <cuda_runtime.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <utility>
#include <vector>

#include "host_stage.h"

using namespace b200q;

#define CHECK(x)                                                       \
  do {                                                                 \
    if (!(x)) {                                                        \
      fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #x);          \
      exit(1);                                                         \
    }                                                                  \
  } while (0)

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

int main(int argc, char** argv) {
  const char* what = argc > 1 ? argv[1] : "";
  if (!strcmp(what, "conversions")) return checks_conversions();
  fprintf(stderr, "unknown check '%s'\n", what);
  return 2;
}
