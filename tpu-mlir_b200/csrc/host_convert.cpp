// Conversions between the interpreter's floats and native storage (host_convert.h).  The vector forms are for x86 hosts; any
// other host (this GPU is sold with ARM ones too) runs the plain loops, which the compiler vectorises for it.
#include "host_convert.h"

#include "../../include/b200q.h"

#if defined(__x86_64__) && !defined(B200Q_PORTABLE_HOST)   // (the macro: for tests of the plain loops on an x86 host)
#define B200Q_HOST_AVX2 1
#include <immintrin.h>
#endif

namespace b200q {
namespace {

// the low byte of x as an int32, out of range to the nearest end and NaN to 0, as the GPU converts
uint8_t f32_low_byte(float x) { return x >= 2147483648.f ? 0xff : (x >= -2147483648.f ? (uint8_t)(int)x : 0); }

void f32_to_bytes_scalar(const float* x, uint8_t* y, size_t n) {
  for (size_t i = 0; i < n; ++i) y[i] = f32_low_byte(x[i]);
}

template <typename T>
void q_to_f32_scalar(const T* x, float* y, size_t n) {
  for (size_t i = 0; i < n; ++i) y[i] = (float)x[i];
}

#ifdef B200Q_HOST_AVX2
// cvttps gives 0x80000000 for what does not fit; above the range the low byte has to be that of 0x7fffffff
__attribute__((target("avx2"))) inline __m256i low_bytes(const float* x) {
  const __m256 v = _mm256_loadu_ps(x);
  const __m256i above = _mm256_castps_si256(_mm256_cmp_ps(v, _mm256_set1_ps(2147483648.f), _CMP_GE_OQ));
  return _mm256_and_si256(_mm256_or_si256(_mm256_cvttps_epi32(v), above), _mm256_set1_epi32(0xff));
}

__attribute__((target("avx2"))) void f32_to_bytes_avx2(const float* x, uint8_t* y, size_t n) {
  const __m256i order = _mm256_setr_epi32(0, 4, 1, 5, 2, 6, 3, 7);   // undo the per-128-bit-lane packing
  size_t i = 0;
  for (; i + 32 <= n; i += 32) {
    const __m256i a = low_bytes(x + i), b = low_bytes(x + i + 8), c = low_bytes(x + i + 16), d = low_bytes(x + i + 24);
    const __m256i p = _mm256_packus_epi16(_mm256_packus_epi32(a, b), _mm256_packus_epi32(c, d));
    _mm256_storeu_si256(reinterpret_cast<__m256i*>(y + i), _mm256_permutevar8x32_epi32(p, order));
  }
  f32_to_bytes_scalar(x + i, y + i, n - i);
}

// 8-bit to float, 32 values per step
template <bool SIGNED, bool PAST_CACHE>
__attribute__((target("avx2"))) void bytes_to_f32_avx2(const uint8_t* x, float* y, size_t n) {
  size_t i = 0;
  while (i < n && (reinterpret_cast<uintptr_t>(y + i) & 31) != 0) {
    y[i] = SIGNED ? (float)(int8_t)x[i] : (float)x[i];
    ++i;
  }
  for (; i + 32 <= n; i += 32) {
    for (int k = 0; k < 4; ++k) {
      const __m128i b = _mm_loadl_epi64(reinterpret_cast<const __m128i*>(x + i + 8 * k));
      const __m256i w = SIGNED ? _mm256_cvtepi8_epi32(b) : _mm256_cvtepu8_epi32(b);
      if (PAST_CACHE) _mm256_stream_ps(y + i + 8 * k, _mm256_cvtepi32_ps(w));
      else _mm256_store_ps(y + i + 8 * k, _mm256_cvtepi32_ps(w));
    }
  }
  for (; i < n; ++i) y[i] = SIGNED ? (float)(int8_t)x[i] : (float)x[i];
  if (PAST_CACHE) _mm_sfence();
}

bool have_avx2() {
  static const bool yes = __builtin_cpu_supports("avx2");
  return yes;
}
#endif

}  // namespace

void host_pause() {
#if defined(B200Q_HOST_AVX2)
  _mm_pause();
#elif defined(__aarch64__)
  asm volatile("yield" ::: "memory");
#else
  asm volatile("" ::: "memory");
#endif
}

void host_f32_to_bytes(const float* x, uint8_t* y, size_t n) {
#ifdef B200Q_HOST_AVX2
  if (have_avx2()) return f32_to_bytes_avx2(x, y, n);
#endif
  f32_to_bytes_scalar(x, y, n);
}

void host_q_to_f32(const void* x, int dt, float* y, size_t n, bool past_cache) {
#ifdef B200Q_HOST_AVX2
  if ((dt == B200Q_DT_I8 || dt == B200Q_DT_U8) && have_avx2()) {
    auto* f = dt == B200Q_DT_I8 ? (past_cache ? bytes_to_f32_avx2<true, true> : bytes_to_f32_avx2<true, false>)
                                : (past_cache ? bytes_to_f32_avx2<false, true> : bytes_to_f32_avx2<false, false>);
    return f(static_cast<const uint8_t*>(x), y, n);
  }
#else
  (void)past_cache;
#endif
  switch (dt) {
    case B200Q_DT_I8: q_to_f32_scalar(static_cast<const int8_t*>(x), y, n); break;
    case B200Q_DT_U8: q_to_f32_scalar(static_cast<const uint8_t*>(x), y, n); break;
    case B200Q_DT_I16: q_to_f32_scalar(static_cast<const int16_t*>(x), y, n); break;
    case B200Q_DT_U16: q_to_f32_scalar(static_cast<const uint16_t*>(x), y, n); break;
    default: q_to_f32_scalar(static_cast<const int32_t*>(x), y, n); break;
  }
}

}  // namespace b200q
