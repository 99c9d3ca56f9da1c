// C ABI of the calibration math: a context that owns the scratch memory of the min/max, histogram and KLD
// kernels, plus the two entry points of the reference's calibration_math.so
// (bindings/kld/calibration_math.cpp:326-337) so that kld_calibrator.py:50-59 can load this library instead.
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "calib.h"
#include "devbuf.h"
#include "internal.h"

namespace b200q {
namespace {

constexpr long long MAX_KLD_BINS = 64 * 2048;  // kld_calibrator.py:338

struct CalibCtx {
  DevBuf mm_scratch, params, work, work2, table, thresholds, kl, stage, mm_out;
  size_t mm_scratch_zeroed = 0;
};

long long pad_to(long long n, long long m) { return (n + m - 1) / m * m; }

// pad + fold plan of find_threshold (kld_calibrator.py:329-342): final length and width
void fold_plan(long long nb, float width, long long dst_bins, long long* len_out, float* width_out, int* folds) {
  long long L = pad_to(nb, dst_bins);
  int f = 0;
  while (L > MAX_KLD_BINS) {
    L = pad_to(L / 2, dst_bins);
    width = width * 2.0f;
    ++f;
  }
  *len_out = L;
  *width_out = width;
  *folds = f;
}

int find_thresholds(CalibCtx* c, int tensors, const int32_t* const* hist_dev, const int64_t* n_bins,
                    const float* widths, long long dst_bins, float* thresholds_host, float* kl_host, cudaStream_t s) {
  if (tensors == 0) return B200Q_OK;
  if (dst_bins != 128 && dst_bins != 8) return set_error(B200Q_ERR_INVALID, "find_threshold: dst_bins must be 128 or 8 (asserted by the reference)");
  // A histogram short enough is searched where it lies (its zero padding is implied by its length); longer ones are
  // folded into `work` first.
  std::vector<KldTensor> tab((size_t)tensors);
  std::vector<int> folds((size_t)tensors);
  std::vector<long long> offs((size_t)tensors);
  long long max_len = 0, max_tmp = 0, folded = 0;
  for (int t = 0; t < tensors; ++t) {
    if (n_bins[t] < 1 || !hist_dev[t]) return set_error(B200Q_ERR_INVALID, "find_threshold: empty histogram %d", t);
    long long L;
    KldTensor& k = tab[(size_t)t];
    fold_plan(n_bins[t], widths[t], dst_bins, &L, &k.width, &folds[(size_t)t]);
    k.hist = hist_dev[t];
    k.n_in = (int)(folds[(size_t)t] ? L : n_bins[t]);
    k.len = (int)L;
    if (L > max_len) max_len = L;
    if (folds[(size_t)t]) {
      offs[(size_t)t] = folded;
      folded += L;
    }
    if (folds[(size_t)t] > 1) {
      const long long tmp = pad_to(pad_to(n_bins[t], dst_bins) / 2, dst_bins);
      if (tmp > max_tmp) max_tmp = tmp;
    }
  }
  if (folded) B200Q_TRY(c->work.ensure((size_t)folded * 4));
  if (max_tmp) {
    B200Q_TRY(c->work2.ensure((size_t)max_tmp * 4));
    B200Q_TRY(c->stage.ensure((size_t)max_tmp * 4));
  }
  for (int t = 0; t < tensors; ++t) {
    if (folds[(size_t)t] == 0) continue;
    // fold chain; intermediate results ping-pong between two scratch buffers, the last step lands in `dst`
    int* dst = c->work.as<int>() + offs[(size_t)t];
    const int* src = hist_dev[t];
    long long n_in = n_bins[t], cur = pad_to(n_bins[t], dst_bins);
    int* bufs[2] = {c->work2.as<int>(), c->stage.as<int>()};
    for (int f = 0; f < folds[(size_t)t]; ++f) {
      const long long n_out = pad_to(cur / 2, dst_bins);
      int* out = (f == folds[(size_t)t] - 1) ? dst : bufs[f & 1];
      B200Q_TRY(fold_launch(src, n_in, out, n_out, s));
      src = out;
      n_in = n_out;
      cur = n_out;
    }
    tab[(size_t)t].hist = dst;
  }
  B200Q_TRY(c->table.upload(tab.data(), tab.size() * sizeof(KldTensor), s));
  B200Q_TRY(c->thresholds.ensure((size_t)tensors * 4));
  B200Q_TRY(c->kl.ensure((size_t)tensors * 1024 * 4));
  B200Q_TRY(kld_launch(c->table.as<KldTensor>(), tensors, (int)dst_bins, max_len, c->thresholds.as<float>(), c->kl.as<float>(), s));
  CUDA_TRY(cudaMemcpyAsync(thresholds_host, c->thresholds.p, (size_t)tensors * 4, cudaMemcpyDeviceToHost, s));
  if (kl_host) CUDA_TRY(cudaMemcpyAsync(kl_host, c->kl.p, (size_t)tensors * 1024 * 4, cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  return B200Q_OK;
}

// Statistics over many tensors: the table (and what follows it) in one upload.
int upload_table(CalibCtx* c, int tensors, const float* const* x, const int64_t* n_per_sample, int64_t samples, int32_t* const* hist,
                 const void* tail, size_t tail_bytes, cudaStream_t s, long long* total, long long* chunks) {
  std::vector<char> packed((size_t)tensors * sizeof(CalibTensor) + tail_bytes);
  CalibTensor* tab = reinterpret_cast<CalibTensor*>(packed.data());
  *total = *chunks = 0;
  for (int t = 0; t < tensors; ++t) {
    if (!x[t] || n_per_sample[t] < 1) return set_error(B200Q_ERR_INVALID, "calib: tensor %d is empty", t);
    tab[t].x = x[t];
    tab[t].hist = hist ? hist[t] : nullptr;
    tab[t].n = n_per_sample[t];
    tab[t].first = *total;
    tab[t].first_chunk = *chunks;
    *total += n_per_sample[t] * samples;
    *chunks += minmax_many_chunks(n_per_sample[t], samples);
  }
  if (tail_bytes) memcpy(packed.data() + (size_t)tensors * sizeof(CalibTensor), tail, tail_bytes);
  return c->params.upload(packed.data(), packed.size(), s);
}

float float_of_ordered(uint32_t u) {
  const uint32_t b = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
  float f;
  memcpy(&f, &b, 4);
  return f;
}

// numpy's floor_divide of two positive finite float32 values (the reference's `//`): the quotient from the exact remainder
float floor_divide_f32(float a, float b) {
  const float mod = fmodf(a, b);
  const float div = (a - mod) / b;
  if (div == 0.f) return 0.f;
  float fl = floorf(div);
  if (div - fl > 0.5f) fl += 1.f;
  return fl;
}

int histogram_many(CalibCtx* c, int tensors, const float* const* x, const int64_t* n_per_sample, int64_t samples, const float* th_host,
                   const int32_t* nbins_host, int32_t* const* hist, const int64_t* hist_len, cudaStream_t s) {
  const size_t rows = (size_t)tensors * (size_t)samples;
  int fit = 0, max_bins = 0;
  for (int t = 0; t < tensors; ++t) {
    if (!hist[t]) return set_error(B200Q_ERR_INVALID, "calib_histogram: null histogram");
    for (int64_t i = 0; i < samples; ++i) {
      const int nb = nbins_host[(size_t)t * samples + i];
      if (nb < 0 || nb > hist_len[t]) return set_error(B200Q_ERR_INVALID, "calib_histogram: nbins[%lld] = %d exceeds the histogram length %lld", (long long)i, nb, (long long)hist_len[t]);
      if (nb == 1) return set_error(B200Q_ERR_INVALID, "calib_histogram: a histogram needs at least 2 bins");
      if (nb > max_bins) max_bins = nb;
      if (nb > fit && nb <= histogram_max_shared_bins()) fit = nb;
    }
  }
  if (max_bins == 0) return B200Q_OK;
  std::vector<char> tail(rows * 8);   // th | nbins
  memcpy(tail.data(), th_host, rows * 4);
  memcpy(tail.data() + rows * 4, nbins_host, rows * 4);
  long long total, chunks;
  B200Q_TRY(upload_table(c, tensors, x, n_per_sample, samples, hist, tail.data(), tail.size(), s, &total, &chunks));
  const char* dev = c->params.as<char>() + (size_t)tensors * sizeof(CalibTensor);
  return histogram_launch(c->params.as<CalibTensor>(), tensors, samples, total, reinterpret_cast<const float*>(dev),
                          reinterpret_cast<const int*>(dev + rows * 4), fit ? fit : max_bins, s);
}

CalibCtx* global_ctx() {
  static CalibCtx* ctx = new (std::nothrow) CalibCtx();
  return ctx;
}
std::mutex g_mutex;

}  // namespace
}  // namespace b200q

using namespace b200q;

extern "C" {

int b200q_calib_create(void** ctx) {
  if (!ctx) return set_error(B200Q_ERR_INVALID, "calib_create: null argument");
  auto* c = new (std::nothrow) CalibCtx();
  if (!c) return set_error(B200Q_ERR_NOMEM, "calib_create: out of host memory");
  *ctx = c;
  return B200Q_OK;
}

void b200q_calib_destroy(void** ctx) {
  if (ctx && *ctx) {
    delete static_cast<CalibCtx*>(*ctx);
    *ctx = nullptr;
  }
}

int b200q_calib_minmax(void* ctx, const float* x_dev, int64_t n_per_sample, int64_t samples, float* out_dev,
                       void* stream) {
  if (!ctx || !x_dev || !out_dev || n_per_sample < 1 || samples < 0) return set_error(B200Q_ERR_INVALID, "calib_minmax: bad argument");
  CalibCtx* c = static_cast<CalibCtx*>(ctx);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int bps = minmax_blocks_per_sample(n_per_sample, samples);
  const size_t need = minmax_scratch_bytes(samples, bps);
  if (need > c->mm_scratch.cap || c->mm_scratch_zeroed < need) {
    B200Q_TRY(c->mm_scratch.ensure(need));
    CUDA_TRY(cudaMemsetAsync(c->mm_scratch.p, 0, c->mm_scratch.cap, s));  // ticket counters start at zero
    c->mm_scratch_zeroed = c->mm_scratch.cap;
  } else {
    // the ticket area moves with (samples, bps): clear it (cheap) so that any layout starts from zero
    CUDA_TRY(cudaMemsetAsync(static_cast<char*>(c->mm_scratch.p) + (size_t)samples * bps * 8, 0, (size_t)samples * 4, s));
  }
  return minmax_launch(x_dev, n_per_sample, samples, out_dev, c->mm_scratch.p, bps, s);
}

int b200q_calib_minmax_noalloc(const float* x_dev, int64_t n_per_sample, int64_t samples, float* out_dev, void* stream) {
  if (!x_dev || !out_dev || n_per_sample < 1 || samples < 0) return set_error(B200Q_ERR_INVALID, "calib_minmax_noalloc: bad argument");
  return minmax_static_launch(x_dev, n_per_sample, samples, out_dev, static_cast<cudaStream_t>(stream));
}

int b200q_calib_histogram(void* ctx, const float* x_dev, int64_t n_per_sample, int64_t samples, const float* th_host,
                          const int32_t* nbins_host, int32_t* hist_dev, int64_t hist_len, void* stream) {
  if (!ctx || !x_dev || !th_host || !nbins_host || !hist_dev || n_per_sample < 1 || samples < 0)
    return set_error(B200Q_ERR_INVALID, "calib_histogram: bad argument");
  return histogram_many(static_cast<CalibCtx*>(ctx), 1, &x_dev, &n_per_sample, samples, th_host, nbins_host, &hist_dev, &hist_len,
                        static_cast<cudaStream_t>(stream));
}

int b200q_calib_minmax_many(void* ctx, int32_t tensors, const float* const* x_dev, const int64_t* n_per_sample, int64_t samples,
                            float* minmax_host, void* stream) {
  if (!ctx || tensors < 1 || !x_dev || !n_per_sample || samples < 1 || samples > 0x7fffffffLL || !minmax_host)
    return set_error(B200Q_ERR_INVALID, "calib_minmax_many: bad argument");
  CalibCtx* c = static_cast<CalibCtx*>(ctx);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t rows = (size_t)tensors * (size_t)samples;
  long long total, chunks;
  B200Q_TRY(upload_table(c, tensors, x_dev, n_per_sample, samples, nullptr, nullptr, 0, s, &total, &chunks));
  B200Q_TRY(c->mm_out.ensure(rows * 8));
  uint32_t* lo = c->mm_out.as<uint32_t>();
  CUDA_TRY(cudaMemsetAsync(lo, 0xff, rows * 4, s));
  CUDA_TRY(cudaMemsetAsync(lo + rows, 0, rows * 4, s));
  B200Q_TRY(minmax_many_launch(c->params.as<CalibTensor>(), tensors, samples, chunks, lo, lo + rows, s));
  std::vector<uint32_t> raw(rows * 2);
  CUDA_TRY(cudaMemcpyAsync(raw.data(), lo, rows * 8, cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  for (size_t i = 0; i < rows; ++i) {
    minmax_host[2 * i] = float_of_ordered(raw[i]);
    minmax_host[2 * i + 1] = float_of_ordered(raw[rows + i]);
  }
  return B200Q_OK;
}

int b200q_calib_histogram_many(void* ctx, int32_t tensors, const float* const* x_dev, const int64_t* n_per_sample, int64_t samples,
                               const float* th_host, const int32_t* nbins_host, int32_t* const* hist_dev, const int64_t* hist_len,
                               void* stream) {
  if (!ctx || tensors < 1 || !x_dev || !n_per_sample || samples < 1 || samples > 0x7fffffffLL || !th_host || !nbins_host || !hist_dev || !hist_len)
    return set_error(B200Q_ERR_INVALID, "calib_histogram_many: bad argument");
  return histogram_many(static_cast<CalibCtx*>(ctx), tensors, x_dev, n_per_sample, samples, th_host, nbins_host, hist_dev, hist_len,
                        static_cast<cudaStream_t>(stream));
}

int b200q_calib_bin_schedule(b200q_bin_state* state, int32_t tensors, int64_t samples, const float* minmax, int64_t first_sample,
                             int32_t bin_num, int64_t max_bins, float* th, int32_t* nbins) {
  if (!state || tensors < 0 || samples < 0 || (tensors > 0 && samples > 0 && (!minmax || !th || !nbins)) || bin_num < 2)
    return set_error(B200Q_ERR_INVALID, "calib_bin_schedule: bad argument");
  for (int32_t t = 0; t < tensors; ++t) {
    b200q_bin_state& st = state[t];
    for (int64_t i = 0; i < samples; ++i) {
      const float lo = minmax[((size_t)t * samples + i) * 2], hi = minmax[((size_t)t * samples + i) * 2 + 1];
      if (lo < st.min) st.min = lo;
      if (hi > st.max) st.max = hi;
      const float abs_value = fmaxf(fabsf(st.min), fabsf(st.max));
      float* const th_i = th + (size_t)t * samples + i;
      int32_t* const nb_i = nbins + (size_t)t * samples + i;
      if (fmaxf(fabsf(lo), fabsf(hi)) < 1e-8f) {   // an all-zero activation contributes nothing
        *th_i = 0.f;
        *nb_i = 0;
        continue;
      }
      bool moved = false;
      if (!st.started) {
        st.th = abs_value;
        st.bins = bin_num;
        st.started = 1;
        moved = true;
      } else if (abs_value > st.th) {
        const float old_step = st.th / (float)st.bins;
        const float grown = floor_divide_f32(abs_value - st.th, old_step) + 1.f;
        const int64_t inc = grown >= 0.f && grown < 9e18f ? (int64_t)grown : (grown >= 9e18f && grown <= 3.402823e38f ? max_bins + 1 : 0);
        if (inc + st.bins > max_bins) {
          st.th = abs_value;
          st.bins = bin_num;
          st.last_reset = first_sample + i;
          for (int64_t j = 0; j < i; ++j) {   // (earlier calls' samples: the caller drops what it counted for them)
            th[(size_t)t * samples + j] = 0.f;
            nbins[(size_t)t * samples + j] = 0;
          }
        } else {
          st.th = (float)inc * old_step + st.th;
          st.bins = inc + st.bins;
        }
        moved = true;
      }
      if (moved) st.width = st.th / (float)(st.bins - 1);
      *th_i = st.th;
      *nb_i = (int32_t)st.bins;
    }
  }
  return B200Q_OK;
}

void b200q_calib_set_histogram_layout(int32_t mode) { histogram_set_mode(mode); }

int b200q_calib_find_thresholds(void* ctx, int32_t tensors, const int32_t* const* hist_dev, const int64_t* n_bins,
                                const float* widths, int64_t dst_bins, float* thresholds_host, float* kl_host,
                                void* stream) {
  if (!ctx || tensors < 0 || (tensors > 0 && (!hist_dev || !n_bins || !widths || !thresholds_host)))
    return set_error(B200Q_ERR_INVALID, "calib_find_thresholds: bad argument");
  return find_thresholds(static_cast<CalibCtx*>(ctx), tensors, hist_dev, n_bins, widths, dst_bins, thresholds_host,
                         kl_host, static_cast<cudaStream_t>(stream));
}

// ---- the reference's calibration_math ABI (calibration_math.cpp:326-337); like the reference these report
// failure only by their return value, here NaN (message through b200q_last_error()).
float kl_diversity_hist(int* data, float width, long long num_bins, long long dst_bins) {
  std::lock_guard<std::mutex> lock(g_mutex);
  CalibCtx* c = global_ctx();
  if (!c || !data || num_bins < dst_bins || num_bins % dst_bins != 0) {
    set_error(B200Q_ERR_INVALID, "kl_diversity_hist: bad argument");
    return NAN;
  }
  cudaStream_t s = 0;
  if (c->stage.upload(data, (size_t)num_bins * 4, s) != B200Q_OK) return NAN;
  // the caller (find_threshold) has already padded and folded: run the search on the histogram as given
  if (num_bins / dst_bins > 1024) {
    set_error(B200Q_ERR_UNSUPPORTED, "kl_diversity_hist: more than 1024 candidates");
    return NAN;
  }
  float th = NAN;
  const KldTensor k{c->stage.as<int>(), (int)num_bins, (int)num_bins, width};
  if (c->table.upload(&k, sizeof(k), s) != B200Q_OK || c->thresholds.ensure(4) != B200Q_OK || c->kl.ensure(1024 * 4) != B200Q_OK) return NAN;
  if (kld_launch(c->table.as<KldTensor>(), 1, (int)dst_bins, num_bins, c->thresholds.as<float>(), c->kl.as<float>(), s) != B200Q_OK) return NAN;
  if (cudaMemcpyAsync(&th, c->thresholds.p, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) {
    cuda_error(cudaGetLastError(), "kl_diversity_hist", __FILE__, __LINE__);
    return NAN;
  }
  return th;
}

float kl_diversity(float* data, long long count, long long num_bins) {
  std::lock_guard<std::mutex> lock(g_mutex);
  CalibCtx* c = global_ctx();
  const long long BINS = 128;
  if (!c || !data || count < 1 || num_bins < BINS || num_bins % BINS != 0 || num_bins / BINS > 1024) {
    set_error(B200Q_ERR_INVALID, "kl_diversity: bad argument");
    return NAN;
  }
  cudaStream_t s = 0;
  // data_max = max |x| (calibration_math.cpp:60-68), width = data_max / (N - 1)
  if (c->work2.upload(data, (size_t)count * 4, s) != B200Q_OK || c->mm_out.ensure(8) != B200Q_OK) return NAN;
  const int bps = minmax_blocks_per_sample(count, 1);
  if (c->mm_scratch.ensure(minmax_scratch_bytes(1, bps)) != B200Q_OK) return NAN;
  cudaMemsetAsync(c->mm_scratch.p, 0, c->mm_scratch.cap, s);
  c->mm_scratch_zeroed = c->mm_scratch.cap;
  if (minmax_launch(c->work2.as<float>(), count, 1, c->mm_out.as<float>(), c->mm_scratch.p, bps, s) != B200Q_OK) return NAN;
  float mm[2];
  if (cudaMemcpyAsync(mm, c->mm_out.p, 8, cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) return NAN;
  const float data_max = fmaxf(fabsf(mm[0]), fabsf(mm[1]));
  const float width = data_max / (float)(num_bins - 1);
  if (c->stage.ensure((size_t)num_bins * 4) != B200Q_OK) return NAN;
  cudaMemsetAsync(c->stage.p, 0, (size_t)num_bins * 4, s);
  if (kl_raw_histogram_launch(c->work2.as<float>(), count, width, (int)num_bins, c->stage.as<int>(), s) != B200Q_OK) return NAN;
  float th = NAN;
  const KldTensor k{c->stage.as<int>(), (int)num_bins, (int)num_bins, width};
  if (c->table.upload(&k, sizeof(k), s) != B200Q_OK || c->thresholds.ensure(4) != B200Q_OK || c->kl.ensure(1024 * 4) != B200Q_OK) return NAN;
  if (kld_launch(c->table.as<KldTensor>(), 1, (int)BINS, num_bins, c->thresholds.as<float>(), c->kl.as<float>(), s) != B200Q_OK) return NAN;
  if (cudaMemcpyAsync(&th, c->thresholds.p, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) return NAN;
  return th;
}

}  // extern "C"
