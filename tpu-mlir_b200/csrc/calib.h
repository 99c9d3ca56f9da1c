// Calibration kernel launchers (calib.cu).  All asynchronous on the given stream.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace b200q {

// One tensor of a call over many: x[samples][n]; `first` / `first_chunk` place it in the flat element / chunk order.
struct CalibTensor {
  const float* x;
  int* hist;
  long long n, first, first_chunk;
};
// One histogram of a KLD call: n_in counts, zeros up to len (a multiple of the bins).
struct KldTensor {
  const int* hist;
  int n_in, len;
  float width;
};

int minmax_blocks_per_sample(long long n, long long samples);
size_t minmax_scratch_bytes(long long samples, int blocks_per_sample);
// out[s] = {min, max} of x[s*n .. (s+1)*n); scratch must be zero-initialised once and is left re-armed
int minmax_launch(const float* x, long long n, long long samples, float* out, void* scratch, int blocks_per_sample,
                  cudaStream_t s);
// Same result as minmax_launch with the scratch in a fixed device array of the library: no allocation.
int minmax_static_launch(const float* x, long long n, long long samples, float* out, cudaStream_t s);
// the same over the tensors of a device table, as order-preserving integers (out_min all ones, out_max zeros before)
long long minmax_many_chunks(long long n, long long samples);
int minmax_many_launch(const CalibTensor* tab_dev, int tensors, long long samples, long long chunks, uint32_t* out_min, uint32_t* out_max,
                       cudaStream_t s);
// hist_t[0 .. nb[t][s]) += histogram of sample s of tensor t with threshold th[t][s]; tab, th and nb are DEVICE arrays, total the
// elements of all tensors, max_bins the largest nb that is at most histogram_max_shared_bins()
int histogram_max_shared_bins();
int histogram_launch(const CalibTensor* tab_dev, int tensors, long long samples, long long total, const float* th, const int* nb,
                     int max_bins, cudaStream_t s);
// Counter layout of the histogram kernel: -1 = chosen per launch (default); 0..4 = 2^mode 32-bit copies per bin;
// 5 = lane-owned 16-bit counters.  A tuning control for measurements; every layout gives the same counts.
void histogram_set_mode(int mode);
int kl_raw_histogram_launch(const float* x, long long n, float width, int bins, int* hist, cudaStream_t s);
int fold_launch(const int* in, long long n_in, int* out, long long n_out, cudaStream_t s);
// thresholds[t] for the histograms of a device table; kl_dev is scratch and output, 1024 floats per tensor
int kld_launch(const KldTensor* tab_dev, int tensors, int dst_bins, long long max_len, float* thresholds_dev, float* kl_dev, cudaStream_t s);

}  // namespace b200q
