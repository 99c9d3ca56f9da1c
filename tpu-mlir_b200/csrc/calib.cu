// Calibration math on the GPU: per-sample min/max, the activation histogram, histogram folding and the
// KLD threshold search.
//
// Reference semantics (paths inside the tpu-mlir tree):
//   histogram            python/calibration/cali_math.py:68-80 (CaliMathCpu.histogram; float32 arithmetic,
//                        zeros excluded, numpy.histogram on float32 input with its float32 bin edges)
//   min/max bookkeeping  python/calibration/kld_calibrator.py:391-398
//   pad + fold           python/calibration/kld_calibrator.py:329-342
//   KLD search           bindings/kld/calibration_math.cpp:158-212 (kl_calc_thread), :273-323, :71-83
#include <math.h>

#include <atomic>
#include <type_traits>

#include "calib.h"
#include "internal.h"

namespace b200q {
namespace {

// ------------------------------------------------------------------------------------------- min / max
constexpr int MM_THREADS = 256;

__device__ __forceinline__ float warp_min(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// grid (blocks_per_sample, samples).  Block partials go to scratch; the last block of a sample to finish
// (ticket counter in scratch) reduces them, writes out[s] = {min, max} and re-arms the counter.
// NaNs are ignored (fminf/fmaxf), where numpy would propagate them.
__global__ void __launch_bounds__(MM_THREADS)
minmax_kernel(const float* __restrict__ x, long long n, float* __restrict__ out, float* __restrict__ partial,
              unsigned int* __restrict__ tickets) {
  const int s = blockIdx.y, nb = gridDim.x;
  const float* xs = x + (long long)s * n;
  float lo = INFINITY, hi = -INFINITY;
  const long long n4 = ((reinterpret_cast<uintptr_t>(xs) & 15) == 0) ? n / 4 : 0;
  const float4* x4 = reinterpret_cast<const float4*>(xs);
  for (long long i = (long long)blockIdx.x * MM_THREADS + threadIdx.x; i < n4; i += (long long)nb * MM_THREADS) {
    const float4 v = x4[i];
    lo = fminf(fminf(lo, v.x), fminf(v.y, fminf(v.z, v.w)));
    hi = fmaxf(fmaxf(hi, v.x), fmaxf(v.y, fmaxf(v.z, v.w)));
  }
  for (long long i = n4 * 4 + (long long)blockIdx.x * MM_THREADS + threadIdx.x; i < n; i += (long long)nb * MM_THREADS) {
    lo = fminf(lo, xs[i]);
    hi = fmaxf(hi, xs[i]);
  }
  __shared__ float slo[MM_THREADS / 32], shi[MM_THREADS / 32];
  __shared__ bool last;
  lo = warp_min(lo);
  hi = warp_max(hi);
  if ((threadIdx.x & 31) == 0) {
    slo[threadIdx.x >> 5] = lo;
    shi[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < MM_THREADS / 32; ++w) {
      lo = fminf(lo, slo[w]);
      hi = fmaxf(hi, shi[w]);
    }
    partial[((long long)s * nb + blockIdx.x) * 2] = lo;
    partial[((long long)s * nb + blockIdx.x) * 2 + 1] = hi;
    __threadfence();
    last = atomicAdd(&tickets[s], 1u) == (unsigned)(nb - 1);
  }
  __syncthreads();
  if (last) {
    __threadfence();
    lo = INFINITY;
    hi = -INFINITY;
    for (int b = threadIdx.x; b < nb; b += MM_THREADS) {
      lo = fminf(lo, partial[((long long)s * nb + b) * 2]);
      hi = fmaxf(hi, partial[((long long)s * nb + b) * 2 + 1]);
    }
    lo = warp_min(lo);
    hi = warp_max(hi);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
      slo[threadIdx.x >> 5] = lo;
      shi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < MM_THREADS / 32; ++w) {
        lo = fminf(lo, slo[w]);
        hi = fmaxf(hi, shi[w]);
      }
      out[2 * s] = lo;
      out[2 * s + 1] = hi;
      tickets[s] = 0;  // ready for the next launch
    }
  }
}

// Many tensors in one launch.  The rows (tensor, sample) are cut into chunks of MANY_CHUNK floats, one block each, so that
// a launch over a network's activations is one wave after another of equal blocks instead of a kernel (and its tail) per
// tensor.  A block's extrema meet in two atomics on an order-preserving integer image of the floats; the host maps them
// back.  73 activations of 16 ResNet-50 samples (711 MB): one launch instead of 73.
constexpr int MANY_CHUNK = 32768;

__device__ __forceinline__ uint32_t ordered_bits(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// the last tensor whose first chunk / element is <= pos
__device__ __forceinline__ int find_tensor(const CalibTensor* __restrict__ tab, int tensors, long long pos, bool by_chunk) {
  int lo = 0, hi = tensors - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((by_chunk ? tab[mid].first_chunk : tab[mid].first) <= pos) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(MM_THREADS)
minmax_many_kernel(const CalibTensor* __restrict__ tab, int tensors, int samples, uint32_t* __restrict__ out_min, uint32_t* __restrict__ out_max) {
  const int t = find_tensor(tab, tensors, blockIdx.x, true);
  const long long n = tab[t].n;
  const int per_row = (int)((n + MANY_CHUNK - 1) / MANY_CHUNK);
  const int c = (int)(blockIdx.x - tab[t].first_chunk);
  const int s = c / per_row, part = c - s * per_row;
  const float* p = tab[t].x + (long long)s * n + (long long)part * MANY_CHUNK;
  const int len = (int)min((long long)MANY_CHUNK, n - (long long)part * MANY_CHUNK);
  float lo = INFINITY, hi = -INFINITY;
  int head = (int)(((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) >> 2);
  if (head > len) head = len;
  if ((int)threadIdx.x < head) lo = hi = p[threadIdx.x];
  const int body4 = (len - head) >> 2;
  const float4* p4 = reinterpret_cast<const float4*>(p + head);
#pragma unroll 8
  for (int i = threadIdx.x; i < body4; i += MM_THREADS) {
    const float4 v = p4[i];
    lo = fminf(fminf(lo, v.x), fminf(v.y, fminf(v.z, v.w)));
    hi = fmaxf(fmaxf(hi, v.x), fmaxf(v.y, fmaxf(v.z, v.w)));
  }
  const int done = head + body4 * 4;
  if (done + (int)threadIdx.x < len) {
    lo = fminf(lo, p[done + threadIdx.x]);
    hi = fmaxf(hi, p[done + threadIdx.x]);
  }
  __shared__ float slo[MM_THREADS / 32], shi[MM_THREADS / 32];
  lo = warp_min(lo);
  hi = warp_max(hi);
  if ((threadIdx.x & 31) == 0) {
    slo[threadIdx.x >> 5] = lo;
    shi[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < MM_THREADS / 32; ++w) {
      lo = fminf(lo, slo[w]);
      hi = fmaxf(hi, shi[w]);
    }
    if (!(lo != lo)) {   // (a chunk of NaNs alone leaves +-infinity, which changes nothing)
      atomicMin(&out_min[(long long)t * samples + s], ordered_bits(lo));
      atomicMax(&out_max[(long long)t * samples + s], ordered_bits(hi));
    }
  }
}

// ------------------------------------------------------------------------------------------- histogram
constexpr int HIST_THREADS = 1024;
constexpr int HIST_SMEM_BYTES = 208 * 1024;        // counters of one block (one block per SM)
constexpr long long HIST_FLUSH_ELEMS = 1998848;    // 488 * 4096 elements: the longest run a block counts without a merge
constexpr long long HIST_MERGE_EVERY = 2040;       // per-thread element budget between merges: 32 warps x 2040 < 2^16
constexpr uint32_t FLOOR_MAGIC = 0x4B000000u;      // bits of 2^23

// Bin of the integer-valued float k in [0, bins-1] under numpy.histogram(k, bins, range=(0, bins-1)) on
// float32 input: bin k, moved up by one when k >= (float)((k+1) * ((bins-1)/bins)) (float32 bin edges).
__device__ __forceinline__ int numpy_bin(float k, int bins, float binsf, double step) {
  int idx = (int)k;
  if (idx >= bins - 1) return bins - 1;
  // the fix-up can only trigger when 1 - (idx+1)/bins <= ulp(idx)/2 <= idx * 2^-24; test with a 2x margin
  if ((float)(bins - 1 - idx) > binsf * k * 1.2e-7f) return idx;
  const float edge = (float)((double)(idx + 1) * step);
  return idx + (k >= edge ? 1 : 0);
}

// How a block keeps its counters in shared memory.
//   LANE16: every lane of a warp owns one bank.  Word (bin >> 1) * 32 + lane holds two 16-bit counters (bins 2j and
//           2j + 1) that only threads with this lane index touch: an update never meets a bank conflict nor another
//           lane's update of the same address, however the values pile up in a few bins.  A counter receives at most
//           32 warps x 2040 elements between two merges, so it cannot carry into its neighbour.
//   copies: 2^L 32-bit counters per bin, copy = lane mod 2^L (L = 0: one privatised copy); for bin counts whose
//           LANE16 form does not fit.  Bin counts that do not fit at all count straight into global memory.
struct HistGeom {
  int lane16;      // 1 = LANE16
  int copies_log2; // otherwise
  int cap_words;   // shared-memory words available
};

// Persistent: the tensors x_t[samples][n_t] of the table lie one behind the other in one flat element order, of which
// block b owns the range [b * piece, (b + 1) * piece).  Sample s of tensor t is histogrammed with its own (threshold
// th[t][s], bins nb[t][s]) and ADDED into the first nb[t][s] entries of the tensor's hist; nb == 0 skips the sample.
// Counters stay in shared memory across samples that share tensor, threshold and bins and are merged into hist when one
// of them changes, before a 16-bit counter could overflow, and at the end.
template <bool LANE16>
__global__ void __launch_bounds__(HIST_THREADS, 1)
histogram_kernel(const CalibTensor* __restrict__ tab, int tensors, int samples, long long total, long long piece,
                 const float* __restrict__ th_all, const int* __restrict__ nb_all, int copies_log2, int cap_words, int zero_words) {
  extern __shared__ unsigned int sh[];
  const int tid = threadIdx.x, lane = tid & 31;
  const long long begin = (long long)blockIdx.x * piece;
  const long long end = begin + piece < total ? begin + piece : total;
  if (begin >= end) return;
  for (int i = tid; i < zero_words; i += HIST_THREADS) sh[i] = 0u;
  __syncthreads();

  int cur_bins = 0;            // geometry of the counters now in shared memory (0: none)
  int* hist = nullptr;         // where they belong
  uint32_t cur_th = 0;
  bool cur_shared = false;
  long long since_merge = 0;
  const int lcopy = lane & ((1 << copies_log2) - 1);

  auto merge = [&]() {
    if (cur_bins == 0 || !cur_shared) return;
    __syncthreads();
    // counters are indexed by k; numpy.histogram puts k into bin k or, by its float32 bin edges, into bin k + 1
    const float cur_binsf = (float)cur_bins;
    const double cur_step = (double)(cur_bins - 1) / (double)cur_bins;
    if (LANE16) {
      const int pairs = (cur_bins + 1) >> 1;
      for (int p = tid; p < pairs; p += HIST_THREADS) {
        unsigned lo = 0, hi = 0;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
          const int w = p * 32 + ((j + lane) & 31);
          const unsigned v = sh[w];
          sh[w] = 0u;
          lo += v & 0xffffu;
          hi += v >> 16;
        }
        if (lo) atomicAdd(&hist[numpy_bin((float)(2 * p), cur_bins, cur_binsf, cur_step)], (int)lo);
        if (hi) atomicAdd(&hist[numpy_bin((float)(2 * p + 1), cur_bins, cur_binsf, cur_step)], (int)hi);
      }
    } else {
      const int R = 1 << copies_log2;
      for (int b = tid; b < cur_bins; b += HIST_THREADS) {
        unsigned c = 0;
        for (int j = 0; j < R; ++j) {
          const int w = (b << copies_log2) + ((j + lane) & (R - 1));
          c += sh[w];
          sh[w] = 0u;
        }
        if (c) atomicAdd(&hist[numpy_bin((float)b, cur_bins, cur_binsf, cur_step)], (int)c);
      }
    }
    __syncthreads();
    since_merge = 0;
  };

  long long pos = begin;
  int t = find_tensor(tab, tensors, begin, false);
  while (pos < end) {
    while (t + 1 < tensors && pos >= tab[t + 1].first) ++t;
    const long long n = tab[t].n, first = tab[t].first;
    const float* const x = tab[t].x - first;   // indexed by flat position
    const long long s = (pos - first) / n;
    long long seg_end = first + (s + 1) * n < end ? first + (s + 1) * n : end;
    const int bins = nb_all[(long long)t * samples + s];
    if (bins <= 0) {
      pos = seg_end;
      continue;
    }
    const float thv = th_all[(long long)t * samples + s];
    if (bins != cur_bins || __float_as_uint(thv) != cur_th || tab[t].hist != hist) {
      merge();
      hist = tab[t].hist;
      cur_bins = bins;
      cur_th = __float_as_uint(thv);
      cur_shared = LANE16 ? (((bins + 1) >> 1) * 32 <= cap_words) : (((long long)bins << copies_log2) <= cap_words);
    }
    if (LANE16 && cur_shared) {
      // elements one thread can add to its lane's counters in this segment (float4 body + scalar head and tail)
      long long per_thread = (((seg_end - pos) >> 2) + HIST_THREADS - 1) / HIST_THREADS * 4 + 14;
      if (per_thread > HIST_MERGE_EVERY) {
        seg_end = pos + HIST_FLUSH_ELEMS;
        per_thread = ((HIST_FLUSH_ELEMS >> 2) + HIST_THREADS - 1) / HIST_THREADS * 4 + 14;
      }
      if (since_merge + per_thread > HIST_MERGE_EVERY) merge();
      since_merge += per_thread;
    }
    const bool shared_now = cur_shared;
    const float binsf = (float)bins;
    const uint32_t top = (uint32_t)(bins - 1);
    const float width = __fdiv_rn(thv, (float)(bins - 1));
    const double step = (double)(bins - 1) / (double)bins;
    // t / width, correctly rounded, without a division per element: with r = RN(1/width), q0 = RN(t*r),
    // rem = t - q0*width (exact in an FMA) and q = RN(q0 + rem*r) is the correctly rounded quotient (Markstein) unless
    // width's significand is all ones; that case, and widths whose reciprocal is not a normal number, divide.
    const float rw = __frcp_rn(width);
    const uint32_t wbits = __float_as_uint(width);
    const bool quick = (wbits & 0x007fffffu) != 0x007fffffu && width >= 1e-30f && width <= 1e30f;
    const uint32_t sh_base = static_cast<uint32_t>(__cvta_generic_to_shared(sh));
    // Per element, branch-free: quotient, k = floor(q + 0.5) as the low mantissa bits of a float, two comparisons,
    // one predicated shared-memory reduction.  FLOOR_MAGIC is folded into the comparison and into the address
    // (arithmetic modulo 2^32).  Shared counters are indexed by k itself; numpy's float32-edge rule, which sends
    // some k to bin k + 1, depends on k alone and is applied when the counters are merged.
    const uint32_t k_limit = FLOOR_MAGIC + top;   // largest valid bit pattern
    const uint32_t lane16_bias = sh_base + (uint32_t)lane * 4u - FLOOR_MAGIC * 64u;
    const uint32_t copies_bias = sh_base + (uint32_t)lcopy * 4u - ((FLOOR_MAGIC << copies_log2) << 2);
    const uint32_t copies_mul = 4u << copies_log2;
    auto run = [&](auto quick_tag, auto shared_tag) {
      constexpr bool QUICK = decltype(quick_tag)::value;
      constexpr bool SHARED = decltype(shared_tag)::value;
      auto one = [&](float v) {
        const float t = fabsf(v);
        float q;
        if (QUICK) {
          const float q0 = __fmul_rn(t, rw);
          q = __fmaf_rn(__fmaf_rn(-q0, width, t), rw, q0);
        } else {
          q = __fdiv_rn(t, width);
        }
        // k = floor(RN(q + 0.5)): adding 2^23 with rounding toward minus infinity leaves floor(y) in the low mantissa
        // bits for 0 <= y < 2^23; larger y (and infinity) give bit patterns above every valid bin and are dropped,
        // like values outside range=(0, bins-1) in numpy.histogram.  Zeros are excluded (cali_math.py:70); a NaN
        // fails t > 0 too.
        const uint32_t ub = __float_as_uint(__fadd_rd(__fadd_rn(q, 0.5f), 8388608.0f));
        if (!SHARED) {
          if (t > 0.f && ub <= k_limit) atomicAdd(&hist[numpy_bin((float)(ub - FLOOR_MAGIC), bins, binsf, step)], 1);
        } else {
          const uint32_t addr = LANE16 ? (ub & ~1u) * 64u + lane16_bias : ub * copies_mul + copies_bias;
          const uint32_t inc = LANE16 ? (ub & 1u) * 65535u + 1u : 1u;
          asm volatile(
              "{\n\t"
              ".reg .pred p, q;\n\t"
              "setp.gt.f32 q, %2, 0f00000000;\n\t"
              "setp.le.and.u32 p, %3, %4, q;\n\t"
              "@p red.shared.add.u32 [%0], %1;\n\t"
              "}\n" ::"r"(addr), "r"(inc), "f"(t), "r"(ub), "r"(k_limit)
              : "memory");
        }
      };
      // the segment [pos, seg_end) of the flat array: scalars up to a 16-byte boundary, float4 body, scalar tail
      const float* p = x + pos;
      const long long len = seg_end - pos;
      long long head = (long long)((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) >> 2;
      if (head > len) head = len;
      if (tid < head) one(p[tid]);
      const long long body4 = (len - head) >> 2;
      const float4* p4 = reinterpret_cast<const float4*>(p + head);
      // three float4 per thread per step, the next step's loads requested before this step's values are counted
      // (positions past the end read as zeros, which the histogram ignores)
      const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
      long long i = tid;
      float4 c0 = i < body4 ? __ldcs(p4 + i) : zero4;
      float4 c1 = i + HIST_THREADS < body4 ? __ldcs(p4 + i + HIST_THREADS) : zero4;
      float4 c2 = i + 2 * HIST_THREADS < body4 ? __ldcs(p4 + i + 2 * HIST_THREADS) : zero4;
      for (; i < body4; i += 3 * HIST_THREADS) {
        const long long j = i + 3 * HIST_THREADS;
        const float4 n0 = j < body4 ? __ldcs(p4 + j) : zero4;
        const float4 n1 = j + HIST_THREADS < body4 ? __ldcs(p4 + j + HIST_THREADS) : zero4;
        const float4 n2 = j + 2 * HIST_THREADS < body4 ? __ldcs(p4 + j + 2 * HIST_THREADS) : zero4;
        one(c0.x); one(c0.y); one(c0.z); one(c0.w);
        one(c1.x); one(c1.y); one(c1.z); one(c1.w);
        one(c2.x); one(c2.y); one(c2.z); one(c2.w);
        c0 = n0; c1 = n1; c2 = n2;
      }
      const long long done = head + body4 * 4;
      if (done + tid < len) one(p[done + tid]);
    };
    if (quick) {
      if (shared_now) run(std::true_type{}, std::true_type{});
      else run(std::true_type{}, std::false_type{});
    } else {
      if (shared_now) run(std::false_type{}, std::true_type{});
      else run(std::false_type{}, std::false_type{});
    }
    pos = seg_end;
  }
  merge();
}

// real_multi_thread_kl_diversity's own histogram (calibration_math.cpp:229-236): every value counts,
// index = floor(fabs(x) / width + 0.5) with the + 0.5 in double.
__global__ void kl_raw_histogram_kernel(const float* __restrict__ x, long long n, float width, int bins, int* hist) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double k = floor((double)__fdiv_rn(fabsf(x[i]), width) + 0.5);
    if (k >= 0.0 && k < (double)bins) atomicAdd(&hist[(long long)k], 1);
  }
}

// out[i] = in[2i] + in[2i+1] (missing entries are zero), i < n_out: one folding step of find_threshold
__global__ void fold_kernel(const int* __restrict__ in, long long n_in, int* __restrict__ out, long long n_out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_out) return;
  const long long a = 2 * i, b = 2 * i + 1;
  out[i] = (a < n_in ? in[a] : 0) + (b < n_in ? in[b] : 0);
}

// ------------------------------------------------------------------------------------------- KLD
// One warp per candidate threshold i = (m+1)*BINS.  Every float sum runs in the reference's order (sequential, left to
// right) because the counts exceed 2^24 and float addition is not associative; the log10 terms are formed in double and
// folded into a float accumulator like the reference.  What can be done in any order is spread over the lanes: the two
// long sums run side by side on two lanes, the bins' sums and logarithms on 32, and of the divergence itself only the
// chain acc = (float)(acc + term) is serial (one conversion, one double addition and one conversion per non-empty bin).
// 73 histograms of 2048 to 3000 bins: 1690 us with one thread per candidate, dominated by two log10 calls per bin in a
// row, 157 us this way.
constexpr int KLD_WARPS = 16;
constexpr int KLD_SMEM_BINS = 40 * 1024;   // histograms up to this length are read from shared memory
constexpr int KLD_QLOG = 128;              // bins whose logarithms a warp keeps; with more (the calibration uses 128 and 8) every
                                           // element works out its bin's

struct KldWarp {
  double qlog[KLD_QLOG];
};

__global__ void __launch_bounds__(KLD_WARPS * 32)
kld_kernel(const KldTensor* __restrict__ tab, int BINS, float* __restrict__ kl_all, int smem_bins) {
  extern __shared__ __align__(16) uint8_t kld_smem[];
  KldWarp* const per_warp = reinterpret_cast<KldWarp*>(kld_smem);
  int* const sh = reinterpret_cast<int*>(kld_smem + KLD_WARPS * sizeof(KldWarp));
  const int t = blockIdx.x;
  const int N = tab[t].len, n_in = tab[t].n_in;
  const int* __restrict__ gh = tab[t].hist;
  const int KL_NUM = N / BINS;
  if ((int)blockIdx.y * KLD_WARPS >= KL_NUM) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool in_smem = N <= smem_bins;
  __shared__ long long scount[KLD_WARPS];
  long long c = 0;   // total count (exact, int64)
  for (int j = threadIdx.x; j < N; j += KLD_WARPS * 32) {
    const int h = j < n_in ? gh[j] : 0;
    if (in_smem) sh[j] = h;
    c += h;
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (lane == 0) scount[warp] = c;
  __syncthreads();
  long long count = 0;
  for (int w = 0; w < KLD_WARPS; ++w) count += scount[w];
  const float fcount = (float)count;
  auto H = [&](int j) { return in_smem ? sh[j] : (j < n_in ? __ldg(gh + j) : 0); };

  const int m = (int)blockIdx.y * KLD_WARPS + warp;
  if (m >= KL_NUM) return;
  const int expand = m + 1, i = expand * BINS;
  // lane 0: P's sum, hist[0 .. i-1]; lane 1: P[i-1], hist[i-1 .. N-1]; both left to right
  float chain = 0.f;
  {
    const int from = lane == 0 ? 0 : i - 1, to = lane == 0 ? i : (lane == 1 ? N : 0);
    int j = from;
    for (; j + 8 <= to; j += 8) {
      int v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = H(j + k);
#pragma unroll
      for (int k = 0; k < 8; ++k) chain = __fadd_rn(chain, (float)v[k]);
    }
    for (; j < to; ++j) chain = __fadd_rn(chain, (float)H(j));
  }
  const float sum = __shfl_sync(0xffffffffu, chain, 0), tail = __shfl_sync(0xffffffffu, chain, 1);
  double* const qlog = per_warp[warp].qlog;
  const bool kept = BINS <= KLD_QLOG;
  auto q_log = [&](int b) {
    float sum_bin = 0.f;
    int positive = 0;
    for (int k = 0; k < expand; ++k) {
      const int h = H(b * expand + k);
      sum_bin = __fadd_rn(sum_bin, (float)h);
      positive += h > 0;
    }
    const float q = __fdiv_rn(__fdiv_rn(sum_bin, positive ? (float)positive : 1.f), sum);
    return log10(__dadd_rn((double)q, 1e-30));
  };
  if (kept)
    for (int b = lane; b < BINS; b += 32) qlog[b] = q_log(b);
  __syncwarp();
  const double qlog0 = log10(__dadd_rn(0.0, 1e-30));
  float acc = 0.f;
  for (int base = 0; base < i; base += 32) {   // BINS is a multiple of 8: i need not be one of 32
    const int idx = base + lane;
    const int h = idx < i ? H(idx) : 0;
    const float p = idx < i ? __fdiv_rn(idx == i - 1 ? tail : (float)h, fcount) : 0.f;
    double term = 0.0;
    if (p != 0.f)
      term = __dmul_rn((double)p, __dsub_rn(log10(__dadd_rn((double)p, 1e-30)), !h ? qlog0 : (kept ? qlog[idx / expand] : q_log(idx / expand))));
    // p == 0: the term is exactly +-0 and leaves the accumulator unchanged
    unsigned live = __ballot_sync(0xffffffffu, p != 0.f);
    if (live == 0xffffffffu) {
#pragma unroll
      for (int k = 0; k < 32; ++k) acc = (float)__dadd_rn((double)acc, __shfl_sync(0xffffffffu, term, k));
    } else {
      while (live) {
        const int k = __ffs((int)live) - 1;
        live &= live - 1;
        acc = (float)__dadd_rn((double)acc, __shfl_sync(0xffffffffu, term, k));
      }
    }
  }
  if (lane == 0) kl_all[(long long)t * 1024 + m] = acc;
}

// the_min_index (calibration_math.cpp:71-83): first strict minimum
__global__ void __launch_bounds__(128)
kld_argmin_kernel(const KldTensor* __restrict__ tab, int BINS, const float* __restrict__ kl_all, float* __restrict__ thresholds) {
  __shared__ float skl[1024];
  const int t = blockIdx.x, KL_NUM = tab[t].len / BINS;
  for (int k = threadIdx.x; k < KL_NUM; k += 128) skl[k] = kl_all[(long long)t * 1024 + k];
  __syncthreads();
  if (threadIdx.x == 0) {
    float best = skl[0];
    int best_m = 0;
    for (int k = 1; k < KL_NUM; ++k)
      if (best > skl[k]) {
        best = skl[k];
        best_m = k;
      }
    thresholds[t] = __fmul_rn(__fmul_rn(tab[t].width, (float)(best_m + 1)), (float)BINS);
  }
}

}  // namespace

size_t minmax_scratch_bytes(long long samples, int blocks_per_sample) {
  return (size_t)samples * blocks_per_sample * 2 * sizeof(float) + (size_t)samples * sizeof(unsigned int);
}

int minmax_blocks_per_sample(long long n, long long samples) {
  long long want = (n + MM_THREADS * 16 - 1) / (MM_THREADS * 16);  // >= 16 float4 per thread... at most
  long long cap = 148LL * 8 / (samples > 0 ? samples : 1);
  if (cap < 1) cap = 1;
  if (want > cap) want = cap;
  if (want < 1) want = 1;
  return (int)want;
}

int minmax_launch(const float* x, long long n, long long samples, float* out, void* scratch, int blocks_per_sample,
                  cudaStream_t s) {
  if (samples == 0) return B200Q_OK;
  if (samples > 65535) return set_error(B200Q_ERR_UNSUPPORTED, "minmax: at most 65535 samples per call");
  float* partial = static_cast<float*>(scratch);
  unsigned int* tickets = reinterpret_cast<unsigned int*>(partial + (size_t)samples * blocks_per_sample * 2);
  dim3 grid(blocks_per_sample, (unsigned)samples);
  minmax_kernel<<<grid, MM_THREADS, 0, s>>>(x, n, out, partial, tickets);
  CUDA_TRY(cudaGetLastError());
  return B200Q_OK;
}


// ------------------------------------------------------------------------------------------- min/max without allocation
// Scratch of the min/max kernel for callers that must not allocate: a fixed array that lives in the module
// image of every GPU that loads this library (36 KB per GPU, held until the process exits).
// Layout: [STATIC_MM_MAX_SAMPLES ticket counters][STATIC_MM_MAX_PARTIALS {min, max} pairs].
constexpr int STATIC_MM_MAX_SAMPLES = 1024;
constexpr int STATIC_MM_MAX_PARTIALS = 4096;
constexpr size_t STATIC_MM_TICKET_BYTES = STATIC_MM_MAX_SAMPLES * sizeof(unsigned int);
constexpr size_t STATIC_MM_BYTES = STATIC_MM_TICKET_BYTES + (size_t)STATIC_MM_MAX_PARTIALS * 2 * sizeof(float);
static __device__ __align__(256) unsigned char g_static_minmax_scratch[STATIC_MM_BYTES];

constexpr int MAX_DEVICES = 64;
static std::atomic<void*> g_static_scratch_addr[MAX_DEVICES];  // device address of the array, per device ordinal

// In host code the array's name is only a handle for the runtime, not a device address: the address a
// kernel can use comes from cudaGetSymbolAddress, asked once per device with that device current.
int static_scratch_for_current_device(void** out) {
  int dev = -1;
  CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES) return set_error(B200Q_ERR_UNSUPPORTED, "minmax_static: device ordinal %d not supported", dev);
  // Threads that make their first call on a device at the same time each ask the runtime and store the same
  // answer; the atomic makes that harmless.  (The cache does not survive a cudaDeviceReset of that device.)
  void* p = g_static_scratch_addr[dev].load(std::memory_order_acquire);
  if (!p) {
    cudaError_t e = cudaGetSymbolAddress(&p, g_static_minmax_scratch);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetSymbolAddress(g_static_minmax_scratch)", __FILE__, __LINE__);
    if (!p) return set_error(B200Q_ERR_CUDA, "minmax_static: the scratch symbol has no device address");
    g_static_scratch_addr[dev].store(p, std::memory_order_release);
  }
  *out = p;
  return B200Q_OK;
}

int minmax_static_launch(const float* x, long long n, long long samples, float* out, cudaStream_t s) {
  if (samples == 0) return B200Q_OK;
  if (samples > STATIC_MM_MAX_SAMPLES)
    return set_error(B200Q_ERR_UNSUPPORTED, "minmax_static: %lld samples exceed the fixed scratch (at most %d per call)",
                     samples, STATIC_MM_MAX_SAMPLES);
  int bps = minmax_blocks_per_sample(n, samples);
  if ((long long)bps * samples > STATIC_MM_MAX_PARTIALS) bps = (int)(STATIC_MM_MAX_PARTIALS / samples);
  if (bps < 1) bps = 1;
  void* base = nullptr;
  B200Q_TRY(static_scratch_for_current_device(&base));
  unsigned int* tickets = static_cast<unsigned int*>(base);
  float* partial = reinterpret_cast<float*>(static_cast<unsigned char*>(base) + STATIC_MM_TICKET_BYTES);
  // the array keeps whatever the previous call left: the ticket counters must start at zero
  CUDA_TRY(cudaMemsetAsync(tickets, 0, (size_t)samples * sizeof(unsigned int), s));
  dim3 grid(bps, (unsigned)samples);
  minmax_kernel<<<grid, MM_THREADS, 0, s>>>(x, n, out, partial, tickets);
  CUDA_TRY(cudaGetLastError());
  return B200Q_OK;
}

static int g_hist_mode = -1;  // -1: chosen per launch; 0..4: 2^mode copies; 5: lane-owned 16-bit counters
void histogram_set_mode(int mode) { g_hist_mode = (mode >= 0 && mode <= 5) ? mode : -1; }

int histogram_launch(const CalibTensor* tab_dev, int tensors, long long samples, long long total, const float* th, const int* nb,
                     int max_bins, cudaStream_t s) {
  if (samples == 0 || total == 0) return B200Q_OK;
  int dev = 0, sms = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // one block per SM; a block's piece is a multiple of one float4 per thread and at least 16 of them
  const long long quantum = 4LL * HIST_THREADS;
  long long blocks = (total + 16 * quantum - 1) / (16 * quantum);
  if (blocks > sms) blocks = sms;
  if (blocks < 1) blocks = 1;
  long long piece = (total + blocks - 1) / blocks;
  piece = (piece + quantum - 1) / quantum * quantum;
  blocks = (total + piece - 1) / piece;
  const int cap_words = HIST_SMEM_BYTES / 4;
  const long long lane16_words = (long long)((max_bins + 1) / 2) * 32;
  // Chosen layout: four copies per bin.  Measured on 64 x 802 816 normal values, 2048 bins: one copy 41.9 us, four
  // 42.2 us, sixteen 43.7 us, lane-owned 16-bit counters 46.3 us (two more instructions per element cost more than the
  // conflicts they avoid); on 64 x 100 352 values four copies are the fastest (20.0 us).  Copies also keep skewed data
  // (everything in a few bins) from serialising on one address.  Fewer copies when the bins do not fit, or when a
  // block would spend more than a quarter of its element count clearing and summing counters.  (max_bins is the largest
  // bin count of the call that fits at all; a sample with more bins than that counts straight into global memory.)
  int mode = g_hist_mode;
  if (mode < 0) {
    mode = 2;
    while (mode > 0 && (((long long)max_bins << mode) > cap_words || ((long long)max_bins << mode) * 4 > piece)) --mode;
  }
  if (mode == 5 && lane16_words > cap_words) mode = 0;
  while (mode > 0 && mode < 5 && ((long long)max_bins << mode) > cap_words) --mode;
  long long zero_words = mode == 5 ? lane16_words : ((long long)max_bins << mode);
  if (zero_words > cap_words) zero_words = 0;  // nothing fits: every sample counts into global memory
  const size_t smem = (size_t)(zero_words > 0 ? zero_words : 1) * 4;
  auto kfn = mode == 5 ? histogram_kernel<true> : histogram_kernel<false>;
  CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, HIST_SMEM_BYTES));
  kfn<<<(unsigned)blocks, HIST_THREADS, smem, s>>>(tab_dev, tensors, (int)samples, total, piece, th, nb, mode == 5 ? 0 : mode,
                                                   (int)zero_words, (int)zero_words);
  CUDA_TRY(cudaGetLastError());
  return B200Q_OK;
}

int histogram_max_shared_bins() { return HIST_SMEM_BYTES / 4; }

long long minmax_many_chunks(long long n, long long samples) { return (n + MANY_CHUNK - 1) / MANY_CHUNK * samples; }

// out_min must hold all ones and out_max zeros; see minmax_many_kernel
int minmax_many_launch(const CalibTensor* tab_dev, int tensors, long long samples, long long chunks, uint32_t* out_min, uint32_t* out_max,
                       cudaStream_t s) {
  if (chunks == 0) return B200Q_OK;
  if (chunks > 0x7fffffffLL) return set_error(B200Q_ERR_UNSUPPORTED, "minmax: too many elements for one call");
  minmax_many_kernel<<<(unsigned)chunks, MM_THREADS, 0, s>>>(tab_dev, tensors, (int)samples, out_min, out_max);
  CUDA_TRY(cudaGetLastError());
  return B200Q_OK;
}

int kl_raw_histogram_launch(const float* x, long long n, float width, int bins, int* hist, cudaStream_t s) {
  if (n == 0) return B200Q_OK;
  long long blocks = (n + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  kl_raw_histogram_kernel<<<(unsigned)blocks, 256, 0, s>>>(x, n, width, bins, hist);
  CUDA_TRY(cudaGetLastError());
  return B200Q_OK;
}

int fold_launch(const int* in, long long n_in, int* out, long long n_out, cudaStream_t s) {
  if (n_out == 0) return B200Q_OK;
  fold_kernel<<<(unsigned)((n_out + 255) / 256), 256, 0, s>>>(in, n_in, out, n_out);
  CUDA_TRY(cudaGetLastError());
  return B200Q_OK;
}

int kld_launch(const KldTensor* tab_dev, int tensors, int dst_bins, long long max_len, float* thresholds_dev, float* kl_dev, cudaStream_t s) {
  if (tensors == 0) return B200Q_OK;
  if (dst_bins < 1 || max_len / dst_bins > 1024)
    return set_error(B200Q_ERR_UNSUPPORTED, "kld: more than 1024 candidates (fold the histogram to at most %d bins first)", 1024 * dst_bins);
  const int smem_bins = max_len < KLD_SMEM_BINS ? (int)max_len : KLD_SMEM_BINS;
  const size_t smem = KLD_WARPS * sizeof(KldWarp) + (size_t)smem_bins * 4;
  CUDA_TRY(cudaFuncSetAttribute(kld_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(KLD_WARPS * sizeof(KldWarp) + KLD_SMEM_BINS * 4)));
  const dim3 grid((unsigned)tensors, (unsigned)((max_len / dst_bins + KLD_WARPS - 1) / KLD_WARPS));
  kld_kernel<<<grid, KLD_WARPS * 32, smem, s>>>(tab_dev, dst_bins, kl_dev, smem_bins);
  CUDA_TRY(cudaGetLastError());
  kld_argmin_kernel<<<tensors, 128, 0, s>>>(tab_dev, dst_bins, kl_dev, thresholds_dev);
  CUDA_TRY(cudaGetLastError());
  return B200Q_OK;
}

}  // namespace b200q
