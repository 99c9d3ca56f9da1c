// fp32 convolution of the Top dialect on the tensor cores: every fp32 operand as the sum of three bf16 numbers.
//
// A float splits exactly into hi + mid + lo (6, 8 and 8 significant bits, round to nearest), a product of two such sums into
// nine bf16 products that are exact in fp32.  Eight of them are multiplied; the ninth, lo*lo, is below 2^-30 of the product.
// The tensor core adds 16 products and its fp32 accumulator exactly and then cuts the sum off at 24 bits.  What that loses has
// the sign of the sum, so that it would add up over a network's layers; three things keep it small:
//   - no accumulator lives longer than 64 products deep: the epilogue warps take it out of tensor memory after every 64 k and
//     add it to their own fp32 sum, rounded to nearest;
//   - hi*hi has an accumulator of its own, so that it does not cut off the low bits of the seven smaller products;
//   - hi has 6 bits instead of the 8 that bf16 holds: a product of 12 bits loses nothing until it is 2^-12 of the sum.
// Sums that are exact in fp32 stay exact (integers, one-hot filters).  Against 64-bit sums the result is closer than a serial
// chain of fp32 FMAs: relative error (2-norm) 2.9e-8 to 9.9e-8 over ResNet-50's layers where the CUDA-core kernel has 1.0e-7
// to 3.1e-7, mean error in the sum's own direction 3e-9 to 4e-9 (4.8e-8 with 8-bit hi parts in one accumulator, 2.7e-8 in two,
// 5e-9 with an accumulator for every 16 k, which is slower); whole network 3.2e-7 against 8.0e-7.
//
// A k chunk of 64 costs 32 MMAs of 128 x BN x 16, an eighth of the bf16 rate: about 200 TFLOP/s of fp32 products where the
// CUDA cores have 74.  Measured at batch 32: 3x3 128 channels 28x28 203 -> 74 us (100 TFLOP/s), 3x3 256 channels 14x14 196 ->
// 67 us, 3x3 64 channels 56x56 285 -> 101 us, 1x1 64 to 256 channels 103 -> 54 us.  Two kernels per call:
//   split_f32_kernel   NCHW fp32 -> three bf16 planes [rows][channels].  Stride 1: rows are the pixels of the padded image,
//                      and the rows of a filter tap are the same rows shifted (one TMA box per tap, no im2col).  Other
//                      strides: rows are the output pixels, one channel run per tap.  10 bytes moved per element.
//   conv_f32_umma_kernel   persistent, one CTA per SM, tiles of 128 rows x BN channels; warp 0 loads (one 3-D box per operand
//                      and chunk carries the three planes), warp 1 issues the MMAs, the others add up and store NCHW fp32.
// Images are taken a group at a time so that the planes stay in the L2 between the two kernels.
//
// Three things are recomputed by a plain FMA loop over the fp32 operands, which gives what the CUDA-core kernel gives: infinities
// and NaN, sums that overflow, and results that underflow may have touched.  The last is decided from the operands: the split
// kernels note the smallest and largest exponents of every 32 rows and of every channel (see `may_be_lost`).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "igemm.h"
#include "internal.h"
#include "ptx_sm100.cuh"
#include "top_f32.h"

namespace b200q {
namespace {

constexpr int TILE_M = 128;                    // rows per CTA
constexpr int CHUNK = 64;                      // k per accumulator: one 128-byte row of bf16
constexpr int PARTS = 2;                       // accumulators of a chunk: the seven small products, hi * hi
constexpr int CHUNK_BYTES = CHUNK * 2;
constexpr int A_STAGES = 2;
constexpr int MAX_SHARE = 3;

// BN: channels of a tile.  PAIR: two CTAs of a cluster compute 256 rows x BN channels (tcgen05 cta_group::2); each loads its
// own 128 rows of A and half of B.
template <int BN, bool PAIR>
struct UmmaLayout {
  static constexpr int BUFS = BN == 256 ? 2 : 4;                 // accumulators in tensor memory: hides the hand-over
  static constexpr int TMEM_COLS = BUFS * BN;
  static constexpr int B_ROWS = PAIR ? BN / 2 : BN;
  static constexpr int B_STAGES = B_ROWS == 128 ? 2 : 4;
  static constexpr int A_PLANE = (TILE_M + 8) * CHUNK_BYTES;     // up to MAX_SHARE - 1 extra rows; 1024-byte multiple
  static constexpr int B_PLANE = B_ROWS * CHUNK_BYTES;
  static constexpr int A_BYTES = 3 * A_PLANE;
  static constexpr int B_BYTES = 3 * B_PLANE;
  static constexpr int B_OFFSET = A_STAGES * A_BYTES;
  static constexpr int BAR_OFFSET = B_OFFSET + B_STAGES * B_BYTES;
  static constexpr int MISC_OFFSET = BAR_OFFSET + (2 * A_STAGES + 2 * B_STAGES + 2 * BUFS + 1) * 8;
  static constexpr int DYN_BYTES = MISC_OFFSET + 16 + 1024;      // slack for the manual 1024-byte alignment
  static constexpr int EPI_WARPS = BN == 64 ? 8 : 16;
  static constexpr int EPI_COLS = BN * 4 / EPI_WARPS;            // a warp: 32 rows x 32 channels (64 at BN = 256)
  static constexpr int THREADS = 96 + 32 * EPI_WARPS;
};

// x = h + m + l, h rounded to nearest to 6 significant bits, m and l to bf16's 8: 18 bits are left for m, 9 of them and a sign
// (or 2^8) for l.  Exact for every float whose low part is not subnormal.  (An infinity and a NaN leave a NaN in m, and values
// that round to an infinite h do too: their sums are recomputed.)
__device__ __forceinline__ void split3(float x, uint16_t& h, uint16_t& m, uint16_t& l) {
  const uint32_t hb = (__float_as_uint(x) + 0x20000u) & 0xfffc0000u;
  const float r1 = x - __uint_as_float(hb);
  const __nv_bfloat16 bm = __float2bfloat16_rn(r1);
  const float r2 = r1 - __bfloat162float(bm);
  h = (uint16_t)(hb >> 16);
  m = __bfloat16_as_ushort(bm);
  l = __bfloat16_as_ushort(__float2bfloat16_rn(r2));
}

// Exponents (biased) of a set of values: largest << 16 | smallest of the non-zero ones.
constexpr uint32_t NO_VALUE = 511;             // "smallest" of a set of zeros
constexpr int RANGE_ROWS = 32;                 // rows that share a range

// (a NaN is left out: what it touches is NaN and recomputed for that)
__device__ __forceinline__ void range_add(float v, float& largest, uint32_t& smallest) {
  largest = fmaxf(largest, fabsf(v));
  smallest = min(smallest, __float_as_uint(v) * 2u - 1u);   // drops the sign; zero wraps round to the largest number
}
__device__ __forceinline__ uint32_t range_pack(float largest, uint32_t smallest) {   // over the warp
  const uint32_t l = __reduce_max_sync(0xffffffffu, __float_as_uint(largest));
  smallest = __reduce_min_sync(0xffffffffu, smallest);
  return ((l >> 23) << 16) | (smallest == 0xffffffffu ? NO_VALUE : (smallest + 1u) >> 24);
}
__device__ __forceinline__ uint32_t range_join(uint32_t a, uint32_t b) {
  return max(a & 0xffff0000u, b & 0xffff0000u) | min(a & 0xffffu, b & 0xffffu);
}

// A sum of `k` products from operands of the given ranges: 0 if underflow cannot have touched it, else the magnitude from
// which on it does not matter.  Nothing is lost while every part is a normal bf16 (the lowest bit of an operand is 2^-23 of its
// leading one: exponents from -102) and every product of operands is at least 2^-90 (what its smallest parts lose is below
// 2^-33 of it).  Otherwise a product can lose 3 * 2^-126 of either operand and eight parts of 2^-126: the sum is off by at most
// k * 2^-124 * (max|x| + max|w| + 2), which is 2^-26 of a result of this size, a quarter of an fp32 rounding.
__device__ __forceinline__ float may_be_lost(uint32_t x, uint32_t w, float k) {
  const uint32_t xs = x & 0xffffu, ws = w & 0xffffu;
  if (xs == NO_VALUE || ws == NO_VALUE || (xs >= 25u && ws >= 25u && xs + ws >= 164u)) return 0.f;
  return k * 0x1p-98f * (ldexpf(1.f, (int)(x >> 16) - 126) + ldexpf(1.f, (int)(w >> 16) - 126) + 2.f);
}

struct SplitArgs {
  int ic, ih, iw;          // input image
  int rh, rw;              // rows of one image: rh x rw
  int sh, sw, dh, dw, pht, pwl, kw;
  int cp;                  // channels per tap, rounded up to 8
  long long rows;          // images x rh x rw
  long long pitch;         // elements per row: taps (of this form) x cp
  uint32_t* range;         // [tap][64 channels][32 rows]
};

// One block: 32 rows x 64 channels of one tap.  Memory bound (4 bytes read, 6 written per element): a warp reads 32
// neighbouring pixels of eight channels, the block turns them in shared memory and writes 128-byte channel runs.
__global__ void __launch_bounds__(256) split_f32_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ out, const SplitArgs a) {
  __shared__ __align__(16) uint16_t tile[3][32][CHUNK + 8];
  __shared__ uint32_t ranges[8];
  ptx::griddep_launch_dependents();   // the second kernel may set itself up meanwhile; it waits for this one's end
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = blockIdx.y * CHUNK + warp * 8;
  const int tap = blockIdx.z, fy = tap / a.kw, fx = tap - fy * a.kw;
  const long long row = (long long)blockIdx.x * 32 + lane;
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = 0.f;
  if (row < a.rows) {
    const int per = a.rh * a.rw;
    const int n = (int)(row / per), r = (int)(row - (long long)n * per);
    const int ra = r / a.rw, rb = r - ra * a.rw;
    const int h = ra * a.sh + fy * a.dh - a.pht, w = rb * a.sw + fx * a.dw - a.pwl;
    if ((unsigned)h < (unsigned)a.ih && (unsigned)w < (unsigned)a.iw) {
      const int hw = a.ih * a.iw;
      const float* src = x + ((long long)n * a.ic + c0) * hw + (long long)h * a.iw + w;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c0 + i < a.ic) v[i] = __ldg(src + (long long)i * hw);
    }
  }
  float largest = 0.f;
  uint32_t smallest = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < 8; ++i) range_add(v[i], largest, smallest);
  const uint32_t range = range_pack(largest, smallest);
  if (lane == 0) ranges[warp] = range;
  uint32_t p[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint16_t h0, m0, l0, h1, m1, l1;
    split3(v[2 * i], h0, m0, l0);
    split3(v[2 * i + 1], h1, m1, l1);
    p[0][i] = (uint32_t)h0 | ((uint32_t)h1 << 16);
    p[1][i] = (uint32_t)m0 | ((uint32_t)m1 << 16);
    p[2][i] = (uint32_t)l0 | ((uint32_t)l1 << 16);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q)
    *reinterpret_cast<uint4*>(&tile[q][lane][warp * 8]) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t all = ranges[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) all = range_join(all, ranges[i]);
    a.range[((long long)tap * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = all;
  }
  const int rr = threadIdx.x >> 3, piece = (threadIdx.x & 7) * 8;
  const long long orow = (long long)blockIdx.x * 32 + rr;
  const int c = blockIdx.y * CHUNK + piece;
  if (orow < a.rows && c < a.cp) {
    __nv_bfloat16* dst = out + orow * a.pitch + (long long)tap * a.cp + c;
#pragma unroll
    for (int q = 0; q < 3; ++q)
      *reinterpret_cast<uint4*>(dst + q * a.rows * a.pitch) = *reinterpret_cast<const uint4*>(&tile[q][rr][piece]);
  }
}

// OIHW fp32 -> planes [3][oc][tap][cp], once per handle
__global__ void split_weight_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ out, int oc, int ic, int taps, int cp) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)oc * taps * cp;
  if (i >= total) return;
  const int c = (int)(i % cp);
  const long long r = i / cp;
  const int t = (int)(r % taps), o = (int)(r / taps);
  uint16_t h, m, l;
  split3(c < ic ? w[((long long)o * ic + c) * taps + t] : 0.f, h, m, l);
  out[i] = __ushort_as_bfloat16(h);
  out[total + i] = __ushort_as_bfloat16(m);
  out[2 * total + i] = __ushort_as_bfloat16(l);
}

// Exponents of every output channel's weights, once per handle: one block per channel
__global__ void __launch_bounds__(128) weight_range_kernel(const float* __restrict__ w, uint32_t* __restrict__ range, long long per_channel) {
  __shared__ uint32_t ranges[4];
  const float* src = w + blockIdx.x * per_channel;
  float largest = 0.f;
  uint32_t smallest = 0xffffffffu;
  for (long long i = threadIdx.x; i < per_channel; i += 128) range_add(src[i], largest, smallest);
  const uint32_t r = range_pack(largest, smallest);
  if ((threadIdx.x & 31) == 0) ranges[threadIdx.x >> 5] = r;
  __syncthreads();
  if (threadIdx.x == 0) range[blockIdx.x] = range_join(range_join(ranges[0], ranges[1]), range_join(ranges[2], ranges[3]));
}

struct UmmaArgs {
  TopConvPlan p;             // n: the images of this launch
  // k is walked in units of (tap group, 64 channels); a unit is `share` chunks, the taps of one filter row on one load of A
  int share, taps_w;         // taps_w: tap groups per filter row (1 when share covers it)
  int tap_h, tap_w;          // rows between vertically / horizontally adjacent taps
  int units_per_tap, tap_k;  // units of one tap group; k (elements) between taps in the weight
  int one_row;               // a row holds all taps one after the other (tap groups: one)
  int cp;
  int rh, rw;                // rows of one image; output pixel (h, w) is row h * rw + w
  int rows, m_tiles, n_tiles, units, splits, units_per_split;
  uint32_t idesc;
  const float* x;
  const float* wt;           // [K][oc], k = (c, kh, kw): the recomputation's operand
  const float* bias;
  float* y;                  // splits > 1: planes of partial sums
  long long plane;           // floats of one plane
  const uint32_t* x_range;   // [x_groups][x_blocks], x_blocks of 32 rows each
  const uint32_t* w_range;   // [oc]
  float k_total;             // products of one output
  int x_blocks, x_groups, halo;   // halo: rows past a tile's last that its last row's taps reach
  int* status;               // set to the wait site if a bounded wait ran out; the results are not valid then
  unsigned long long wait_budget_ns;
  int expect_extra;          // test aid: bytes a stage's barrier expects beyond what its loads deliver (0 in normal use)
};

// Units [u0, u1) of k as runs of channels of one tap: f(tap, first channel, end), until it returns false
template <typename F>
__device__ __forceinline__ void for_runs(const UmmaArgs& a, int u0, int u1, F f) {
  const int taps = a.p.kh * a.p.kw;
  for (int u = u0; u < u1; ++u) {
    const int group = u / a.units_per_tap, e0 = (u - group * a.units_per_tap) * CHUNK;
    if (!a.one_row) {
      for (int tap = group * a.share; tap < min(taps, (group + 1) * a.share); ++tap)
        if (e0 < a.p.ic && !f(tap, e0, min(e0 + CHUNK, a.p.ic))) return;
    } else {
      const int end = min(e0 + CHUNK, taps * a.cp);
      for (int e = e0; e < end;) {
        const int tap = e / a.cp, c = e - tap * a.cp, n = min(end - e, a.cp - c);
        if (c < a.p.ic && !f(tap, c, min(c + n, a.p.ic))) return;
        e += n;
      }
    }
  }
}

// Results of a warp's rows (`row` is this lane's) in 32 channels from `co` on, by fp32 FMAs: `again` has this lane's.  Four channels at a time from one value of x, so that a layer full of infinities costs a few times what the
// CUDA-core kernel takes for it; a group of four leaves off when nothing but NaN is left.
__device__ __noinline__ void recompute(const UmmaArgs& a, int row, int co, int split, uint32_t again) {
  const TopConvPlan& p = a.p;
  const int per = a.rh * a.rw, img = row / per, rem = row - img * per, h = rem / a.rw, w = rem - h * a.rw;
  const bool valid = row < a.rows && h < p.oh && w < p.ow;
  const long long hw = (long long)p.ih * p.iw, w_step = (long long)p.kh * p.kw * p.oc;
  const int u0 = split * a.units_per_split, u1 = min(a.units, u0 + a.units_per_split);
  const bool partial = a.splits > 1;
  float* const out = a.y + (partial ? split * a.plane : 0) + ((long long)img * p.oc + co) * p.oh * p.ow + h * p.ow + w;
  const float ceiling = p.relu_limit > 0.f ? p.relu_limit : INFINITY;
  if (!valid) again = 0u;
  if (p.oc - co < 32) again &= (1u << max(p.oc - co, 0)) - 1u;
  uint32_t columns = __reduce_or_sync(0xffffffffu, again);
  while (columns != 0u) {
    int col[4];   // the next four channels (the last one again where fewer are left)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      col[q] = columns != 0u ? __ffs((int)columns) - 1 : col[q > 0 ? q - 1 : 0];
      columns &= columns - 1u;
    }
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    for_runs(a, u0, u1, [&](int tap, int c0, int c1) {
      const int fy = tap / p.kw, fx = tap - fy * p.kw;
      const int y = h * p.sh + fy * p.dh - p.pht, x = w * p.sw + fx * p.dw - p.pwl;
      const bool inside = valid && (unsigned)y < (unsigned)p.ih && (unsigned)x < (unsigned)p.iw;   // the border is zeros: 0 * inf is NaN
      const float* xp = a.x + (inside ? (((long long)img * p.ic + c0) * p.ih + y) * p.iw + x : 0);
      const float* wp = a.wt + c0 * w_step + (long long)tap * p.oc + co;
#pragma unroll 4
      for (int c = c0; c < c1; ++c, wp += w_step) {
        const float xv = inside ? __ldg(xp) : 0.f;
        if (inside) xp += hw;
#pragma unroll
        for (int q = 0; q < 4; ++q) s[q] = fmaf(__ldg(wp + col[q]), xv, s[q]);
      }
      return !__all_sync(0xffffffffu, !valid || (s[0] != s[0] && s[1] != s[1] && s[2] != s[2] && s[3] != s[3]));
    });
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float v = s[q] + (a.bias && !partial ? __ldg(a.bias + co + col[q]) : 0.f);
      if (!partial && p.do_relu) v = fminf(fmaxf(v, 0.f), ceiling);
      if ((again >> col[q]) & 1u) out[(long long)col[q] * p.oh * p.ow] = v;
    }
  }
}

// Waits until the phase is complete, but not for long: what is on its way here arrives within microseconds.
__device__ __forceinline__ void drain(uint32_t bar, uint32_t parity) {
  const uint64_t t0 = ptx::globaltimer_ns();
  while (!ptx::mbar_try_wait_hint(bar, parity, 20000u) && ptx::globaltimer_ns() - t0 < 200000u) {}
}

template <int BN, bool PAIR>
__global__ void __launch_bounds__(UmmaLayout<BN, PAIR>::THREADS, 1)
conv_f32_umma_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ UmmaArgs args) {
  using L = UmmaLayout<BN, PAIR>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t smem_base = ptx::smem_u32(smem);
  const uint32_t bar_base = smem_base + L::BAR_OFFSET;
  auto full_a = [&](int s) { return bar_base + 8u * s; };
  auto empty_a = [&](int s) { return bar_base + 8u * (A_STAGES + s); };
  auto full_b = [&](int s) { return bar_base + 8u * (2 * A_STAGES + s); };
  auto empty_b = [&](int s) { return bar_base + 8u * (2 * A_STAGES + L::B_STAGES + s); };
  auto tmem_full_bar = [&](int b) { return bar_base + 8u * (2 * A_STAGES + 2 * L::B_STAGES + b); };
  auto tmem_empty_bar = [&](int b) { return bar_base + 8u * (2 * A_STAGES + 2 * L::B_STAGES + L::BUFS + b); };
  const uint32_t mma_done_bar = bar_base + 8u * (2 * A_STAGES + 2 * L::B_STAGES + 2 * L::BUFS);   // used after a wait ran out
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem + L::MISC_OFFSET);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::MISC_OFFSET + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? ptx::cluster_ctarank() : 0u;      // CTA 0 leads: its barriers count both CTAs' loads
  const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  constexpr int CTAS = PAIR ? 2 : 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < A_STAGES; ++s) {
      ptx::mbar_init(full_a(s), 1);
      ptx::mbar_init(empty_a(s), 1);
    }
    for (int s = 0; s < L::B_STAGES; ++s) {
      ptx::mbar_init(full_b(s), 1);
      ptx::mbar_init(empty_b(s), 1);
    }
    for (int b = 0; b < L::BUFS; ++b) {
      ptx::mbar_init(tmem_full_bar(b), 1);
      ptx::mbar_init(tmem_empty_bar(b), CTAS * L::EPI_WARPS);
    }
    ptx::mbar_init(mma_done_bar, 1);
    *abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async_smem();
    ptx::prefetch_tensormap(&tmap_a);
    ptx::prefetch_tensormap(&tmap_b);
  }
  if (PAIR) {
    __syncthreads();
    ptx::cluster_sync_all();   // the peer's barriers exist before anything can signal them
  }
  if (warp == 1) {
    if (PAIR) {
      ptx::tmem_alloc_pair(ptx::smem_u32(tmem_ptr_smem), L::TMEM_COLS);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(ptx::smem_u32(tmem_ptr_smem), L::TMEM_COLS);
      ptx::tmem_relinquish();
    }
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  const int tiles = args.m_tiles * args.n_tiles * args.splits;
  const int share = args.share;

  if (warp == 0 || warp == 2) {
    // ---- loaders: warp 0 the activations, warp 2 the weights (each runs as far ahead as its own ring allows)
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      if (warp == 0) ptx::griddep_wait();   // the planes are the previous kernel's output; the weights are not
      for (int tile = worker; tile < tiles && ok; tile += workers) {
        const int nt = tile % args.n_tiles, r = tile / args.n_tiles;
        const int mt = r % args.m_tiles, split = r / args.m_tiles;
        const int u0 = split * args.units_per_split, u1 = min(args.units, u0 + args.units_per_split);
        int group = u0 / args.units_per_tap, kc = u0 - group * args.units_per_tap;
        for (int u = u0; u < u1 && ok; ++u) {
          if (warp == 0) {
            ok = ptx::mbar_wait_bounded_fast<20>(empty_a(stage), phase ^ 1u, abort_flag, 1, args.wait_budget_ns);
            if (!ok) break;
            const int fy = group / args.taps_w, fx = group - fy * args.taps_w;
            const int row = mt * (CTAS * TILE_M) + (int)rank * TILE_M + fy * args.tap_h + fx * args.tap_w;
            const uint32_t sa = smem_base + stage * L::A_BYTES;
            if (rank == 0) ptx::mbar_arrive_expect_tx(full_a(stage), CTAS * 3 * (TILE_M + share - 1) * CHUNK_BYTES + args.expect_extra);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
              if (PAIR) ptx::tma_load_3d_pair(sa + q * L::A_PLANE, &tmap_a, ptx::map_to_cta(full_a(stage), 0), kc * CHUNK_BYTES, row, q);
              else ptx::tma_load_3d(sa + q * L::A_PLANE, &tmap_a, full_a(stage), kc * CHUNK_BYTES, row, q);
            }
            if (++stage == A_STAGES) {
              stage = 0;
              phase ^= 1u;
            }
          } else {
            for (int t = 0; t < share; ++t) {
              ok = ptx::mbar_wait_bounded_fast<20>(empty_b(stage), phase ^ 1u, abort_flag, 2, args.wait_budget_ns);
              if (!ok) break;
              const int col = (group * share + t) * args.tap_k * 2 + kc * CHUNK_BYTES;
              const uint32_t sb = smem_base + L::B_OFFSET + stage * L::B_BYTES;
              if (rank == 0) ptx::mbar_arrive_expect_tx(full_b(stage), CTAS * L::B_BYTES);
              if (PAIR) ptx::tma_load_3d_pair(sb, &tmap_b, ptx::map_to_cta(full_b(stage), 0), col, nt * BN + (int)rank * L::B_ROWS, 0);
              else ptx::tma_load_3d(sb, &tmap_b, full_b(stage), col, nt * BN, 0);
              if (++stage == L::B_STAGES) {
                stage = 0;
                phase ^= 1u;
              }
            }
          }
          if (++kc == args.units_per_tap) {
            kc = 0;
            ++group;
          }
        }
      }
      if (!ok && rank == 0) {
        // a wait ran out: do not leave while copies of this pair may still be on their way (stages from `stage` on were last
        // filled in the phase before)
        const int stages = warp == 0 ? A_STAGES : L::B_STAGES;
        for (int i = 0; i < stages; ++i) drain(warp == 0 ? full_a(i) : full_b(i), i < stage ? phase : phase ^ 1u);
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      int sa = 0, sb = 0, buf = 0;
      uint32_t pa = 0, pb = 0, buf_phase = 0;
      bool ok = true;
      const uint64_t desc0 = ptx::make_smem_desc_kmajor(smem_base, 1024, 2);
      const uint32_t hi = (uint32_t)(desc0 >> 32), a_lo0 = (uint32_t)desc0;
      const uint32_t b_lo0 = (uint32_t)ptx::make_smem_desc_kmajor(smem_base + L::B_OFFSET, 1024, 2);
      constexpr uint32_t AP = L::A_PLANE >> 4, BP = L::B_PLANE >> 4;   // descriptor address units of 16 bytes
      auto mma = [&](uint32_t d, uint32_t al, uint32_t bl, uint32_t first) {
        if (PAIR) ptx::umma_kblock_f16_pair(d, al, bl, hi, hi, args.idesc, first);
        else ptx::umma_kblock_f16(d, al, bl, hi, hi, args.idesc, first);
      };
      auto commit = [&](uint32_t bar) {
        if (PAIR) ptx::umma_commit_pair(bar, 3);
        else ptx::umma_commit(bar);
      };
      for (int tile = worker; tile < tiles && ok; tile += workers) {
        const int split = tile / args.n_tiles / args.m_tiles;
        const int u0 = split * args.units_per_split, u1 = min(args.units, u0 + args.units_per_split);
        for (int u = u0; u < u1 && ok; ++u) {
          ok = ptx::mbar_wait_bounded_fast<20>(full_a(sa), pa, abort_flag, 3, args.wait_budget_ns);
          for (int t = 0; t < share && ok; ++t) {
            ok = ptx::mbar_wait_bounded_fast<20>(full_b(sb), pb, abort_flag, 5, args.wait_budget_ns);
            // tap t reads the block from row t on: the swizzle follows the address bits, only the start moves
            const uint32_t al = a_lo0 + (uint32_t)(sa * (L::A_BYTES >> 4) + t * (CHUNK_BYTES >> 4));
            const uint32_t bl = b_lo0 + (uint32_t)(sb * (L::B_BYTES >> 4));
#pragma unroll
            for (int part = 0; part < PARTS && ok; ++part) {
              ok = ptx::mbar_wait_bounded_fast<20>(tmem_empty_bar(buf), buf_phase ^ 1u, abort_flag, 4, args.wait_budget_ns);
              if (!ok) break;
              ptx::tc_fence_after_sync();
              const uint32_t d = tmem_base + (uint32_t)(buf * BN);
              if (part == 0) {                           // the small products, the smallest first
                mma(d, al + AP, bl + 2 * BP, 0u);        // mid * lo
                mma(d, al + 2 * AP, bl + BP, 1u);        // lo * mid
                mma(d, al, bl + 2 * BP, 1u);             // hi * lo
                mma(d, al + 2 * AP, bl, 1u);             // lo * hi
                mma(d, al + AP, bl + BP, 1u);            // mid * mid
                mma(d, al, bl + BP, 1u);                 // hi * mid
                mma(d, al + AP, bl, 1u);                 // mid * hi
              } else {
                mma(d, al, bl, 0u);                      // hi * hi
                commit(empty_b(sb));
                if (t == share - 1) commit(empty_a(sa));
              }
              commit(tmem_full_bar(buf));
              if (++buf == L::BUFS) {
                buf = 0;
                buf_phase ^= 1u;
              }
            }
            if (++sb == L::B_STAGES) {
              sb = 0;
              pb ^= 1u;
            }
          }
          if (++sa == A_STAGES) {
            sa = 0;
            pa ^= 1u;
          }
        }
      }
      if (!ok) {   // nor while products are being written to the tensor memory that is freed below
        if (PAIR) ptx::umma_commit_pair(mma_done_bar, 1);
        else ptx::umma_commit(mma_done_bar);
        drain(mma_done_bar, 0u);
      }
    }
  } else {
    const int quarter = warp & 3;                 // a warp reads the tensor-memory lanes of its number mod 4
    const int col0 = ((warp - 3) >> 2) * L::EPI_COLS;
    const TopConvPlan& p = args.p;
    const int ohow = p.oh * p.ow;
    const uint32_t lead_empty0 = PAIR ? ptx::map_to_cta(tmem_empty_bar(0), 0) : 0u;
    const uint32_t t_warp = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)col0;
    int buf = 0;
    uint32_t buf_phase = 0;
    bool ok = true;
    ptx::griddep_wait();   // before the first write of the output
    for (int tile = worker; tile < tiles; tile += workers) {
      const int nt = tile % args.n_tiles, r = tile / args.n_tiles;
      const int mt = r % args.m_tiles, split = r / args.m_tiles;
      const int u0 = split * args.units_per_split, u1 = min(args.units, u0 + args.units_per_split);
      const int row = mt * (CTAS * TILE_M) + (int)rank * TILE_M + quarter * 32 + lane;
      const int per = args.rh * args.rw;
      const int img = row / per, rem = row - img * per;
      const int h = rem / args.rw, w = rem - h * args.rw;
      const int co0 = nt * BN + col0;
      const bool partial = args.splits > 1;
      float bias[L::EPI_COLS / 32];               // lane j holds channel j's; handed round when the results are stored
#pragma unroll
      for (int i = 0; i < L::EPI_COLS / 32; ++i)
        bias[i] = (args.bias && co0 + i * 32 + lane < p.oc) ? __ldg(args.bias + co0 + i * 32 + lane) : 0.f;
      // ranges of the rows this warp's taps read (lane by lane) and of its channels; first looked at after the sums
      uint32_t x_range = NO_VALUE, w_range[L::EPI_COLS / 32];
      {
        const int row0 = min(row - lane, args.rows - 1), b0 = row0 / RANGE_ROWS;
        const int nb = min(row0 + 31 + args.halo, args.rows - 1) / RANGE_ROWS - b0 + 1;
        for (int i = lane; i < nb * args.x_groups; i += 32) {
          const int gr = i / nb;
          const uint32_t v = __ldcg(args.x_range + (long long)gr * args.x_blocks + b0 + (i - gr * nb));
          x_range = i < 32 ? v : range_join(x_range, v);
        }
      }
#pragma unroll
      for (int i = 0; i < L::EPI_COLS / 32; ++i) w_range[i] = co0 + i * 32 + lane < p.oc ? __ldg(args.w_range + co0 + i * 32 + lane) : NO_VALUE;
      float acc[L::EPI_COLS];
#pragma unroll
      for (int j = 0; j < L::EPI_COLS; ++j) acc[j] = 0.f;
      const int sums = (u1 - u0) * share * PARTS;
      for (int q = 0; q < sums && ok; ++q) {
        ok = __all_sync(0xffffffffu, ptx::mbar_wait_bounded_fast<20>(tmem_full_bar(buf), buf_phase, abort_flag, 6, args.wait_budget_ns));
        if (!ok) break;
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int part = 0; part < L::EPI_COLS / 16; ++part) {
          uint32_t v[16];
          ptx::tmem_ld_32x32b_x16(t_warp + (uint32_t)(buf * BN + part * 16), v);
          ptx::tmem_ld_wait_16(v);
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[part * 16 + j] += __uint_as_float(v[j]);
        }
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) ptx::mbar_arrive_cluster_relaxed(lead_empty0 + 8u * buf);
          else ptx::mbar_arrive_relaxed(tmem_empty_bar(buf));
        }
        if (++buf == L::BUFS) {
          buf = 0;
          buf_phase ^= 1u;
        }
      }
      const bool valid = row < args.rows && h < p.oh && w < p.ow;
      const int ncols = min(L::EPI_COLS, p.oc - co0);
      float* const out0 = args.y + (partial ? split * args.plane : 0) + ((long long)img * p.oc + co0) * ohow + h * p.ow + w;
      const bool relu = !partial && p.do_relu;
      const float ceiling = p.relu_limit > 0.f ? p.relu_limit : INFINITY;
      x_range = (__reduce_max_sync(0xffffffffu, x_range >> 16) << 16) | __reduce_min_sync(0xffffffffu, x_range & 0xffffu);
      uint32_t again[L::EPI_COLS / 32];           // results to recompute
      float* o = out0;
#pragma unroll
      for (int i = 0; i < L::EPI_COLS / 32; ++i) {
        again[i] = 0u;
        float lost = may_be_lost(x_range, w_range[i], args.k_total);   // lane j: channel j's
        if (fabsf(bias[i]) >= lost) lost = 0.f;     // the bias swallows it (a dead channel: weights near zero, any bias)
        if (partial) bias[i] = 0.f;                 // added with the partial sums
        if (__any_sync(0xffffffffu, lost > 0.f)) {
          for (int j = 0; j < 32; ++j) {
            const float from = __shfl_sync(0xffffffffu, lost, j);
            float s = 0.f;
#pragma unroll
            for (int q = 0; q < 32; ++q) s = q == j ? acc[i * 32 + q] : s;   // (rare: no indexing of registers)
            if (fabsf(s) < from) again[i] |= 1u << j;
          }
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float s = acc[i * 32 + j];
          if (!(fabsf(s) <= 3.402823466e38f)) again[i] |= 1u << j;
          const float v = s + __shfl_sync(0xffffffffu, bias[i], j);
          if (valid && i * 32 + j < ncols) *o = relu ? fminf(fmaxf(v, 0.f), ceiling) : v;
          o += ohow;
          asm volatile("" : "+l"(o));   // one running address: 64 of them kept ahead spilled the sums
        }
      }
      // the rare ones, and everything if a wait ran out (the sums are lost: NaN, and the status word)
#pragma unroll
      for (int i = 0; i < L::EPI_COLS / 32; ++i) {
        if (!ok) {
          for (int j = i * 32; valid && j < min(i * 32 + 32, ncols); ++j) out0[(long long)j * ohow] = __int_as_float(0x7fffffff);
        } else if (__any_sync(0xffffffffu, valid && again[i] != 0u)) {
          recompute(args, row, co0 + i * 32, split, again[i]);
        }
      }
    }
  }
  if (PAIR && *abort_flag != 0) ptx::st_shared_cluster_u32(ptx::map_to_cta(ptx::smem_u32((const void*)abort_flag), rank ^ 1u), (uint32_t)*abort_flag);
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && args.status != nullptr) atomicCAS(args.status, 0, *abort_flag);
  if (PAIR) ptx::cluster_sync_all();   // neither CTA frees tensor memory or exits while the other can still signal or read it
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    if (PAIR) ptx::tmem_dealloc_pair(tmem_base, L::TMEM_COLS);
    else ptx::tmem_dealloc(tmem_base, L::TMEM_COLS);
  }
}

// Form of the rows: stride 1 -> the padded image (taps are shifted rows); anything else -> output pixels with all taps
bool shifted_rows(const TopConvPlan& p) { return p.sh == 1 && p.sw == 1; }

int cp_of(const TopConvPlan& p) { return (p.ic + 7) & ~7; }

size_t image_bytes(const TopConvPlan& p) {
  const size_t taps = (size_t)p.kh * p.kw, cp = cp_of(p);
  if (shifted_rows(p)) return 6 * cp * (size_t)(p.oh + (p.kh - 1) * p.dh) * (p.ow + (p.kw - 1) * p.dw);
  return 6 * cp * taps * (size_t)p.oh * p.ow;
}

size_t image_rows(const TopConvPlan& p) {
  return shifted_rows(p) ? (size_t)(p.oh + (p.kh - 1) * p.dh) * (p.ow + (p.kw - 1) * p.dw) : (size_t)p.oh * p.ow;
}

size_t scratch_plane_bytes(const TopConvPlan& p, int images) { return ((size_t)images * image_bytes(p) + 1023) & ~(size_t)1023; }

size_t scratch_range_bytes(const TopConvPlan& p, int images) {
  const size_t blocks = (images * image_rows(p) + RANGE_ROWS - 1) / RANGE_ROWS;
  const size_t groups = (size_t)((cp_of(p) + CHUNK - 1) / CHUNK) * (shifted_rows(p) ? 1 : p.kh * p.kw);
  return (blocks * groups * sizeof(uint32_t) + 1023) & ~(size_t)1023;
}

// Planes of one group of images: half of the L2, so that the second kernel finds what the first one wrote
constexpr size_t GROUP_BYTES = 64u << 20;

int group_images(const TopConvPlan& p) {
  const size_t per = image_bytes(p);
  long long g = (long long)(GROUP_BYTES / per);
  if (g < 1) g = 1;
  if (g >= p.n) return p.n;
  const long long groups = (p.n + g - 1) / g;
  return (int)((p.n + groups - 1) / groups);
}

struct UmmaChoice {
  int bn, splits, m_tiles, n_tiles, units, share;
  bool pair;
};

// Tile form and K splits of a launch over `images` images, by a model in nanoseconds.  A chunk costs what its operands cost
// to bring in (75 bytes per ns and SM, measured) or its 32 MMAs, whichever is more.  These read both operands from shared
// memory, which sets their pace (128 bytes per clock: 62 clocks measured at 256 x 128 x 16 where the tensor pipe needs 32), so
// that 256 channels cost little more than 128.  A round of tiles costs its chunks, or its stores, plus 1.5 us for the
// pipeline's start; partial sums cost a launch and a pass over the output's planes.
UmmaChoice choose(const TopConvPlan& p, int images, int sms) {
  const bool shifted = shifted_rows(p);
  const long long rows = shifted ? (long long)images * (p.oh + (p.kh - 1) * p.dh) * (p.ow + (p.kw - 1) * p.dw) : (long long)images * p.oh * p.ow;
  const int taps = p.kh * p.kw, cp = cp_of(p);
  UmmaChoice best{};
  best.share = shifted && p.kw == MAX_SHARE && p.dw == 1 ? MAX_SHARE : 1;
  best.units = shifted ? taps / best.share * ((cp + CHUNK - 1) / CHUNK) : (int)(((long long)taps * cp + CHUNK - 1) / CHUNK);
  double best_cost = -1;
  for (int form = 0; form < 4; ++form) {   // 128 x 64, 128 x 128, 256 x 128 (pair), 256 x 256 (pair)
    const int bn = form == 0 ? 64 : (form == 3 ? 256 : 128);
    const bool pair = form >= 2;
    if (bn > 64 && p.oc <= bn / 2) break;
    const int tile_m = pair ? 2 * TILE_M : TILE_M;
    const int m_tiles = (int)((rows + tile_m - 1) / tile_m), n_tiles = (p.oc + bn - 1) / bn;
    const double bytes = 3.0 * CHUNK_BYTES * ((double)TILE_M / best.share + (pair ? bn / 2 : bn));
    const double mma = bn == 64 ? 800 : (bn == 128 ? 1070 : 1470), chunk = bytes / 75.0 > mma ? bytes / 75.0 : mma;
    const double store = TILE_M * bn * 4.0 / 20.0;
    for (int sp = 1; sp <= 8 && sp <= best.units; ++sp) {
      const long long tiles = (long long)m_tiles * n_tiles * sp, slots = pair ? sms / 2 : sms;
      const double k_time = (best.units + sp - 1) / sp * best.share * chunk;
      double cost = (double)((tiles + slots - 1) / slots) * ((k_time > store ? k_time : store) + 1500.0);
      if (sp > 1) cost += 3000.0 + (2.0 * sp + 1) * 4.0 * images * p.oc * p.oh * p.ow / 5000.0;
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        best.bn = bn;
        best.pair = pair;
        best.splits = sp;
        best.m_tiles = m_tiles;
        best.n_tiles = n_tiles;
      }
    }
  }
  return best;
}

template <int BN, bool PAIR>
int launch_umma(const CUtensorMap& ta, const CUtensorMap& tb, const UmmaArgs& a, int sms, cudaStream_t s) {
  using L = UmmaLayout<BN, PAIR>;
  auto kfn = conv_f32_umma_kernel<BN, PAIR>;
  CUDA_TRY(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, L::DYN_BYTES));
  const long long tiles = (long long)a.m_tiles * a.n_tiles * a.splits, slots = PAIR ? sms / 2 : sms;
  const unsigned workers = (unsigned)(tiles < slots ? tiles : slots);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(PAIR ? 2 * workers : workers);
  cfg.blockDim = dim3(L::THREADS);
  cfg.dynamicSmemBytes = L::DYN_BYTES;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = PAIR ? 2 : 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  CUDA_TRY(cudaLaunchKernelEx(&cfg, kfn, ta, tb, a));
  return B200Q_OK;
}

}  // namespace

// the planes, then the channels' ranges
size_t weight_plane_bytes(const TopConvPlan& p) { return ((size_t)3 * 2 * p.oc * p.kh * p.kw * cp_of(p) + 255) & ~(size_t)255; }
size_t top_conv_umma_weight_bytes(const TopConvPlan& p) { return weight_plane_bytes(p) + (size_t)p.oc * sizeof(uint32_t); }

bool top_conv_umma_takes(const TopConvPlan& p) {
  if (p.groups != 1 || p.ic < 32 || p.oc < 32) return false;
  const long long Hp = p.oh + (long long)(p.kh - 1) * p.dh, Wp = p.ow + (long long)(p.kw - 1) * p.dw;
  const long long taps = (long long)p.kh * p.kw;
  const long long rows = shifted_rows(p) ? Hp * Wp : (long long)p.oh * p.ow;
  const long long k = taps * cp_of(p);
  return rows * 2 < (1ll << 30) && k < (1 << 24) && (shifted_rows(p) || taps <= 65535) && image_bytes(p) <= (size_t)1 << 30 && p.oc < (1 << 24);
}

int top_conv_umma_prepare(const TopConvPlan& p, const float* w_oihw, void* planes, cudaStream_t s) {
  const int taps = p.kh * p.kw, cp = cp_of(p);
  const long long total = (long long)p.oc * taps * cp;
  split_weight_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(w_oihw, static_cast<__nv_bfloat16*>(planes), p.oc, p.ic, taps, cp);
  CUDA_TRY(cudaGetLastError());
  weight_range_kernel<<<(unsigned)p.oc, 128, 0, s>>>(w_oihw, reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(planes) + weight_plane_bytes(p)),
                                                     (long long)p.ic * taps);
  CUDA_TRY(cudaGetLastError());
  return B200Q_OK;
}

// The scratch a call needs: the planes of one group of images and their ranges, then the partial sums of one group (if it
// splits K).
size_t top_conv_umma_scratch(const TopConvPlan& p, int sms) {
  const int g = group_images(p);
  const UmmaChoice c = choose(p, g, sms);
  size_t need = scratch_plane_bytes(p, g) + scratch_range_bytes(p, g);
  if (c.splits > 1) need += (size_t)c.splits * g * p.oc * p.oh * p.ow * 4;
  return need;
}

int top_conv_umma_launch(const TopConvPlan& plan, const float* x, const float* wt, const void* w_planes, const float* bias, float* y,
                         void* scratch, int* status, int sms, cudaStream_t s) {
  const int g = group_images(plan), cp = cp_of(plan), taps = plan.kh * plan.kw;
  const bool shifted = shifted_rows(plan);
  const UmmaChoice c = choose(plan, g, sms);
  const size_t plane_bytes = scratch_plane_bytes(plan, g);
  uint32_t* const range = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(scratch) + plane_bytes);
  float* partial = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + plane_bytes + scratch_range_bytes(plan, g));
  for (int i0 = 0; i0 < plan.n; i0 += g) {
    TopConvPlan p = plan;
    p.n = plan.n - i0 < g ? plan.n - i0 : g;
    const float* xg = x + (size_t)i0 * p.ic * p.ih * p.iw;
    float* yg = y + (size_t)i0 * p.oc * p.oh * p.ow;
    SplitArgs sa{};
    sa.ic = p.ic; sa.ih = p.ih; sa.iw = p.iw; sa.cp = cp; sa.pht = p.pht; sa.pwl = p.pwl;
    sa.dh = p.dh; sa.dw = p.dw; sa.kw = p.kw;
    if (shifted) {
      sa.rh = p.oh + (p.kh - 1) * p.dh; sa.rw = p.ow + (p.kw - 1) * p.dw; sa.sh = sa.sw = 1; sa.pitch = cp;
    } else {
      sa.rh = p.oh; sa.rw = p.ow; sa.sh = p.sh; sa.sw = p.sw; sa.pitch = (long long)taps * cp;
    }
    sa.rows = (long long)p.n * sa.rh * sa.rw;
    sa.range = range;
    dim3 grid((unsigned)((sa.rows + RANGE_ROWS - 1) / RANGE_ROWS), (unsigned)((cp + CHUNK - 1) / CHUNK), (unsigned)(shifted ? 1 : taps));
    split_f32_kernel<<<grid, 256, 0, s>>>(xg, static_cast<__nv_bfloat16*>(scratch), sa);
    CUDA_TRY(cudaGetLastError());

    UmmaArgs a{};
    a.p = p;
    a.cp = cp;
    a.rh = sa.rh; a.rw = sa.rw; a.rows = (int)sa.rows;
    a.share = c.share;
    a.taps_w = shifted ? p.kw / c.share : 1;
    a.tap_h = p.dh * sa.rw; a.tap_w = p.dw;
    a.one_row = shifted ? 0 : 1;
    a.tap_k = shifted ? cp : taps * cp;
    a.units_per_tap = (a.tap_k + CHUNK - 1) / CHUNK;
    a.units = c.units;
    const int tile_m = c.pair ? 2 * TILE_M : TILE_M;
    a.m_tiles = (int)((sa.rows + tile_m - 1) / tile_m);
    a.n_tiles = c.n_tiles;
    a.units_per_split = (a.units + c.splits - 1) / c.splits;
    a.splits = (a.units + a.units_per_split - 1) / a.units_per_split;
    a.idesc = ptx::make_idesc(1u, 1u, 1u, (uint32_t)tile_m, (uint32_t)c.bn);
    a.x = xg; a.wt = wt; a.bias = bias;
    a.plane = (long long)p.n * p.oc * p.oh * p.ow;
    a.y = a.splits > 1 ? partial : yg;
    a.x_range = range;
    a.w_range = reinterpret_cast<const uint32_t*>(static_cast<const uint8_t*>(w_planes) + weight_plane_bytes(p));
    a.x_blocks = (int)grid.x;
    a.x_groups = (int)(grid.y * grid.z);
    a.halo = shifted ? (p.kh - 1) * a.tap_h + (p.kw - 1) * a.tap_w : 0;
    a.k_total = (float)taps * (float)p.ic;
    a.status = status;
    igemm_wait_test(&a.expect_extra, &a.wait_budget_ns);

    CUtensorMap ta, tb;
    {
      const uint64_t dims[3] = {(uint64_t)sa.pitch * 2, (uint64_t)sa.rows, 3};
      const uint64_t st[2] = {(uint64_t)sa.pitch * 2, (uint64_t)sa.rows * sa.pitch * 2};
      const uint32_t box[3] = {CHUNK_BYTES, (uint32_t)(TILE_M + c.share - 1), 1};
      B200Q_TRY(make_tmap_u8(&ta, scratch, 3, dims, st, box));
    }
    {
      const uint64_t k2 = (uint64_t)taps * cp * 2;
      const uint64_t dims[3] = {k2, (uint64_t)p.oc, 3};
      const uint64_t st[2] = {k2, k2 * p.oc};
      const uint32_t box[3] = {CHUNK_BYTES, (uint32_t)(c.pair ? c.bn / 2 : c.bn), 3};
      B200Q_TRY(make_tmap_u8(&tb, w_planes, 3, dims, st, box));
    }
    if (c.bn == 64) B200Q_TRY((launch_umma<64, false>(ta, tb, a, sms, s)));
    else if (!c.pair) B200Q_TRY((launch_umma<128, false>(ta, tb, a, sms, s)));
    else if (c.bn == 128) B200Q_TRY((launch_umma<128, true>(ta, tb, a, sms, s)));
    else B200Q_TRY((launch_umma<256, true>(ta, tb, a, sms, s)));
    if (a.splits > 1)
      B200Q_TRY(top_conv_reduce_launch(partial, bias, yg, a.plane, a.splits, p.oc, p.oh * p.ow, p.do_relu, p.relu_limit, s));
  }
  return B200Q_OK;
}

}  // namespace b200q
