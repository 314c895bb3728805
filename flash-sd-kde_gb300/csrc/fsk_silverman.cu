// fsk_silverman.cu - Silverman bandwidth rules on the GPU.
//
// h = 0.9 * mean_k min(std_k, IQR_k / 1.34) * n^(-1/(d+4))   (FSK_RULE_SILVERMAN)
//   flash_sd_kde/reference.py:171-184 (d-D) and :24-36 (1-D, same formula, d=1)
// h = 0.4 * min(std, IQR / 1.34) * n^(-1/9)                   (FSK_RULE_SDKDE_1D)
//   kernels/flash_sd_kde/empirical.py:328-333
//
// std is the population standard deviation (ddof=0) in FP64, two passes.  The
// 25th/75th percentiles use numpy's default linear interpolation between the order
// statistics floor(p(n-1)) and floor(p(n-1))+1, which are found exactly by a
// 4-pass, 8-bit radix selection on order-preserving integer keys.
//
// Five launches: column sums and the first digits' histogram; deviations and
// the second histogram; two more histograms; the result.  Each kernel finishes
// the previous one's work itself - every block adds up the per-block sums it
// needs and picks the next digit of every order statistic from the previous
// histogram, a warp per statistic - where single-block kernels with one thread
// per statistic scanning 256 bins took 28 us a pass (n = 10007, d = 16: 230 us
// in 14 launches).
#include <math.h>

#include "fsk_kernels.cuh"

namespace fsk {

namespace {
constexpr int SV_MAXD = 64;
constexpr int SV_TARGETS = 4;        // ranks: lo25, hi25, lo75, hi75
constexpr int SV_THREADS = 256;
constexpr int SV_WARPS = SV_THREADS / 32;
constexpr int SV_BLOCKS = 304;
constexpr int SV_BINS = 256;
constexpr int SV_PASSES = 4;
constexpr int SV_SLICE = 48;         // columns per block: 4 x 256 counters each in shared memory

// A selection's state after some digits: the digits chosen so far and the rank
// among the elements that share them.
struct SvPick {
  uint32_t prefix;
  uint32_t rank;
};

struct SvBufs {
  unsigned int* hist;     // [SV_PASSES][d][SV_TARGETS][SV_BINS], cleared before the first kernel
  SvPick* pick;           // [SV_PASSES][d][SV_TARGETS] after 1, 2, ... digits
  double* sum;            // [2][SV_BLOCKS][SV_MAXD] per-block column sums, then squared deviations
};
}  // namespace

// Order-preserving key; positive NaNs come last.  As a xor and not as a choice
// between ~u and u | sign bit: the latter can be compiled to a negation of the
// float, which does not keep a NaN's bits (its key came out as 0x7FFFFFFF, -0).
__device__ __forceinline__ uint32_t sortable_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return u ^ ((uint32_t)((int32_t)u >> 31) | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
  uint32_t u = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
  return __uint_as_float(u);
}

// floor(p (n - 1)) and its successor for p = 1/4, 3/4
__device__ __forceinline__ int64_t target_rank(int64_t n, int t) {
  const int64_t i = t < 2 ? (n - 1) / 4 : (3 * (n - 1)) / 4;
  return (t & 1) ? imin<int64_t>(i + 1, n - 1) : i;
}

// Digit of one statistic from its 256-bin histogram, by one warp holding 8 bins
// per lane: the bin where the running count passes the rank.  RANK: the type of
// ranks and running counts, 64 bits for the first digit of more than 2^32 rows
// (a rank inside one bin fits 32).
template <typename RANK>
__device__ __forceinline__ SvPick pick_digit(uint4 u, uint4 v, uint32_t prefix, RANK rank) {
  const int lane = threadIdx.x & 31;
  const unsigned int c[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
  RANK total = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) total += c[i];
  RANK below = total;   // inclusive scan over lanes
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const RANK w = __shfl_up_sync(0xffffffffu, below, o);
    if (lane >= o) below += w;
  }
  below -= total;
  const bool mine = rank >= below && rank - below < total;
  RANK left = rank - below;
  int bin = 0;
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    const bool past = mine && bin == i && left >= c[i];
    if (past) {
      left -= c[i];
      bin = i + 1;
    }
  }
  const unsigned int who = __ballot_sync(0xffffffffu, mine);
  const int src = who ? __ffs(who) - 1 : 31;
  const uint32_t digit = (uint32_t)__shfl_sync(0xffffffffu, 8 * lane + bin, src);
  return SvPick{(prefix << 8) | digit, (uint32_t)__shfl_sync(0xffffffffu, left, src)};
}

// The selections after `digits` digits of columns [c0, c0 + dc) into shared
// memory, a warp per statistic, from those after one digit less (written by
// the previous kernel) and that kernel's histogram.  `keep`: write them for
// the next kernel.
__device__ __forceinline__ void block_picks(const SvBufs& b, int64_t n, int d, int c0, int dc, int digits, bool keep,
                                            SvPick* pick) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = digits - 1, stats = dc * SV_TARGETS;
  constexpr int U = 4;   // statistics in flight per warp
  for (int s0 = warp * U; s0 < stats; s0 += SV_WARPS * U) {
    uint4 u[U], v[U];
    SvPick p[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const int s = c0 * SV_TARGETS + min(s0 + i, stats - 1);
      // in the first pass all statistics of a column share one histogram
      const int at = q == 0 ? s - s % SV_TARGETS : s;
      const uint4* h = reinterpret_cast<const uint4*>(b.hist + ((int64_t)q * d * SV_TARGETS + at) * SV_BINS) + 2 * lane;
      u[i] = h[0];
      v[i] = h[1];
      p[i] = q == 0 ? SvPick{0u, (uint32_t)target_rank(n, s % SV_TARGETS)}
                    : b.pick[(int64_t)(q - 1) * d * SV_TARGETS + s];
    }
#pragma unroll
    for (int i = 0; i < U; ++i) {
      if (q == 0 && n > 0xffffffffll)
        p[i] = pick_digit<uint64_t>(u[i], v[i], 0u, (uint64_t)target_rank(n, min(s0 + i, stats - 1) % SV_TARGETS));
      else
        p[i] = pick_digit<uint32_t>(u[i], v[i], p[i].prefix, p[i].rank);
      if (lane == 0 && s0 + i < stats) {
        pick[s0 + i] = p[i];
        if (keep) b.pick[(int64_t)q * d * SV_TARGETS + c0 * SV_TARGETS + s0 + i] = p[i];
      }
    }
  }
}

// Column sums of the per-block sums, by all threads of the block: thread t
// adds column t % d of blocks t / d, t / d + rows, ..., thread k < d then its
// column's strided sums, in a fixed order (same bits in every block).
__device__ __forceinline__ double block_column_sum(const double* __restrict__ part, int blocks, int d,
                                                   double (&sh)[SV_THREADS]) {
  const int rows = SV_THREADS / d, k = threadIdx.x % d, l = threadIdx.x / d;
  double s = 0.0;
  if (l < rows) {
#pragma unroll 4
    for (int i = l; i < blocks; i += rows) s += part[(int64_t)i * SV_MAXD + k];
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < d) {
    for (int j = 1; j < rows; ++j) s += sh[j * d + threadIdx.x];
  }
  __syncthreads();
  return s;   // threads below d
}

// Pass 0: column sums; pass 1: squared deviations; all passes: histogram of
// digit `pass` of the elements that match a statistic's earlier digits.
__global__ void __launch_bounds__(SV_THREADS) sv_pass_kernel(const float* __restrict__ x, int64_t n, int d, int pass,
                                                             SvBufs b) {
  extern __shared__ unsigned int hist[];   // [d][SV_TARGETS][SV_BINS] (pass 0: [d][SV_BINS])
  __shared__ SvPick pick[SV_SLICE * SV_TARGETS];
  __shared__ double mean[SV_SLICE];
  __shared__ double sums[SV_THREADS];
  if (pass > 0) pdl_wait();   // (pass 0 follows an ordinary operation)
  pdl_launch_dependents();
  const int c0 = blockIdx.y * SV_SLICE, dc = min(SV_SLICE, d - c0);   // this block's columns
  const int per = pass == 0 ? 1 : SV_TARGETS;
  const int nb = dc * per * SV_BINS;
  for (int i = threadIdx.x; i < nb; i += SV_THREADS) hist[i] = 0u;
  if (pass > 0) block_picks(b, n, d, c0, dc, pass, blockIdx.x == 0, pick);
  if (pass == 1) {
    const double total = block_column_sum(b.sum + c0, gridDim.x, dc, sums);
    if (threadIdx.x < dc) mean[threadIdx.x] = total / (double)n;
  }
  __syncthreads();
  // thread t owns column t % dc of rows t / dc, t / dc + rows, ...
  const int rows = SV_THREADS / dc, k = threadIdx.x % dc, lane_row = threadIdx.x / dc;
  double acc = 0.0;
  if (lane_row < rows) {
    const int shift = 24 - 8 * pass;
    const double mk = pass == 1 ? mean[k] : 0.0;
    uint32_t want[SV_TARGETS];
#pragma unroll
    for (int t = 0; t < SV_TARGETS; ++t) want[t] = pass > 0 ? pick[k * SV_TARGETS + t].prefix : 0u;
    unsigned int* h = hist + k * per * SV_BINS;
    for (int64_t r = (int64_t)blockIdx.x * rows + lane_row; r < n; r += (int64_t)gridDim.x * rows) {
      const float v = x[r * d + c0 + k];
      const uint32_t key = sortable_key(v);
      const uint32_t digit = (key >> shift) & 255u;
      if (pass == 0) {
        atomicAdd(&h[digit], 1u);
        acc += (double)v;
      } else {
        const uint32_t top = key >> (shift + 8);
#pragma unroll
        for (int t = 0; t < SV_TARGETS; ++t)
          if (top == want[t]) atomicAdd(&h[t * SV_BINS + digit], 1u);
        if (pass == 1) {
          const double c = (double)v - mk;
          acc += c * c;
        }
      }
    }
  }
  sums[threadIdx.x] = acc;
  __syncthreads();
  unsigned int* out = b.hist + ((int64_t)pass * d + c0) * SV_TARGETS * SV_BINS;
  for (int i = threadIdx.x; i < nb; i += SV_THREADS) {
    const unsigned int c = hist[i];
    if (c) atomicAdd(&out[pass == 0 ? (i / SV_BINS) * SV_TARGETS * SV_BINS + i % SV_BINS : i], c);
  }
  if (pass < 2 && threadIdx.x < dc) {
    double s = sums[threadIdx.x];
    for (int j = 1; j < rows; ++j) s += sums[j * dc + threadIdx.x];
    b.sum[((int64_t)pass * SV_BLOCKS + blockIdx.x) * SV_MAXD + c0 + threadIdx.x] = s;
  }
}

__global__ void __launch_bounds__(SV_THREADS) sv_finish_kernel(int64_t n, int d, int rule, int blocks, double factor,
                                                               SvBufs b, double* __restrict__ h_out) {
  __shared__ SvPick pick[SV_MAXD * SV_TARGETS];
  __shared__ double sig[SV_MAXD];
  __shared__ double sums[SV_THREADS];
  pdl_wait();
  block_picks(b, n, d, 0, d, SV_PASSES, false, pick);
  const double m2 = block_column_sum(b.sum + (int64_t)SV_BLOCKS * SV_MAXD, blocks, d, sums);
  if (threadIdx.x < d) {
    const int k = threadIdx.x;
    const double sd = sqrt(m2 / (double)n);
    // weights of the upper order statistic: the fraction of p (n - 1)
    const double g25 = 0.25 * (double)((n - 1) % 4), g75 = 0.25 * (double)((3 * (n - 1)) % 4);
    auto lerp = [](double a, double c, double t) {
      const double diff = c - a;
      return t >= 0.5 ? c - diff * (1.0 - t) : a + diff * t;
    };
    const double a25 = key_to_float(pick[k * 4].prefix), b25 = key_to_float(pick[k * 4 + 1].prefix);
    const double a75 = key_to_float(pick[k * 4 + 2].prefix), b75 = key_to_float(pick[k * 4 + 3].prefix);
    sig[k] = fmin(sd, (lerp(a75, b75, g75) - lerp(a25, b25, g25)) / 1.34);
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  double sum = 0.0;
  for (int k = 0; k < d; ++k) sum += sig[k];
  double sigma = sum / (double)d;
  if (rule != FSK_RULE_SDKDE_1D && sigma <= 0.0) sigma = 1.0;
  *h_out = factor * sigma;
}

static SvBufs take_silverman(WsCarver& c, int d) {
  SvBufs b;
  b.hist = c.take<unsigned int>((size_t)SV_PASSES * d * SV_TARGETS * SV_BINS);
  b.pick = c.take<SvPick>((size_t)SV_PASSES * d * SV_TARGETS);
  b.sum = c.take<double>((size_t)2 * SV_BLOCKS * SV_MAXD);
  return b;
}

size_t silverman_ws_bytes(int64_t n, int d) {
  (void)n;
  WsCarver c(nullptr, 0);
  take_silverman(c, d);
  return align_up(c.used, 256);
}

int run_silverman(const float* x, int64_t n, int d, int rule, double* h_out, void* ws, size_t ws_bytes,
                  cudaStream_t s) {
  if (d < 1 || d > SV_MAXD) return FSK_ERR_INVALID_ARGUMENT;
  WsCarver c(ws, ws_bytes);
  const SvBufs b = take_silverman(c, d);
  if (!c.fits()) return FSK_ERR_WORKSPACE_TOO_SMALL;
  const int slices = (d + SV_SLICE - 1) / SV_SLICE;
  const int rows = SV_THREADS / imin(d, SV_SLICE);
  const int blocks = (int)imax<int64_t>(1, imin<int64_t>(SV_BLOCKS, (n + 4 * rows - 1) / (4 * rows)));
  cudaError_t e = cudaMemsetAsync(b.hist, 0, (size_t)SV_PASSES * d * SV_TARGETS * SV_BINS * sizeof(unsigned int), s);
  if (e != cudaSuccess) return cuda_status(e);
  const size_t hsm = (size_t)imin(d, SV_SLICE) * SV_TARGETS * SV_BINS * sizeof(unsigned int);
  if (hsm > 32 * 1024) {
    e = cudaFuncSetAttribute(sv_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hsm);
    if (e != cudaSuccess) return cuda_status(e);
  }
  const dim3 grid((unsigned)blocks, (unsigned)slices);
  sv_pass_kernel<<<grid, SV_THREADS, hsm / SV_TARGETS, s>>>(x, n, d, 0, b);
  count_launch();
  for (int pass = 1; pass < SV_PASSES; ++pass) {
    launch_pdl(sv_pass_kernel, grid, SV_THREADS, hsm, s, x, n, d, pass, b);
    count_launch();
  }
  const double factor = rule == FSK_RULE_SDKDE_1D ? 0.4 * pow((double)n, -1.0 / 9.0)
                                                  : 0.9 * pow((double)n, -1.0 / (double)(d + 4));
  e = launch_pdl(sv_finish_kernel, 1, SV_THREADS, 0, s, n, d, rule, blocks, factor, b, h_out);
  count_launch();
  return e != cudaSuccess ? cuda_status(e) : cuda_status(cudaGetLastError());
}

}  // namespace fsk
