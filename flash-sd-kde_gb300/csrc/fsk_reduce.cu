// fsk_reduce.cu - O(n) kernels: column means for centering, the fixed-order
// cross-split reduction of partial sums with the FP64 normalisation (and
// optional log), the empirical-score reduction, and the SD-KDE debias shift.
// The CUDA-core kernels' partials are FP64, the tensor-core kernels' FP32
// (value, error) pairs, added as double-float (~48 bits).  The split reduction replaces kernels/reduce_partials.py:6-58 (which
// sums splits in FP32); normalisation follows flash_sd_kde/kde.py:93-94,
// :119-122; the debias shift follows flash_sd_kde/kde.py:319-322.
#include "fsk_kernels.cuh"
#include "fsk_tc.cuh"

namespace fsk {

namespace {
constexpr int MEAN_THREADS = 256;
constexpr int MEAN_MAX_BLOCKS = 512;
}  // namespace

size_t mean_scratch_doubles(int64_t n) {
  (void)n;
  return (size_t)MEAN_MAX_BLOCKS * FSK_D;
}

__global__ void __launch_bounds__(MEAN_THREADS) mean16_partial_kernel(const float* __restrict__ x,
                                                                      int64_t n, double* __restrict__ part) {
  // thread layout: 16 features x 16 row lanes
  const int k = threadIdx.x % FSK_D;
  const int lane = threadIdx.x / FSK_D;
  double acc = 0.0;
  for (int64_t r = (int64_t)blockIdx.x * (MEAN_THREADS / FSK_D) + lane; r < n;
       r += (int64_t)gridDim.x * (MEAN_THREADS / FSK_D))
    acc += (double)x[r * FSK_D + k];
  __shared__ double sh[MEAN_THREADS];
  sh[threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.x < FSK_D) {
    double s = 0.0;
    for (int l = 0; l < MEAN_THREADS / FSK_D; ++l) s += sh[l * FSK_D + threadIdx.x];
    part[(int64_t)blockIdx.x * FSK_D + threadIdx.x] = s;
  }
}

// One block of MEAN_THREADS: thread t sums the partials b = t/16, t/16 + 16, ...
// of feature t%16, then each feature's 16 strided sums are added in a fixed
// order (deterministic).
__global__ void __launch_bounds__(MEAN_THREADS) mean16_final_kernel(const double* __restrict__ part, int blocks,
                                                                    int64_t n, float* __restrict__ mu,
                                                                    double* __restrict__ mu64) {
  const int k = threadIdx.x % FSK_D;
  const int l = threadIdx.x / FSK_D;
  constexpr int L = MEAN_THREADS / FSK_D;
  double s = 0.0;
  for (int b = l; b < blocks; b += L) s += part[b * FSK_D + k];
  __shared__ double sh[MEAN_THREADS];
  sh[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < FSK_D) {
    double t = 0.0;
    for (int j = 0; j < L; ++j) t += sh[j * FSK_D + threadIdx.x];
    const float mf = (float)(t / (double)n);
    mu[threadIdx.x] = mf;
    if (mu64) mu64[threadIdx.x] = (double)mf;  // the shift actually applied (exactly representable)
  }
}

void launch_mean16(const float* x, int64_t n, double* scratch, float* mu, double* mu64,
                   cudaStream_t s) {
  int blocks = (int)imin<int64_t>(MEAN_MAX_BLOCKS, (n + 255) / 256);
  blocks = imax(blocks, 1);
  mean16_partial_kernel<<<blocks, MEAN_THREADS, 0, s>>>(x, n, scratch);
  count_launch();
  mean16_final_kernel<<<1, MEAN_THREADS, 0, s>>>(scratch, blocks, n, mu, mu64);
  count_launch();
}

// Cross-split sums with the FP64 normalisation (and log).  RL threads share a
// row (split k goes to thread k % RL) so that a query's few hundred partials
// are not one chain of dependent loads: 49 us for 2048 rows x 300 partials by
// one thread per row, 8-thread rows take the reduction to launch cost.  The
// threads' sums are added in thread order, so the result is deterministic.
constexpr int RED_THREADS = tc::TC_RED_THREADS;
constexpr int RED_LANES = 8;

template <int RL>
__global__ void __launch_bounds__(RED_THREADS) reduce_rows_kernel(const double* __restrict__ partials, int splits,
                                                                  int64_t m, double scale, double eps, int log_out,
                                                                  float* __restrict__ out,
                                                                  const int* __restrict__ skip) {
  if (skip != nullptr && *skip != 0) return;
  constexpr int ROWS = RED_THREADS / RL;
  const int r = threadIdx.x % ROWS, l = threadIdx.x / ROWS;
  for (int64_t i0 = (int64_t)blockIdx.x * ROWS; i0 < m; i0 += (int64_t)gridDim.x * ROWS) {
    const int64_t i = i0 + r;
    double s = 0.0;
    if (i < m) {
#pragma unroll 4
      for (int k = l; k < splits; k += RL) s += partials[(int64_t)k * m + i];
    }
    if (RL > 1) {
      __shared__ double sh[RL][ROWS];
      __syncthreads();   // the rows before are out
      sh[l][r] = s;
      __syncthreads();
      if (l > 0 || i >= m) continue;
#pragma unroll
      for (int j = 1; j < RL; ++j) s += sh[j][r];
    }
    if (i >= m) continue;
    double v = s * scale;
    if (log_out) v = log(v + eps);
    out[i] = (float)v;
  }
}

void launch_reduce_rows(const double* partials, int splits, int64_t m, double scale, double eps,
                        bool log_out, float* out, const int* skip, cudaStream_t s) {
  // one thread per row while the chain is short, or the rows alone fill the
  // GPU (100000 rows x 6 splits: 4 us more with 8 threads per row); where the
  // launch may turn out to have nothing to do, no more blocks than fit at once
  // (32768 that return at once take 19 us)
  const bool single = splits <= 4 || (splits <= 32 && m >= 65536);
  const int rows = single ? RED_THREADS : RED_THREADS / RED_LANES;
  int64_t blocks = (m + rows - 1) / rows;
  if (skip != nullptr) blocks = imin<int64_t>(blocks, 8LL * sm_count());
  if (single)
    reduce_rows_kernel<1><<<(unsigned)blocks, RED_THREADS, 0, s>>>(partials, splits, m, scale, eps, log_out ? 1 : 0, out, skip);
  else
    reduce_rows_kernel<RED_LANES><<<(unsigned)blocks, RED_THREADS, 0, s>>>(partials, splits, m, scale, eps, log_out ? 1 : 0, out,
                                                                           skip);
  count_launch();
}

template <int RL>
__global__ void __launch_bounds__(RED_THREADS) reduce_tc_rows_kernel(tc::TcPartials p, int64_t m, double scale,
                                                                     double eps, int log_out,
                                                                     float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * (RED_THREADS / RL) + threadIdx.x % (RED_THREADS / RL);
  double sum;
  pdl_wait();
  if (!tc::reduce_tc_row<RL>(p, i, m, sum)) return;
  double v = sum * scale;
  if (log_out) v = log(v + eps);
  out[i] = (float)v;
}

void launch_reduce_tc_rows(const tc::TcPartials& p, int64_t m, double scale, double eps, bool log_out, float* out,
                           cudaStream_t s) {
  if (tc::tc_short_rows(p))
    launch_pdl(reduce_tc_rows_kernel<1>, (int)((m + RED_THREADS - 1) / RED_THREADS), RED_THREADS, 0, s, p, m, scale,
               eps, log_out ? 1 : 0, out);
  else
    launch_pdl(reduce_tc_rows_kernel<RED_LANES>,
               (int)((m + RED_THREADS / RED_LANES - 1) / (RED_THREADS / RED_LANES)), RED_THREADS, 0, s, p, m, scale,
               eps, log_out ? 1 : 0, out);
  count_launch();
}

// Tensor-core score partials -> any of pdf_sum, weighted_sum, the debiased
// point and the score, 16 threads per row (thread k: feature k of every
// segment's centred weighted sum, and the pdf pairs k, k + 16, ... of the row,
// added across the 16 threads by shuffles).  The self pair, which the
// partials leave out, is added exactly (phi = 1, weight x_i), then mu * pdf
// undoes the centring; the shift is (x + W / (pdf + eps)) / 2.  Everything is
// carried as double-float and rounded to FP32 once; in FP64 the reduction and
// the shift were bound by the FP64 unit (26 + 18 us at n = 65536).
__global__ void __launch_bounds__(RED_THREADS) reduce_score_tc_kernel(tc::ScPartials p, int64_t n,
                                                                      const float* __restrict__ x, ScoreOut o,
                                                                      float eps_hi, float eps_lo, int eps_wide,
                                                                      double eps64, double inv_h2) {
  constexpr int QB = 256;   // rows per query block
  pdl_wait();
  const int64_t e = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x;
  const int64_t i = e / FSK_D;
  const int k = (int)(threadIdx.x % FSK_D);
  if (i >= n) return;   // a row's 16 threads leave together
  const unsigned group = 0xFFFFu << (threadIdx.x & 16);
  const int64_t qb = i / QB;
  const int r = (int)(i % QB);
  int segs;
  const int64_t seg0 = p.line.segments_of(qb, segs);
  float2 ps = make_float2(0.f, 0.f);
  for (int j = k; j < 2 * segs; j += FSK_D) ps = df_add(ps, p.ppdf[(2 * seg0 + j) * QB + r]);
#pragma unroll
  for (int d = 1; d < FSK_D; d <<= 1)
    ps = df_add(ps, make_float2(__shfl_xor_sync(group, ps.x, d), __shfl_xor_sync(group, ps.y, d)));
  float2 ws = make_float2(0.f, 0.f);
  const float2* wp = p.pw + (seg0 * QB + r) * FSK_D + k;
#pragma unroll 4
  for (int j = 0; j < segs; ++j) ws = df_add(ws, wp[(int64_t)j * QB * FSK_D]);
  constexpr float phi_unscale = 1.0f / 32768.0f;   // 2^-PHI_LOG2_SCALE
  static_assert(tc::PHI_LOG2_SCALE == 15.0f, "weight scale");
  const float w_unscale = ldexpf(1.f, -p.scales->pad[2]);
  ps.x *= phi_unscale;
  ps.y *= phi_unscale;
  ws.x = ws.x * phi_unscale * w_unscale;
  ws.y = ws.y * phi_unscale * w_unscale;
  // pdf = p + 1, W + mu * p + x_i
  const float mk = p.mu[k], xi = x[e];
  float2 mp = two_prod(mk, ps.x);
  mp.y = fmaf(mk, ps.y, mp.y);
  const float2 wt = df_add(df_add(ws, mp), make_float2(xi, 0.f));
  const float2 pdf = df_add(ps, make_float2(1.0f, 0.f));
  // beyond the pairs' range (eps, a weighted sum past the largest float, a point
  // whose double is): FP64
  constexpr float LARGE = 8.5e37f;   // 2^126
  const bool wide = eps_wide != 0 || !(fabsf(wt.x) < LARGE) || !(fabsf(xi) < LARGE);
  float w = wt.x;
  double off = 0.0;   // W / (pdf + eps) - x
  if (__builtin_expect(wide, 0)) {
    const double p64 = (double)ps.x + (double)ps.y, c64 = (double)ws.x + (double)ws.y;
    w = (float)(c64 + (double)mk * p64 + (double)xi);
    off = (c64 + ((double)mk - (double)xi) * p64) / (p64 + 1.0 + eps64) - (double)xi / (1.0 + (p64 + 1.0) / eps64);
  }
  if (o.w) {
    const int64_t at = i * o.ws_row + k * o.ws_col;
    if (in_bounds(at, n * FSK_D, 53)) o.w[at] = w;
  }
  if (o.pdf && k == 0) o.pdf[i] = pdf.x;
  if (o.debiased) {
    if (__builtin_expect(wide, 0)) {
      o.debiased[e] = (float)(0.5 * off + (double)xi);
      if (o.score) o.score[e] = (float)(off * inv_h2);
      return;
    }
    // m = W / (pdf + eps) as a quotient and its remainder over the divisor (pdf >= 1)
    const float2 d = df_add(pdf, make_float2(eps_hi, eps_lo));
    const float q = wt.x / d.x;
    const float rem = (fmaf(-q, d.x, wt.x) + wt.y) - q * d.y;
    const float2 m = two_sum(q, rem / d.x);
    o.debiased[e] = 0.5f * df_add(m, make_float2(xi, 0.f)).x;
    if (o.score) {
      const float2 df = df_add(m, make_float2(-xi, 0.f));
      o.score[e] = (float)(((double)df.x + (double)df.y) * inv_h2);
    }
  }
}

void launch_reduce_score_tc(const tc::ScPartials& p, int64_t n, const float* x, const ScoreOut& o, double h, double eps,
                            cudaStream_t s) {
  const float eps_hi = (float)eps, eps_lo = (float)(eps - (double)eps_hi);
  launch_pdl(reduce_score_tc_kernel, (int)((n * FSK_D + RED_THREADS - 1) / RED_THREADS), RED_THREADS, 0, s, p, n, x, o,
             eps_hi, eps_lo, eps < 1e30 ? 0 : 1, eps, 1.0 / (h * h));
  count_launch();
}

// CUDA-core score partials (FP64): pdf = sum of pdf partials (thread per row;
// the FP64 sum is kept for the weighted pass), then weighted = sum of centred
// partials + mu * pdf (thread per element, coalesced over the
// [split][row][16] partials).
__global__ void reduce_score_pdf_kernel(const double* __restrict__ ppdf, int pdf_splits, int64_t n,
                                        float* __restrict__ pdf, double* __restrict__ p_sum) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double p = 0.0;
  for (int s = 0; s < pdf_splits; ++s) p += ppdf[(int64_t)s * n + i];
  p_sum[i] = p;
  pdf[i] = (float)p;
}

__global__ void reduce_score_w_kernel(const double* __restrict__ pw, int w_splits, int64_t n,
                                      const double* __restrict__ mu64, const double* __restrict__ p_sum,
                                      float* __restrict__ w, int64_t ws_row, int64_t ws_col) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n * FSK_D) return;
  const int64_t i = e / FSK_D;
  const int k = (int)(e % FSK_D);
  double a = 0.0;
  for (int s = 0; s < w_splits; ++s) a += pw[(int64_t)s * n * FSK_D + e];
  const double v = a + mu64[k] * p_sum[i];
  const int64_t o = i * ws_row + k * ws_col;
  if (in_bounds(o, n * FSK_D, 53)) w[o] = (float)v;
}

size_t reduce_score_scratch_doubles(int64_t n) { return (size_t)n; }

void launch_reduce_score(const double* ppdf, const double* pw, int splits, int64_t n, const double* mu64, float* pdf,
                         float* w, int64_t ws_row, int64_t ws_col, double* scratch, cudaStream_t s) {
  const int T = 256;
  reduce_score_pdf_kernel<<<(unsigned)((n + T - 1) / T), T, 0, s>>>(ppdf, splits, n, pdf, scratch);
  count_launch();
  reduce_score_w_kernel<<<(unsigned)((n * FSK_D + T - 1) / T), T, 0, s>>>(pw, splits, n, mu64, scratch, w, ws_row,
                                                                         ws_col);
  count_launch();
}

// Thread per row, FP64: one reciprocal of (pdf + eps) per row; then per
// feature score = (w / (pdf + eps) - x) / h^2 and x + h^2/2 * score, which is
// (x + w / (pdf + eps)) / 2.
__global__ void debias16_kernel(const float* __restrict__ x, int64_t n, const float* __restrict__ pdf,
                                const float* __restrict__ w, int64_t ws_row, int64_t ws_col, double inv_h2,
                                double eps, float* __restrict__ deb, float* __restrict__ score) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double inv = 1.0 / ((double)pdf[i] + eps);
#pragma unroll
  for (int k = 0; k < FSK_D; ++k) {
    const double xi = (double)x[i * FSK_D + k];
    const int64_t o = i * ws_row + k * ws_col;
    const double m = in_bounds(o, n * FSK_D, 54) ? (double)w[o] * inv : 0.0;
    deb[i * FSK_D + k] = (float)(0.5 * (xi + m));
    if (score) score[i * FSK_D + k] = (float)((m - xi) * inv_h2);
  }
}

void launch_debias16(const float* x, int64_t n, const float* pdf, const float* w, int64_t ws_row,
                     int64_t ws_col, double h, double eps, float* debiased, float* score,
                     cudaStream_t s) {
  const int T = 128;
  debias16_kernel<<<(unsigned)((n + T - 1) / T), T, 0, s>>>(x, n, pdf, w, ws_row, ws_col, 1.0 / (h * h), eps,
                                                           debiased, score);
  count_launch();
}

__global__ void reduce_kde1d_score_kernel(const double* __restrict__ p0, const double* __restrict__ p1,
                                          int splits, int64_t m, double inv_norm, double h,
                                          float* __restrict__ score, float* __restrict__ pdf,
                                          float* __restrict__ deriv) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  double s0 = 0.0, s1 = 0.0;
  for (int s = 0; s < splits; ++s) {
    s0 += p0[(int64_t)s * m + i];
    s1 += p1[(int64_t)s * m + i];
  }
  // p1 holds sum (x - q) phi = -h * sum z phi
  const double pd = s0 * inv_norm;
  const double dv = s1 * inv_norm / (h * h);
  const float pdf_f = (float)pd, dv_f = (float)dv;
  if (pdf) pdf[i] = pdf_f;
  if (deriv) deriv[i] = dv_f;
  if (score) score[i] = dv_f / (pdf_f + 1e-12f);
}

void launch_reduce_kde1d_score(const double* p0, const double* p1, int splits, int64_t m,
                               int64_t n, double h, float* score, float* pdf, float* deriv,
                               cudaStream_t s) {
  const int T = 256;
  const double inv_norm = 1.0 / (sqrt(2.0 * 3.14159265358979323846) * (double)n * h);
  reduce_kde1d_score_kernel<<<(unsigned)((m + T - 1) / T), T, 0, s>>>(p0, p1, splits, m, inv_norm, h,
                                                                     score, pdf, deriv);
  count_launch();
}

__global__ void reduce_f32_partials_kernel(const float* __restrict__ partials, int64_t splits,
                                           int64_t count, float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  double s = 0.0;
  for (int64_t k = 0; k < splits; ++k) s += (double)partials[k * count + i];
  out[i] = (float)s;
}

void launch_reduce_f32_partials(const float* partials, int64_t splits, int64_t count, float* out,
                                cudaStream_t s) {
  const int T = 256;
  reduce_f32_partials_kernel<<<(unsigned)((count + T - 1) / T), T, 0, s>>>(partials, splits, count, out);
  count_launch();
}

__global__ void zero_kernel(double* p, int64_t count) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x)
    p[i] = 0.0;
}

void launch_zero(double* p, int64_t count, cudaStream_t s) {
  if (count <= 0) return;
  int blocks = (int)imin<int64_t>(4096, (count + 255) / 256);
  zero_kernel<<<blocks, 256, 0, s>>>(p, count);
  count_launch();
}

unsigned int reduce_take_device_error() { return take_unit_device_error(); }

}  // namespace fsk
