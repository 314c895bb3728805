// fsk_cell1d.cu - 1-D Gaussian KDE of many points at many queries by cell
// expansions (the Taylor form of the fast Gauss transform, Greengard and
// Strain, SIAM J. Sci. Stat. Comput. 12 (1991) 79-94).
//
// With cells of width w = h / 4, centre c, t = (x - c) / h and u = (q - c) / h,
//   exp(-(q - x)^2 / 2h^2) = exp(-u^2 / 2) sum_k u^k [exp(-t^2 / 2) t^k / k!],
// so a cell's points enter a query through P moments M_k = sum of the bracket:
// n + m * cells * P operations instead of n * m exps (2^22 points x 2^20
// queries: 532 ms for the pair sums at 88 % of the ex2 rate).
//
// Accuracy: |u t| <= |u| / 8; a query visits cells until every remaining term
// together is below 2^-34 of its sum, i.e. |u| <= ~10, where the first dropped
// Taylor term (u t)^14 / 14! is below 3e-10 and near the query below 1e-20.
// Moments are summed in fixed point (31 fractional bits per point, exact and
// order-independent, so the result is deterministic), the exponent u^2 / 2 in
// double-float.  A model against FP64 over mixtures and tails: 2-norm error
// 1.1e-8 (direct FP32 pairs 1.6e-8), largest relative error 1.4e-7 at
// densities down to 1e-30 of the peak (direct: 4.9e-6, the rounding of the far
// pairs' exponents).
//
// The number of cells, (max x - min x) / w, is known on the device only.  The
// tables hold CELLS_MAX; data spread wider than that against h (or not
// finite) is left to the direct kernel: `use` in the state decides, and the
// kernels of the path not taken return at once.
#include "fsk_common.cuh"
#include "fsk_kernels.cuh"

namespace fsk {

namespace {
constexpr int P = 14;                 // moments per cell
constexpr int ROW = 16;               // floats per cell in the moment table
constexpr int CELLS_MAX = 1792;       // P * CELLS_MAX * 8 B of shared memory per block
constexpr float CELL_H = 0.25f;       // cell width / h
constexpr int MM_THREADS = 256;
constexpr int MM_MAX_BLOCKS = 304;
constexpr int MO_THREADS = 1024;
constexpr int MO_MAX_POINTS = 1 << 15;   // points per block: their 16-bit parts (x (1 + 1/32)^13) sum below 2^31
constexpr int Q_THREADS = 128;
constexpr int MO_SMEM = P * CELLS_MAX * 8;
static_assert(MO_SMEM <= 227 * 1024, "shared memory");

struct CellState {
  float lo, w;
  int cells;
  int use;
};

struct CellBufs {
  float2* minmax;              // [MM_MAX_BLOCKS]
  unsigned long long* acc;     // [P][CELLS_MAX] fixed-point moments
  float* table;                // [CELLS_MAX][ROW]
  CellState* st;
};

__device__ __forceinline__ float cell_centre(const CellState& s, int i) { return fmaf((float)i + 0.5f, s.w, s.lo); }

// Per-block extent of the data; also clears the accumulators.
__global__ void __launch_bounds__(MM_THREADS) cell_extent_kernel(const float* __restrict__ x, int64_t n, CellBufs b) {
  for (int i = blockIdx.x * MM_THREADS + threadIdx.x; i < P * CELLS_MAX; i += gridDim.x * MM_THREADS) b.acc[i] = 0ull;
  const float inf = __int_as_float(0x7f800000);
  float lo = inf, hi = -inf;
  bool bad = false;
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * MM_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * MM_THREADS) {
    const float v = x[i];
    bad |= !(fabsf(v) < inf);
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
  }
  if (bad) hi = inf;   // an infinite extent: no cells
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  __shared__ float2 sh[MM_THREADS / 32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = make_float2(lo, hi);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < MM_THREADS / 32; ++w) {
      lo = fminf(lo, sh[w].x);
      hi = fmaxf(hi, sh[w].y);
    }
    b.minmax[blockIdx.x] = make_float2(lo, hi);
  }
}

// Fixed-point moments of one block's points: two 32-bit shared-memory
// accumulators per moment (bits above and below 2^-15 of a value around [-1, 1]),
// added into the 64-bit global ones at the end.
__global__ void __launch_bounds__(MO_THREADS, 1) cell_moment_kernel(const float* __restrict__ x, int64_t n, float h,
                                                                    int extent_blocks, CellBufs b) {
  extern __shared__ int tab[];   // [2][P][cells]
  __shared__ CellState st;
  pdl_wait();
  if (threadIdx.x < 32) {
    float lo = __int_as_float(0x7f800000), hi = -lo;
    for (int i = threadIdx.x; i < extent_blocks; i += 32) {
      const float2 v = b.minmax[i];
      lo = fminf(lo, v.x);
      hi = fmaxf(hi, v.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (threadIdx.x == 0) {
      st.lo = lo;
      st.w = CELL_H * h;
      // 64 ulps of the data's magnitude at least, so that rounded centres
      // leave positions within 1 + 1/32 of a half cell
      const float need = (hi - lo) / st.w;
      st.use = need < (float)(CELLS_MAX - 1) && st.w > 64.f * 1.2e-7f * fmaxf(fabsf(lo), fabsf(hi)) && st.w > 1e-30f;
      st.cells = st.use ? (int)need + 1 : 0;
      if (blockIdx.x == 0) *b.st = st;
    }
  }
  __syncthreads();
  if (!st.use) return;
  const int cells = st.cells, size = P * cells;
  for (int i = threadIdx.x; i < 2 * size; i += MO_THREADS) tab[i] = 0;
  __syncthreads();
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  const int64_t i0 = (int64_t)blockIdx.x * per, i1 = imin<int64_t>(n, i0 + per);
  const float inv_w = 1.0f / st.w, inv_half = 2.0f / st.w;
  constexpr float HALF = 0.5f * CELL_H;   // half a cell in units of h
  for (int64_t i = i0 + threadIdx.x; i < i1; i += MO_THREADS) {
    const float v = x[i];
    int c = min(cells - 1, (int)((v - st.lo) * inv_w));
    float t = (v - cell_centre(st, c)) * inv_half;   // position in half cells
    if (fabsf(t) > 1.f) {   // the index was rounded across an edge
      c = max(0, min(cells - 1, c + (t > 0.f ? 1 : -1)));
      t = (v - cell_centre(st, c)) * inv_half;
    }
    const float th = t * HALF;
    float f = exp2f(-0.72134752044448170f * th * th);   // exp(-t^2 / 2)
#pragma unroll
    for (int k = 0; k < P; ++k) {
      const float hi = rintf(f * 32768.f);
      const float lo = rintf(fmaf(hi, -1.f / 32768.f, f) * 2147483648.f);
      atomicAdd(&tab[k * cells + c], (int)hi);
      atomicAdd(&tab[size + k * cells + c], (int)lo);
      f *= t;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < size; i += MO_THREADS) {
    const long long v = ((long long)tab[i] << 16) + tab[size + i];
    if (v != 0) atomicAdd(&b.acc[(i / cells) * CELLS_MAX + i % cells], (unsigned long long)v);
  }
}

// Moment table: M_k = acc 2^-31 (1/8)^k / k!
__global__ void __launch_bounds__(MM_THREADS) cell_table_kernel(CellBufs b) {
  pdl_wait();
  const CellState st = *b.st;
  if (!st.use) return;
  for (int i = blockIdx.x * MM_THREADS + threadIdx.x; i < st.cells * ROW; i += gridDim.x * MM_THREADS) {
    const int c = i / ROW, k = i % ROW;
    float v = 0.f;
    if (k < P) {
      double f = 1.0 / 2147483648.0;
      for (int j = 1; j <= k; ++j) f *= 0.5 * CELL_H / j;
      v = (float)((double)(long long)b.acc[k * CELLS_MAX + c] * f);
    }
    b.table[i] = v;
  }
}

// One query per thread: cells outward from the query's own, right and left,
// until the rest cannot matter.  ~60 cells x ~45 instructions at n = 2^22.
__global__ void __launch_bounds__(Q_THREADS) cell_query_kernel(const float* __restrict__ q, int64_t m, float log2n,
                                                               float inv_h, float c2, float c2_lo, double scale,
                                                               double eps, int log_out, CellBufs b,
                                                               float* __restrict__ out) {
  pdl_wait();
  const CellState st = *b.st;
  if (!st.use) return;
  const int64_t i = (int64_t)blockIdx.x * Q_THREADS + threadIdx.x;
  if (i >= m) return;
  const float qv = q[i];
  Comp acc{0.f, 0.f};
  // terms beyond the gap g (in h) total at most n 2^(-g^2 log2(e) / 2); stop at
  // 2^-34 of the sum so far, and where even n of them are below 2^-150
  float limit = 150.f + log2n;
  auto visit = [&](int c) {
    const float4* row = reinterpret_cast<const float4*>(b.table + (int64_t)c * ROW);
    const float4 r0 = row[0];
    if (r0.x == 0.f) return;   // no points
    const float4 r1 = row[1], r2 = row[2], r3 = row[3];
    const float2 d = two_sum(qv, -cell_centre(st, c));
    const float u = d.x * inv_h;
    float s = r3.y;
    s = fmaf(s, u, r3.x);
    s = fmaf(s, u, r2.w);
    s = fmaf(s, u, r2.z);
    s = fmaf(s, u, r2.y);
    s = fmaf(s, u, r2.x);
    s = fmaf(s, u, r1.w);
    s = fmaf(s, u, r1.z);
    s = fmaf(s, u, r1.y);
    s = fmaf(s, u, r1.x);
    s = fmaf(s, u, r0.w);
    s = fmaf(s, u, r0.z);
    s = fmaf(s, u, r0.y);
    s = fmaf(s, u, r0.x);
    // 2^(-c2 d^2), exponent in double-float
    const float2 dd = two_prod(d.x, d.x);
    const float p = dd.x * c2;
    const float e = fmaf(dd.x, c2, -p) + fmaf(dd.x, c2_lo, fmaf(2.f * d.x, d.y, dd.y) * c2);
    const float y = exp2f(-p);
    acc.add(fmaf(y, -e * 0.69314718055994531f, y) * s);
  };
  const float pos = (qv - st.lo) / st.w;
  const int own = (int)fminf(fmaxf(pos, 0.f), (float)(st.cells - 1));
  int right = own, left = own - 1;
  bool go_r = right < st.cells, go_l = left >= 0;
  if (fabsf(qv) == __int_as_float(0x7f800000)) go_r = go_l = false;   // no mass at infinity
  while (go_r || go_l) {
    if (go_r) {
      const float g = fmaxf(0.f, fmaf((float)right, st.w, st.lo) - qv) * inv_h;
      if (g * g * 0.72134752f > limit) go_r = false;
      else visit(right);
      if (++right >= st.cells) go_r = false;
    }
    if (go_l) {
      const float g = fmaxf(0.f, qv - fmaf((float)(left + 1), st.w, st.lo)) * inv_h;
      if (g * g * 0.72134752f > limit) go_l = false;
      else visit(left);
      if (--left < 0) go_l = false;
    }
    if (acc.s > 0.f) limit = fminf(150.f + log2n, 34.f + log2n - __log2f(acc.s));
  }
  double v = ((double)acc.s + (double)acc.c) * scale;
  if (log_out) v = log(v + eps);
  if (in_bounds(i, m, 57)) out[i] = (float)v;
}

CellBufs take_cells(WsCarver& c) {
  CellBufs b;
  b.minmax = c.take<float2>(MM_MAX_BLOCKS);
  b.acc = c.take<unsigned long long>((size_t)P * CELLS_MAX);
  b.table = c.take<float>((size_t)CELLS_MAX * ROW);
  b.st = c.take<CellState>(1);
  return b;
}
}  // namespace

// Where the expansions are tried: their launches (~15 us) and ~60 cells per
// query pay above ~600 points and ~1e8 pairs; from 2^30 pairs (131 us of pair
// sums) on, data that turns out too spread for the tables loses at most a few
// per cent to the attempt.
bool cell1d_applies(int64_t m, int64_t n) { return n >= 4096 && (double)m * (double)n >= 1073741824.0; }

void take_cell1d(WsCarver& c) { take_cells(c); }

int launch_cell1d(const float* q, int64_t m, const float* x, int64_t n, double h, double scale, double eps,
                  bool log_out, WsCarver& c, float* out, const int** taken, cudaStream_t s) {
  const CellBufs b = take_cells(c);
  if (!c.fits()) return FSK_ERR_WORKSPACE_TOO_SMALL;
  *taken = &b.st->use;
  cudaError_t e = cudaFuncSetAttribute(cell_moment_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MO_SMEM);
  if (e != cudaSuccess) return cuda_status(e);
  const int eb = (int)imin<int64_t>(MM_MAX_BLOCKS, (n + MM_THREADS - 1) / MM_THREADS);
  cell_extent_kernel<<<eb, MM_THREADS, 0, s>>>(x, n, b);
  count_launch();
  const int mb = (int)imax<int64_t>(imin<int64_t>(sm_count(), (n + MO_THREADS - 1) / MO_THREADS),
                                    (n + MO_MAX_POINTS - 1) / MO_MAX_POINTS);
  launch_pdl(cell_moment_kernel, mb, MO_THREADS, MO_SMEM, s, x, n, (float)h, eb, b);
  count_launch();
  launch_pdl(cell_table_kernel, 64, MM_THREADS, 0, s, b);
  count_launch();
  const double c2d = FSK_LOG2E / (2.0 * h * h);
  const float c2 = (float)c2d, c2_lo = (float)(c2d - (double)c2);
  {
    TimerScope ts(K_KDE1D_CELL, (double)m * (double)n, s);
    e = launch_pdl(cell_query_kernel, (int)((m + Q_THREADS - 1) / Q_THREADS), Q_THREADS, 0, s, q, m,
                   (float)log2((double)n), (float)(1.0 / h), c2, c2_lo, scale, eps, log_out ? 1 : 0, b, out);
    count_launch();
  }
  return cuda_status(e);
}

unsigned int cell1d_take_device_error() { return take_unit_device_error(); }

}  // namespace fsk
