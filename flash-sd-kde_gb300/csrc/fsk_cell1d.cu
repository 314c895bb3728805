// fsk_cell1d.cu - 1-D Gaussian KDE of many points at many queries by cell
// expansions (the Taylor form of the fast Gauss transform, Greengard and
// Strain, SIAM J. Sci. Stat. Comput. 12 (1991) 79-94).
//
// With cells of width w = h / 4, centre c, t = (x - c) / h and u = (q - c) / h,
//   exp(-(q - x)^2 / 2h^2) = exp(-u^2 / 2) sum_k u^k [exp(-t^2 / 2) t^k / k!],
// so a cell's points enter a query through P moments M_k = sum of the bracket,
// and a cell's queries share one polynomial through 12 nodes: n P + cells^2 + m
// operations instead of n * m exps.  2^22 points x 2^20 queries: 532 ms for
// the pair sums (88 % of the ex2 rate), 238 us with every query visiting its
// cells, 89 us this way.
//
// Accuracy: |u t| <= |u| / 8; a query visits cells until every remaining term
// together is below 2^-34 of its sum, i.e. |u| <= ~10, where the first dropped
// Taylor term (u t)^14 / 14! is below 3e-10 and near the query below 1e-20.
// Moments are summed in fixed point (31 or 15 fractional bits per point, exact
// and order-independent, so the result is deterministic), the exponent u^2 / 2 in
// double-float.  A model against FP64 over mixtures and tails: 2-norm error
// 1.1e-8 (direct FP32 pairs 1.6e-8), largest relative error 1.4e-7 at
// densities down to 1e-30 of the peak (direct: 4.9e-6, the rounding of the far
// pairs' exponents).  The nodes' sums are double-float, which leaves a
// polynomial 1e-8 before its rounding to FP32 (2-norm, rounded: 2.3e-8 to
// 3.2e-8 over the shapes tried; direct pairs 2.9e-8 to 5.4e-8).
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
constexpr int CELLS_MAX = 1792;       // (P + P_LOW) * CELLS_MAX * 4 B of shared memory per block
constexpr float CELL_H = 0.25f;       // cell width / h
constexpr int MM_THREADS = 256;
constexpr int MM_MAX_BLOCKS = 1216;
constexpr int MO_THREADS = 1024;
constexpr int MO_MAX_POINTS = 1 << 15;   // points per block: their 16-bit parts (x (1 + 1/32)^13) sum below 2^31
constexpr int Q_THREADS = 256;
constexpr int NODES = 12;             // Chebyshev nodes per cell of the local polynomials
constexpr int NODE_LANES = 8;         // threads that share a node's source cells
constexpr int REACH = 40;             // source cells to either side of a node's
constexpr int LOCAL_THREADS = 2 * NODES * NODE_LANES;   // two cells per block
constexpr float FAST_LOG2 = 38.f;     // polynomials hold where the sum is above n 2^-38
constexpr int P_LOW = 7;              // moments that keep bits below 2^-15 of a point's value
constexpr int MO_SMEM = (P + P_LOW) * CELLS_MAX * 4;
static_assert(MO_SMEM <= 227 * 1024, "shared memory");

struct CellState {
  float lo, w;
  int cells;
  int use;
};

struct CellBufs {
  float2* minmax;              // [MM_MAX_BLOCKS]
  unsigned long long* acc;     // [P][CELLS_MAX] fixed-point moments
  float* table;                // [CELLS_MAX][ROW]: moments, then the errors of the first two
  float* local;                // [CELLS_MAX][ROW]: polynomial (b_0, its error, b_1 .. b_11), then 1 where it holds
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

// Fixed-point moments of one block's points in 32-bit shared-memory
// accumulators (bits above and, for the first P_LOW moments, below 2^-15 of a
// value around [-1, 1]), added into the 64-bit global ones at the end.  Moment k enters
// a sum times (u / 8)^k / k!: from k = 7 on that is below 1e-3 even at |u| = 10
// and below 2e-6 at 4, so 2^-16 of a point's value there is 7e-9 of the far
// tail and 1e-11 of the bulk.  Bound by the shared-memory atomics: 28 per
// point took 51 us for 2^22 points, 21 take 41.
__global__ void __launch_bounds__(MO_THREADS, 1) cell_moment_kernel(const float* __restrict__ x, int64_t n, float h,
                                                                    int extent_blocks, CellBufs b) {
  extern __shared__ int tab[];   // [P][cells], then [P_LOW][cells]
  __shared__ CellState st;
  __shared__ float2 warp_mm[MO_THREADS / 32];
  pdl_wait();
  {
    float lo = __int_as_float(0x7f800000), hi = -lo;
    for (int i = threadIdx.x; i < extent_blocks; i += MO_THREADS) {
      const float2 v = b.minmax[i];
      lo = fminf(lo, v.x);
      hi = fmaxf(hi, v.y);
    }
    auto across = [&]() {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
    };
    across();
    if ((threadIdx.x & 31) == 0) warp_mm[threadIdx.x >> 5] = make_float2(lo, hi);
    __syncthreads();
    if (threadIdx.x < 32) {
      lo = warp_mm[threadIdx.x].x;
      hi = warp_mm[threadIdx.x].y;
      across();
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
  for (int i = threadIdx.x; i < size + P_LOW * cells; i += MO_THREADS) tab[i] = 0;
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
      atomicAdd(&tab[k * cells + c], (int)hi);
      if (k < P_LOW) atomicAdd(&tab[size + k * cells + c], (int)rintf(fmaf(hi, -1.f / 32768.f, f) * 2147483648.f));
      f *= t;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < size; i += MO_THREADS) {
    const long long v = ((long long)tab[i] << 16) + (i < P_LOW * cells ? tab[size + i] : 0);
    if (v != 0) atomicAdd(&b.acc[(i / cells) * CELLS_MAX + i % cells], (unsigned long long)v);
  }
}

// Constants of the kernels below, computed on the host in FP64.
struct CellConsts {
  double moment[P];               // 2^-31 (1/8)^k / k!
  double coef[NODES][NODES];      // polynomial coefficient j in z from the node values
  float z[NODES];                 // node positions in half cells
  float2 exp2_tab[32];            // 2^(-j/32) as (value, error)
  float inv_h, inv_h_lo, c2, c2_lo;
};

// Moment table: M_k = acc 2^-31 (1/8)^k / k!
__global__ void __launch_bounds__(MM_THREADS) cell_table_kernel(CellBufs b, const __grid_constant__ CellConsts k) {
  pdl_wait();
  const CellState st = *b.st;
  if (!st.use) return;
  for (int c = blockIdx.x * MM_THREADS + threadIdx.x; c < st.cells; c += gridDim.x * MM_THREADS) {
    float4* row = reinterpret_cast<float4*>(b.table + (int64_t)c * ROW);
    float v[ROW], err[2];
#pragma unroll
    for (int j = 0; j < P; ++j) {
      const double d = (double)(long long)b.acc[j * CELLS_MAX + c] * k.moment[j];
      v[j] = (float)d;
      if (j < 2) err[j] = (float)(d - (double)v[j]);
    }
    v[P] = err[0];
    v[P + 1] = err[1];
#pragma unroll
    for (int j = 0; j < ROW / 4; ++j) row[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  }
}

// Local polynomials: the sum at 12 Chebyshev nodes of every cell (source
// expansions of the cells within REACH, in double-float where it matters) and
// from them f(c + z w / 2) = sum_j b_j z^j.  A query then costs one row of 64
// bytes and 12 FMAs instead of ~60 cells: 147 us for 2^20 queries of 2^22
// points, 23 us this way plus 13 here (bound by the gather of the rows, and by
// the latency of a node's ~10 cells per thread).  The polynomial is used where
// the dropped cells cannot matter (f >= n 2^-38; they hold below n 2^-72) and
// f changes by less than a factor of two over the cell, so that node and
// rounding errors stay relative to the sum: everywhere but in tails and gaps.
__global__ void __launch_bounds__(LOCAL_THREADS) cell_local_kernel(CellBufs b, float log2n,
                                                                   const __grid_constant__ CellConsts k) {
  __shared__ double value[2][NODES];
  pdl_wait();
  const CellState st = *b.st;
  if (!st.use || (int)blockIdx.x * 2 >= st.cells) return;
  const int half = threadIdx.x / (NODES * NODE_LANES), node = threadIdx.x % (NODES * NODE_LANES) / NODE_LANES;
  const int cell = blockIdx.x * 2 + half, l = threadIdx.x % NODE_LANES;
  float2 sum = make_float2(0.f, 0.f);
  if (cell < st.cells) {
    const float delta = k.z[node] * (0.5f * st.w);
    const float centre = cell_centre(st, cell);
    const int last = min(st.cells - 1, cell + REACH);
    for (int c = max(0, cell - REACH) + l; c <= last; c += NODE_LANES) {
      const float4* row = reinterpret_cast<const float4*>(b.table + (int64_t)c * ROW);
      const float4 r0 = row[0];
      if (r0.x == 0.f) continue;   // no points
      const float4 r1 = row[1], r2 = row[2], r3 = row[3];
      // distance node - source centre, and u = distance / h
      const float2 dc = two_sum(centre, -cell_centre(st, c));
      float2 d = two_sum(dc.x, delta);
      d.y += dc.y;
      const float uh = d.x * k.inv_h;
      const float ul = fmaf(d.x, k.inv_h, -uh) + fmaf(d.x, k.inv_h_lo, d.y * k.inv_h);
      float s = r3.y;
      s = fmaf(s, uh, r3.x);
      s = fmaf(s, uh, r2.w);
      s = fmaf(s, uh, r2.z);
      s = fmaf(s, uh, r2.y);
      s = fmaf(s, uh, r2.x);
      s = fmaf(s, uh, r1.w);
      s = fmaf(s, uh, r1.z);
      s = fmaf(s, uh, r1.y);
      s = fmaf(s, uh, r1.x);
      s = fmaf(s, uh, r0.w);
      s = fmaf(s, uh, r0.z);
      // M_0 + u (M_1 + u s), pairs
      float2 t = two_prod(s, uh);
      float2 v = two_sum(r0.y, t.x);
      v.y += t.y + fmaf(s, ul, r3.w);
      t = two_prod(v.x, uh);
      t.y += fmaf(v.x, ul, v.y * uh);
      float2 w = two_sum(r0.x, t.x);
      w.y += t.y + r3.z;
      // 2^(-c2 d^2): 2^(-j/32) from the table, the rest by its Taylor series
      const float2 dd = two_prod(d.x, d.x);
      const float p = dd.x * k.c2;
      const float pl = fmaf(dd.x, k.c2, -p) + fmaf(dd.x, k.c2_lo, fmaf(2.f * d.x, d.y, dd.y) * k.c2);
      const float j = rintf(p * 32.f);
      const float r = -0.69314718055994531f * (fmaf(j, -0.03125f, p) + pl);   // |r| <= ln 2 / 64
      const float q = r * fmaf(r, fmaf(r, fmaf(r, 1.f / 24.f, 1.f / 6.f), 0.5f), 1.f);
      const float2 e = k.exp2_tab[(int)j & 31];
      const float scale = exp2f(-(float)((int)j >> 5));   // a power of two
      const float el = fmaf(e.x, q, e.y);
      t = two_prod(e.x, w.x);
      t.y += fmaf(e.x, w.y, el * w.x);
      sum = df_add(sum, make_float2(t.x * scale, t.y * scale));
    }
  }
#pragma unroll
  for (int o = NODE_LANES / 2; o > 0; o >>= 1)
    sum = df_add(sum, make_float2(__shfl_xor_sync(0xffffffffu, sum.x, o), __shfl_xor_sync(0xffffffffu, sum.y, o)));
  if (l == 0) value[half][node] = (double)sum.x + (double)sum.y;
  __syncthreads();
  if (l != 0 || cell >= st.cells) return;
  double c = 0.0;
#pragma unroll
  for (int i = 0; i < NODES; ++i) c += k.coef[node][i] * value[half][i];
  float* row = b.local + (int64_t)cell * ROW;
  if (node > 0) {
    row[node + 1] = (float)c;
    return;
  }
  float lo = (float)value[half][0], hi = lo;
#pragma unroll
  for (int i = 1; i < NODES; ++i) {
    lo = fminf(lo, (float)value[half][i]);
    hi = fmaxf(hi, (float)value[half][i]);
  }
  const float top = (float)c;
  row[0] = top;
  row[1] = (float)(c - (double)top);
  row[NODES + 1] = lo > exp2f(log2n - FAST_LOG2) && hi < 2.f * lo ? 1.f : 0.f;
}

// One query per thread: its cell's polynomial, or, where that does not hold,
// cells outward from the query's own, right and left, until the rest cannot
// matter (~60 cells x ~45 instructions).  scale as (value, error) in FP32
// where it fits there: the FP64 unit runs 2 lanes per clock per SM.
__global__ void __launch_bounds__(Q_THREADS) cell_query_kernel(const float* __restrict__ q, int64_t m, float log2n,
                                                               float inv_h, float c2, float c2_lo, double scale,
                                                               double eps, int log_out, float2 scale2, CellBufs b,
                                                               float* __restrict__ out) {
  pdl_wait();
  const CellState st = *b.st;
  if (!st.use) return;
  const int64_t i = (int64_t)blockIdx.x * Q_THREADS + threadIdx.x;
  if (i >= m) return;
  const float qv = q[i];
  const float pos = (qv - st.lo) / st.w;
  const int own = (int)fminf(fmaxf(pos, 0.f), (float)(st.cells - 1));
  if (pos >= 0.f && pos < (float)st.cells) {
    const float4* row = reinterpret_cast<const float4*>(b.local + (int64_t)own * ROW);
    const float4 r3 = row[3];
    if (r3.y != 0.f) {
      const float4 r0 = row[0], r1 = row[1], r2 = row[2];
      const float z = (qv - cell_centre(st, own)) * (2.f / st.w);
      float s = r3.x;
      s = fmaf(s, z, r2.w);
      s = fmaf(s, z, r2.z);
      s = fmaf(s, z, r2.y);
      s = fmaf(s, z, r2.x);
      s = fmaf(s, z, r1.w);
      s = fmaf(s, z, r1.z);
      s = fmaf(s, z, r1.y);
      s = fmaf(s, z, r1.x);
      s = fmaf(s, z, r0.w);
      s = fmaf(s, z, r0.z);
      const float2 v = two_sum(r0.x, fmaf(s, z, r0.y));
      if (scale2.x != 0.f) {
        const float2 t = two_prod(v.x, scale2.x);
        if (in_bounds(i, m, 57)) out[i] = t.x + (t.y + fmaf(v.x, scale2.y, v.y * scale2.x));
      } else {
        double y = ((double)v.x + (double)v.y) * scale;
        if (log_out) y = log(y + eps);
        if (in_bounds(i, m, 57)) out[i] = (float)y;
      }
      return;
    }
  }
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
  // from the query to cell c's interval, in h: 0 inside it, so that a query
  // far outside the data stops at the first cell on either side (visited at
  // 1e5 h the moments' polynomial overflows; its weight there is 0)
  auto gap = [&](int c) {
    const float below = fmaf((float)c, st.w, st.lo) - qv, above = qv - fmaf((float)(c + 1), st.w, st.lo);
    return fmaxf(0.f, fmaxf(below, above)) * inv_h;
  };
  int right = own, left = own - 1;
  bool go_r = right < st.cells, go_l = left >= 0;
  while (go_r || go_l) {
    if (go_r) {
      const float g = gap(right);
      if (g * g * 0.72134752f > limit) go_r = false;
      else visit(right);
      if (++right >= st.cells) go_r = false;
    }
    if (go_l) {
      const float g = gap(left);
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
  b.local = c.take<float>((size_t)CELLS_MAX * ROW);
  b.st = c.take<CellState>(1);
  return b;
}

CellConsts fixed_consts() {
  CellConsts k = {};
  double f = 1.0 / 2147483648.0;
  for (int j = 0; j < P; ++j) {
    k.moment[j] = f;
    f *= 0.5 * CELL_H / (j + 1);
  }
  // Chebyshev polynomials T_j in powers of z, then the interpolation through the nodes
  const double pi = 3.14159265358979323846;
  double t[NODES][NODES] = {};
  t[0][0] = t[1][1] = 1.0;
  for (int j = 2; j < NODES; ++j)
    for (int i = 0; i < NODES; ++i) t[j][i] = (i > 0 ? 2.0 * t[j - 1][i - 1] : 0.0) - t[j - 2][i];
  for (int j = 0; j < NODES; ++j) {
    const double angle = pi * (2 * j + 1) / (2 * NODES);
    k.z[j] = (float)cos(angle);
    for (int i = 0; i < NODES; ++i) {
      double c = 0.0;
      for (int d = 0; d < NODES; ++d) c += (d ? 2.0 : 1.0) / NODES * cos(d * angle) * t[d][i];
      k.coef[i][j] = c;
    }
  }
  for (int j = 0; j < 32; ++j) {
    const double e = exp2(-j / 32.0);
    k.exp2_tab[j].x = (float)e;
    k.exp2_tab[j].y = (float)(e - (double)k.exp2_tab[j].x);
  }
  return k;
}

CellConsts cell_consts(double h) {
  static const CellConsts fixed = fixed_consts();
  CellConsts k = fixed;
  const double c2 = FSK_LOG2E / (2.0 * h * h), ih = 1.0 / h;
  k.c2 = (float)c2;
  k.c2_lo = (float)(c2 - (double)k.c2);
  k.inv_h = (float)ih;
  k.inv_h_lo = (float)(ih - (double)k.inv_h);
  return k;
}
}  // namespace

// Where the expansions are tried.  Both sides, us per call (pair sums /
// expansions / data too spread, which pays for the attempt):
//   0.10e9 pairs: 4096 x 25000 41 / 43 / 49, 100000 x 1000 41 / 36 / 51
//   0.34e9:       4096 x 80000 76 / 47 / 84, 100000 x 3500 78 / 38 / 86
//   0.70e9:       4096 x 170000 117 / 47 / 125
//   1.07e9:       4095 x 262144 154 / 45 / 162, 4096 x 262144 154 / 47 / 162
//   4.3e9:        4095 x 1048576 544 / 54 / 554
// The expansions win from ~1.5e8 pairs on; the line at 2^30 keeps what spread
// data loses (3 to 10 us) at 5 % or less.  The limit of 4096 points has no
// reason in time (2000 x 2000000: 518 / 64 / 531; 500 x 1000000: 85 / 77 / 97).
// n <= 2^31: a point adds up to 1.5 x 2^31 to the signed 64-bit moments.
bool cell1d_applies(int64_t m, int64_t n) {
  return n >= 4096 && n <= (int64_t(1) << 31) && (double)m * (double)n >= 1073741824.0;
}

// Bandwidths whose squares the FP32 tables hold: a visited cell's d^2 reaches
// (16 h)^2, its rounding error and c2 = log2(e) / 2 h^2 have to stay normal.
// Others take the pair kernel alone.
bool cell1d_holds(double h) { return h >= 1e-15 && h <= 1e18; }

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
  const CellConsts k = cell_consts(h);
  launch_pdl(cell_table_kernel, (CELLS_MAX + MM_THREADS - 1) / MM_THREADS, MM_THREADS, 0, s, b, k);
  count_launch();
  launch_pdl(cell_local_kernel, CELLS_MAX / 2, LOCAL_THREADS, 0, s, b, (float)log2((double)n), k);
  count_launch();
  float2 scale2 = make_float2(0.f, 0.f);
  // (a sum is at most n: no product beyond FP32, whose error would be infinite)
  if (!log_out && fabs(scale) > 1e-30 && fabs(scale) * (double)n < 1e38) {
    scale2.x = (float)scale;
    scale2.y = (float)(scale - (double)scale2.x);
  }
  e = launch_pdl(cell_query_kernel, (int)((m + Q_THREADS - 1) / Q_THREADS), Q_THREADS, 0, s, q, m, (float)log2((double)n),
                 k.inv_h, k.c2, k.c2_lo, scale, eps, log_out ? 1 : 0, scale2, b, out);
  count_launch();
  return cuda_status(e);
}

unsigned int cell1d_take_device_error() { return take_unit_device_error(); }

}  // namespace fsk
