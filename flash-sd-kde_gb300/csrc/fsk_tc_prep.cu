// fsk_tc_prep.cu - operand preparation of the tensor-core kernels: column
// means, scale selection and the fp16 operand images of fsk_tc_kde16.cu and
// fsk_tc_score16.cu, in three launches.
//
// The chain mean -> maxima of the centred coordinates -> images has two
// grid-wide dependencies.  Each is one launch boundary: every block of the
// next kernel adds up the per-block results of the previous one itself (a few
// hundred pairs, in a fixed order, so all blocks get the same bits), which
// takes the place of the single-block kernels in between (final mean, scale
// state, scale selection in FP64: 4 + 2 + 6 us).  With programmatic dependent
// launch the start-up of a kernel overlaps the end of the one before.  Sums
// are double-float, exponents come from bit fields: nothing uses the FP64
// unit.  The preparation of a 4096 / 1024 KDE took 40 us in 8 kernels.
#include <cuda_fp16.h>

#include "fsk_kernels.cuh"
#include "fsk_tc.cuh"
#include "fsk_tc_ops.cuh"

namespace fsk {
namespace tc {

namespace {
constexpr int PT = 256;               // threads per block
constexpr int PW = PT / 32;
constexpr int MEAN_MAX_BLOCKS = 304;
constexpr int STATS_MAX_BLOCKS = 304; // per point set

struct PrepBufs {
  float2* mean_part;   // [MEAN_MAX_BLOCKS][16]
  float4* stats;       // [2 * STATS_MAX_BLOCKS] (max |v|, max beta, max alpha)
  float* mu;
  TcScales* sc;
};

// One row's 16 coordinates; 16-byte loads where the caller's rows allow them.
__device__ __forceinline__ void load_row(const float* __restrict__ p, bool vec, float (&v)[FSK_D]) {
  if (vec) {
    const float4* p4 = reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 t = p4[k];
      v[4 * k] = t.x; v[4 * k + 1] = t.y; v[4 * k + 2] = t.z; v[4 * k + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < FSK_D; ++k) v[k] = p[k];
  }
}

// Per-block column sums of x * down as (value, error) pairs: thread t adds
// feature t % 16 of the rows t / 16, t / 16 + 16, ... of the block's share.
// down: a power of two below 1 / (2 n), so that no partial sum overflows where
// a column holds values near the largest float.
__global__ void __launch_bounds__(PT) tc_mean_kernel(const float* __restrict__ x, int64_t n, float down,
                                                     float2* __restrict__ part) {
  pdl_launch_dependents();
  constexpr int L = PT / FSK_D;
  const int k = threadIdx.x % FSK_D, l = threadIdx.x / FSK_D;
  Comp a{0.f, 0.f};
#pragma unroll 4
  for (int64_t r = (int64_t)blockIdx.x * L + l; r < n; r += (int64_t)gridDim.x * L)
    a.add(x[r * FSK_D + k] * down);
  __shared__ float2 sh[PT];
  sh[threadIdx.x] = make_float2(a.s, a.c);
  __syncthreads();
  if (threadIdx.x < FSK_D) {
    float2 s = sh[threadIdx.x];
#pragma unroll
    for (int j = 1; j < L; ++j) s = df_add(s, sh[j * FSK_D + threadIdx.x]);
    part[blockIdx.x * FSK_D + threadIdx.x] = s;
  }
}

// The mean from the per-block sums into shared memory (every block, same
// order, same bits).  Any centre would do: it is subtracted exactly as
// rounded here and added back by the reductions.
__device__ __forceinline__ void block_mean(const float2* __restrict__ part, int blocks, int64_t n, float down,
                                           float (&mu)[FSK_D], float2 (&sh)[PT]) {
  constexpr int L = PT / FSK_D;
  const int k = threadIdx.x % FSK_D, l = threadIdx.x / FSK_D;
  float2 s = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int b = l; b < blocks; b += L) s = df_add(s, part[b * FSK_D + k]);
  sh[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < FSK_D) {
#pragma unroll
    for (int j = 1; j < L; ++j) s = df_add(s, sh[j * FSK_D + threadIdx.x]);
    const float n2 = (float)n * (2.f * down);   // half the mean, which cannot round to infinity
    const float q = s.x / n2;
    mu[threadIdx.x] = 2.f * (q + (fmaf(-q, n2, s.x) + s.y) / n2);
  }
  __syncthreads();
}

// Maxima for the scale selection over one block's rows: |v| (v centred), the
// norm term beta = c2 |v|^2 and alpha = |beta - alpha_off|.  Blocks below
// `data_blocks` take the data, the others the queries (none for the score,
// whose queries are the data).
__global__ void __launch_bounds__(PT) tc_stats_kernel(const float* __restrict__ x, int64_t n,
                                                      const float* __restrict__ q, int64_t m, int vec, int data_blocks,
                                                      int mean_blocks, float down, float c2, float alpha_off,
                                                      PrepBufs b) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float mu[FSK_D];
  __shared__ float2 sh[PT];
  block_mean(b.mean_part, mean_blocks, n, down, mu, sh);
  if (blockIdx.x == 0 && threadIdx.x < FSK_D) b.mu[threadIdx.x] = mu[threadIdx.x];
  const bool data = (int)blockIdx.x < data_blocks;
  const float* pts = data ? x : q;
  const int64_t count = data ? n : m;
  const int blk = data ? blockIdx.x : blockIdx.x - data_blocks;
  const int blks = data ? data_blocks : gridDim.x - data_blocks;
  float vmax = 0.f, bmax = 0.f, amax = 0.f;
  for (int64_t i = (int64_t)blk * PT + threadIdx.x; i < count; i += (int64_t)blks * PT) {
    float p[FSK_D];
    load_row(pts + i * FSK_D, vec, p);
    float nrm = 0.f;
#pragma unroll
    for (int k = 0; k < FSK_D; ++k) {
      const float v = p[k] - mu[k];
      nrm = fmaf(v, v, nrm);
      vmax = fmaxf(vmax, fabsf(v));
    }
    bmax = fmaxf(bmax, c2 * nrm);
    amax = fmaxf(amax, fabsf(c2 * nrm - alpha_off));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  }
  __shared__ float4 wmax[PW];
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = make_float4(vmax, bmax, amax, 0.f);
  __syncthreads();
  if (threadIdx.x == 0) {
    float4 t = wmax[0];
    for (int w = 1; w < PW; ++w) {
      t.x = fmaxf(t.x, wmax[w].x);
      t.y = fmaxf(t.y, wmax[w].y);
      t.z = fmaxf(t.z, wmax[w].z);
    }
    b.stats[blockIdx.x] = t;
  }
}

// smallest e with v <= 2^e (v > 0, normal)
__device__ __forceinline__ int ceil_log2(float v) {
  const uint32_t u = __float_as_uint(v);
  return (int)((u >> 23) & 255u) - 127 + ((u & 0x7FFFFFu) != 0u ? 1 : 0);
}

// Power-of-two operand scales.  q' max and x' max are balanced around
// sqrt(Lq Lx 2^-es) <= T = 2^13 (FP16_TARGET); es > 0 scales the whole
// product down where the operands or the norm terms would not fit; alpha and
// beta parts are scaled into range against exact powers of two (<= 2^15) in
// the other operand's bias columns.
__device__ __forceinline__ TcScales select_scales(float vq, float vx, float am, float bm) {
  static_assert(FP16_TARGET == 8192.0f, "T = 2^13");
  constexpr int T = 13;
  const float lq = fmaxf(vq, 1e-30f), lx = fmaxf(vx, 1e-30f);
  const float am1 = fmaxf(am, 1e-30f), bm1 = fmaxf(bm, 1e-30f);
  // ceil log2 of lq * lx: exponents plus that of the mantissa product in [1, 4)
  const int e_q = (int)(__float_as_uint(lq) >> 23) - 127, e_x = (int)(__float_as_uint(lx) >> 23) - 127;
  const float m_q = __uint_as_float((__float_as_uint(lq) & 0x7FFFFFu) | 0x3F800000u);
  const float m_x = __uint_as_float((__float_as_uint(lx) & 0x7FFFFFu) | 0x3F800000u);
  const float mp = __fmul_ru(m_q, m_x);   // rounded up: exact powers stay, everything above stays above
  const int e_prod = e_q + e_x + (mp > 2.0f ? 2 : (mp > 1.0f ? 1 : 0));
  const int es = min(64, max(max(0, e_prod - 2 * T), max(ceil_log2(am1), ceil_log2(bm1)) - T - 15));
  const int ea = max(0, ceil_log2(am1) - es - T), eb = max(0, ceil_log2(bm1) - es - T);
  // x' = (x - mu) 2^ex, q' = 2 c2 (q - mu) 2^eq, eq + ex = -es, balanced:
  // ex = floor((log2(lq / lx) - es) / 2)
  const int ex = (e_q - e_x - (m_q < m_x ? 1 : 0) - es) >> 1;
  const int eq = -es - ex;
  TcScales s;
  s.x_scale = ldexpf(1.f, ex);
  s.q_scale = ldexpf(1.f, eq);          // times 2 c2, applied to the query rows
  s.a_scale = ldexpf(1.f, -es - ea);    // alpha * a_scale in A, 2^ea in B
  s.b_scale = ldexpf(1.f, -es - eb);    // beta * b_scale in B, 2^eb in A
  s.pad[0] = ea;
  s.pad[1] = eb;
  s.pad[2] = T - ceil_log2(lx);         // (x - mu) operand of the weighted sum: max |x'| <= T
  s.out_mul = ldexpf(1.f, es);
  return s;
}

// Query tile image of row i: [H (QT x 32 fp16) | M | L (QT x 16 fp16)] and
// (score) the original coordinates, padded to whole query blocks.
__device__ __forceinline__ void query_image_row(int64_t i, bool ok, const float (&xo)[FSK_D], const float* mu, float c2,
                                                float alpha_off, const TcScales& sc, uint8_t* __restrict__ img,
                                                float* __restrict__ qexact) {
  float v[FSK_D], nrm = 0.f;
  const float qs = 2.0f * c2 * sc.q_scale;
#pragma unroll
  for (int k = 0; k < FSK_D; ++k) {
    const float cv = xo[k] - mu[k];
    nrm = fmaf(cv, cv, nrm);
    v[k] = ok ? cv * qs : 0.f;
  }
  uint8_t* tile = img + (i / QT) * (int64_t)A_TILE_BYTES;
  const float alpha = ok ? (alpha_off - c2 * nrm) * sc.a_scale : 0.f;
  write_operand_row(tile, tile + A_M_OFFSET, tile + A_L_OFFSET, (int)(i % QT), v, alpha,
                    ok ? ldexpf(1.f, sc.pad[1]) : 0.f, false);
  if (qexact == nullptr) return;
  float4* qe = reinterpret_cast<float4*>(qexact + i * FSK_D);
#pragma unroll
  for (int k = 0; k < 4; ++k) qe[k] = make_float4(xo[4 * k], xo[4 * k + 1], xo[4 * k + 2], xo[4 * k + 3]);
}

// Data image of row j.  KDE tile (128 points): [H | M | L | x (FP32)]; score
// stage (64 points): [H | M | L | XT hi (16 x 64 fp16) | XT lo | x (FP32)],
// XT rows being features, K-major over the points.
template <bool SCORE>
__device__ __forceinline__ void data_image_row(int64_t j, bool ok, const float (&xo)[FSK_D], const float* mu, float c2,
                                               const TcScales& sc, uint8_t* __restrict__ img) {
  constexpr int ROWS = SCORE ? NT : KNT;
  uint8_t* tile = img + (j / ROWS) * (int64_t)(SCORE ? S_STAGE_BYTES : KB_STAGE_BYTES);
  const int r = (int)(j % ROWS);
  float v[FSK_D], nrm = 0.f;
  const float ws = ldexpf(1.f, sc.pad[2]);
#pragma unroll
  for (int k = 0; k < FSK_D; ++k) {
    const float cv = xo[k] - mu[k];
    nrm = fmaf(cv, cv, nrm);
    v[k] = ok ? cv * sc.x_scale : 0.f;
    if (SCORE) {
      const float w = ok ? cv * ws : 0.f;
      const __half wh = __float2half_rn(w);
      put_h(tile + S_XTH_OFFSET, k, r, XT_ROW_BYTES, wh);
      put_h(tile + S_XTL_OFFSET, k, r, XT_ROW_BYTES, __float2half_rn(w - __half2float(wh)));
    }
  }
  const float beta = ok ? -c2 * nrm * sc.b_scale : 0.f;
  write_operand_row(tile, tile + (SCORE ? B_M_OFFSET : KB_M_OFFSET), tile + (SCORE ? B_L_OFFSET : KB_L_OFFSET), r, v,
                    beta, ok ? ldexpf(1.f, sc.pad[0]) : 0.f, true);
  float4* xr = reinterpret_cast<float4*>(tile + (SCORE ? S_X_OFFSET : KB_X_OFFSET) + r * (FSK_D * 4));
#pragma unroll
  for (int k = 0; k < 4; ++k) xr[k] = make_float4(xo[4 * k], xo[4 * k + 1], xo[4 * k + 2], xo[4 * k + 3]);
}

struct ImageArgs {
  const float* x;
  const float* q;
  int64_t n, n_pad, m, m_pad;
  int vec;
  int stats_blocks, data_stats;   // blocks of the stats kernel, of which data
  float c2, alpha_off;
  uint8_t* ximg;
  uint8_t* qimg;
  float* qexact;
};

// Row images.  KDE: rows [0, n_pad) data, [n_pad, n_pad + m_pad) queries.
// Score: row i < m_pad writes its query row and, below n_pad, its data row.
template <bool SCORE>
__global__ void __launch_bounds__(PT) tc_image_kernel(ImageArgs a, PrepBufs b) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float mu[FSK_D];
  __shared__ TcScales sc;
  __shared__ float4 wx[PW], wq[PW];
  if (threadIdx.x < FSK_D) mu[threadIdx.x] = b.mu[threadIdx.x];
  // maxima over the stats blocks (order does not matter)
  float4 tx = make_float4(0.f, 0.f, 0.f, 0.f), tq = tx;
  for (int i = threadIdx.x; i < a.stats_blocks; i += PT) {
    const float4 s = b.stats[i];
    if (i < a.data_stats) {
      tx.x = fmaxf(tx.x, s.x);
      tx.y = fmaxf(tx.y, s.y);
    }
    if (SCORE || i >= a.data_stats) {
      tq.x = fmaxf(tq.x, s.x);
      tq.z = fmaxf(tq.z, s.z);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    tx.x = fmaxf(tx.x, __shfl_xor_sync(0xffffffffu, tx.x, o));
    tx.y = fmaxf(tx.y, __shfl_xor_sync(0xffffffffu, tx.y, o));
    tq.x = fmaxf(tq.x, __shfl_xor_sync(0xffffffffu, tq.x, o));
    tq.z = fmaxf(tq.z, __shfl_xor_sync(0xffffffffu, tq.z, o));
  }
  if ((threadIdx.x & 31) == 0) {
    wx[threadIdx.x >> 5] = tx;
    wq[threadIdx.x >> 5] = tq;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < PW; ++w) {
      tx.x = fmaxf(tx.x, wx[w].x);
      tx.y = fmaxf(tx.y, wx[w].y);
      tq.x = fmaxf(tq.x, wq[w].x);
      tq.z = fmaxf(tq.z, wq[w].z);
    }
    sc = select_scales(2.0f * a.c2 * tq.x, tx.x, tq.z, tx.y);
    if (blockIdx.x == 0) *b.sc = sc;
  }
  __syncthreads();
  const int64_t rows = SCORE ? a.m_pad : a.n_pad + a.m_pad;
  for (int64_t e = (int64_t)blockIdx.x * PT + threadIdx.x; e < rows; e += (int64_t)gridDim.x * PT) {
    float xo[FSK_D];
#pragma unroll
    for (int k = 0; k < FSK_D; ++k) xo[k] = 0.f;
    if (SCORE) {
      const bool ok = e < a.n;
      if (ok) load_row(a.x + e * FSK_D, a.vec, xo);
      if (e < a.n_pad) data_image_row<true>(e, ok, xo, mu, a.c2, sc, a.ximg);
      query_image_row(e, ok, xo, mu, a.c2, a.alpha_off, sc, a.qimg, a.qexact);
    } else if (e < a.n_pad) {
      const bool ok = e < a.n;
      if (ok) load_row(a.x + e * FSK_D, a.vec, xo);
      data_image_row<false>(e, ok, xo, mu, a.c2, sc, a.ximg);
    } else {
      const int64_t i = e - a.n_pad;
      const bool ok = i < a.m;
      if (ok) load_row(a.q + i * FSK_D, a.vec, xo);
      query_image_row(i, ok, xo, mu, a.c2, a.alpha_off, sc, a.qimg, nullptr);
    }
  }
}

PrepBufs take_prep(WsCarver& c) {
  PrepBufs b;
  b.mean_part = c.take<float2>((size_t)MEAN_MAX_BLOCKS * FSK_D);
  b.stats = c.take<float4>((size_t)2 * STATS_MAX_BLOCKS);
  b.mu = c.take<float>(FSK_D);
  b.sc = c.take<TcScales>(1);
  return b;
}

int blocks_for(int64_t rows, int limit) { return (int)imax<int64_t>(1, imin<int64_t>(limit, (rows + PT - 1) / PT)); }

template <bool SCORE>
int launch_prep(const float* x, int64_t n, const float* q, int64_t m, double h, const TcPlan& pl, float alpha_off,
                uint8_t* ximg, uint8_t* qimg, float* qexact, WsCarver& c, TcPrep* out, cudaStream_t s) {
  const PrepBufs b = take_prep(c);
  if (!c.fits()) return FSK_ERR_WORKSPACE_TOO_SMALL;
  out->mu = b.mu;
  out->scales = b.sc;
  const float c2 = (float)(FSK_LOG2E / (2.0 * h * h));
  const int vec = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(q)) & 15) == 0;
  const int mean_blocks = blocks_for(n, MEAN_MAX_BLOCKS);
  const float down = ldexpf(1.f, -2 - (int)log2((double)n));
  tc_mean_kernel<<<mean_blocks, PT, 0, s>>>(x, n, down, b.mean_part);
  count_launch();
  const int data_stats = blocks_for(n, STATS_MAX_BLOCKS);
  const int stats_blocks = data_stats + (SCORE ? 0 : blocks_for(m, STATS_MAX_BLOCKS));
  launch_pdl(tc_stats_kernel, stats_blocks, PT, 0, s, x, n, q, m, vec, data_stats, mean_blocks, down, c2, alpha_off, b);
  count_launch();
  ImageArgs a;
  a.x = x;
  a.q = q;
  a.n = n;
  a.n_pad = pl.n_pad;
  a.m = m;
  a.m_pad = pl.m_pad;
  a.vec = vec;
  a.stats_blocks = stats_blocks;
  a.data_stats = data_stats;
  a.c2 = c2;
  a.alpha_off = alpha_off;
  a.ximg = ximg;
  a.qimg = qimg;
  a.qexact = qexact;
  launch_pdl(tc_image_kernel<SCORE>, blocks_for(SCORE ? pl.m_pad : pl.n_pad + pl.m_pad, 8 * sm_count()), PT, 0, s, a,
             b);
  count_launch();
  return FSK_OK;
}

}  // namespace

void take_tc_prep(WsCarver& c) { take_prep(c); }

int launch_kde16_prep(const float* x, int64_t n, const float* q, int64_t m, double h, const TcPlan& pl, uint8_t* ximg,
                      uint8_t* qimg, WsCarver& c, TcPrep* out, cudaStream_t s) {
  return launch_prep<false>(x, n, q, m, h, pl, 0.f, ximg, qimg, nullptr, c, out, s);
}

int launch_score16_prep(const float* x, int64_t n, double h, const TcPlan& pl, uint8_t* ximg, uint8_t* qimg,
                        float* qexact, WsCarver& c, TcPrep* out, cudaStream_t s) {
  return launch_prep<true>(x, n, x, n, h, pl, PHI_LOG2_SCALE, ximg, qimg, qexact, c, out, s);
}

}  // namespace tc
}  // namespace fsk
