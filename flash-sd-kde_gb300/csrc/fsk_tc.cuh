// fsk_tc.cuh - tile geometry, parameters and launchers of the tcgen05 kernels.
#pragma once
#include "fsk_common.cuh"

namespace fsk {
namespace tc {

// ---- geometry -----------------------------------------------------------------
constexpr int QT = 128;                 // queries per MMA tile (M, one TMEM lane each)
constexpr int NT = 64;                  // data points per 64-row operand image (score kernel stages)
// KDE kernel: 2 query tiles x 128 data points per tile (an M=128, K=16 MMA
// costs ~46 cycles for any N <= 64 and 64 cycles at N = 128, so N = 128
// halves the instruction count of the S product per pair).
constexpr int NQT = 2;                  // KDE: query tiles per work unit (256 queries)
constexpr int KNT = 128;                // KDE: data points per stage (MMA N)
constexpr int NS = 6;                   // KDE: shared-memory data stages
constexpr int KH = 32;                  // K of the "hi" operand: 16 features + 16 bias columns
// Operand images, fp16, no-swizzle K-major core-matrix layout: 8-row groups,
// each group = (K/8) core matrices of 8 rows x 16 B stored back to back.
constexpr int H_ROW_BYTES = KH * 2;     // 64 B: features (2 K-chunks) + bias (2 K-chunks)
constexpr int L_ROW_BYTES = 16 * 2;     // 32 B: features only (mid and lo parts)
// Operands are split in three fp16 parts v = hi + mid + lo (~33 significant
// bits): H holds hi and the bias columns, M the mid parts, L the lo parts.
constexpr int A_H_BYTES = QT * H_ROW_BYTES;       // 8 KB
constexpr int A_M_BYTES = QT * L_ROW_BYTES;       // 4 KB
constexpr int A_L_BYTES = QT * L_ROW_BYTES;       // 4 KB
constexpr int A_M_OFFSET = A_H_BYTES;
constexpr int A_L_OFFSET = A_H_BYTES + A_M_BYTES;
constexpr int A_TILE_BYTES = A_L_OFFSET + A_L_BYTES;  // 16 KB
constexpr int A_BYTES = NQT * A_TILE_BYTES;       // 32 KB per KDE unit
constexpr int B_H_BYTES = NT * H_ROW_BYTES;       // 4 KB
constexpr int B_M_BYTES = NT * L_ROW_BYTES;       // 2 KB
constexpr int B_L_BYTES = NT * L_ROW_BYTES;       // 2 KB
constexpr int B_M_OFFSET = B_H_BYTES;
constexpr int B_L_OFFSET = B_H_BYTES + B_M_BYTES;
constexpr int B_X_OFFSET = B_L_OFFSET + B_L_BYTES; // original FP32 rows, 64 B each
// KDE data stage: [H (128 x 32 fp16) | M (128 x 16) | L (128 x 16) | x (128 x 16 FP32)]
constexpr int KB_H_BYTES = KNT * H_ROW_BYTES;                 // 8 KB
constexpr int KB_M_OFFSET = KB_H_BYTES;
constexpr int KB_L_OFFSET = KB_M_OFFSET + KNT * L_ROW_BYTES;  // 12 KB
constexpr int KB_X_OFFSET = KB_L_OFFSET + KNT * L_ROW_BYTES;  // 16 KB
constexpr int KB_STAGE_BYTES = KB_X_OFFSET + KNT * FSK_D * 4; // 24 KB
constexpr int EPI_WARPS = 8 * NQT;      // KDE: (lane quarter, column half) per query tile
constexpr int PRODUCER_WARP = EPI_WARPS;
constexpr int MMA_WARP = EPI_WARPS + 1;   // owns TMEM, issues the MMAs
constexpr int THREADS = (EPI_WARPS + 2) * 32;
constexpr int NACC = 3;                  // KDE: accumulators, taken in turn by the query tiles
constexpr int T_KA = NACC * KNT;         // KDE: query operand in tensor memory, [NQT][hi 16 | mid 8 | lo 8]
constexpr int TMEM_COLS = 512;
constexpr int K_BAR_OFFSET = A_BYTES + NS * KB_STAGE_BYTES;
// KDE: one 64-byte slot per epilogue thread for its query's FP32 row (read by
// the exact recompute; each thread writes its own slot at the start of a unit)
constexpr int K_QX_OFFSET = K_BAR_OFFSET + 512;
constexpr int SMEM_BYTES = K_QX_OFFSET + EPI_WARPS * 32 * FSK_D * 4;
// A term is recomputed exactly when its 32-column chunk holds more than this
// fraction of the running sum of its query (the chunk included).  With the
// three-part operands the exponent of any other term is off by at most
// ~2^-25 * 2 c2 |q - mu| |x - mu| (one FP32 rounding at the magnitude of the
// cross product), so a term below an eighth of the sum moves it by well
// under 1e-6.
constexpr float NEAR_FRACTION = 1.0f / 8.0f;
constexpr float PHI_LOG2_SCALE = 15.0f;   // score weights are phi * 2^15
constexpr float FP16_TARGET = 8192.0f;  // largest operand magnitude aimed for

static_assert(T_KA + NQT * 32 <= TMEM_COLS, "TMEM budget");
static_assert(NQT == 2 && NACC == 3, "the accumulator's predecessor and the depth of its barriers");
static_assert((2 * NS + 8 * NQT + 4) * 8 + 4 <= 512, "barrier area");
static_assert(KB_STAGE_BYTES % 16 == 0 && A_BYTES % 16 == 0, "bulk copy granularity");
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");

// Score kernel data stage (64 points):
// [H | M | L | XT hi (16 x 64 fp16) | XT lo | x (64 x 16 FP32)]
constexpr int XT_ROW_BYTES = NT * 2;                       // one feature row over 64 points, fp16
constexpr int XT_BYTES = FSK_D * XT_ROW_BYTES;             // 2 KB
constexpr int S_XTH_OFFSET = B_L_OFFSET + B_L_BYTES;       // 8 KB
constexpr int S_XTL_OFFSET = S_XTH_OFFSET + XT_BYTES;      // 10 KB
constexpr int S_X_OFFSET = S_XTL_OFFSET + XT_BYTES;        // 12 KB: original FP32 rows
constexpr int S_STAGE_BYTES = S_X_OFFSET + NT * FSK_D * 4; // 16 KB

// Device-side scale state written by the prep kernels (see fsk_tc_prep.cu).
struct TcScales {
  float q_scale;   // q' = q_scale * (q - mu)       (= 2 c2 2^eq)
  float x_scale;   // x' = x_scale * (x - mu)       (= 2^ex)
  float a_scale;   // alpha part scale  2^-ea  (A bias col holds alpha*a_scale, B holds 1/a_scale)
  float b_scale;   // beta part scale   2^-eb
  float out_mul;   // a2 = out_mul * D  (1 unless the product had to be scaled down)
  int pad[3];      // ea, eb, ew: x'' = (x - mu) 2^ew is the weighted-sum operand
};

// ---- work split -------------------------------------------------------------------
// Query blocks x data tiles over `grid` CTAs, in segments: a segment is a run
// of data tiles of one query block, one accumulation and one row of partial
// sums.  CTA b first takes the `whole` query blocks b, b + grid, ... from
// their first to their last tile; all CTAs then walk the data roughly in step,
// and a wave of 152 blocks reads the score's 268 MB data image at n = 2^20, which
// exceeds the L2, 5.7 times from DRAM (ranges that start anywhere made that
// kernel 5 % slower).  The remaining rest < grid blocks form one line of rest * n_tiles
// tiles of which every CTA takes an equal contiguous range, so small problems
// neither leave the last wave empty nor pay for many short units (equal
// splits of every query block gave the score kernel 5 units of 9 tiles per
// CTA at n = 10007: 254 us against 49 us for its tiles at the large-n rate).
struct WorkLine {
  int64_t n_tiles;
  int grid, whole, rest;
  int line_grid;   // CTAs that share the line: min(grid, rest * n_tiles), at least 1
  __host__ __device__ int64_t begin(int64_t b) const {
    return imin<int64_t>(b, line_grid) * (rest * n_tiles) / line_grid;
  }
  // CTA holding tile L of the line: the largest b with begin(b) <= L
  __host__ __device__ int64_t cta_of(int64_t L) const {
    const int64_t total = rest * n_tiles;
    return ((L + 1) * line_grid + total - 1) / total - 1;
  }
  // Segments of query block qb: numbers [first, first + count).  In the line
  // both the CTA and the query block grow from one segment to the next, so
  // their sum numbers them.
  __host__ __device__ int64_t segments_of(int64_t qb, int& count) const {
    const int64_t r = qb - (int64_t)whole * grid;
    if (r < 0) {
      count = 1;
      return qb;
    }
    const int64_t b0 = cta_of(r * n_tiles);
    count = (int)(cta_of((r + 1) * n_tiles - 1) - b0) + 1;
    return qb + b0;
  }
  // number of the segment of query block qb that CTA b runs
  __host__ __device__ int64_t segment_id(int qb, int b) const { return qb < whole * grid ? qb : (int64_t)qb + b; }
  __host__ __device__ int64_t segment_bound() const { return (int64_t)(whole + 1) * grid + rest; }
};

struct Segment {
  int qb, t0, count;   // query block, first data tile, tiles
};

// Segment k of CTA b: its whole query blocks, then the one or two that its
// share of the line (at most n_tiles tiles) falls into; count = 0 at the end.
// (k is the only state a role keeps across its tile loop, where the epilogue
// warps have no registers to spare, and stays small: a count of tiles would
// pass 2^31 at 1e8 points and queries.)
__host__ __device__ inline Segment segment_at(const WorkLine& w, int b, int k) {
  Segment g;
  if (k < w.whole) {
    g.qb = b + k * w.grid;
    g.t0 = 0;
    g.count = (int)w.n_tiles;
  } else {
    const int64_t L0 = w.begin(b), L1 = w.begin((int64_t)b + 1);
    const int64_t r = L0 / w.n_tiles + (k - w.whole);   // query block of the line
    const int64_t L = imax<int64_t>(L0, r * w.n_tiles);
    g.qb = (int)r + w.whole * w.grid;
    g.t0 = (int)(L - r * w.n_tiles);
    g.count = (int)imax<int64_t>(0, imin<int64_t>((r + 1) * w.n_tiles, L1) - L);
  }
  return g;
}

struct TcParams {
  const uint8_t* qimg;
  const uint8_t* ximg;
  const float* q;         // original query rows (m, 16), for the exact recompute
  const TcScales* scales;
  int64_t m, n;
  WorkLine line;
  float c2, c2_lo, c1;
  float2* partials;       // [segment][column half][row_stride] (value, error) pairs
  int row_stride;         // rows per query block in the partials: min(m, 256)
  double* atomic_acc;
};

struct TcPlan {
  int64_t m_pad, n_pad, n_tiles, q_blocks;
  WorkLine line;
};

// Fills line from q_blocks and n_tiles.
void plan_line(TcPlan& pl);
TcPlan plan_kde16(int64_t m, int64_t n);
// Partial sums of the tensor-core KDE as the reductions read them.
struct TcPartials {
  const float2* part;
  WorkLine line;
  int row_stride;
};

// Operand preparation (fsk_tc_prep.cu): data mean, scale state and images.
struct TcPrep {
  const float* mu;
  const TcScales* scales;
};
void take_tc_prep(WsCarver& c);   // its scratch in the workspace
int launch_kde16_prep(const float* x, int64_t n, const float* q, int64_t m, double h, const TcPlan& pl, uint8_t* ximg,
                      uint8_t* qimg, WsCarver& c, TcPrep* out, cudaStream_t s);
int launch_score16_prep(const float* x, int64_t n, double h, const TcPlan& pl, uint8_t* ximg, uint8_t* qimg,
                        float* qexact, WsCarver& c, TcPrep* out, cudaStream_t s);
size_t tc_kde16_ws_bytes(const TcPlan& pl, int64_t m, bool atomic);
int launch_kde16_tc(const float* q, int64_t m, const float* x, int64_t n, double h,
                    bool laplace, bool single, bool poly, const TcPlan& pl, WsCarver& c, TcPartials* partials_out,
                    double** atomic_out, cudaStream_t s);
TcPlan plan_score16(int64_t n);
size_t tc_score16_ws_bytes(const TcPlan& pl);
// Empirical-score partials as (value, error) pairs, self pair excluded:
// ppdf [segment][column half][256], pw [segment][256][16] (centred); both in
// the kernel's scaled units (phi 2^15, x 2^ew).
struct ScPartials {
  const float2* ppdf;
  const float2* pw;
  const TcScales* scales;
  const float* mu;
  WorkLine line;
};
int launch_score16_tc(const float* x, int64_t n, double h, const TcPlan& pl, WsCarver& c,
                      ScPartials* out, cudaStream_t s);
int launch_mma_probe(const float* a, const float* b, float* d, cudaStream_t s);
int launch_mma_ts_probe(const float* a, const float* b, float* d, cudaStream_t s);
int launch_tmem_cp_probe(const float* a, uint32_t* out, cudaStream_t s);
int launch_wait_timeout_probe(int* out, cudaStream_t s);

// Sum of query i's partials (row = threadIdx.x % (blockDim.x / RL) of the
// block's rows; RL threads per row take pairs l, l + RL, ... and are added in
// thread order through shared memory).  True for the one thread that holds
// the sum of a row i < m.  Call with blockDim.x = 256 and all threads.
constexpr int TC_RED_THREADS = 256;
// One thread per row where most query blocks have at most ~3 segments.
inline bool tc_short_rows(const TcPartials& p) { return p.line.whole >= 8 || 2 * p.line.rest >= p.line.grid; }
template <int RL>
__device__ __forceinline__ bool reduce_tc_row(const TcPartials& p, int64_t i, int64_t m, double& sum) {
  constexpr int ROWS = TC_RED_THREADS / RL;
  const int l = threadIdx.x / ROWS;
  float2 a = make_float2(0.f, 0.f);
  if (i < m) {
    const int64_t qb = i / (NQT * QT);
    int segs;
    const int64_t seg0 = p.line.segments_of(qb, segs);
    const float2* row = p.part + seg0 * 2 * p.row_stride + i % (NQT * QT);
    const int pairs = 2 * segs;
#pragma unroll 4
    for (int k = l; k < pairs; k += RL) a = df_add(a, row[(int64_t)k * p.row_stride]);
  }
  if (RL > 1) {
    __shared__ float2 sh[RL][ROWS];
    const int r = threadIdx.x % ROWS;
    sh[l][r] = a;
    __syncthreads();
    if (l > 0) return false;
#pragma unroll
    for (int j = 1; j < RL; ++j) a = df_add(a, sh[j][r]);
  }
  sum = (double)a.x + (double)a.y;
  return i < m;
}

// fp16 core-matrix offset of element (row r, k) in an image whose rows are
// `row_bytes` wide (K = row_bytes / 2).
__host__ __device__ __forceinline__ uint32_t cm_offset(int r, int k, int row_bytes) {
  return (uint32_t)(r >> 3) * (uint32_t)(8 * row_bytes) + (uint32_t)(k >> 3) * 128u +
         (uint32_t)(r & 7) * 16u + (uint32_t)(k & 7) * 2u;
}

}  // namespace tc
}  // namespace fsk
