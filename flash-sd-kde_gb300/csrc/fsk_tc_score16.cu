// fsk_tc_score16.cu - tensor-core (tcgen05 / TMEM) empirical-score
// accumulators of the 16-D SD-KDE, GB300-native.
//
// What it computes, for every data point x_i (queries = data):
//   pdf_sum_i      = sum_j phi_ij,          phi_ij = exp(-||x_i - x_j||^2 / (2 h^2))
//   weighted_sum_i = sum_j phi_ij x_j
// the accumulators of kernels/flash_sd_kde/empirical.py:72-131 and
// kernels/emp_score_16d_ordered_splitk.py:20-95 (both tl.dot products with
// allow_tf32), as (value, error) partials per segment (see WorkLine); the weighted sum is kept
// centred (sum_j phi_ij (x_j - mu)) and mu * pdf_sum is added back by the
// reduction, in double-float.
//
// How (per 256-query x 64-point tile):
//  * S = the log2-domain exponent a2 + 15, three-part fp16 product of the
//    operand images of the KDE kernel (fsk_tc_kde16.cu): seven tcgen05.mma
//    per query tile, the query operand (hi | mid | lo rows) read from tensor
//    memory, where the epilogue warps copy it at the start of each unit (an
//    M=128, K=16 MMA with both operands in shared memory costs ~44 cycles
//    more).  The +15 rides in the query's bias term, so 2^S = phi * 2^15 and
//    the weights keep fp16 normal range down to phi ~ 2^-29.
//  * Epilogue: tcgen05.ld, ex2.approx, pdf chunk sums, the exact near-pair
//    recompute of the KDE kernel (the recomputed value also replaces the
//    approximate one in the weights), then the weights are split into fp16
//    hi + lo and stored with tcgen05.st over the tensor-memory columns their
//    S came from.
//  * W += Phi_hi [X_hi | X_lo] + Phi_lo X_hi: tcgen05.mma with the A operand
//    (weights, M=128 x K=16 per step) read from tensor memory and the B
//    operand ((x_j - mu) 2^ew as fp16 hi and lo rows, K-major over the data
//    points) from the data stage, FP32 accumulation over a group of tiles
//    (score_group), then added into compensated FP32 sums.
//
// Pipeline (one persistent CTA per SM, 19 warps of 96 registers):
//   warp 16 : producer (bulk copies of query images per unit, data stages).
//   warp 17 : issues S for both query tiles, up to NBUF tiles ahead of W;
//             owns TMEM.
//   warp 18 : issues the weighted-sum MMAs of both query tiles.
//   warps 0-15: epilogue; warp w: query tile w/8, data-column half (w/4)&1,
//             TMEM lane quarter w&3.  The two column halves of a row keep
//             separate pdf partials (two rows per segment) and
//             read disjoint halves of the weighted-sum features.
//
// What bounds it: the epilogue's instructions.  Per tile a warp runs ~250 of
// them for 32 columns; issue slots are 70 % busy, exp pipe 36 %, tensor core
// 45 %.  So the tile loop is kept short: rare work (scaled sums, ragged and
// diagonal columns in one block, near pairs, group read-out) is marked
// unlikely and stays behind the straight path, and the weights are stored
// before the sums, whose latency covers that of the stores.  n = 262144:
// 24.1 ms with seven issuing warps of 80 registers and separate ragged and
// diagonal blocks, 20.6 this way, 20.0 with one weighted-sum issuer instead
// of one per query tile (its polling took issue slots) and five data stages
// (2^20: 381, 328, 318), 19.8 (316) with the waits' slow path out of line.
// Tried and slower: one warp for all MMAs (29.9), eight
// warps of 64 columns (28.6 ms), S and weights in separate columns with one
// buffer each (25.9), the rare blocks as calls (21.6-22.3), the next tile's S
// loaded ahead (25.0, spills).
// TMEM: A operands [2 query tiles][hi 16 | mid 8 | lo 8]  (columns 0-63)
//       | S / weights [NBUF buffers][2 query tiles][64]  (64-319)
//       | W [2 group parities][2 query tiles][hi part 32 | lo part 16]  (320-511).
#include <cuda_fp16.h>

#include "fsk_kernels.cuh"
#include "fsk_tc.cuh"
#include "fsk_tc_ops.cuh"

namespace fsk {
namespace tc {

namespace {

constexpr int SNQT = 2;                                    // query tiles per unit (256 queries)
constexpr int SNS = 5;                                     // data stages
constexpr int S_A_BYTES = SNQT * A_TILE_BYTES;             // 32 KB
constexpr int S_EPI_WARPS = 8 * SNQT;
constexpr int S_PRODUCER_WARP = S_EPI_WARPS;
constexpr int S_MMA_WARP = S_EPI_WARPS + 1;     // issues the S MMAs, owns TMEM
constexpr int W_MMA_WARP = S_EPI_WARPS + 2;     // issues the weighted-sum MMAs
constexpr int S_THREADS = (S_EPI_WARPS + 3) * 32;
constexpr int NBUF = 2;                                    // S / weight buffers in TMEM
constexpr int WN = 2 * FSK_D;                              // W MMA N, hi weights: X_hi and X_lo rows
constexpr int WN_LO = FSK_D;                               // W MMA N, lo weights: X_hi rows
constexpr int T_A = 0;                                     // [SNQT][32]: hi 16 | mid 8 | lo 8
constexpr int T_S = 64;
constexpr int T_W = T_S + NBUF * SNQT * NT;                // 320
constexpr int W_TILE_COLS = WN + WN_LO;                    // 48 per (parity, query tile)
constexpr int S_TMEM_COLS = 512;
// exact-recompute corrections of the weighted sums: [unit parity][column half][256 rows][16] FP32
// original coordinates of the unit's 256 queries (exact near-pair recompute)
constexpr int S_QX_OFFSET = S_A_BYTES;
constexpr int S_QX_BYTES = SNQT * QT * FSK_D * 4;                    // 16 KB
constexpr int S_B_OFFSET = S_QX_OFFSET + S_QX_BYTES;
constexpr int S_BAR_OFFSET = S_B_OFFSET + SNS * S_STAGE_BYTES;
constexpr int S_WCORR_OFFSET = S_BAR_OFFSET + 512;
constexpr int S_WCORR_BYTES = 2 * 2 * SNQT * QT * FSK_D * 4;          // 64 KB
// compensated per-thread weighted-sum accumulators (8 features, value + error),
// float4 planes [s0-3, s4-7, c0-3, c4-7][epilogue thread]
constexpr int S_WACC_OFFSET = S_WCORR_OFFSET + S_WCORR_BYTES;
constexpr int S_WACC_BYTES = 4 * S_EPI_WARPS * 32 * 16;                // 32 KB
constexpr int S_MU_OFFSET = S_WACC_OFFSET + S_WACC_BYTES;             // data mean, 16 FP32
constexpr int S_SMEM_BYTES = S_MU_OFFSET + FSK_D * 4;
// Three-part S product as in the KDE kernel, so the same near-pair threshold
// (1/8 of the running sum, the excluded self pair's weight included).
constexpr float SCORE_NEAR_FRACTION = NEAR_FRACTION;
static_assert(T_W + 2 * SNQT * W_TILE_COLS <= S_TMEM_COLS, "TMEM budget");
static_assert(S_XTL_OFFSET == S_XTH_OFFSET + 16 * XT_ROW_BYTES, "X_lo rows follow X_hi rows (one N=32 operand)");
static_assert(S_STAGE_BYTES % 16 == 0 && S_A_BYTES % 16 == 0 && S_QX_BYTES % 16 == 0, "bulk copy granularity");
static_assert(S_SMEM_BYTES <= 227 * 1024, "shared memory");
static_assert((2 * SNS + 3 * NBUF * SNQT + 4 * SNQT + SNQT + 4) * 8 + 4 <= 512, "barrier area");

struct ScParams {
  const uint8_t* qimg;
  const uint8_t* ximg;
  const float* qexact;
  const TcScales* scales;
  const float* mu;
  int64_t n;
  WorkLine line;
  int group;      // data tiles per W accumulation in tensor memory
  float c2, c2_lo;
  // (value, error) pairs per segment, self pair excluded, in the kernel's
  // scaled units: pdf [segment][column half][256], centred weighted sums
  // [segment][256][16]
  float2* ppdf;
  float2* pw;
};

// f32 pair -> packed fp16 hi and lo parts (hi + lo = v to ~22 bits).  The
// residual v - hi is exact in FP32 (hi holds v's leading 11 bits) and comes
// from one mixed-precision FMA per value, fp16 hi times -1 plus the FP32 v.
__device__ __forceinline__ void split_pack(float v0, float v1, uint32_t& hi, uint32_t& lo) {
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(v1), "f"(v0));
  float r0, r1;
  const unsigned short minus_one = 0xBC00;   // fp16 -1
  asm("{\n\t.reg .b16 h0, h1;\n\tmov.b32 {h0, h1}, %2;\n\t"
      "fma.rn.f32.f16 %0, h0, %5, %3;\n\tfma.rn.f32.f16 %1, h1, %5, %4;\n\t}"
      : "=f"(r0), "=f"(r1)
      : "r"(hi), "f"(v0), "f"(v1), "h"(minus_one));
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(r1), "f"(r0));
}

__global__ void __launch_bounds__(S_THREADS, 1) score16_tc_kernel(ScParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sA = smem_raw;
  const float* sQ = reinterpret_cast<const float*>(smem_raw + S_QX_OFFSET);
  uint8_t* sB = smem_raw + S_B_OFFSET;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + S_BAR_OFFSET);
  float* sMu = reinterpret_cast<float*>(smem_raw + S_MU_OFFSET);
  uint64_t* full = bars;                          // [SNS] stage loaded
  uint64_t* empty = bars + SNS;                   // [SNS] stage consumed (W MMAs + epilogue)
  uint64_t* tfull = bars + 2 * SNS;               // [NBUF][SNQT] S written
  // [NBUF][SNQT] weights stored.  One barrier per buffer and query tile: a
  // buffer's barrier cannot complete again before its weights are consumed.
  uint64_t* pready = tfull + NBUF * SNQT;
  uint64_t* sfree = pready + NBUF * SNQT;         // [NBUF][SNQT] weights read by the W MMAs
  uint64_t* wfull = sfree + NBUF * SNQT;          // [2 parities][SNQT] W group accumulated
  uint64_t* wempty = wfull + 2 * SNQT;            // [2 parities][SNQT] W group read
  uint64_t* aready = wempty + 2 * SNQT;           // [SNQT] unit's A operand in TMEM
  uint64_t* qready = aready + SNQT;
  uint64_t* qempty = qready + 1;
  uint64_t* drain = qready + 2;                   // all MMAs of this CTA finished (exit path)
  uint64_t* cready = qready + 3;                  // unit's W corrections written (epilogue warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(qready + 4);
  float* wcorr = reinterpret_cast<float*>(smem_raw + S_WCORR_OFFSET);
  float4* wacc = reinterpret_cast<float4*>(smem_raw + S_WACC_OFFSET);
  int64_t n_stage_copies = 0, n_query_copies = 0;   // producer: bulk copies issued

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < SNS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], SNQT + S_EPI_WARPS);   // W commits of both query tiles + every epilogue warp
    }
    for (int i = 0; i < NBUF * SNQT; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&pready[i], 8);
      mbar_init(&sfree[i], 1);
    }
    for (int i = 0; i < 2 * SNQT; ++i) {
      mbar_init(&wfull[i], 1);
      mbar_init(&wempty[i], 8);
    }
    for (int a = 0; a < SNQT; ++a) mbar_init(&aready[a], 8);
    mbar_init(qready, 1);
    mbar_init(qempty, S_EPI_WARPS);
    mbar_init(drain, 2);   // the S and the W issuer
    mbar_init(cready, S_EPI_WARPS);
    fence_barrier_init();
  }
  if (warp == S_MMA_WARP) {
    tmem_alloc(tmem_slot, S_TMEM_COLS);
    tmem_relinquish();
  }
  pdl_wait();   // the images, mean and scales of the preparation
  if (threadIdx.x < FSK_D) sMu[threadIdx.x] = p.mu[threadIdx.x];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == S_PRODUCER_WARP) {
    // whole warp runs the loop (32-bit stage / phase counters), lane 0 copies
    {
      int64_t& g = n_stage_copies;
      int64_t& k = n_query_copies;
      int st = 0;
      uint32_t ph = 0;
      for (int k_seg = 0;; ++k_seg) {
        const Segment sg = segment_at(p.line, blockIdx.x, k_seg);
        if (sg.count == 0) break;
        if (!__all_sync(0xffffffffu, mbar_wait_cold(qempty, (uint32_t)((k & 1) ^ 1), 21))) goto done;
        if (lane == 0) {
          mbar_arrive_expect_tx(qready, S_A_BYTES + S_QX_BYTES);
          bulk_g2s(sA, p.qimg + sg.qb * (int64_t)S_A_BYTES, S_A_BYTES, qready);
          bulk_g2s(smem_raw + S_QX_OFFSET, p.qexact + sg.qb * (int64_t)(SNQT * QT * FSK_D), S_QX_BYTES, qready);
        }
        ++k;
        const uint8_t* src = p.ximg + sg.t0 * (int64_t)S_STAGE_BYTES;
        for (int i = 0; i < sg.count; ++i, src += S_STAGE_BYTES) {
          if (!__all_sync(0xffffffffu, mbar_wait_cold(&empty[st], ph ^ 1u, 22))) goto done;
          if (lane == 0) {
            mbar_arrive_expect_tx(&full[st], S_STAGE_BYTES);
            bulk_g2s(sB + st * S_STAGE_BYTES, src, S_STAGE_BYTES, &full[st]);
          }
          ++g;
          if (++st == SNS) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
    }
  } else if (warp == S_MMA_WARP) {
    // S(g) of both query tiles for every tile, up to NBUF tiles ahead of W:
    // buffer g % NBUF is reused once the W MMAs of tile g - NBUF have read its
    // weights (sfree).  S and W are issued by different threads because
    // tcgen05.commit tracks every earlier MMA of its thread.  The whole warp
    // runs the loop (warp-uniform values stay in uniform registers), one lane
    // issues the MMAs and commits.
    {
      const uint32_t idesc_s = idesc_f16_f32(QT, NT);
      // descriptors are advanced by adding (bytes >> 4) to the start-address
      // field (shared addresses stay below 2^18 B, so the field cannot carry)
      const uint32_t b0 = smem_u32(sB);
      const uint64_t dh0 = smem_desc_kmajor(b0, 128, 8 * H_ROW_BYTES);
      const uint64_t dm0 = smem_desc_kmajor(b0 + B_M_OFFSET, 128, 8 * L_ROW_BYTES);
      const uint64_t dl0 = smem_desc_kmajor(b0 + B_L_OFFSET, 128, 8 * L_ROW_BYTES);
      uint32_t gs = 0;     // data tile (modulo 2^32: only its low bits are used)
      int s = 0;           // its stage
      uint32_t sph = 0;    // and that one's phase
      for (int ku = 0;; ++ku) {
        const int count = segment_at(p.line, blockIdx.x, ku).count;
        if (count == 0) break;
        for (int i = 0; i < count; ++i, ++gs) {
          const uint32_t b = gs % NBUF;
          if (!__all_sync(0xffffffffu, mbar_wait_cold(&full[s], sph, 24))) goto done;
          const uint64_t so = (uint64_t)((s * S_STAGE_BYTES) >> 4);
          const uint64_t b_h = dh0 + so, b_m = dm0 + so, b_l = dl0 + so;
#pragma unroll
          for (int a = 0; a < SNQT; ++a) {
            // the segment's A operand in TMEM
            if (i == 0 && !__all_sync(0xffffffffu, mbar_wait_cold(&aready[a], (uint32_t)(ku & 1), 23))) goto done;
            // (before the first tiles: a phase that has passed)
            if (!__all_sync(0xffffffffu, mbar_wait_cold(&sfree[b * SNQT + a], ((gs / NBUF) & 1u) ^ 1u, 25))) goto done;
            tc_fence_after();
            const uint32_t a_h = tmem_base + (uint32_t)(T_A + a * 32);   // hi: features | bias; mid at +16, lo at +24
            const uint32_t d = tmem_base + T_S + b * (SNQT * NT) + (uint32_t)(a * NT);
            // three-part product, small terms first (the order of mma_s_tile)
            if (elect_one()) {
              mma_s_tile(d, a_h, b_h, b_m, b_l, idesc_s);
              mma_commit(&tfull[b * SNQT + a]);
            }
            __syncwarp();
          }
          if (++s == SNS) {
            s = 0;
            sph ^= 1u;
          }
        }
      }
    }
  } else if (warp == W_MMA_WARP) {
    // W(g) of both query tiles in turn, each once its epilogue warps have
    // stored tile g's weights (whole warp runs the loop, one lane issues).
    {
      const uint32_t idesc_hi = idesc_f16_f32(QT, WN), idesc_lo = idesc_f16_f32(QT, WN_LO);
      const uint64_t dx0 = smem_desc_kmajor(smem_u32(sB) + S_XTH_OFFSET, 128, 8 * XT_ROW_BYTES);
      uint32_t gw = 0, grp = 0;   // data tile and group (modulo 2^32)
      int s = 0;                  // the tile's stage
      for (int k_seg = 0;; ++k_seg) {
        const int count = segment_at(p.line, blockIdx.x, k_seg).count;
        if (count == 0) break;
        int left = 0;   // tiles left in the group
        for (int i = 0; i < count; ++i, ++gw, s = (s + 1 == SNS) ? 0 : s + 1) {
          const uint32_t b = gw % NBUF;
          const bool first = left == 0;
          if (first) left = p.group;
          const bool last = --left == 0 || i == count - 1;
          const uint32_t par = grp & 1u;
#pragma unroll
          for (int a = 0; a < SNQT; ++a) {
            if (first &&
                !__all_sync(0xffffffffu, mbar_wait_cold(&wempty[par * SNQT + a], ((grp >> 1) & 1u) ^ 1u, 26)))
              goto done;
            if (!__all_sync(0xffffffffu, mbar_wait_cold(&pready[b * SNQT + a], (gw / NBUF) & 1u, 27))) goto done;
            tc_fence_after();
            const uint64_t xd0 = dx0 + (uint64_t)((s * S_STAGE_BYTES) >> 4);
            const uint32_t ph = tmem_base + T_S + b * (SNQT * NT) + (uint32_t)(a * NT);
            const uint32_t d = tmem_base + T_W + par * (SNQT * W_TILE_COLS) + (uint32_t)(a * W_TILE_COLS);
            if (elect_one()) {
#pragma unroll
              for (int ks = 0; ks < NT / 16; ++ks) {
                // data columns 16 ks .. +15: column half ks/2; weights hi at +0, lo at +16
                const uint32_t wa = ph + (uint32_t)(32 * (ks >> 1) + 8 * (ks & 1));
                const uint64_t xd = xd0 + (uint64_t)(ks * (256 >> 4));
                const uint32_t add = ks > 0 || !first;
                mma_f16_ts(d, wa, xd, idesc_hi, add);              // hi weights x [X_hi | X_lo]
                mma_f16_ts(d + WN, wa + 16u, xd, idesc_lo, add);   // lo weights x X_hi
              }
              mma_commit(&sfree[b * SNQT + a]);
              mma_commit(&empty[s]);
              if (last) mma_commit(&wfull[par * SNQT + a]);
            }
            __syncwarp();
          }
          if (last) ++grp;
        }
      }
    }
  } else {
    // ---------------- epilogue warps ----------------
    // The self pair (data index == query index) is left out of every sum
    // here; the reduce pass adds it exactly (phi = 1, weight x_i).  Its
    // weight still counts in the near-pair threshold: pdf_sum >= 1.
    const int qt = warp >> 3;             // query tile
    const int half = (warp >> 2) & 1;     // data-column half
    const int quarter = warp & 3;         // TMEM lane quarter
    const int row = quarter * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const float out_mul = p.scales->out_mul;
    const bool scaled = out_mul != 1.0f;
    const float phi_scale = 32768.0f;     // 2^PHI_LOG2_SCALE
    // correction rows: wcorr[parity][half][qt*128 + row][16]
    const int wc_row = (qt * QT + row) * FSK_D;
    constexpr int WC_HALF = SNQT * QT * FSK_D, WC_PAR = 2 * WC_HALF;
#pragma unroll
    for (int par = 0; par < 2; ++par)
#pragma unroll
      for (int k = 0; k < FSK_D; k += 4)
        *reinterpret_cast<float4*>(wcorr + par * WC_PAR + half * WC_HALF + wc_row + k) =
            make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t g = 0, grp = 0;   // data tile and W group (modulo 2^32)
    int s = 0;   // data stage of tile g (g % SNS, advanced per tile)
    // valid columns of the last (possibly ragged) data tile; every other tile has NT
    const int last_t = (int)p.line.n_tiles - 1;
    const int last_valid = (int)(p.n - (int64_t)last_t * NT);
    for (int k_unit = 0;; ++k_unit) {
      const Segment sg = segment_at(p.line, blockIdx.x, k_unit);
      if (sg.count == 0) break;
      const int qb = sg.qb;
      const int gi = qb * (SNQT * QT) + qt * QT + row;
      const int diag_col = qb * (SNQT * QT) + qt * QT + quarter * 32;   // this warp's rows
      float* wc = wcorr + (k_unit & 1) * WC_PAR + half * WC_HALF + wc_row;
      // The unit's query images: this row's A operand to TMEM (column half 0
      // copies the hi row, half 1 the mid and lo rows).  The S MMAs of the previous
      // unit have all completed: this warp consumed their accumulators.
      if (!__all_sync(0xffffffffu, mbar_wait_cold(qready, (uint32_t)(k_unit & 1), 36))) goto done;
      {
        const uint8_t* tile = sA + qt * A_TILE_BYTES;
        const uint32_t ta = tmem_base + lane_off + (uint32_t)(T_A + qt * 32);
        if (half == 0) {
          uint32_t w[16];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 v = *reinterpret_cast<const uint4*>(tile + cm_offset(row, 8 * c, H_ROW_BYTES));
            w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
          }
          tmem_st16(ta, w);
        } else {
          uint32_t w[16];   // mid row, then lo row
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 v = *reinterpret_cast<const uint4*>(tile + (c < 2 ? A_M_OFFSET : A_L_OFFSET) +
                                                            cm_offset(row, 8 * (c & 1), L_ROW_BYTES));
            w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
          }
          tmem_st16(ta + 16u, w);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&aready[qt]);
      }
      Comp acc{0.f, 0.f};
      float corr = 0.f;
      constexpr int EPI_T = S_EPI_WARPS * 32;
#pragma unroll
      for (int k = 0; k < 4; ++k) wacc[k * EPI_T + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
      auto read_group = [&]() -> bool {
        const int par = grp & 1;
        if (!__all_sync(0xffffffffu, mbar_wait_cold(&wfull[par * SNQT + qt], (uint32_t)((grp >> 1) & 1), 30))) return false;
        tc_fence_after();
        // this warp's 8 features: hi weights x X_hi, hi weights x X_lo, lo weights x X_hi
        uint32_t wv[8], wl[8], wm[8];
        const uint32_t wcol = tmem_base + lane_off + (uint32_t)(T_W + par * (SNQT * W_TILE_COLS) + qt * W_TILE_COLS + half * 8);
        tmem_ld8(wcol, wv);
        tmem_ld8(wcol + FSK_D, wl);
        tmem_ld8(wcol + WN, wm);
        tmem_ld_wait();
#pragma unroll
        for (int k = 0; k < 8; ++k)
          wv[k] = __float_as_uint(__uint_as_float(wv[k]) + (__uint_as_float(wl[k]) + __uint_as_float(wm[k])));
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&wempty[par * SNQT + qt]);
        {
          float4 s0 = wacc[threadIdx.x], s1 = wacc[EPI_T + threadIdx.x];
          float4 e0 = wacc[2 * EPI_T + threadIdx.x], e1 = wacc[3 * EPI_T + threadIdx.x];
          Comp c;
#define FSK_WADD(S, E, V) c = Comp{S, E}; c.add(__uint_as_float(V)); S = c.s; E = c.c;
          FSK_WADD(s0.x, e0.x, wv[0]) FSK_WADD(s0.y, e0.y, wv[1])
          FSK_WADD(s0.z, e0.z, wv[2]) FSK_WADD(s0.w, e0.w, wv[3])
          FSK_WADD(s1.x, e1.x, wv[4]) FSK_WADD(s1.y, e1.y, wv[5])
          FSK_WADD(s1.z, e1.z, wv[6]) FSK_WADD(s1.w, e1.w, wv[7])
#undef FSK_WADD
          wacc[threadIdx.x] = s0;
          wacc[EPI_T + threadIdx.x] = s1;
          wacc[2 * EPI_T + threadIdx.x] = e0;
          wacc[3 * EPI_T + threadIdx.x] = e1;
        }
        ++grp;
        return true;
      };
      const int t0 = sg.t0;
      const int t1 = t0 + sg.count;
      bool pend = false;     // a W group ended at the previous tile and is not read yet
      int left = p.group;    // tiles left in the group
      for (int t = t0; t < t1; ++t, ++g, s = (s + 1 == SNS) ? 0 : s + 1) {
        const int b = g % NBUF;
        const int valid = t == last_t ? last_valid : NT;
        if (!__all_sync(0xffffffffu, mbar_wait_cold(&tfull[b * SNQT + qt], (uint32_t)((g / NBUF) & 1), 28))) goto done;
        tc_fence_after();
        const uint8_t* stage = sB + s * S_STAGE_BYTES;
        // this warp's 32 S columns; its weights go back into the same columns
        const uint32_t my_cols = tmem_base + lane_off + (uint32_t)(T_S + b * (SNQT * NT) + qt * NT + half * 32);
        uint32_t r[32];
        tmem_ld32(my_cols, r);
        tmem_ld_wait();
        float e[32];
        if (__builtin_expect(scaled, 0)) {
#pragma unroll
          for (int j = 0; j < 32; ++j) e[j] = __uint_as_float(r[j]) * out_mul;
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) e[j] = __uint_as_float(r[j]);
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) e[j] = ex2_approx(e[j]);
        const bool diag = t * NT + half * 32 == diag_col;   // these 32 columns are this warp's 32 rows
        if (__builtin_expect(diag || valid < NT, 0)) {
          // columns past the data and the self pair
          const int n_ok = imin(32, imax(0, valid - half * 32));
          const uint32_t drop = ~(n_ok == 32 ? 0xffffffffu : (1u << n_ok) - 1u) | (diag ? 1u << lane : 0u);
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (drop & (1u << j)) e[j] = 0.f;
        }
        // fp16 hi / lo weights for the W product, written over this warp's
        // S columns (hi: 16 columns of packed pairs, then lo), eight pairs at
        // a time to keep the register peak low
#pragma unroll
        for (int h8 = 0; h8 < 2; ++h8) {
          uint32_t hi[8], lo[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) split_pack(e[16 * h8 + 2 * j], e[16 * h8 + 2 * j + 1], hi[j], lo[j]);
          tmem_st8(my_cols + (uint32_t)(8 * h8), hi);
          tmem_st8(my_cols + (uint32_t)(16 + 8 * h8), lo);
        }
        float2 pa = make_float2(e[0], e[1]), pb = make_float2(e[2], e[3]);
#pragma unroll
        for (int j = 4; j < 32; j += 4) {
          pa = __fadd2_rn(pa, make_float2(e[j], e[j + 1]));
          pb = __fadd2_rn(pb, make_float2(e[j + 2], e[j + 3]));
        }
        pa = __fadd2_rn(pa, pb);
        const float cs = pa.x + pa.y;
        const bool trig = cs > (phi_scale + acc.s + cs) * SCORE_NEAR_FRACTION;   // phi_scale: the self pair
        if (__builtin_expect(__any_sync(0xffffffffu, trig), 0)) {
          // The chunk's largest weight A is recomputed exactly (argmax on keys =
          // value bits with the column in the low 5 bits; A is then taken from the
          // column, since the key is up to 31 ulps off the value in the sum).  The
          // pdf gets ex - A (corr) and the weighted sum (ex - A)(x_j - mu)
          // (shared-memory corrections).
          if (trig) {
            // (an opaque copy for the compiler: 2932 us at n = 100000 with it, 2985
            // without)
#pragma unroll
            for (int k = 0; k < 32; ++k) asm volatile("" : "+f"(e[k]));
            uint32_t k0 = 0u, k1 = 0u, k2 = 0u, k3 = 0u;
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              k0 = max(k0, (__float_as_uint(e[j]) & ~31u) | (uint32_t)j);
              k1 = max(k1, (__float_as_uint(e[j + 1]) & ~31u) | (uint32_t)(j + 1));
              k2 = max(k2, (__float_as_uint(e[j + 2]) & ~31u) | (uint32_t)(j + 2));
              k3 = max(k3, (__float_as_uint(e[j + 3]) & ~31u) | (uint32_t)(j + 3));
            }
            const int j = (int)(max(max(k0, k1), max(k2, k3)) & 31u);
            // column j of e, which is not needed after this: halves until one is left
#pragma unroll
            for (int w = 16; w > 0; w >>= 1)
#pragma unroll
              for (int k = 0; k < w; ++k) e[k] = (j & w) ? e[k + w] : e[k];
            const float top = e[0];
            const int col = half * 32 + j;
            const float4* xr = reinterpret_cast<const float4*>(stage + S_X_OFFSET + col * (FSK_D * 4));
            // exact squared distance, four features at a time
            const float4* qr = reinterpret_cast<const float4*>(sQ + (qt * QT + row) * FSK_D);
            float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const float4 qv = qr[kk], xv = xr[kk];
              const float a0 = qv.x - xv.x, a1 = qv.y - xv.y, a2 = qv.z - xv.z, a3 = qv.w - xv.w;
              d0 = fmaf(a0, a0, d0);
              d1 = fmaf(a1, a1, d1);
              d2 = fmaf(a2, a2, d2);
              d3 = fmaf(a3, a3, d3);
            }
            const float dist = (d0 + d1) + (d2 + d3);
            float ex = exp2_neg_scaled(dist, p.c2, p.c2_lo) * phi_scale;
            if (col >= valid || t * NT + col == gi) ex = 0.f;
            const float delta = ex - top;
            corr += delta;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const float4 xv = xr[kk];
              const float4 mv = reinterpret_cast<const float4*>(sMu)[kk];
              float4 cv = *reinterpret_cast<float4*>(wc + 4 * kk);
              cv.x = fmaf(delta, xv.x - mv.x, cv.x);
              cv.y = fmaf(delta, xv.y - mv.y, cv.y);
              cv.z = fmaf(delta, xv.z - mv.z, cv.z);
              cv.w = fmaf(delta, xv.w - mv.w, cv.w);
              *reinterpret_cast<float4*>(wc + 4 * kk) = cv;
            }
          }
          __syncwarp();
        }
        acc.add(cs);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&pready[b * SNQT + qt]);
          mbar_arrive(&empty[s]);
        }
        // read a W group that ended at the previous tile (its MMAs were
        // issued after that tile's weights, so by now they are usually done)
        if (__builtin_expect(pend, 0) && !read_group()) goto done;
        pend = --left == 0;
        if (pend) left = p.group;
      }
      if (!read_group()) goto done;   // the segment's last group
      // Combine the two column halves' corrections of this row for the 8
      // features this warp outputs.  Buffers alternate by unit parity; the
      // previous parity is cleared once every warp has passed this unit's
      // barrier (so has finished reading it).
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(cready);
        mbar_arrive(qempty);   // done with this unit's query images and rows in shared memory
      }
      if (!__all_sync(0xffffffffu, mbar_wait_cold(cready, (uint32_t)(k_unit & 1), 35))) goto done;
      {
        float* wc_next = wcorr + ((k_unit + 1) & 1) * WC_PAR + half * WC_HALF + wc_row;
#pragma unroll
        for (int k = 0; k < FSK_D; k += 4)
          *reinterpret_cast<float4*>(wc_next + k) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      if (gi < p.n) {
        // (value, error) pairs in the kernel's units: the FP64 unit (2 lanes
        // per clock per SM) took ~8 us per unit here when these were FP64 sums
        const float w_mul = ldexpf(1.f, p.scales->pad[2]);   // weighted-sum operand scale 2^ew
        const int64_t seg = p.line.segment_id(qb, blockIdx.x);
        const int64_t n_seg = p.line.segment_bound();
        const int64_t pidx = (2 * seg + half) * (SNQT * QT) + qt * QT + row;
        if (in_bounds(pidx, 2 * n_seg * (SNQT * QT), 42)) p.ppdf[pidx] = make_float2(acc.s, acc.c + corr);
        const int64_t wbase = (seg * (SNQT * QT) + qt * QT + row) * FSK_D + half * 8;   // 8 features from here
        const bool w_ok = in_bounds(wbase, n_seg * (SNQT * QT) * FSK_D - 7, 43);
        float4* wrow = reinterpret_cast<float4*>(p.pw + wbase);
        const float4* c0 = reinterpret_cast<const float4*>(wcorr + (k_unit & 1) * WC_PAR + wc_row + half * 8);
        const float4* c1 = c0 + WC_HALF / 4;
        if (w_ok) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float4 v = wacc[k * EPI_T + threadIdx.x], e = wacc[(2 + k) * EPI_T + threadIdx.x];
            const float4 a = c0[k], b = c1[k];
            wrow[2 * k] = make_float4(v.x, fmaf(a.x + b.x, w_mul, e.x), v.y, fmaf(a.y + b.y, w_mul, e.y));
            wrow[2 * k + 1] = make_float4(v.z, fmaf(a.z + b.z, w_mul, e.z), v.w, fmaf(a.w + b.w, w_mul, e.w));
          }
        }
      }
    }
  }
done:
  pdl_launch_dependents();
  // Exit path (also after a timed-out wait): let this CTA's bulk copies and
  // MMAs finish before shared and tensor memory are released.
  if (warp == S_PRODUCER_WARP && lane == 0) {
    for (int64_t i = imax<int64_t>(0, n_stage_copies - SNS); i < n_stage_copies; ++i)
      mbar_wait_cold(&full[i % SNS], (uint32_t)((i / SNS) & 1), 32);
    if (n_query_copies > 0) mbar_wait_cold(qready, (uint32_t)((n_query_copies - 1) & 1), 33);
  }
  if (warp >= S_MMA_WARP && elect_one()) {
    mma_commit(drain);   // one arrival per issuing thread, when its MMAs have finished
    mbar_wait_cold(drain, 0, 34);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == S_MMA_WARP) tmem_dealloc(tmem_base, S_TMEM_COLS);
}

}  // namespace

// Data tiles per W accumulation.  The tensor core's FP32 accumulation over a
// group is the largest error of the weighted sums and grows with its length
// (debiased points against FP64, rows sorted by a feature: ~4e-8 per tile of
// the group); each group's read-out costs about half a tile.  Small problems,
// bound by launches and not by tiles, take short groups.  The lengths are
// those of equal splits of every query block (2 or 3 tiles at n = 8000 to
// 10000, 10 at 19500, 13 to 16 above) at the sizes where those were shortest:
// with tiles / 8 here the error was up to twice as large between them.
static int score_group(const TcPlan& pl) {
  const int64_t tiles = pl.q_blocks * pl.n_tiles / pl.line.grid;   // per CTA
  if (tiles >= 16384) return 16;
  if (tiles >= 1024) return 15;
  return (int)imin<int64_t>(13, imax<int64_t>(1, tiles / 15));
}

TcPlan plan_score16(int64_t n) {
  TcPlan pl;
  pl.m_pad = (n + SNQT * QT - 1) / (SNQT * QT) * (SNQT * QT);
  pl.n_tiles = (n + NT - 1) / NT;
  pl.n_pad = pl.n_tiles * NT;
  pl.q_blocks = pl.m_pad / (SNQT * QT);
  plan_line(pl);
  return pl;
}

size_t tc_score16_ws_bytes(const TcPlan& pl) {
  WsCarver c(nullptr, 0);
  c.take<uint8_t>((size_t)pl.q_blocks * S_A_BYTES);
  c.take<float>((size_t)pl.m_pad * FSK_D);
  c.take<uint8_t>((size_t)pl.n_tiles * S_STAGE_BYTES);
  c.take<float2>((size_t)pl.line.segment_bound() * 2 * SNQT * QT);
  c.take<float2>((size_t)pl.line.segment_bound() * SNQT * QT * FSK_D);
  take_tc_prep(c);
  return align_up(c.used, 256);
}

int launch_score16_tc(const float* x, int64_t n, double h, const TcPlan& pl, WsCarver& c,
                      ScPartials* out, cudaStream_t s) {
  uint8_t* qimg = c.take<uint8_t>((size_t)pl.q_blocks * S_A_BYTES);
  float* qexact = c.take<float>((size_t)pl.m_pad * FSK_D);
  uint8_t* ximg = c.take<uint8_t>((size_t)pl.n_tiles * S_STAGE_BYTES);
  float2* ppdf = c.take<float2>((size_t)pl.line.segment_bound() * 2 * SNQT * QT);
  float2* pw = c.take<float2>((size_t)pl.line.segment_bound() * SNQT * QT * FSK_D);
  if (!c.fits()) return FSK_ERR_WORKSPACE_TOO_SMALL;
  TcPrep prep;
  const int st = launch_score16_prep(x, n, h, pl, ximg, qimg, qexact, c, &prep, s);
  if (st) return st;
  *out = ScPartials{ppdf, pw, prep.scales, prep.mu, pl.line};
  const double c2d = FSK_LOG2E / (2.0 * h * h);
  const float c2 = (float)c2d;
  const float c2_lo = (float)(c2d - (double)c2);

  ScParams p;
  p.qimg = qimg;
  p.ximg = ximg;
  p.qexact = qexact;
  p.scales = prep.scales;
  p.mu = prep.mu;
  p.n = n;
  p.line = pl.line;
  p.group = score_group(pl);
  p.c2 = c2;
  p.c2_lo = c2_lo;
  p.ppdf = ppdf;
  p.pw = pw;
  cudaError_t e = cudaFuncSetAttribute(score16_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       S_SMEM_BYTES);
  if (e != cudaSuccess) return cuda_status(e);
  TimerScope ts(K_SCORE16_TC, (double)n * (double)n, s);
  const cudaError_t le = launch_pdl(score16_tc_kernel, pl.line.grid, S_THREADS, S_SMEM_BYTES, s, p);
  count_launch();
  return cuda_status(le);
}

// ---- layout probe: D (128 x 16) = A (128 x 64) . B (16 x 64)^T, fp16 ------------
// A is stored to tensor memory with tcgen05.st (two fp16 per 32-bit column,
// row = TMEM lane) and read by tcgen05.mma as its A operand; B uses the
// transposed-feature image layout of the score kernel's data stages (rows of
// 64 points, 128 B).  Four K=16 steps.  Inputs FP32, rounded to fp16 here.
namespace {
__global__ void __launch_bounds__(128, 1) mma_ts_probe_kernel(const float* __restrict__ a,
                                                              const float* __restrict__ b,
                                                              float* __restrict__ d) {
  __shared__ __align__(1024) uint8_t sb[XT_BYTES];
  __shared__ uint64_t bar;
  __shared__ uint32_t slot;
  const int t = threadIdx.x;
  const int warp = t >> 5;
  for (int i = t; i < FSK_D * NT; i += 128)
    put_h(sb, i / NT, i % NT, XT_ROW_BYTES, __float2half_rn(b[i]));
  if (t == 0) {
    mbar_init(&bar, 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&slot, 128);
    tmem_relinquish();
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = slot;
  const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const __half2 h2 = __floats2half2_rn(a[t * NT + c * 32 + 2 * j], a[t * NT + c * 32 + 2 * j + 1]);
      v[j] = *reinterpret_cast<const uint32_t*>(&h2);
    }
    tmem_st16(tbase + lane_off + (uint32_t)(c * 16), v);
  }
  tmem_st_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (t == 0) {
    const uint32_t idesc = idesc_f16_f32(QT, FSK_D);
    for (int ks = 0; ks < NT / 16; ++ks)
      mma_f16_ts(tbase + 64, tbase + (uint32_t)(8 * ks),
                 smem_desc_kmajor(smem_u32(sb) + 256 * ks, 128, 8 * XT_ROW_BYTES), idesc, ks ? 1u : 0u);
    mma_commit(&bar);
  }
  __syncwarp();
  const bool ok = mbar_wait(&bar, 0, 31);
  tc_fence_after();
  if (ok) {
    uint32_t r[16];
    tmem_ld16(tbase + lane_off + 64u, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) d[t * FSK_D + j] = __uint_as_float(r[j]);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tbase, 128);
}
}  // namespace

// ---- layout probe: tcgen05.cp of a query operand image into tensor memory -----
// A (128 x 32, rounded to fp16) is written in the "hi" operand image layout
// (64-byte rows, no-swizzle K-major core matrices), copied to TMEM columns
// 0-15 with two 128x256b copies (K 0-15 at +0 B, K 16-31 at +256 B) and read
// back with tcgen05.ld: out[r][c] is column c of lane r (two fp16 per word).
namespace {
__global__ void __launch_bounds__(128, 1) tmem_cp_probe_kernel(const float* __restrict__ a,
                                                               uint32_t* __restrict__ out) {
  __shared__ __align__(1024) uint8_t sa[QT * H_ROW_BYTES];
  __shared__ uint64_t bar;
  __shared__ uint32_t slot;
  const int t = threadIdx.x;
  const int warp = t >> 5;
#pragma unroll 4
  for (int k = 0; k < KH; ++k) put_h(sa, t, k, H_ROW_BYTES, __float2half_rn(a[t * KH + k]));
  if (t == 0) {
    mbar_init(&bar, 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&slot, 32);
    tmem_relinquish();
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = slot;
  if (t == 0) {
    tmem_cp_128x256b(tbase, smem_desc_kmajor(smem_u32(sa), 128, 8 * H_ROW_BYTES));
    tmem_cp_128x256b(tbase + 8u, smem_desc_kmajor(smem_u32(sa) + 256, 128, 8 * H_ROW_BYTES));
    mma_commit(&bar);
  }
  __syncwarp();
  const bool ok = mbar_wait(&bar, 0, 37);
  tc_fence_after();
  if (ok) {
    uint32_t r[16];
    tmem_ld16(tbase + ((uint32_t)(warp * 32) << 16), r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) out[t * 16 + j] = r[j];
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tbase, 32);
}
}  // namespace

}  // namespace tc

unsigned int score16_take_device_error() { return take_unit_device_error(); }

namespace tc {

int launch_tmem_cp_probe(const float* a, uint32_t* out, cudaStream_t s) {
  tmem_cp_probe_kernel<<<1, 128, 0, s>>>(a, out);
  count_launch();
  return cuda_status(cudaGetLastError());
}

int launch_mma_ts_probe(const float* a, const float* b, float* d, cudaStream_t s) {
  mma_ts_probe_kernel<<<1, 128, 0, s>>>(a, b, d);
  count_launch();
  return cuda_status(cudaGetLastError());
}

}  // namespace tc
}  // namespace fsk
