// fsk_tc_kde16.cu - tensor-core (tcgen05 / TMEM) 16-D Gaussian KDE, the
// "fast_tf32" precision mode of the reference, GB300-native.
//
// What it computes (per query q_i): sum_j exp(-||q_i - x_j||^2 / (2 h^2)),
// optionally times the Laplace factor (1 + d/2 - ||q_i-x_j||^2/(2h^2)); the
// quantity of kernels/kde_eval_16d_stream_splitk.py:14-81 (pass A) and
// kernels/flash_sd_kde/kde.py:103-144, as partial sums per segment (fsk_reduce.cu adds them).
//
// How:
//  * Coordinates are centred on the data mean mu (FP32).  With c2 =
//    log2(e)/(2h^2), the log2-domain exponent of a pair is
//        a2 = 2 c2 (q-mu).(x-mu) + beta_j + alpha_i,
//    beta_j = -c2 |x_j-mu|^2, alpha_i = -c2 |q_i-mu|^2.
//  * Operands are fp16 triples v = hi + mid + lo (~33 significant bits): queries as
//    q' = 2 c2 (q-mu) 2^eq, data as x' = (x-mu) 2^ex with power-of-two
//    scales chosen on the device so every operand stays in fp16 range and
//    eq + ex = 0 (or the product is scaled down and multiplied back).  Each
//    hi operand row carries 16 extra "bias" K-columns holding beta_j and
//    alpha_i as three fp16 parts each against exact powers of two, so one
//    accumulator D = mid.mid + hi.lo + lo.hi + hi.mid + mid.hi + hi.hi +
//    bias.bias (seven tcgen05.mma kind::f16, M=128, N=128, FP32 accumulation
//    in tensor memory) *is* a2, to one FP32 rounding at the magnitude of the
//    cross product.
//  * Epilogue: tcgen05.ld one query row per thread, 2^D on the SFU
//    (ex2.approx), 32-column chunk sums, compensated (TwoSum) per query.
//  * Exact near-pair recompute: when a 32-column chunk holds more than 1/8
//    of its query's running sum (of its segment: the data tiles one CTA runs
//    for the query block), the chunk's largest term is recomputed from
//    direct FP32 differences of the original coordinates (kept in the data
//    stage) with the exponent product in double-float, and replaces its
//    approximation; all triggered lanes of a warp recompute one pair each in
//    lock-step.  Other
//    terms carry the ~2^-25 relative error of the accumulation, which
//    averages out.
//
// Pipeline (one persistent CTA per SM, 18 warps):
//   warp 16 : producer - bulk (TMA) copies of query images per unit and of
//             data-tile images (128 points) per stage into shared memory
//             (mbarrier tx).
//   warp 17 : copies the query operands to tensor memory once per segment
//             and issues all MMAs (one lane); owns TMEM.
//   warps 0-15: epilogue; warp w reads TMEM lanes 32*(w%4).. and columns
//             64*((w/4)%2).. of query tile w/8.
// A work unit (segment, see WorkLine) is 256 queries (two M=128 tiles) x a run
// of data tiles.  TMEM holds three accumulators of 128 columns, taken in turn
// by the two query tiles, and the query operands (hi | mid | lo, 32 columns a
// tile).  With both operands in shared memory an M=128, N=128, K=16 MMA takes
// ~100 cycles (44 of them for A, whatever N is), with A in tensor memory 64:
// four double-buffered accumulators and A in shared memory took 11.95 ms at
// n = m = 262144, this 11.24 (2^20: 184.3, 173).  The exp pipe is then busy
// 62 % of the time, the tensor core 54 %, issue slots 55 %; the rest is the
// latency of waits, TMEM loads and add chains that 16 warps of 96 registers
// cannot hide.  Each query's sum is kept as two column halves by two threads
// and written as two rows of (value, error) pairs per segment.
#include <cuda_fp16.h>

#include "fsk_kernels.cuh"
#include "fsk_tc.cuh"
#include "fsk_tc_ops.cuh"

namespace fsk {
namespace tc {

// Out of line: inlined into the three roles it costs the epilogue 8 bytes of
// spills per tile (192 against 186 ms at n = m = 2^20).
static __device__ __noinline__ Segment next_segment(const WorkLine& w, int k) {
  return segment_at(w, blockIdx.x, k);
}

// SINGLE: the single-pass precision rung (FSK_PREC_FP16_SINGLE) - only the
// hi.hi cross product (one fp16 product per feature, FP32 accumulation) and
// the bias step, no exact near-pair recompute.
// POLY: the last POLY_COLS columns of every 32-column chunk take the FMA-pipe
// exp2 (exp2_poly2) instead of ex2.approx, moving a quarter of the exps off
// the exp pipe (the FP32 pipe carries ~one lane operation per pair here).
constexpr int POLY_COLS = 8;
template <bool LAPLACE, bool SINGLE, bool POLY>
__global__ void __launch_bounds__(THREADS, 1) kde16_tc_kernel(TcParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sA = smem_raw;                               // NQT query tiles: H | M | L
  uint8_t* sB = smem_raw + A_BYTES;                     // NS data stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + K_BAR_OFFSET);
  uint64_t* full = bars;                 // [NS] data stage loaded
  uint64_t* empty = bars + NS;           // [NS] data stage consumed (MMAs + epilogue)
  // [NQT][4], by the tile's number modulo 4: one phase of a barrier must not
  // pass before every waiter of the phase before has seen it, and an
  // accumulator's three predecessors run up to two tiles ahead of it
  uint64_t* tfull = bars + 2 * NS;       // accumulator written
  uint64_t* tempty = tfull + 4 * NQT;    // accumulator drained
  uint64_t* qready = tempty + 4 * NQT;   // query images loaded
  uint64_t* qempty = qready + 1;         // query images copied to tensor memory
  uint64_t* sdone = qready + 2;          // the MMAs of the segment finished
  uint64_t* drain = sdone + 1;           // all MMAs of this CTA finished (exit path)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  uint32_t n_stage_copies = 0;   // producer: bulk copies issued
  uint32_t n_query_copies = 0;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1 + EPI_WARPS);
    }
    for (int i = 0; i < 4 * NQT; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], EPI_WARPS / NQT);
    }
    mbar_init(qready, 1);
    mbar_init(sdone, 1);
    mbar_init(qempty, 1);
    mbar_init(drain, 1);
    fence_barrier_init();
  }
  if (warp == MMA_WARP) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();   // the images and scales of the preparation
  if (warp == PRODUCER_WARP) {
    // the whole warp runs the loop (warp-uniform values stay in uniform
    // registers); lane 0 issues the copies
    {
      uint32_t& g = n_stage_copies;
      uint32_t& k = n_query_copies;
      int s = 0;
      uint32_t ph = 0;
      for (int k_seg = 0;; ++k_seg) {
        const Segment sg = next_segment(p.line, k_seg);
        if (sg.count == 0) break;
        if (g >= 1u << 30) g = 2 * NS + g % (2 * NS);   // stage and phase of the last copies are kept
        if (!__all_sync(0xffffffffu, mbar_wait_cold(qempty, (k & 1u) ^ 1u, 1))) goto done;
        if (lane == 0) {
          mbar_arrive_expect_tx(qready, A_BYTES);
          bulk_g2s(sA, p.qimg + sg.qb * (int64_t)A_BYTES, A_BYTES, qready);
        }
        ++k;
        const uint8_t* src = p.ximg + sg.t0 * (int64_t)KB_STAGE_BYTES;
        for (int i = 0; i < sg.count; ++i, src += KB_STAGE_BYTES) {
          if (!__all_sync(0xffffffffu, mbar_wait_cold(&empty[s], ph ^ 1u, 2))) goto done;
          if (lane == 0) {
            mbar_arrive_expect_tx(&full[s], KB_STAGE_BYTES);
            bulk_g2s(sB + s * KB_STAGE_BYTES, src, KB_STAGE_BYTES, &full[s]);
          }
          ++g;
          if (++s == NS) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    }
  } else if (warp == MMA_WARP) {
    // Accumulation u = 2 g + a (data tile g of this CTA's run, query tile a)
    // goes to accumulator u % NACC, so the query tiles take the accumulators
    // in turn and a tile's MMAs wait only for the 8 warps reading the one
    // before them there: u - NACC, tile g - 2 + a of the other query tile.  The
    // query operand is copied to tensor memory once per segment.  The per-tile
    // path is kept to the waits, the MMAs and the commits (descriptors of
    // stage s = stage 0 + s * KB_STAGE_BYTES in the 16-byte address field).
    // One warp issues for both query tiles: a second one's polling took issue
    // slots from the epilogue (11.5 against 11.35 ms at n = m = 262144).
    {
      const uint32_t idesc = idesc_f16_f32(QT, KNT);
      const uint32_t as = smem_u32(sA);
      const uint64_t a_h = smem_desc_kmajor(as, 128, 8 * H_ROW_BYTES);
      const uint64_t a_m = smem_desc_kmajor(as + A_M_OFFSET, 128, 8 * L_ROW_BYTES);
      const uint64_t a_l = smem_desc_kmajor(as + A_L_OFFSET, 128, 8 * L_ROW_BYTES);
      const uint32_t bs0 = smem_u32(sB);
      const uint64_t b_h0 = smem_desc_kmajor(bs0, 128, 8 * H_ROW_BYTES);
      const uint64_t b_m0 = smem_desc_kmajor(bs0 + KB_M_OFFSET, 128, 8 * L_ROW_BYTES);
      const uint64_t b_l0 = smem_desc_kmajor(bs0 + KB_L_OFFSET, 128, 8 * L_ROW_BYTES);
      const uint32_t ta = tmem_base + (uint32_t)T_KA;   // per query tile, hi: features | bias; mid at +16, lo at +24
      uint32_t ph = 0;
      int s = 0;
      int g = 0;            // data tile
      int acc = 0;          // u % NACC
      for (int k = 0;; ++k) {
        const int nt = next_segment(p.line, k).count;
        if (nt == 0) break;
        if (g >= 1 << 30) g = 8 + (g & 7);   // its low bits count; a segment has fewer than 2^30 tiles
        if (!__all_sync(0xffffffffu, mbar_wait_cold(qready, (uint32_t)k & 1u, 3))) goto done;
        // the previous segment's MMAs have read its operand
        if (k > 0 && !__all_sync(0xffffffffu, mbar_wait_cold(sdone, (uint32_t)(k - 1) & 1u, 10))) goto done;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int a = 0; a < NQT; ++a) {
            const uint64_t at = (uint64_t)(a * A_TILE_BYTES >> 4);
            tmem_cp_128x256b(ta + 32u * a, a_h + at);
            tmem_cp_128x256b(ta + 32u * a + 8u, a_h + at + (256 >> 4));
            if (!SINGLE) {
              tmem_cp_128x256b(ta + 32u * a + 16u, a_m + at);
              tmem_cp_128x256b(ta + 32u * a + 24u, a_l + at);
            }
          }
          mma_commit(qempty);
        }
        __syncwarp();
        for (int i = 0; i < nt; ++i) {
          if (!__all_sync(0xffffffffu, mbar_wait_cold(&full[s], ph, 4))) goto done;
          const uint64_t so = (uint64_t)(s * (KB_STAGE_BYTES >> 4));
#pragma unroll
          for (int a = 0; a < NQT; ++a) {
            const int prev = g - 2 + a;
            if (prev >= 0 && !__all_sync(0xffffffffu, mbar_wait_cold(&tempty[(1 - a) * 4 + (prev & 3)], (uint32_t)(prev >> 2) & 1u, 5)))
              goto done;
            tc_fence_after();
            if (elect_one()) {
              const uint32_t d = tmem_base + (uint32_t)(acc * KNT);
              if (SINGLE)
                mma_s_tile_single(d, ta + 32u * a, b_h0 + so, idesc);
              else
                mma_s_tile(d, ta + 32u * a, b_h0 + so, b_m0 + so, b_l0 + so, idesc);
              mma_commit(&tfull[a * 4 + (g & 3)]);
              if (a == NQT - 1) mma_commit(&empty[s]);
              if (a == NQT - 1 && i == nt - 1) mma_commit(sdone);
            }
            __syncwarp();
            if (++acc == NACC) acc = 0;
          }
          ++g;
          if (++s == NS) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    }
  } else {
    // ---------------- epilogue warps ----------------
    const int qt = warp >> 3;          // query tile within the unit
    const int half = (warp >> 2) & 1;  // column half of the 128-point data tile
    const int quarter = warp & 3;      // TMEM lane quarter
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const float out_mul = p.scales->out_mul;
    const bool scaled = out_mul != 1.0f;
    // slot float4 kk of thread t at [kk][t]: a warp's 16-byte accesses are contiguous
    float4* qslot = reinterpret_cast<float4*>(smem_raw + K_QX_OFFSET) + (warp * 32 + lane);
    constexpr int QS_STRIDE = EPI_WARPS * 32;
    uint32_t g = 0;   // data tile
    int ab = qt;   // its accumulator, (2 g + qt) % NACC
    int s = 0;
    const int last_t = (int)p.line.n_tiles - 1;
    // valid columns of this thread's half of the last (possibly ragged) data
    // tile; every other tile has KNT / 2
    const int last_valid = (int)imin<int64_t>(KNT / 2, p.n - ((int64_t)last_t * KNT + half * (KNT / 2)));
    for (int k_seg = 0;; ++k_seg) {
      const Segment sg = next_segment(p.line, k_seg);
      if (sg.count == 0) break;
      const int qrow = qt * QT + quarter * 32 + lane;                   // row in the query block
      const int64_t gi = (int64_t)sg.qb * (NQT * QT) + qrow;            // padded query index
      // this query's FP32 row into the thread's own shared-memory slot (read
      // only by the exact recompute; the slot is rewritten only by this thread)
      {
        // scalar loads: the caller's rows need only 4-byte alignment
        const float* src = p.q + (gi < p.m ? gi : 0) * FSK_D;
#pragma unroll
        for (int kk = 0; kk < FSK_D / 4; ++kk)
          qslot[kk * QS_STRIDE] = make_float4(src[4 * kk], src[4 * kk + 1], src[4 * kk + 2], src[4 * kk + 3]);
      }
      Comp acc{0.f, 0.f};
      float corr = 0.f;
      const int last_i = last_t - sg.t0;
      const int nt = sg.count;
      for (int i = 0; i < nt; ++i, ++g) {
        const int valid = i == last_i ? last_valid : KNT / 2;   // may be <= 0 on the last tile
        // (a timed-out wait ends the whole warp: it must stay converged)
        if (!__all_sync(0xffffffffu, mbar_wait_cold(&tfull[qt * 4 + (g & 3)], (g >> 2) & 1u, 6))) goto done;
        tc_fence_after();
        const uint8_t* xrows = sB + s * KB_STAGE_BYTES + KB_X_OFFSET + half * (KNT / 2) * (FSK_D * 4);
        float tsum = 0.f;
        // Both 32-column chunks are loaded before either is processed, so the
        // accumulator buffer goes back to the MMA issuer as early as possible.
        uint32_t ra[32], rb[32];
        {
          const uint32_t col = tmem_base + lane_off + (uint32_t)(ab * KNT + half * (KNT / 2));
          tmem_ld32(col, ra);
          tmem_ld32(col + 32u, rb);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[qt * 4 + (g & 3)]);
          ab += NQT;
          if (ab >= NACC) ab -= NACC;
        }
        auto chunk = [&](const uint32_t (&r)[32], const int c) {
            float e[32];
            if (scaled) {
#pragma unroll
              for (int j = 0; j < 32; j += 2) {
                const float2 v = __fmul2_rn(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])),
                                            make_float2(out_mul, out_mul));
                e[j] = v.x;
                e[j + 1] = v.y;
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) e[j] = __uint_as_float(r[j]);
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (POLY && j >= 32 - POLY_COLS) continue;
              float v = ex2_approx(e[j]);
              // Laplace factor 1 + d/2 - dist/(2h^2) = 9 + a2 ln 2   (a2 = -c2 dist)
              if (LAPLACE) v *= fmaf(e[j], 0.69314718055994531f, 1.0f + 0.5f * FSK_D);
              e[j] = v;
            }
            if (POLY) {
#pragma unroll
              for (int j = 32 - POLY_COLS; j < 32; j += 2) {
                const float2 v = exp2_poly2(make_float2(e[j], e[j + 1]));
                e[j] = v.x;
                e[j + 1] = v.y;
              }
            }
            const int cvalid = valid - c * 32;   // valid columns of this chunk (may be <= 0 or > 32)
            if (cvalid < 32) {  // ragged last data tile: drop padding columns
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (j >= cvalid) e[j] = 0.f;
            }
            // packed pairwise sum (f32x2 adds on register pairs)
            float2 pa = make_float2(e[0], e[1]), pb = make_float2(e[2], e[3]);
#pragma unroll
            for (int j = 4; j < 32; j += 4) {
              pa = __fadd2_rn(pa, make_float2(e[j], e[j + 1]));
              pb = __fadd2_rn(pb, make_float2(e[j + 2], e[j + 3]));
            }
            pa = __fadd2_rn(pa, pb);
            float cs = pa.x + pa.y;
            // Near-pair test: a chunk holding more than NEAR_FRACTION of the
            // running sum (this chunk included) may contain a dominant term.
            const float run = fabsf(acc.s) + fabsf(tsum);
            const bool trig = !SINGLE && fabsf(cs) > (run + fabsf(cs)) * NEAR_FRACTION;
            if (!SINGLE && __any_sync(0xffffffffu, trig)) {
              // Triggered lanes replace their chunk's largest term by its exact
              // value, one pair each, in lock-step.  The term is found by
              // value (its bits are what the sum holds, so subtracting it
              // removes exactly what was added).
              if (trig) {
                float mx = LAPLACE ? fabsf(e[0]) : e[0];   // terms are >= 0 except with the Laplace factor
#pragma unroll
                for (int jj = 1; jj < 32; ++jj) mx = fmaxf(mx, LAPLACE ? fabsf(e[jj]) : e[jj]);
                int j = 0;
                float approx = mx;
#pragma unroll
                for (int jj = 0; jj < 32; ++jj) {
                  const bool hit = (LAPLACE ? fabsf(e[jj]) : e[jj]) == mx;
                  j = hit ? jj : j;
                  if (LAPLACE) approx = hit ? e[jj] : approx;
                }
                float qx[FSK_D];
#pragma unroll
                for (int kk = 0; kk < FSK_D; kk += 4) {
                  const float4 v = qslot[(kk / 4) * QS_STRIDE];
                  qx[kk] = v.x; qx[kk + 1] = v.y; qx[kk + 2] = v.z; qx[kk + 3] = v.w;
                }
                const float dist = exact_dist(xrows, c * 32 + j, qx, 0);
                float ex = exp2_neg_scaled(dist, p.c2, p.c2_lo);
                if (LAPLACE) ex *= fmaf(-p.c1, dist, 1.0f + 0.5f * FSK_D);
                if (j >= cvalid) ex = 0.f;
                corr += ex - approx;
              }
              __syncwarp();
            }
            tsum += cs;
        };
        chunk(ra, 0);
        chunk(rb, 1);
        acc.add(tsum);
        // the stage's x rows are no longer read by this warp
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        if (++s == NS) s = 0;
      }
      if (gi < p.m) {
        if (p.atomic_acc) {
          const double v = (double)acc.s + (double)acc.c + (double)corr;
          if (in_bounds(gi, p.m, 40)) atomicAdd(&p.atomic_acc[gi], v);
        } else {
          // (value, error) pair: the FP64 unit (2 lanes per clock per SM) stays out of the segment's end
          const int64_t idx = (p.line.segment_id(sg.qb, blockIdx.x) * 2 + half) * p.row_stride + qrow;
          if (in_bounds(idx, p.line.segment_bound() * 2 * p.row_stride, 41))
            p.partials[idx] = make_float2(acc.s, acc.c + corr);
        }
      }
    }
  }
done:
  pdl_launch_dependents();
  // Exit path (also after a timed-out wait): let this CTA's bulk copies and
  // MMAs finish before shared and tensor memory are released.
  if (warp == PRODUCER_WARP && lane == 0) {
    for (uint32_t i = n_stage_copies > NS ? n_stage_copies - NS : 0u; i < n_stage_copies; ++i)
      mbar_wait_cold(&full[i % NS], (uint32_t)(i / NS) & 1u, 7);
    if (n_query_copies > 0) mbar_wait_cold(qready, (n_query_copies - 1) & 1u, 8);
  }
  if (warp == MMA_WARP && elect_one()) {
    mma_commit(drain);   // one arrival per issuing thread, when its MMAs have finished
    mbar_wait_cold(drain, 0, 9);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == MMA_WARP) tmem_dealloc(tmem_base, TMEM_COLS);
}

void plan_line(TcPlan& pl) {
  pl.line.n_tiles = pl.n_tiles;
  pl.line.grid = (int)imin<int64_t>(pl.q_blocks * pl.n_tiles, sm_count());
  pl.line.whole = (int)(pl.q_blocks / pl.line.grid);
  pl.line.rest = (int)(pl.q_blocks % pl.line.grid);
  pl.line.line_grid = (int)imax<int64_t>(1, imin<int64_t>(pl.line.grid, pl.line.rest * pl.n_tiles));
}

TcPlan plan_kde16(int64_t m, int64_t n) {
  TcPlan pl;
  pl.m_pad = (m + NQT * QT - 1) / (NQT * QT) * (NQT * QT);
  pl.n_tiles = (n + KNT - 1) / KNT;
  pl.n_pad = pl.n_tiles * KNT;
  pl.q_blocks = pl.m_pad / (NQT * QT);
  plan_line(pl);
  return pl;
}

static int kde16_row_stride(int64_t m) { return (int)imin<int64_t>(m, NQT * QT); }

size_t tc_kde16_ws_bytes(const TcPlan& pl, int64_t m, bool atomic) {
  WsCarver c(nullptr, 0);
  c.take<uint8_t>((size_t)pl.q_blocks * A_BYTES);
  c.take<uint8_t>((size_t)pl.n_tiles * KB_STAGE_BYTES);
  if (atomic) c.take<double>((size_t)m);
  else c.take<float2>((size_t)pl.line.segment_bound() * 2 * kde16_row_stride(m));
  take_tc_prep(c);
  return align_up(c.used, 256);
}

template <bool LAPLACE, bool SINGLE, bool POLY = false>
static cudaError_t launch_kde16_tc_kernel(const TcPlan& pl, const TcParams& p, cudaStream_t s) {
  const cudaError_t e = cudaFuncSetAttribute(kde16_tc_kernel<LAPLACE, SINGLE, POLY>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  if (e != cudaSuccess) return e;
  return launch_pdl(kde16_tc_kernel<LAPLACE, SINGLE, POLY>, pl.line.grid, THREADS, SMEM_BYTES, s, p);
}

int launch_kde16_tc(const float* q, int64_t m, const float* x, int64_t n, double h,
                    bool laplace, bool single, bool poly, const TcPlan& pl, WsCarver& c, TcPartials* partials_out,
                    double** atomic_out, cudaStream_t s) {
  uint8_t* qimg = c.take<uint8_t>((size_t)pl.q_blocks * A_BYTES);
  uint8_t* ximg = c.take<uint8_t>((size_t)pl.n_tiles * KB_STAGE_BYTES);
  const bool atomic = atomic_out != nullptr;
  const int row_stride = kde16_row_stride(m);
  double* acc = atomic ? c.take<double>((size_t)m) : nullptr;
  float2* part = atomic ? nullptr : c.take<float2>((size_t)pl.line.segment_bound() * 2 * row_stride);
  if (!c.fits()) return FSK_ERR_WORKSPACE_TOO_SMALL;
  if (atomic) *atomic_out = acc;
  *partials_out = TcPartials{part, pl.line, row_stride};

  TcPrep prep;
  const int st = launch_kde16_prep(x, n, q, m, h, pl, ximg, qimg, c, &prep, s);
  if (st) return st;
  const double c2d = FSK_LOG2E / (2.0 * h * h);
  const float c2 = (float)c2d;
  const float c2_lo = (float)(c2d - (double)c2);
  if (atomic) launch_zero(acc, m, s);

  TcParams p;
  p.qimg = qimg;
  p.ximg = ximg;
  p.q = q;
  p.scales = prep.scales;
  p.m = m;
  p.n = n;
  p.line = pl.line;
  p.c2 = c2;
  p.c2_lo = c2_lo;
  p.c1 = (float)(1.0 / (2.0 * h * h));
  p.partials = part;
  p.row_stride = row_stride;
  p.atomic_acc = acc;
  cudaError_t e;
  TimerScope ts(K_KDE16_TC, (double)m * (double)n, s);
  if (laplace)
    e = single ? launch_kde16_tc_kernel<true, true>(pl, p, s) : launch_kde16_tc_kernel<true, false>(pl, p, s);
  else if (single)
    e = launch_kde16_tc_kernel<false, true>(pl, p, s);
  else
    e = poly ? launch_kde16_tc_kernel<false, false, true>(pl, p, s) : launch_kde16_tc_kernel<false, false>(pl, p, s);
  count_launch();
  return cuda_status(e);
}

// ---- layout probe: D (128 x 64) = A (128 x 32) . B (64 x 32)^T, fp16 ----------------
// Two K=16 tcgen05.mma steps over the 64-byte-row core-matrix images used by
// the KDE kernel (the second step at +256 B, like its bias columns).  Inputs
// are FP32, rounded to fp16 here; D is written row-major FP32.
__global__ void __launch_bounds__(128, 1) mma_probe_kernel(const float* __restrict__ a,
                                                           const float* __restrict__ b,
                                                           float* __restrict__ d) {
  __shared__ __align__(1024) uint8_t sa[QT * H_ROW_BYTES];
  __shared__ __align__(1024) uint8_t sb[NT * H_ROW_BYTES];
  __shared__ uint64_t bar;
  __shared__ uint32_t slot;
  const int t = threadIdx.x;
#pragma unroll 4
  for (int k = 0; k < KH; ++k) {
    put_h(sa, t, k, H_ROW_BYTES, __float2half_rn(a[t * KH + k]));
    if (t < NT) put_h(sb, t, k, H_ROW_BYTES, __float2half_rn(b[t * KH + k]));
  }
  if (t == 0) {
    mbar_init(&bar, 1);
    fence_barrier_init();
  }
  const int warp = t >> 5;
  if (warp == 0) {
    tmem_alloc(&slot, 64);
    tmem_relinquish();
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = slot;
  if (t == 0) {
    const uint32_t idesc = idesc_f16_f32(QT, NT);
    mma_f16_ss(tbase, smem_desc_kmajor(smem_u32(sa), 128, 8 * H_ROW_BYTES),
               smem_desc_kmajor(smem_u32(sb), 128, 8 * H_ROW_BYTES), idesc, 0u);
    mma_f16_ss(tbase, smem_desc_kmajor(smem_u32(sa) + 256, 128, 8 * H_ROW_BYTES),
               smem_desc_kmajor(smem_u32(sb) + 256, 128, 8 * H_ROW_BYTES), idesc, 1u);
    mma_commit(&bar);
  }
  __syncwarp();
  const bool ok = mbar_wait(&bar, 0, 20);
  tc_fence_after();
  if (ok) {
    for (int c = 0; c < NT / 32; ++c) {
      uint32_t r[32];
      tmem_ld32(tbase + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c * 32), r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) d[(int64_t)t * NT + c * 32 + j] = __uint_as_float(r[j]);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tbase, 64);
}

int launch_mma_probe(const float* a, const float* b, float* d, cudaStream_t s) {
  mma_probe_kernel<<<1, 128, 0, s>>>(a, b, d);
  count_launch();
  return cuda_status(cudaGetLastError());
}

// Waits on an mbarrier that nothing arrives on: the bounded wait gives up
// (about 2 s), records FSK_ERR_DEVICE_TIMEOUT in the device error word and
// the kernel returns normally.  Tests the failure path without a GPU fault.
__global__ void wait_timeout_probe_kernel(int* out) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) *out = mbar_wait(&bar, 0, 30) ? 1 : 0;
}

}  // namespace tc

unsigned int kde16_take_device_error() { return take_unit_device_error(); }

namespace tc {

int launch_wait_timeout_probe(int* out, cudaStream_t s) {
  wait_timeout_probe_kernel<<<1, 32, 0, s>>>(out);
  count_launch();
  return cuda_status(cudaGetLastError());
}

}  // namespace tc
}  // namespace fsk
