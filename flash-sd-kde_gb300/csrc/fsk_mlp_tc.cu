// fsk_mlp_tc.cu - tensor-core (tcgen05 / TMEM) inference of the surrogate
// MLP ensemble: 16 -> 256 -> 256 -> 256 -> 1, SiLU, bf16 weights and
// activations, FP32 accumulation, one ensemble member per CTA.
//
// Per tile of 128 queries (one TMEM lane each):
//   A0 = bf16((x - mean) * inv_std)         epilogue warps -> TMEM
//   D  = A0 . W1^T                           1 MMA, M=128, N=256, K=16
//   A1 = bf16(silu(D + b1))                  TMEM -> registers -> TMEM
//   D  = A1 . W2^T                           16 MMAs (K steps), N=256
//   A2 = bf16(silu(D + b2)); D = A2 . W3^T   16 MMAs
//   y  = bf16(silu(D + b3)) . bf16(w4) + b4  per-thread dot, four feature quarters combined
// The activations stay in tensor memory as the A operand of the next layer
// (tcgen05.mma with A in TMEM), so nothing is transposed through shared
// memory.  W2 and W3 (128 KB each in bf16) do not fit in shared memory next
// to anything else, so they stream from L2 as 8 KB K slices ([256 out][16 in],
// core-matrix K-major), four to a copy, through a ring of RING 32 KB slots; W1,
// the biases, w4 and the input normalisation are loaded once per CTA.
//
// Two tiles run in turn on one accumulator: the epilogue warps drain the whole
// accumulator of one tile into registers (64 per thread) and hand it to the
// other tile's MMAs before they start on bias and SiLU, so tensor core and
// tanh unit work at the same time, and each weight slice serves both tiles.
// 2^20 queries x 4 members: 3.06 ms with one tile at a time and a wait and a
// release per slice (the issuing thread then takes 250-400 cycles per MMA, of
// which the tensor core needs 133); 1.82 ms with two tiles, 1.04 with four
// slices per wait, inputs by bulk copy and one bf16 conversion per pair, 0.94
// with packed FMAs.  The tanh unit is busy 0.69 ms of that (3.2e9 tanh at 16
// per cycle and SM), the tensor core 0.47.  Where every block has one tile
// there is nothing to pair and it runs alone.
//
// TMEM: accumulator 256 columns | activations of tile 0, 128 | of tile 1, 128.
// Warps: 0-15 epilogue (warp w: TMEM lane quarter w&3, feature quarter
// w>>2), 16 producer (bulk copies), 17 MMA issue + TMEM owner.
#include <cuda_bf16.h>

#include "fsk_kernels.cuh"
#include "fsk_mlp.cuh"
#include "fsk_tc.cuh"
#include "fsk_tc_ops.cuh"

namespace fsk {
namespace mlp {

namespace {

constexpr int QT = 128;                         // queries per tile
constexpr int SLICE_BYTES = MLP_H * 16 * 2;     // one K slice: [256][16] bf16 = 8 KB
constexpr int N_SLICES = MLP_H / 16;            // 16 per hidden layer
constexpr int CHUNK = 4;                        // slices per copy, per wait and per release
constexpr int CHUNK_BYTES = CHUNK * SLICE_BYTES;   // 32 KB
constexpr int LAYER_CHUNKS = N_SLICES / CHUNK;  // 4
constexpr int RING = 6;                         // chunks in flight: a layer and half of the next
constexpr int X_BYTES = QT * MLP_IN * 4;        // a tile's inputs, 8 KB
// packed member image (global):
//   header 256 B: in_mean[16] in_inv_std[16] out_scale out_shift b4 (FP32)
//   b1 b2 b3 w4 (FP32, w4 bf16-rounded) 4 KB
//   W1 image [256][16] bf16 8 KB, W2 slices 16 x 8 KB, W3 slices 16 x 8 KB
constexpr int HDR_BYTES = 256;
constexpr int VEC_BYTES = 4 * MLP_H * 4;
constexpr int W1_OFF = HDR_BYTES + VEC_BYTES;
constexpr int W2_OFF = W1_OFF + SLICE_BYTES;
constexpr int W3_OFF = W2_OFF + N_SLICES * SLICE_BYTES;
constexpr int MEMBER_BYTES = W3_OFF + N_SLICES * SLICE_BYTES;
// shared memory
constexpr int SM_CONST_BYTES = W2_OFF;                     // header + vectors + W1 image (one copy)
constexpr int SM_RING_OFF = SM_CONST_BYTES;
constexpr int SM_X_OFF = SM_RING_OFF + RING * CHUNK_BYTES;
constexpr int SM_HB_OFF = SM_X_OFF + 2 * X_BYTES;
constexpr int SM_YSUM_OFF = SM_HB_OFF + 3 * MLP_H * 4;
constexpr int SM_BAR_OFF = SM_YSUM_OFF + 2 * 3 * QT * 4;
constexpr int N_BARS = 12 + 2 * RING;   // cready, ring, aready 2, dfull, dfree, ycomb 2, x full 2, x empty 2, drain
constexpr int SMEM_BYTES = SM_BAR_OFF + (N_BARS + 1) * 8;   // + the TMEM address slot
constexpr int EPI_WARPS = 16;
constexpr int PROD_WARP = 16;
constexpr int MMA_WARP = 17;
constexpr int THREADS = 18 * 32;
constexpr int T_D = 0;       // accumulator: 256 FP32 columns
constexpr int T_A = 256;     // activations: 128 columns of packed bf16 pairs per tile
constexpr int T_A_TILE = 128;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
static_assert(MEMBER_BYTES % 16 == 0 && W1_OFF % 16 == 0, "bulk copy alignment");

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// bf16 pair of silu(z + b) = h (1 + tanh h), h = (z + b) / 2, from the
// accumulators and the halved biases: h = z / 2 + hb in one rounding is the
// halved sum (a power of two), so a pair takes two packed FMAs, two tanh and
// one conversion.
__device__ __forceinline__ uint32_t silu_pair(uint32_t z0, uint32_t z1, float hb0, float hb1) {
  const float2 h = __ffma2_rn(make_float2(__uint_as_float(z0), __uint_as_float(z1)), make_float2(0.5f, 0.5f), make_float2(hb0, hb1));
  const float2 a = __ffma2_rn(h, make_float2(tanh_approx(h.x), tanh_approx(h.y)), h);
  return pack_bf16(a.x, a.y);
}

struct InferParams {
  const uint8_t* packed;
  int members;
  const float* x;
  int64_t batch;
  float* y;            // [members][batch]
  int tiles;
  int per;             // tiles per turn: 2, or 1 where every CTA has one tile at most
};

__global__ void __launch_bounds__(THREADS, 1) mlp_infer_kernel(InferParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const float* hdr = reinterpret_cast<const float*>(smem);
  const float* vec = reinterpret_cast<const float*>(smem + HDR_BYTES);   // b1 b2 b3 w4
  float* half_b = reinterpret_cast<float*>(smem + SM_HB_OFF);            // b1 b2 b3, halved
  uint8_t* ring = smem + SM_RING_OFF;
  float* ysum = reinterpret_cast<float*>(smem + SM_YSUM_OFF);            // [2 tiles][3][QT]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM_BAR_OFF);
  uint64_t* cready = bars;                 // constants loaded
  uint64_t* full = bars + 1;               // [RING]
  uint64_t* empty = bars + 1 + RING;       // [RING] chunk read for every tile of the turn
  uint64_t* aready = bars + 1 + 2 * RING;  // [2] a tile's activations (or inputs) stored, all epilogue warps
  uint64_t* dfull = aready + 2;            // accumulator complete
  uint64_t* dfree = aready + 3;            // accumulator drained into registers, all epilogue warps
  uint64_t* ycomb = aready + 4;            // [2] a tile's partial dots of feature quarters 1-3 stored, 12 warps
  uint64_t* xfull = aready + 6;            // [2] a tile's inputs in shared memory
  uint64_t* xempty = aready + 8;           // [2] and read, all epilogue warps
  uint64_t* drain = aready + 10;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aready + 11);
  unsigned n_ring_copies = 0, n_x_copies[2] = {0, 0};
  int n_const_copies = 0;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int member = blockIdx.x % p.members;
  const int group = blockIdx.x / p.members, groups = gridDim.x / p.members;
  const uint8_t* img = p.packed + (int64_t)member * MEMBER_BYTES;

  if (threadIdx.x == 0) {
    mbar_init(cready, 1);
    for (int i = 0; i < RING; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&aready[i], EPI_WARPS);
      mbar_init(&ycomb[i], 12);
      mbar_init(&xfull[i], 1);
      mbar_init(&xempty[i], EPI_WARPS);
    }
    mbar_init(dfull, 1);
    mbar_init(dfree, EPI_WARPS);
    mbar_init(drain, 1);
    fence_barrier_init();
  }
  for (int i = threadIdx.x; i < 3 * MLP_H; i += THREADS)
    half_b[i] = 0.5f * reinterpret_cast<const float*>(img + HDR_BYTES)[i];
  if (warp == MMA_WARP) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // turns of this CTA: tiles t0 .. t0 + per - 1, t0 = per (group + i groups)
  const int t_first = group * p.per, t_step = groups * p.per;

  if (warp == PROD_WARP) {
    if (lane == 0) {
      mbar_arrive_expect_tx(cready, SM_CONST_BYTES);
      bulk_g2s(smem, img, SM_CONST_BYTES, cready);
      n_const_copies = 1;
      int s = 0;
      uint32_t ph = 0;
      for (int t = t_first; t < p.tiles; t += t_step) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (k >= p.per || t + k >= p.tiles) continue;
          if (!mbar_wait(&xempty[k], (n_x_copies[k] & 1u) ^ 1u, 51)) goto done;
          const int64_t q = (int64_t)(t + k) * QT;
          const uint32_t bytes = (uint32_t)imin<int64_t>(QT, p.batch - q) * (MLP_IN * 4);
          mbar_arrive_expect_tx(&xfull[k], bytes);
          bulk_g2s(smem + SM_X_OFF + k * X_BYTES, p.x + q * MLP_IN, bytes, &xfull[k]);
          ++n_x_copies[k];
        }
        for (int c = 0; c < 2 * LAYER_CHUNKS; ++c) {
          if (!mbar_wait(&empty[s], ph ^ 1u, 62)) goto done;
          mbar_arrive_expect_tx(&full[s], CHUNK_BYTES);
          bulk_g2s(ring + s * CHUNK_BYTES, img + W2_OFF + c * CHUNK_BYTES, CHUNK_BYTES, &full[s]);
          ++n_ring_copies;
          if (++s == RING) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    }
  } else if (warp == MMA_WARP) {
    if (elect_one()) {
      const uint32_t idesc = idesc_bf16_f32(QT, MLP_H);
      const uint64_t w1d = smem_desc_kmajor(smem_u32(smem + W1_OFF), 128, 8 * 32);
      const uint64_t r0 = smem_desc_kmajor(smem_u32(ring), 128, 8 * 32);
      if (!mbar_wait(cready, 0, 52)) goto done;
      int s0 = 0;              // ring slot of the layer's first chunk
      uint32_t ph0 = 0;        // and its phase
      uint32_t step = 0;       // accumulations issued
      uint32_t ka[2] = {0, 0}; // activations taken per tile slot
      for (int t = t_first; t < p.tiles; t += t_step) {
        const int n = t + 1 < p.tiles ? p.per : 1;   // tiles of this turn
        for (int layer = 0; layer < 3; ++layer) {
          for (int k = 0; k < n; ++k, ++step) {
            if (!mbar_wait(&aready[k], ka[k] & 1u, 53)) goto done;
            ++ka[k];
            // the previous accumulation is in the epilogue's registers
            if (step > 0 && !mbar_wait(dfree, (step - 1) & 1u, 54)) goto done;
            tc_fence_after();
            const uint32_t a = tmem + T_A + (uint32_t)(k * T_A_TILE);
            if (layer == 0) {
              mma_f16_ts(tmem + T_D, a, w1d, idesc, 0u);
            } else {
              int s = s0;
              uint32_t ph = ph0;
#pragma unroll
              for (int c = 0; c < LAYER_CHUNKS; ++c) {
                if (k == 0) {
                  if (!mbar_wait(&full[s], ph, 55)) goto done;
                }
                const uint64_t w = r0 + (uint64_t)((uint32_t)(s * CHUNK_BYTES) >> 4);
#pragma unroll
                for (int i = 0; i < CHUNK; ++i)
                  mma_f16_ts(tmem + T_D, a + 8 * (CHUNK * c + i), w + (uint64_t)(i * (SLICE_BYTES >> 4)), idesc,
                             c + i ? 1u : 0u);
                if (k == n - 1) mma_commit(&empty[s]);
                if (++s == RING) {
                  s = 0;
                  ph ^= 1u;
                }
              }
              if (k == n - 1) {
                s0 = s;
                ph0 = ph;
              }
            }
            mma_commit(dfull);
          }
        }
      }
    }
  } else {
    // ---------------- epilogue: thread = one query, one feature quarter ----------------
    const int quarter = warp & 3, fq = warp >> 2;   // TMEM lane quarter, feature quarter (64 features)
    const int row = quarter * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    if (!mbar_wait(cready, 0, 56)) goto done;
    const float* mean = hdr;
    const float* inv_std = hdr + 16;
    // this thread's 4 input features of a tile (features 4 fq .. 4 fq + 3) into
    // the tile slot's activations; `turn` is the tile's
    auto put_inputs = [&](int tile, int k, uint32_t turn) -> bool {
      const int f = 4 * fq;
      if (!mbar_wait(&xfull[k], turn & 1u, 63)) return false;
      float4 v = make_float4(mean[f], mean[f + 1], mean[f + 2], mean[f + 3]);
      if ((int64_t)tile * QT + row < p.batch)
        v = *reinterpret_cast<const float4*>(smem + SM_X_OFF + k * X_BYTES + (row * MLP_IN + f) * 4);
      uint32_t pk[2];
      pk[0] = pack_bf16((v.x - mean[f]) * inv_std[f], (v.y - mean[f + 1]) * inv_std[f + 1]);
      pk[1] = pack_bf16((v.z - mean[f + 2]) * inv_std[f + 2], (v.w - mean[f + 3]) * inv_std[f + 3]);
      tmem_st2(tmem + lane_off + T_A + k * T_A_TILE + 2 * fq, pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&aready[k]);
        mbar_arrive(&xempty[k]);
      }
      return true;
    };
    for (int k = 0; k < p.per; ++k)
      if (t_first + k < p.tiles && !put_inputs(t_first + k, k, 0)) goto done;
    uint32_t step = 0, turn = 0;
    for (int t = t_first; t < p.tiles; t += t_step, ++turn) {
      const int n = t + 1 < p.tiles ? p.per : 1;
      for (int layer = 0; layer < 3; ++layer) {
        const float* bias = half_b + layer * MLP_H + 64 * fq;
#pragma unroll 1
        for (int k = 0; k < n; ++k, ++step) {
          if (!mbar_wait(dfull, step & 1u, 57)) goto done;
          tc_fence_after();
          uint32_t r[2][32];
          tmem_ld32(tmem + lane_off + T_D + 64 * fq, r[0]);
          tmem_ld32(tmem + lane_off + T_D + 64 * fq + 32, r[1]);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(dfree);
          if (layer < 2) {
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              uint32_t pk[4];
#pragma unroll
              for (int j = 0; j < 4; j += 2) {
                const uint32_t* z = r[c >> 2] + 8 * (c & 3) + 2 * j;
                const float4 bb = *reinterpret_cast<const float4*>(bias + 8 * c + 2 * j);
                pk[j] = silu_pair(z[0], z[1], bb.x, bb.y);
                pk[j + 1] = silu_pair(z[2], z[3], bb.z, bb.w);
              }
              tmem_st4(tmem + lane_off + T_A + k * T_A_TILE + 32 * fq + 4 * c, pk);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&aready[k]);
          } else {
            const float* w4 = vec + 3 * MLP_H + 64 * fq;
            float acc_y = 0.f;
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int j = 0; j < 32; j += 4) {
                const float4 bb = *reinterpret_cast<const float4*>(bias + 32 * c + j);
                const float4 ww = *reinterpret_cast<const float4*>(w4 + 32 * c + j);
                const uint32_t lo = silu_pair(r[c][j], r[c][j + 1], bb.x, bb.y);
                const uint32_t hi = silu_pair(r[c][j + 2], r[c][j + 3], bb.z, bb.w);
                acc_y = fmaf(__uint_as_float(lo << 16), ww.x, acc_y);
                acc_y = fmaf(__uint_as_float(lo & 0xffff0000u), ww.y, acc_y);
                acc_y = fmaf(__uint_as_float(hi << 16), ww.z, acc_y);
                acc_y = fmaf(__uint_as_float(hi & 0xffff0000u), ww.w, acc_y);
              }
            // this tile slot's MMAs are done: the next turn's inputs
            if (t + t_step + k < p.tiles && !put_inputs(t + t_step + k, k, turn + 1)) goto done;
            // combine the four feature quarters of each query's dot product
            float* ys = ysum + k * 3 * QT;
            if (fq != 0) {
              ys[(fq - 1) * QT + row] = acc_y;
              __syncwarp();
              if (lane == 0) mbar_arrive(&ycomb[k]);
            } else {
              if (!mbar_wait(&ycomb[k], turn & 1u, 58)) goto done;
              const float v = acc_y + ys[row] + ys[QT + row] + ys[2 * QT + row] + hdr[34];
              const int64_t q = (int64_t)(t + k) * QT + row;
              if (q < p.batch) p.y[(int64_t)member * p.batch + q] = fmaf(v, hdr[32], hdr[33]);
            }
          }
        }
      }
    }
  }
done:
  if (warp == PROD_WARP && lane == 0) {
    for (unsigned i = n_ring_copies > RING ? n_ring_copies - RING : 0u; i < n_ring_copies; ++i)
      mbar_wait(&full[i % RING], (i / RING) & 1u, 59);
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (n_x_copies[k]) mbar_wait(&xfull[k], (n_x_copies[k] - 1u) & 1u, 64);
    if (n_const_copies) mbar_wait(cready, 0, 60);
  }
  if (warp == MMA_WARP && elect_one()) {
    mma_commit(drain);
    mbar_wait(drain, 0, 61);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == MMA_WARP) tmem_dealloc(tmem, 512);
}

// ---- packing: FP32 member parameters -> the image above -------------------------
__device__ __forceinline__ void put_bf16(uint8_t* img, int r, int k, float v) {
  // [256 rows][16 K] core-matrix K-major, 32-byte rows
  const uint32_t off = (uint32_t)(r >> 3) * 256u + (uint32_t)(k >> 3) * 128u + (uint32_t)(r & 7) * 16u +
                       (uint32_t)(k & 7) * 2u;
  *reinterpret_cast<__nv_bfloat16*>(img + off) = __float2bfloat16_rn(v);
}

__global__ void pack_kernel(const float* __restrict__ params, int members, const float* __restrict__ in_mean,
                            const float* __restrict__ in_inv_std, float out_scale, float out_shift,
                            uint8_t* __restrict__ packed) {
  const int member = blockIdx.y;
  const float* P = params + (int64_t)member * MLP_PARAMS;
  uint8_t* img = packed + (int64_t)member * MEMBER_BYTES;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  float* hdr = reinterpret_cast<float*>(img);
  float* vec = reinterpret_cast<float*>(img + HDR_BYTES);
  if (i < 64) {
    float v = 0.f;
    if (i < 16) v = in_mean[i];
    else if (i < 32) v = in_inv_std[i - 16];
    else if (i == 32) v = out_scale;
    else if (i == 33) v = out_shift;
    else if (i == 34) v = P[OFF_B4];
    hdr[i] = v;
  }
  if (i < MLP_H) {
    vec[i] = P[OFF_B1 + i];
    vec[MLP_H + i] = P[OFF_B2 + i];
    vec[2 * MLP_H + i] = P[OFF_B3 + i];
    vec[3 * MLP_H + i] = __bfloat162float(__float2bfloat16_rn(P[OFF_W4 + i]));
  }
  if (i < MLP_H * MLP_IN) {
    const int r = (int)(i / MLP_IN), kk = (int)(i % MLP_IN);
    put_bf16(img + W1_OFF, r, kk, P[OFF_W1 + i]);
  }
  if (i < MLP_H * MLP_H) {
    const int r = (int)(i / MLP_H), kk = (int)(i % MLP_H);
    const int sl = kk / 16, kin = kk % 16;
    put_bf16(img + W2_OFF + sl * SLICE_BYTES, r, kin, P[OFF_W2 + i]);
    put_bf16(img + W3_OFF + sl * SLICE_BYTES, r, kin, P[OFF_W3 + i]);
  }
}

// Ensemble statistics and the serving gate, per query b:
//   r2 = |(x_b - mean) * inv_std|^2 (whitened radius, if x is given)
//   mean[b] = average over members of y + base_a + base_b r2
//   spread[b] = max - min over members
//   served[b] = spread <= spread_tol and r2 <= r2_max
__global__ void combine_kernel(const float* __restrict__ y, int members, int64_t batch, const float* __restrict__ x,
                               const float* __restrict__ in_mean, const float* __restrict__ in_inv_std, float base_a,
                               float base_b, float spread_tol, float r2_max, float* __restrict__ mean,
                               float* __restrict__ spread, uint8_t* __restrict__ served) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  float s = 0.f, lo = INFINITY, hi = -INFINITY;
  for (int m = 0; m < members; ++m) {
    const float v = y[(int64_t)m * batch + b];
    s += v;
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
  }
  float r2 = 0.f;
  if (x) {
#pragma unroll
    for (int k = 0; k < MLP_IN; ++k) {
      const float u = (x[b * MLP_IN + k] - in_mean[k]) * in_inv_std[k];
      r2 = fmaf(u, u, r2);
    }
  }
  const float sp = hi - lo;
  if (mean) mean[b] = s / (float)members + base_a + base_b * r2;
  if (spread) spread[b] = sp;
  if (served) served[b] = (sp <= spread_tol && r2 <= r2_max) ? 1 : 0;
}

}  // namespace

size_t packed_bytes(int members) { return (size_t)members * MEMBER_BYTES; }

int launch_pack(const float* params, int members, const float* in_mean, const float* in_inv_std, float out_scale,
                float out_shift, void* packed, cudaStream_t s) {
  const int64_t n = (int64_t)MLP_H * MLP_H;
  pack_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)members), 256, 0, s>>>(
      params, members, in_mean, in_inv_std, out_scale, out_shift, static_cast<uint8_t*>(packed));
  count_launch();
  return cuda_status(cudaGetLastError());
}

int launch_infer(const void* packed, int members, const float* x, int64_t batch, float* y, cudaStream_t s) {
  InferParams p;
  p.packed = static_cast<const uint8_t*>(packed);
  p.members = members;
  p.x = x;
  p.batch = batch;
  p.y = y;
  p.tiles = (int)((batch + QT - 1) / QT);
  const int sms = sm_count();
  int groups = imax(1, imin(sms / members, p.tiles));
  p.per = p.tiles > groups ? 2 : 1;
  cudaError_t e = cudaFuncSetAttribute(mlp_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  if (e != cudaSuccess) return cuda_status(e);
  TimerScope ts(K_MLP_INFER, (double)batch * members, s);
  mlp_infer_kernel<<<groups * members, THREADS, SMEM_BYTES, s>>>(p);
  count_launch();
  return cuda_status(cudaGetLastError());
}

void launch_combine(const float* y, int members, int64_t batch, const float* x, const float* in_mean,
                    const float* in_inv_std, float base_a, float base_b, float spread_tol, float r2_max, float* mean,
                    float* spread, uint8_t* served, cudaStream_t s) {
  combine_kernel<<<(unsigned)((batch + 255) / 256), 256, 0, s>>>(y, members, batch, x, in_mean, in_inv_std, base_a,
                                                                 base_b, spread_tol, r2_max, mean, spread, served);
  count_launch();
}

}  // namespace mlp

unsigned int mlp_tc_take_device_error() { return take_unit_device_error(); }

}  // namespace fsk
