// fsk_mlp.cu - training kernels of the learned surrogate: an ensemble of
// MLPs 16 -> 256 -> 256 -> 256 -> 1 with SiLU, bf16 weights and activations,
// FP32 accumulation (the model of the tensor-core inference kernel in
// fsk_mlp_tc.cu), trained on (query, exact log-density) pairs.
//
// Forward (per member, batch rows b):
//   a0 = bf16((x - in_mean) * in_inv_std)
//   z_l = bf16(W_l) a_{l-1} + b_l,  a_l = bf16(silu(z_l))   l = 1..3
//   y = bf16(w4) . a3 + b4
// Backward treats the bf16 roundings as identity (straight-through); weight
// gradients are FP32 with split-batch atomics.  AdamW with bias correction.
//
// Every product is an FP32 FMA chain in k order on the CUDA cores
// (gemm_kernel): training runs on after its roundings, so they stay what they
// are whatever the tile.  (A tensor-core version with dz in three bf16 parts
// halved the step's time, but the tensor cores' accumulation left the
// gradients 7e-6 apart from these.)
#include <cuda_bf16.h>

#include "fsk_kernels.cuh"
#include "fsk_mlp.cuh"

namespace fsk {
namespace mlp {

namespace {

__device__ __forceinline__ float bf16r(float v) {   // round to nearest bf16 (ties to even), as FP32
  const uint32_t u = __float_as_uint(v);
  if ((u & 0x7F800000u) == 0x7F800000u) return v;  // inf / nan unchanged
  const uint32_t r = (u + 0x7FFFu + ((u >> 16) & 1u)) & 0xFFFF0000u;
  return __uint_as_float(r);
}

// SiLU through tanh.approx, the same arithmetic as the inference kernel:
// silu(z) = h + h tanh(h), h = z / 2; sigmoid(z) = (1 + tanh(h)) / 2.
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float silu(float z) {
  const float h = 0.5f * z;
  return fmaf(h, tanh_approx(h), h);
}
__device__ __forceinline__ float silu_grad(float z) {
  const float s = fmaf(0.5f, tanh_approx(0.5f * z), 0.5f);
  return s * (1.0f + z * (1.0f - s));
}

enum Epi { EPI_FWD = 0, EPI_DGRAD = 1, EPI_ATOMIC = 2 };

// bf16 weight matrices of one member in the workspace (16-byte aligned rows)
constexpr int64_t WQ_W1 = 0, WQ_W2 = WQ_W1 + MLP_H * MLP_IN, WQ_W3 = WQ_W2 + MLP_H * MLP_H;
constexpr int64_t WQ_MEMBER = WQ_W3 + MLP_H * MLP_H;

struct GemmArgs {
  const void* A;                 // opA (M x K)
  const __nv_bfloat16* B;        // opB (K x N)
  int64_t lda, ldb;              // leading dimensions of the stored arrays (N: of C)
  int64_t sA, sB;                // per-member strides (0: shared)
  int M, K;
  int k_chunk;                   // split-K chunk (multiple of FK); gridDim.z = members * splits
  int splits;
  float* C;  int64_t ldc, sC;    // FWD: z, DGRAD: dz, ATOMIC: grad (accumulated)
  const float* bias;             // FWD, per-member stride MLP_PARAMS
  __nv_bfloat16* Anext;          // FWD: bf16(silu(z)), same layout as C
  const float* Zprev;            // DGRAD: z of the layer below, same layout as C
  float* bias_grad;              // ATOMIC: += row sums of opA, stride sC
};

__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Four consecutive stored elements (all in range, or none), kept as stored
// until they go to shared memory as FP32.
template <typename E> struct Stored4;
template <> struct Stored4<float> {
  float4 u;
  __device__ __forceinline__ void load(const float* p, bool ok) {
    u = ok ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ float4 value() const { return u; }
};
template <> struct Stored4<__nv_bfloat16> {
  uint2 u;
  __device__ __forceinline__ void load(const __nv_bfloat16* p, bool ok) {
    u = ok ? *reinterpret_cast<const uint2*>(p) : make_uint2(0u, 0u);
  }
  __device__ __forceinline__ float4 value() const {
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xFFFF0000u));
  }
};

// C[m][n] = sum_k opA[m][k] opB[k][n] on a 64 x FN tile, 128 threads, two
// columns per f32x2 instruction.  Every C is one FMA chain over its k range
// from 0 in order (then the epilogue), the bits of the 64 x 64 tile with 4 x 4
// per thread that this replaces.  FP32 FMA bound: the 2.1e9 FMAs of an
// 8192 x 4 x 256 x 256 product are 58 us at the measured FMA rate; 8 x 8 per
// thread takes 89 (forward) to 99 us (data gradient) where 4 x 4 took 159 to 175.  64
// rows: 1024 tiles over 152 SMs fill 96 % of the last wave, 128 rows 84 %.
// T: the row index of the operand is contiguous in memory (element (k, row) at
// k * ld + row), else k is.
constexpr int FM = 64, FK = 16, FT = 128;
template <bool TA, bool TB, int EPI, int FN, typename EA>
__global__ void __launch_bounds__(FT, 4) gemm_kernel(GemmArgs g) {
  constexpr int TX = FN == 128 ? 16 : 8;          // threads along columns
  constexpr int CG = FN == 128 ? 2 : 1;           // column groups per thread
  constexpr int CW = FN / TX / CG;                // columns per group (4, or 2)
  constexpr int RG = FM / (FT / TX) / 4;          // row groups of 4 per thread
  __shared__ __align__(16) float As[2][FK][FM + 4];
  __shared__ __align__(16) float Bs[2][FK][FN + 4];
  const int member = blockIdx.z / g.splits, split = blockIdx.z % g.splits;
  const int m0 = blockIdx.y * FM, n0 = blockIdx.x * FN;
  const EA* A = static_cast<const EA*>(g.A) + member * g.sA;
  const __nv_bfloat16* B = g.B + member * g.sB;
  const int k_begin = split * g.k_chunk, k_end = min(g.K, k_begin + g.k_chunk);
  const int t = threadIdx.x, tx = t % TX, ty = t / TX;
  // staging: items of 4 stored elements, lanes along the contiguous index
  constexpr int AI = FM * FK / 4 / FT, BI = (FN * FK / 4 + FT - 1) / FT;
  Stored4<EA> ra[AI];
  Stored4<__nv_bfloat16> rb[BI];
  auto place = [](bool T, int rows, int e, int& row, int& k) {
    row = T ? 4 * (e % (rows / 4)) : e / (FK / 4);
    k = T ? e / (rows / 4) : 4 * (e % (FK / 4));
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < AI; ++i) {
      int row, k;
      place(TA, FM, t + i * FT, row, k);
      ra[i].load(TA ? A + (int64_t)(k0 + k) * g.lda + m0 + row : A + (int64_t)(m0 + row) * g.lda + k0 + k,
                 m0 + row < g.M && k0 + k < k_end);
    }
#pragma unroll
    for (int i = 0; i < BI; ++i) {
      int row, k;
      place(TB, FN, t + i * FT, row, k);
      if (FN * FK / 4 % FT == 0 || t + i * FT < FN * FK / 4)
        rb[i].load(TB ? B + (int64_t)(k0 + k) * g.ldb + n0 + row : B + (int64_t)(n0 + row) * g.ldb + k0 + k,
                   k0 + k < k_end);
    }
  };
  auto put = [](bool T, float* s, int stride, int row, int k, float4 v) {
    if (T) {
      *reinterpret_cast<float4*>(s + k * stride + row) = v;
    } else {
      s[k * stride + row] = v.x;
      s[(k + 1) * stride + row] = v.y;
      s[(k + 2) * stride + row] = v.z;
      s[(k + 3) * stride + row] = v.w;
    }
  };
  auto stage = [&](int s) {
#pragma unroll
    for (int i = 0; i < AI; ++i) {
      int row, k;
      place(TA, FM, t + i * FT, row, k);
      put(TA, &As[s][0][0], FM + 4, row, k, ra[i].value());
    }
#pragma unroll
    for (int i = 0; i < BI; ++i) {
      int row, k;
      place(TB, FN, t + i * FT, row, k);
      if (FN * FK / 4 % FT == 0 || t + i * FT < FN * FK / 4) put(TB, &Bs[s][0][0], FN + 4, row, k, rb[i].value());
    }
  };
  // rows 32 h + 4 ty + i (h < RG), columns 64 h + CW tx + j (h < CG)
  float2 acc[4 * RG][CG * CW / 2];
#pragma unroll
  for (int i = 0; i < 4 * RG; ++i)
#pragma unroll
    for (int j = 0; j < CG * CW / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);
  float row_sum = 0.f;   // ATOMIC: sum of opA's row t over the k range
  fetch(k_begin);
  stage(0);
  __syncthreads();
  for (int k0 = k_begin, s = 0; k0 < k_end; k0 += FK, s ^= 1) {
    const bool more = k0 + FK < k_end;
    if (more) fetch(k0 + FK);
#pragma unroll
    for (int kk = 0; kk < FK; ++kk) {
      float av[4 * RG];
      float2 bv[CG * CW / 2];
#pragma unroll
      for (int h = 0; h < RG; ++h) {
        const float4 p = *reinterpret_cast<const float4*>(&As[s][kk][32 * h + 4 * ty]);
        av[4 * h] = p.x;
        av[4 * h + 1] = p.y;
        av[4 * h + 2] = p.z;
        av[4 * h + 3] = p.w;
      }
#pragma unroll
      for (int h = 0; h < CG; ++h)
#pragma unroll
        for (int j = 0; j < CW / 2; ++j)
          bv[h * CW / 2 + j] = *reinterpret_cast<const float2*>(&Bs[s][kk][64 * h + CW * tx + 2 * j]);
#pragma unroll
      for (int i = 0; i < 4 * RG; ++i)
#pragma unroll
        for (int j = 0; j < CG * CW / 2; ++j) acc[i][j] = __ffma2_rn(make_float2(av[i], av[i]), bv[j], acc[i][j]);
    }
    if (EPI == EPI_ATOMIC && blockIdx.x == 0 && t < FM) {
#pragma unroll
      for (int kk = 0; kk < FK; ++kk) row_sum += As[s][kk][t];
    }
    if (more) stage(s ^ 1);
    __syncthreads();
  }
  if (EPI == EPI_ATOMIC && blockIdx.x == 0 && t < FM && m0 + t < g.M)
    atomicAdd(&g.bias_grad[member * g.sC + m0 + t], row_sum);
#pragma unroll
  for (int i = 0; i < 4 * RG; ++i) {
    const int m = m0 + 32 * (i >> 2) + 4 * ty + (i & 3);
    if (m >= g.M) continue;
#pragma unroll
    for (int h = 0; h < CG; ++h) {
      const int n = n0 + 64 * h + CW * tx;
      const int64_t o = member * g.sC + (int64_t)m * g.ldc + n;
      float v[CW];
#pragma unroll
      for (int j = 0; j < CW; j += 2) {
        v[j] = acc[i][(h * CW + j) / 2].x;
        v[j + 1] = acc[i][(h * CW + j) / 2].y;
      }
      if constexpr (EPI == EPI_ATOMIC) {
#pragma unroll
        for (int j = 0; j < CW; ++j) atomicAdd(&g.C[o + j], v[j]);
      } else {
        static_assert(CW == 4, "16-byte rows");
        if constexpr (EPI == EPI_FWD) {
          const float* b = g.bias + member * MLP_PARAMS + n;
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] += b[j];
          *reinterpret_cast<uint2*>(g.Anext + o) =
              make_uint2(bf16_pair(silu(v[0]), silu(v[1])), bf16_pair(silu(v[2]), silu(v[3])));
        } else {
          const float4 z = *reinterpret_cast<const float4*>(g.Zprev + o);
          v[0] *= silu_grad(z.x);
          v[1] *= silu_grad(z.y);
          v[2] *= silu_grad(z.z);
          v[3] *= silu_grad(z.w);
        }
        *reinterpret_cast<float4*>(g.C + o) = make_float4(v[0], v[1], v[2], v[3]);
      }
    }
  }
}

template <bool TA, bool TB, int EPI, int FN, typename EA>
void gemm(const GemmArgs& g, int n, int members, cudaStream_t s) {
  const dim3 grid((unsigned)(n / FN), (unsigned)((g.M + FM - 1) / FM), (unsigned)(members * g.splits));
  gemm_kernel<TA, TB, EPI, FN, EA><<<grid, FT, 0, s>>>(g);
  count_launch();
}

// First launch of a pass: bf16 copies of the weight matrices, and
//   forward (a0 != null): a0 = bf16((x - mean) * inv_std), shared by all members;
//   backward: gradients cleared.
__global__ void setup_kernel(const float* __restrict__ params, int members, __nv_bfloat16* __restrict__ w,
                             const float* __restrict__ x, int64_t batch, const float* __restrict__ mean,
                             const float* __restrict__ inv_std, __nv_bfloat16* __restrict__ a0,
                             float* __restrict__ grads) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t e = first; e < members * MLP_PARAMS; e += step) {
    const int64_t member = e / MLP_PARAMS, o = e - member * MLP_PARAMS;
    const float v = params[e];
    int64_t at = -1;
    if (o < OFF_B1) at = WQ_W1 + o;
    else if (o >= OFF_W2 && o < OFF_B2) at = WQ_W2 + o - OFF_W2;
    else if (o >= OFF_W3 && o < OFF_B3) at = WQ_W3 + o - OFF_W3;
    if (at >= 0) w[member * WQ_MEMBER + at] = __float2bfloat16_rn(v);
    if (grads != nullptr) grads[e] = 0.f;
  }
  if (a0 == nullptr) return;
  for (int64_t e = first; e < batch * MLP_IN; e += step) {
    const int k = (int)(e % MLP_IN);
    a0[e] = __float2bfloat16_rn((x[e] - mean[k]) * inv_std[k]);
  }
}

// y[member][b] = bf16(w4) . a3[b] + b4, one warp per (member, row).
// Lane l adds features l, l + 32, ... in order.
__global__ void output_kernel(const float* __restrict__ params, const __nv_bfloat16* __restrict__ a3, int64_t batch,
                              int members, float* __restrict__ y) {
  const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= batch * members) return;
  const int member = (int)(wid / batch);
  const float* w4 = params + (int64_t)member * MLP_PARAMS + OFF_W4;
  const __nv_bfloat16* row = a3 + wid * MLP_H;
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < MLP_H; k += 32) s = fmaf(bf16r(w4[k + lane]), __bfloat162float(row[k + lane]), s);
#pragma unroll
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) y[wid] = s + params[(int64_t)member * MLP_PARAMS + OFF_B4];
}

// Output layer backward: grads of w4 (atomics over rows), b4, and
// dz3[b][k] = dy[b] bf16(w4[k]) silu'(z3[b][k]).
__global__ void output_bwd_kernel(const float* __restrict__ params, const __nv_bfloat16* __restrict__ a3,
                                  const float* __restrict__ z3, const float* __restrict__ dy, int64_t batch,
                                  int members, float* __restrict__ dz3, float* __restrict__ grads) {
  const int member = blockIdx.y;
  const int k = threadIdx.x;               // 256 threads = features
  const int64_t rows_per_block = (batch + gridDim.x - 1) / gridDim.x;
  const int64_t b0 = blockIdx.x * rows_per_block, b1 = min(batch, b0 + rows_per_block);
  const float w = bf16r(params[(int64_t)member * MLP_PARAMS + OFF_W4 + k]);
  float gw = 0.f, gb = 0.f;
#pragma unroll 4
  for (int64_t b = b0; b < b1; ++b) {
    const int64_t r = (int64_t)member * batch + b;
    const float d = dy[r];
    gw = fmaf(d, __bfloat162float(a3[r * MLP_H + k]), gw);
    gb += d;
    dz3[r * MLP_H + k] = d * w * silu_grad(z3[r * MLP_H + k]);
  }
  atomicAdd(&grads[(int64_t)member * MLP_PARAMS + OFF_W4 + k], gw);
  if (k == 0) atomicAdd(&grads[(int64_t)member * MLP_PARAMS + OFF_B4], gb);
}

__global__ void mse_kernel(const float* __restrict__ y, const float* __restrict__ target, int64_t batch,
                           int members, float* __restrict__ dy, double* __restrict__ loss) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double l = 0.0;
  if (i < batch * members) {
    const float r = y[i] - target[i % batch];
    dy[i] = 2.0f * r / (float)batch;
    l = (double)r * r;
  }
  if (loss) {
#pragma unroll
    for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0 && l != 0.0) atomicAdd(loss, l / (double)batch);
  }
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, int64_t count, float lr, float beta1, float beta2, float eps,
                            float wd, float bc1, float bc2) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const float gi = g[i];
  const float mi = fmaf(beta1, m[i], (1.0f - beta1) * gi);
  const float vi = fmaf(beta2, v[i], (1.0f - beta2) * gi * gi);
  m[i] = mi;
  v[i] = vi;
  const float mh = mi / bc1, vh = vi / bc2;
  p[i] -= lr * (mh / (sqrtf(vh) + eps) + wd * p[i]);
}

}  // namespace

TrainBufs carve_train(WsCarver& c, int members, int64_t batch) {
  TrainBufs t;
  t.a0 = c.take<__nv_bfloat16>((size_t)batch * MLP_IN);
  t.w = c.take<__nv_bfloat16>((size_t)members * WQ_MEMBER);
  const size_t act = (size_t)members * batch * MLP_H;
  for (int l = 0; l < 3; ++l) {
    t.z[l] = c.take<float>(act);
    t.a[l] = c.take<__nv_bfloat16>(act);
  }
  for (int l = 0; l < 2; ++l) t.dz[l] = c.take<float>(act);
  return t;
}

void launch_forward(const float* params, int members, const float* x, int64_t batch, const float* in_mean,
                   const float* in_inv_std, const TrainBufs& t, float* y, cudaStream_t s) {
  setup_kernel<<<4 * sm_count(), 256, 0, s>>>(params, members, t.w, x, batch, in_mean, in_inv_std, t.a0, nullptr);
  count_launch();
  const int64_t act = batch * MLP_H;
  const int64_t wq_off[3] = {WQ_W1, WQ_W2, WQ_W3}, b_off[3] = {OFF_B1, OFF_B2, OFF_B3};
  for (int l = 0; l < 3; ++l) {
    GemmArgs g{};
    g.A = l == 0 ? t.a0 : t.a[l - 1];
    g.lda = g.ldb = l == 0 ? MLP_IN : MLP_H;
    g.sA = l == 0 ? 0 : act;
    g.B = t.w + wq_off[l];
    g.sB = WQ_MEMBER;
    g.M = (int)batch;
    g.K = g.k_chunk = l == 0 ? MLP_IN : MLP_H;
    g.splits = 1;
    g.C = t.z[l];
    g.ldc = MLP_H;
    g.sC = act;
    g.bias = params + b_off[l];
    g.Anext = t.a[l];
    gemm<false, false, EPI_FWD, 128, __nv_bfloat16>(g, MLP_H, members, s);
  }
  const int64_t warps = batch * members;
  output_kernel<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, s>>>(params, t.a[2], batch, members, y);
  count_launch();
}

void launch_backward(const float* params, int members, int64_t batch, const TrainBufs& t, const float* dy,
                    float* grads, cudaStream_t s) {
  setup_kernel<<<4 * sm_count(), 256, 0, s>>>(params, members, t.w, nullptr, batch, nullptr, nullptr, nullptr, grads);
  count_launch();
  const int64_t act = batch * MLP_H;
  const int row_blocks = (int)imin<int64_t>(512, (batch + 63) / 64);
  output_bwd_kernel<<<dim3((unsigned)row_blocks, (unsigned)members), MLP_H, 0, s>>>(params, t.a[2], t.z[2], dy,
                                                                                     batch, members, t.dz[0], grads);
  count_launch();
  const int64_t w_off[3] = {OFF_W1, OFF_W2, OFF_W3}, b_off[3] = {OFF_B1, OFF_B2, OFF_B3};
  const int64_t wq_off[3] = {WQ_W1, WQ_W2, WQ_W3};
  const int64_t splits = imax<int64_t>(1, imin<int64_t>(64, batch / 256));
  for (int l = 2; l >= 0; --l) {
    // weight gradient: dW_l[o][k] = sum_b dz[b][o] a_{l-1}[b][k], split over the batch
    GemmArgs g{};
    g.A = t.dz[l & 1];
    g.lda = MLP_H;
    g.sA = act;
    g.B = l == 0 ? t.a0 : t.a[l - 1];
    g.ldb = g.ldc = l == 0 ? MLP_IN : MLP_H;
    g.sB = l == 0 ? 0 : act;
    g.M = MLP_H;
    g.K = (int)batch;
    g.k_chunk = (int)(((batch + splits - 1) / splits + FK - 1) / FK * FK);
    g.splits = (int)((batch + g.k_chunk - 1) / g.k_chunk);
    g.C = grads + w_off[l];
    g.sC = MLP_PARAMS;
    g.bias_grad = grads + b_off[l];
    if (l == 0) {
      gemm<true, true, EPI_ATOMIC, 16, float>(g, MLP_IN, members, s);
      break;
    }
    gemm<true, true, EPI_ATOMIC, 128, float>(g, MLP_H, members, s);
    // data gradient into the layer below: dz_{l-1} = (dz W_l) * silu'(z_{l-1})
    GemmArgs d{};
    d.A = t.dz[l & 1];
    d.lda = d.ldb = d.ldc = MLP_H;
    d.sA = act;
    d.B = t.w + wq_off[l];
    d.sB = WQ_MEMBER;
    d.M = (int)batch;
    d.K = d.k_chunk = MLP_H;
    d.splits = 1;
    d.C = t.dz[(l - 1) & 1];
    d.sC = act;
    d.Zprev = t.z[l - 1];
    gemm<false, true, EPI_DGRAD, 128, float>(d, MLP_H, members, s);
  }
}

void launch_mse(const float* y, const float* target, int64_t batch, int members, float* dy, double* loss,
                cudaStream_t s) {
  const int64_t n = batch * members;
  mse_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(y, target, batch, members, dy, loss);
  count_launch();
}

void launch_adam(float* p, const float* g, float* m, float* v, int64_t count, float lr, float beta1, float beta2,
                 float eps, float wd, int step, cudaStream_t s) {
  const float bc1 = 1.0f - powf(beta1, (float)step), bc2 = 1.0f - powf(beta2, (float)step);
  adam_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(p, g, m, v, count, lr, beta1, beta2, eps, wd, bc1, bc2);
  count_launch();
}

}  // namespace mlp
}  // namespace fsk
