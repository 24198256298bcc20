// Learned subgrid-scale closure: a per-cell MLP that predicts the eddy viscosity.
//
//   inputs  x[8]  = 100 * S_ab (6 strain-rate components xx yy zz xy xz yz, estimated
//                   from the non-equilibrium stress), 100 * (rho - 1), wall distance / 16
//   hidden  h1 = GELU(W1 x + b1)  (32),  h2 = GELU(W2 h1 + b2)  (32)
//   output  nu_t / nu_0 = softplus(W3 h2 + b3)
//
// GELU is the tanh form 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3))) (Hendrycks &
// Gimpel, 2016).  Parameters (FP32 master copy, this order): W1[32][8], b1[32],
// W2[32][32], b2[32], W3[32], b3.  In the step kernel the weights are BF16 and the
// products accumulate in FP32 on the tensor cores.
#pragma once
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>
#include <cuda_bf16.h>

namespace aerosim {

constexpr int kMlpIn = 8, kMlpHidden = 32;
constexpr int kMlpW1 = 0, kMlpB1 = kMlpW1 + kMlpHidden * kMlpIn, kMlpW2 = kMlpB1 + kMlpHidden,
              kMlpB2 = kMlpW2 + kMlpHidden * kMlpHidden, kMlpW3 = kMlpB2 + kMlpHidden, kMlpB3 = kMlpW3 + kMlpHidden,
              kMlpParams = kMlpB3 + 1;
constexpr float kGeluK = 0.7978845608028654f;  // sqrt(2 / pi)

__host__ __device__ inline float gelu_f(float x) {
  return 0.5f * x * (1.0f + tanhf(kGeluK * (x + 0.044715f * x * x * x)));
}
__host__ __device__ inline float softplus_f(float o) { return o > 20.0f ? o : log1pf(expf(o)); }
__host__ __device__ inline float sigmoid_f(float o) { return 1.0f / (1.0f + expf(-o)); }

// Model inputs of a cell from its non-equilibrium stress: the strain-rate estimate
// S = -3 Pi^neq / (2 rho tau) with tau the Smagorinsky relaxation time the reference
// computes from |Pi^neq| (lbmCpuReference.ts:264-282), so the closure sees the same
// strain-rate field a box-filtered fine-grid run provides for training.
__host__ __device__ inline void mlp_features(float pxx, float pyy, float pzz, float pxy, float pxz, float pyz,
                                             float rho, float tau_s, float wall_dist, float (&x)[kMlpIn]) {
  const float k = -150.0f / (rho * tau_s);  // 100 * (-3 / (2 rho tau))
  x[0] = k * pxx; x[1] = k * pyy; x[2] = k * pzz;
  x[3] = k * pxy; x[4] = k * pxz; x[5] = k * pyz;
  x[6] = 100.0f * (rho - 1.0f);
  x[7] = wall_dist * (1.0f / 16.0f);
}

// ---- in-kernel inference on the tensor cores ---------------------------------------
// A warp evaluates the MLP for its 32 cells (lane = cell) as BF16 m16n8k16 tile
// contractions with FP32 accumulation: two 16-cell M tiles, hidden width 32 = four
// N tiles, the 8 inputs padded to K = 16.  The D fragments of a layer are, pair by
// pair, the A fragments of the next, so activations never leave the registers.
//
// Weight fragments are pre-packed per lane (mlp_pack_fragments) in six 16-byte vectors:
// word j of vector g of lane l at frag[(g * 32 + l) * 4 + j]:
//   g 0           layer 1, j = N tile t:             (W1[n][k], W1[n][k+1]),  n = 8t + l/4, k = 2(l%4)
//   g 1..4        layer 2, t = g - 1, j = 2kt+half:  (W2[n][k], W2[n][k+1]),  k = 16kt + 2(l%4) + 8 half
//   g 5           layer 3, j = 2kt+half:             (W3[k], W3[k+1]) for l/4 == 0, else 0
// W2 and W3 are packed as halves: their inputs are twice the GELU (gelu2_bf16x2).
// Biases: bias[0..31] = b1, bias[32..63] = b2, bias[64] = b3; from kMlpBiasQuads on the
// accumulators' start values of layer 1 and 2, N tile t, lanes l with l % 4 = q, as the vectors
// (b[8t+2q], b[8t+2q+1], the same again) at 4 * (16 (layer - 1) + 4t + q).
constexpr int kMlpFragWords = 24;
constexpr int kMlpBiasQuads = 68;
constexpr int kMlpBias = kMlpBiasQuads + 128;

__host__ inline uint16_t bf16_bits_rn(float f) {  // round to nearest even
  uint32_t u;
  std::memcpy(&u, &f, 4);
  if ((u & 0x7f800000u) == 0x7f800000u) return (uint16_t)(u >> 16);  // inf / nan
  u += 0x7fffu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}

__host__ inline void mlp_pack_fragments(const float* P, uint32_t* frag /*[24 * 32]*/, float* bias /*[kMlpBias]*/) {
  auto pair = [](float lo, float hi) { return (uint32_t)bf16_bits_rn(lo) | ((uint32_t)bf16_bits_rn(hi) << 16); };
  for (int l = 0; l < 32; ++l) {
    const int k0 = 2 * (l % 4), n0 = l / 4;
    for (int t = 0; t < 4; ++t) {
      const int n = 8 * t + n0;
      frag[l * 4 + t] = pair(P[kMlpW1 + n * kMlpIn + k0], P[kMlpW1 + n * kMlpIn + k0 + 1]);
    }
    for (int kt = 0; kt < 2; ++kt)
      for (int t = 0; t < 4; ++t)
        for (int h = 0; h < 2; ++h) {
          const int n = 8 * t + n0, k = 16 * kt + k0 + 8 * h;
          frag[((1 + t) * 32 + l) * 4 + 2 * kt + h] =
              pair(0.5f * P[kMlpW2 + n * kMlpHidden + k], 0.5f * P[kMlpW2 + n * kMlpHidden + k + 1]);
        }
    for (int kt = 0; kt < 2; ++kt)
      for (int h = 0; h < 2; ++h) {
        const int k = 16 * kt + k0 + 8 * h;
        frag[(5 * 32 + l) * 4 + 2 * kt + h] = n0 == 0 ? pair(0.5f * P[kMlpW3 + k], 0.5f * P[kMlpW3 + k + 1]) : 0u;
      }
  }
  for (int j = 0; j < 32; ++j) {
    bias[j] = P[kMlpB1 + j];
    bias[32 + j] = P[kMlpB2 + j];
  }
  bias[64] = P[kMlpB3];
  for (int j = 65; j < kMlpBiasQuads; ++j) bias[j] = 0.0f;
  for (int i = 0; i < 128; ++i) {
    const int layer = i / 64, t = i / 16 % 4, q = i / 4 % 4;
    bias[kMlpBiasQuads + i] = bias[32 * layer + 8 * t + 2 * q + (i & 1)];
  }
}

#ifdef __CUDACC__
// D = A B + C; C in registers of its own, so that start values shared by tiles need no copies.
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1, const float4& c) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c.x), "f"(c.y), "f"(c.z), "f"(c.w));
}
__device__ __forceinline__ void mma_bf16_1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, const float4& c) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0), "f"(c.x), "f"(c.y), "f"(c.z), "f"(c.w));
}
__device__ __forceinline__ uint32_t bf16x2_of(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// GELU of two pre-activations as one packed BF16 pair, the operand type of the next
// layer: the pair is rounded to BF16 first and the tanh form is evaluated in bf16x2
// arithmetic (x/2 (1 + tanh(x (k + k c x^2))), k = sqrt(2/pi) and k c = k * 0.044715 as
// BF16 constants 0x3f4c and 0x3d12), about a third of the instructions of two FP32 GELUs.
__device__ __forceinline__ uint32_t gelu_bf16x2(float a, float b) {
  const uint32_t x = bf16x2_of(a, b);
  uint32_t x2, u, t, r;
  asm("mul.rn.bf16x2 %0, %1, %1;" : "=r"(x2) : "r"(x));
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(u) : "r"(x2), "r"(0x3d123d12u), "r"(0x3f4c3f4cu));
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(u) : "r"(u), "r"(x));
  asm("tanh.approx.bf16x2 %0, %1;" : "=r"(t) : "r"(u));
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(u) : "r"(x), "r"(0x3f003f00u));
  asm("fma.rn.bf16x2 %0, %1, %2, %1;" : "=r"(r) : "r"(u), "r"(t));
  return r;
}

// Twice the GELU of a pair: x (1 + tanh(...)), the factor 1/2 (an exact scaling of BF16) in the
// weights of the next layer instead of one more multiplication per pair.
__device__ __forceinline__ uint32_t gelu2_bf16x2(float a, float b) {
  const uint32_t x = bf16x2_of(a, b);
  uint32_t x2, u, t, r;
  asm("mul.rn.bf16x2 %0, %1, %1;" : "=r"(x2) : "r"(x));
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(u) : "r"(x2), "r"(0x3d123d12u), "r"(0x3f4c3f4cu));
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(u) : "r"(u), "r"(x));
  asm("tanh.approx.bf16x2 %0, %1;" : "=r"(t) : "r"(u));
  asm("fma.rn.bf16x2 %0, %1, %2, %1;" : "=r"(r) : "r"(x), "r"(t));
  return r;
}

// What bounds it (256x128x128 FP32 step, ncu): issue, about 740 instructions for 32 cells of the
// closure and the step together, of them 64 MUFU.TANH (66 us of that unit) and 28 tensor
// instructions (12 % of theirs).  Fragments and start values as 16-byte shared loads, the
// accumulators' start values not copied and layer 1 at its own K took the two-cell step from
// 189.5 to 168.3 us, and with items of 256 pairs to 162.5.
//
// nu_t / nu_0 of this lane's cell.  All 32 lanes must call it together.  x: the lane's
// 8 inputs; frag / bias: the packed weights (shared memory, 16-byte aligned); stage: 32 x 8
// BF16 of shared memory owned by the warp, 16-byte aligned.
__device__ __forceinline__ float mlp_nut_warp(const float (&x)[kMlpIn], const uint32_t* __restrict__ frag,
                                              const float* __restrict__ bias, uint32_t* __restrict__ stage,
                                              int lane) {
  // inputs to the A-fragment layout through shared memory (row = cell, 4 words each)
  reinterpret_cast<uint4*>(stage)[lane] =
      make_uint4(bf16x2_of(x[0], x[1]), bf16x2_of(x[2], x[3]), bf16x2_of(x[4], x[5]), bf16x2_of(x[6], x[7]));
  __syncwarp();
  const int r = lane >> 2, q = lane & 3;
  const uint4* const fv = reinterpret_cast<const uint4*>(frag) + lane;
  const float4* const cv = reinterpret_cast<const float4*>(bias + kMlpBiasQuads) + q;
  uint32_t a1[2][2];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) {
    a1[mt][0] = stage[(16 * mt + r) * 4 + q];
    a1[mt][1] = stage[(16 * mt + r + 8) * 4 + q];
  }
  __syncwarp();
  // layer 1: 8 -> 32
  float h[2][4][4];
  const uint4 w1 = fv[0];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const float4 c = cv[4 * t];
    const uint32_t b = t == 0 ? w1.x : t == 1 ? w1.y : t == 2 ? w1.z : w1.w;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) mma_bf16_1688(h[mt][t], a1[mt][0], a1[mt][1], b, c);
  }
  uint32_t a2[2][2][4];  // [mt][kt][reg]
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int kt = 0; kt < 2; ++kt) {
      const float* lo = h[mt][2 * kt];
      const float* hi = h[mt][2 * kt + 1];
      a2[mt][kt][0] = gelu2_bf16x2(lo[0], lo[1]);
      a2[mt][kt][1] = gelu2_bf16x2(lo[2], lo[3]);
      a2[mt][kt][2] = gelu2_bf16x2(hi[0], hi[1]);
      a2[mt][kt][3] = gelu2_bf16x2(hi[2], hi[3]);
    }
  // layer 2: 32 -> 32
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const float4 c = cv[16 + 4 * t];
    const uint4 w = fv[32 * (1 + t)];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      mma_bf16_16816(h[mt][t], a2[mt][0][0], a2[mt][0][1], a2[mt][0][2], a2[mt][0][3], w.x, w.y, c);
      const float4 d = make_float4(h[mt][t][0], h[mt][t][1], h[mt][t][2], h[mt][t][3]);
      mma_bf16_16816(h[mt][t], a2[mt][1][0], a2[mt][1][1], a2[mt][1][2], a2[mt][1][3], w.z, w.w, d);
    }
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int kt = 0; kt < 2; ++kt) {
      const float* lo = h[mt][2 * kt];
      const float* hi = h[mt][2 * kt + 1];
      a2[mt][kt][0] = gelu2_bf16x2(lo[0], lo[1]);
      a2[mt][kt][1] = gelu2_bf16x2(lo[2], lo[3]);
      a2[mt][kt][2] = gelu2_bf16x2(hi[0], hi[1]);
      a2[mt][kt][3] = gelu2_bf16x2(hi[2], hi[3]);
    }
  // layer 3: 32 -> 1 (N padded to 8; column 0 is the output)
  float o[2][4];
  const float c3 = q == 0 ? bias[64] : 0.0f;
  const uint4 w3 = fv[32 * 5];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt) {
    mma_bf16_16816(o[mt], a2[mt][0][0], a2[mt][0][1], a2[mt][0][2], a2[mt][0][3], w3.x, w3.y,
                   make_float4(c3, 0.0f, c3, 0.0f));
    const float4 d = make_float4(o[mt][0], o[mt][1], o[mt][2], o[mt][3]);
    mma_bf16_16816(o[mt], a2[mt][1][0], a2[mt][1][1], a2[mt][1][2], a2[mt][1][3], w3.z, w3.w, d);
  }
  // cell i's output sits in lane 4 (i % 8): o[i / 16][0] for i % 16 < 8, else o[i / 16][2]
  const int src = 4 * (lane & 7);
  const float v00 = __shfl_sync(0xffffffffu, o[0][0], src), v02 = __shfl_sync(0xffffffffu, o[0][2], src);
  const float v10 = __shfl_sync(0xffffffffu, o[1][0], src), v12 = __shfl_sync(0xffffffffu, o[1][2], src);
  const float out = lane < 16 ? (lane < 8 ? v00 : v02) : (lane < 24 ? v10 : v12);
  return softplus_f(out);
}
#endif

}  // namespace aerosim
