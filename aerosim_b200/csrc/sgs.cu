// Learned SGS closure support: training of the eddy-viscosity MLP on the GPU (forward,
// backward, Adam), its FP32 evaluation, the wall-distance field of a voxel grid (jump
// flooding) and the training samples of a box-filtered fine-grid flow.  No counterpart
// in the reference, whose only closure is Smagorinsky (lbmCpuReference.ts:264-282).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/aerosim.h"
#include "common.cuh"
#include "engine_internal.h"
#include "sgs_mlp.cuh"
#include "sgs_umma.cuh"

namespace aerosim {
namespace {

// Forward pass of one sample in FP32.
__device__ __forceinline__ float mlp_forward_one(const float* P, const float (&x)[kMlpIn]) {
  float h1[kMlpHidden];
#pragma unroll
  for (int j = 0; j < kMlpHidden; ++j) {
    float s = P[kMlpB1 + j];
#pragma unroll
    for (int i = 0; i < kMlpIn; ++i) s = fmaf(P[kMlpW1 + j * kMlpIn + i], x[i], s);
    h1[j] = gelu_f(s);
  }
  float o = P[kMlpB3];
#pragma unroll 4
  for (int j = 0; j < kMlpHidden; ++j) {
    float s = P[kMlpB2 + j];
#pragma unroll
    for (int i = 0; i < kMlpHidden; ++i) s = fmaf(P[kMlpW2 + j * kMlpHidden + i], h1[i], s);
    o = fmaf(P[kMlpW3 + j], gelu_f(s), o);
  }
  return softplus_f(o);
}

// ---- training: loss and gradient of the mean squared error (prediction - target)^2 ----
// One warp takes kGradRows samples at a time, lane = hidden unit: the lane's rows of W1 and
// W2 and its share of the gradient (rows of dW1 and dW2, the biases, dW3) stay in registers
// over all samples of the warp; activations and back-propagated errors pass between the
// lanes through a few hundred bytes of shared memory per warp as broadcast loads.  The
// contractions over a row pair run as packed FP32 (f32x2) FMAs.  Nothing is accumulated
// with atomics: a CTA adds its warps' registers in order and writes one row of partial sums,
// and the kernel that applies them adds the CTAs' rows in a fixed order, so a training run
// is reproducible bit for bit.  The work is far too small to fill the chip's FP32 pipes
// (65 MFMA a batch of 16384): what bounds it is the latency of a sample's chain (gather,
// two layers, the output sum, two layers back), which kGradRows samples in flight per warp
// and 16 warps per SM hide.  Batch of 16384 (B200): one thread per sample with shared-memory
// atomics 6360 us an iteration, now 27 us with the parameter update (batch 512: 10.7 us).
constexpr int kGradRows = 4;
constexpr int kGradWarps = 16;
static_assert(kGradRows == 4, "a group of samples is one float4 of back-propagated errors");
// Partial sums of a CTA: column c, lane j at c * 32 + j (coalesced for both kernels).
// c = 0..7: dW1[j][c]; 8: db1[j]; 9..40: dW2[j][c - 9]; 41: db2[j]; 42: dW3[j]; 43: db3 (lane 0).
constexpr int kGradCols = 44, kGradSlots = kGradCols * 32;
constexpr int kGradStage = kGradRows * (kMlpIn + 2 * kMlpHidden);  // floats of a warp's exchange area
constexpr int kGradW2Row = kMlpHidden + 4;  // padded row of W2 in shared memory: rows and columns read without conflicts
constexpr int kGradSmem = (kMlpHidden * kGradW2Row + kGradWarps * (kGradStage + kGradSlots)) * 4;

// Parameter of column c, lane j; -1 where there is none.
__host__ __device__ constexpr int grad_param(int c, int j) {
  return c < 8 ? kMlpW1 + j * kMlpIn + c : c == 8 ? kMlpB1 + j : c < 41 ? kMlpW2 + j * kMlpHidden + (c - 9)
       : c == 41 ? kMlpB2 + j : c == 42 ? kMlpW3 + j : (j == 0 ? kMlpB3 : -1);
}

// GELU and its derivative from one tanh.
__device__ __forceinline__ float gelu_both(float x, float& grad) {
  const float t = tanhf(kGeluK * (x + 0.044715f * x * x * x));
  grad = 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * kGeluK * (1.0f + 3.0f * 0.044715f * x * x);
  return 0.5f * x * (1.0f + t);
}

// Row of sample i of a mini-batch: a splitmix64 hash of (seed, iteration, i) modulo n.
struct BatchRows {
  unsigned long long seed;
  unsigned long long n;      // rows to draw from; 0: sample i is row i
  unsigned long long recip;  // (2^64 - 1) / n
  int it;
  __device__ __forceinline__ long long row(long long i) const {
    if (n == 0) return i;
    unsigned long long z = seed + 0x9e3779b97f4a7c15ull * ((unsigned long long)it * 1000003ull + (unsigned long long)i + 1ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    // z mod n: the quotient from the reciprocal is at most two too small
    unsigned long long r = z - __umul64hi(z, recip) * n;
    if (r >= n) r -= n;
    if (r >= n) r -= n;
    return (long long)r;
  }
};

__global__ void __launch_bounds__(kGradWarps * 32, 1)
    mlp_grad_kernel(const float* __restrict__ Pg, const float* __restrict__ X, const float* __restrict__ Y,
                    const BatchRows rows, long long n, float inv_n, float* __restrict__ partial,
                    double* __restrict__ loss_partial) {
  extern __shared__ __align__(16) float gsm[];
  __shared__ double s_loss[kGradWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* const sW2 = gsm;                                              // [j][k]
  float* const red = gsm + kMlpHidden * kGradW2Row;                    // [warp][slot]
  float* const sx = red + kGradWarps * kGradSlots + warp * kGradStage;  // [row][8]
  float* const sh = sx + kGradRows * kMlpIn;                           // [row][k]
  float* const sd = sh + kGradRows * kMlpHidden;                       // [j][row]
  const long long groups = (n + kGradRows - 1) / kGradRows;
  const long long stride = (long long)gridDim.x * kGradWarps;
  long long g = (long long)blockIdx.x * kGradWarps + warp;
  // the samples of a group: lane l holds input l % 8 of its row l / 8; lane l < kGradRows its target
  auto load = [&](long long gi, float& x, float& y) {
    const long long i = gi * kGradRows + (lane >> 3);
    x = i < n ? X[rows.row(i) * kMlpIn + (lane & 7)] : 0.0f;
    const long long iy = gi * kGradRows + lane;
    y = (lane < kGradRows && iy < n) ? Y[rows.row(iy)] : 0.0f;
  };
  float xn = 0.0f, yn = 0.0f;
  if (g < groups) load(g, xn, yn);  // the samples do not change between iterations
  // launched as a programmatic dependent of the kernel that updates the parameters
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  for (int i = threadIdx.x; i < kMlpHidden * kMlpHidden; i += blockDim.x)
    sW2[(i / kMlpHidden) * kGradW2Row + i % kMlpHidden] = __ldcg(&Pg[kMlpW2 + i]);
  float w1[kMlpIn], a1[kMlpIn];
  float2 w2[kMlpHidden / 2], a2[kMlpHidden / 2];
#pragma unroll
  for (int i = 0; i < kMlpIn; ++i) {
    w1[i] = __ldcg(&Pg[kMlpW1 + lane * kMlpIn + i]);
    a1[i] = 0.0f;
  }
  const float b1 = __ldcg(&Pg[kMlpB1 + lane]), b2 = __ldcg(&Pg[kMlpB2 + lane]), w3 = __ldcg(&Pg[kMlpW3 + lane]),
              b3 = __ldcg(&Pg[kMlpB3]);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kMlpHidden / 4; ++k) {
    const float4 w = *reinterpret_cast<const float4*>(sW2 + lane * kGradW2Row + 4 * k);
    w2[2 * k] = make_float2(w.x, w.y);
    w2[2 * k + 1] = make_float2(w.z, w.w);
    a2[2 * k] = a2[2 * k + 1] = make_float2(0.0f, 0.0f);
  }
  float ab1 = 0.0f, ab2 = 0.0f, aw3 = 0.0f, ab3 = 0.0f;
  double l = 0.0;
  for (; g < groups; g += stride) {
    sx[lane] = xn;
    const float yc = yn;
    __syncwarp();
    if (g + stride < groups) load(g + stride, xn, yn);
    float g1[kGradRows], d[kGradRows];
#pragma unroll
    for (int r = 0; r < kGradRows; ++r) {
      const float4 xa = *reinterpret_cast<const float4*>(sx + r * kMlpIn), xb = *reinterpret_cast<const float4*>(sx + r * kMlpIn + 4);
      float s = b1;
      s = fmaf(w1[0], xa.x, s); s = fmaf(w1[1], xa.y, s); s = fmaf(w1[2], xa.z, s); s = fmaf(w1[3], xa.w, s);
      s = fmaf(w1[4], xb.x, s); s = fmaf(w1[5], xb.y, s); s = fmaf(w1[6], xb.z, s); s = fmaf(w1[7], xb.w, s);
      sh[r * kMlpHidden + lane] = gelu_both(s, g1[r]);
    }
    __syncwarp();
    float h2[kGradRows], g2[kGradRows], o[kGradRows];
#pragma unroll
    for (int r = 0; r < kGradRows; ++r) {
      float2 s = make_float2(b2, 0.0f);
#pragma unroll
      for (int k = 0; k < kMlpHidden / 4; ++k) {
        const float4 h = *reinterpret_cast<const float4*>(sh + r * kMlpHidden + 4 * k);
        s = __ffma2_rn(w2[2 * k], make_float2(h.x, h.y), s);
        s = __ffma2_rn(w2[2 * k + 1], make_float2(h.z, h.w), s);
      }
      h2[r] = gelu_both(s.x + s.y, g2[r]);
      o[r] = w3 * h2[r];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
      for (int r = 0; r < kGradRows; ++r) o[r] += __shfl_xor_sync(0xffffffffu, o[r], off);
    }
#pragma unroll
    for (int r = 0; r < kGradRows; ++r) {
      const float ov = o[r] + b3;
      const float e = softplus_f(ov) - __shfl_sync(0xffffffffu, yc, r);
      const bool in = g * kGradRows + r < n;
      if (in) l += (double)e * e;
      const float d_o = in ? 2.0f * e * sigmoid_f(ov) * inv_n : 0.0f;
      ab3 += d_o;
      aw3 = fmaf(d_o, h2[r], aw3);
      d[r] = d_o * w3 * g2[r];
      ab2 += d[r];
    }
    *reinterpret_cast<float4*>(sd + lane * kGradRows) = make_float4(d[0], d[1], d[2], d[3]);
    __syncwarp();
    // dW2[j][k] += d2[j] h1[k], lane j
#pragma unroll
    for (int r = 0; r < kGradRows; ++r) {
      const float2 dd = make_float2(d[r], d[r]);
#pragma unroll
      for (int k = 0; k < kMlpHidden / 4; ++k) {
        const float4 h = *reinterpret_cast<const float4*>(sh + r * kMlpHidden + 4 * k);
        a2[2 * k] = __ffma2_rn(dd, make_float2(h.x, h.y), a2[2 * k]);
        a2[2 * k + 1] = __ffma2_rn(dd, make_float2(h.z, h.w), a2[2 * k + 1]);
      }
    }
    // d1[k] = sum_j d2[j] W2[j][k], lane k, two samples to a packed pair
    float2 e01 = make_float2(0.0f, 0.0f), e23 = e01;
#pragma unroll 8
    for (int j = 0; j < kMlpHidden; ++j) {
      const float w = sW2[j * kGradW2Row + lane];
      const float4 dj = *reinterpret_cast<const float4*>(sd + j * kGradRows);
      e01 = __ffma2_rn(make_float2(w, w), make_float2(dj.x, dj.y), e01);
      e23 = __ffma2_rn(make_float2(w, w), make_float2(dj.z, dj.w), e23);
    }
    const float e1[kGradRows] = {e01.x * g1[0], e01.y * g1[1], e23.x * g1[2], e23.y * g1[3]};
#pragma unroll
    for (int r = 0; r < kGradRows; ++r) {
      const float4 xa = *reinterpret_cast<const float4*>(sx + r * kMlpIn), xb = *reinterpret_cast<const float4*>(sx + r * kMlpIn + 4);
      ab1 += e1[r];
      a1[0] = fmaf(e1[r], xa.x, a1[0]); a1[1] = fmaf(e1[r], xa.y, a1[1]);
      a1[2] = fmaf(e1[r], xa.z, a1[2]); a1[3] = fmaf(e1[r], xa.w, a1[3]);
      a1[4] = fmaf(e1[r], xb.x, a1[4]); a1[5] = fmaf(e1[r], xb.y, a1[5]);
      a1[6] = fmaf(e1[r], xb.z, a1[6]); a1[7] = fmaf(e1[r], xb.w, a1[7]);
    }
    __syncwarp();  // the exchange area is free for the next group
  }
  float* const rw = red + warp * kGradSlots + lane;
#pragma unroll
  for (int i = 0; i < kMlpIn; ++i) rw[i * 32] = a1[i];
  rw[8 * 32] = ab1;
#pragma unroll
  for (int k = 0; k < kMlpHidden / 2; ++k) {
    rw[(9 + 2 * k) * 32] = a2[k].x;
    rw[(10 + 2 * k) * 32] = a2[k].y;
  }
  rw[41 * 32] = ab2;
  rw[42 * 32] = aw3;
  rw[43 * 32] = lane == 0 ? ab3 : 0.0f;
  if (lane == 0) s_loss[warp] = l;
  __syncthreads();
  for (int i = threadIdx.x; i < kGradSlots; i += blockDim.x) {
    float s = 0.0f;
#pragma unroll
    for (int w = 0; w < kGradWarps; ++w) s += red[w * kGradSlots + i];
    partial[(size_t)blockIdx.x * kGradSlots + i] = s;
  }
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < kGradWarps; ++w) s += s_loss[w];
    loss_partial[blockIdx.x] = s;
  }
}

// Adds the partial sums of `ctas` CTAs in a fixed order (CTA c: one column of 32
// parameters) and either writes the gradient (G) or takes an Adam step (Kingma & Ba, 2015)
// on the FP32 parameters; CTA 0 adds the loss.
struct AdamState {
  float *P, *m, *v;
  float lr, b1t, b2t;
};
constexpr int kApplyThreads = 512;
__global__ void __launch_bounds__(kApplyThreads)
    mlp_apply_kernel(const float* __restrict__ partial, const double* __restrict__ loss_partial, int ctas, float inv_n,
                     float* __restrict__ G, const AdamState st, double* __restrict__ loss) {
  __shared__ float s[kApplyThreads];
  __shared__ double sl[32];
  const int c = blockIdx.x, lane = threadIdx.x & 31, part = threadIdx.x >> 5;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  float acc = 0.0f;
#pragma unroll 4
  for (int k = part; k < ctas; k += kApplyThreads / 32) acc += __ldcg(&partial[(size_t)k * kGradSlots + c * 32 + lane]);
  s[threadIdx.x] = acc;
  if (c == 0 && part == 0) {
    double d = 0.0;
    for (int k = lane; k < ctas; k += 32) d += __ldcg(&loss_partial[k]);
    sl[lane] = d;
  }
  __syncthreads();
  if (part == 0) {
    float g = 0.0f;
#pragma unroll
    for (int k = 0; k < kApplyThreads / 32; ++k) g += s[k * 32 + lane];
    const int p = grad_param(c, lane);
    if (p >= 0) {
      if (G) {
        G[p] = g;
      } else {
        const float mp = 0.9f * st.m[p] + 0.1f * g;
        const float vp = 0.999f * st.v[p] + 0.001f * g * g;
        st.m[p] = mp;
        st.v[p] = vp;
        const float mh = mp / (1.0f - st.b1t), vh = vp / (1.0f - st.b2t);
        st.P[p] -= st.lr * mh / (sqrtf(vh) + 1e-8f);
      }
    }
    if (c == 0 && lane == 0) {
      double d = 0.0;
      for (int k = 0; k < 32; ++k) d += sl[k];
      *loss = d * (double)inv_n;
    }
  }
}

__global__ void mlp_forward_kernel(const float* __restrict__ Pg, const float* __restrict__ X, long long n,
                                   float* __restrict__ out) {
  __shared__ float P[kMlpParams];
  for (int p = threadIdx.x; p < kMlpParams; p += blockDim.x) P[p] = Pg[p];
  __syncthreads();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  float x[kMlpIn];
#pragma unroll
  for (int i = 0; i < kMlpIn; ++i) x[i] = X[t * kMlpIn + i];
  out[t] = mlp_forward_one(P, x);
}

// The step kernel's tensor-core evaluation (mlp_nut_warp) over rows of X: one warp per
// 32 rows, rows past n evaluated on zeros and discarded.
__global__ void mlp_forward_tc_kernel(const uint32_t* __restrict__ frag_g, const float* __restrict__ bias_g,
                                      const float* __restrict__ X, long long n, float* __restrict__ out) {
  __shared__ __align__(16) uint32_t frag[kMlpFragWords * 32];
  __shared__ __align__(16) float bias[kMlpBias];
  __shared__ __align__(16) uint32_t stage[4][32 * 4];
  for (int i = threadIdx.x; i < kMlpFragWords * 32; i += blockDim.x) frag[i] = frag_g[i];
  for (int i = threadIdx.x; i < kMlpBias; i += blockDim.x) bias[i] = bias_g[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row = ((long long)blockIdx.x * 4 + warp) * 32 + lane;
  float x[kMlpIn];
#pragma unroll
  for (int i = 0; i < kMlpIn; ++i) x[i] = row < n ? X[row * kMlpIn + i] : 0.0f;
  const float y = mlp_nut_warp(x, frag, bias, stage[warp], lane);
  if (row < n) out[row] = y;
}

// The MLP over rows of X on the 5th-generation tensor cores: a CTA of 4 warps takes
// 128-row tiles (grid-stride); thread t owns row t of the tile and TMEM lane t.  The
// dynamic shared memory (kUmmaSmem) caps residency at 8 CTAs per SM, so the 8 x 64
// allocated TMEM columns always fit: D1 in columns 0..31, D2 in 32..63, and D3 back in
// 0..15 once D1 has been read.  Every mbarrier wait is bounded: on a timeout the
// CTA records the error, waits (bounded) for its last commit and frees its TMEM.
constexpr int kUmmaCols = 64;
constexpr int kUmmaSmem = 27 * 1024;
constexpr int kUmmaWaitLimit = 1 << 22;

__global__ void __launch_bounds__(kUmmaRows) mlp_forward_umma_kernel(const uint4* __restrict__ bimg,
                                                                     const float* __restrict__ bias_g,
                                                                     const float* __restrict__ X, long long n,
                                                                     float* __restrict__ out, int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* sA1 = sm;                                          // 128 x 16 BF16
  uint8_t* sA2 = sm + 4096;                                   // 128 x 32 BF16
  uint8_t* sB = sm + 12288;                                   // weight image
  float* sbias = reinterpret_cast<float*>(sm + 16384);        // [65]
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + 16384 + 512);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + 16384 + 520);
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int i = tid; i < kUmmaBBytes / 16; i += kUmmaRows) reinterpret_cast<uint4*>(sB)[i] = bimg[i];
  for (int i = tid; i < 65; i += kUmmaRows) sbias[i] = bias_g[i];
  *reinterpret_cast<uint4*>(sA1 + umma_off(tid, 8, 16)) = make_uint4(0u, 0u, 0u, 0u);  // K padding
  const uint32_t mb = (uint32_t)__cvta_generic_to_shared(mbar);
  if (tid == 0) umma_mbar_init(mb);
  if (warp == 0) {
    tmem_alloc((uint32_t)__cvta_generic_to_shared(tslot), kUmmaCols);
    tmem_relinquish();
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  const uint32_t a1 = (uint32_t)__cvta_generic_to_shared(sA1), a2 = (uint32_t)__cvta_generic_to_shared(sA2),
                 b = (uint32_t)__cvta_generic_to_shared(sB);
  const uint64_t dA1 = umma_smem_desc(a1, 128, 256);
  const uint64_t dA2[2] = {umma_smem_desc(a2, 128, 512), umma_smem_desc(a2 + 256, 128, 512)};
  const uint64_t dB1 = umma_smem_desc(b + kUmmaB1, 128, 256);
  const uint64_t dB2[2] = {umma_smem_desc(b + kUmmaB2, 128, 512), umma_smem_desc(b + kUmmaB2 + 256, 128, 512)};
  const uint64_t dB3[2] = {umma_smem_desc(b + kUmmaB3, 128, 512), umma_smem_desc(b + kUmmaB3 + 256, 128, 512)};
  constexpr uint32_t id32 = umma_idesc_bf16(kUmmaRows, 32), id16 = umma_idesc_bf16(kUmmaRows, 16);
  const uint32_t lane_base = tbase + ((uint32_t)(warp * 32) << 16);
  uint32_t phase = 0;
  int issued = 0;  // commits issued (thread 0)
  bool failed = false;
  const long long tiles = (n + kUmmaRows - 1) / kUmmaRows;
  // one layer: thread 0 issues, everyone waits; false when the CTA timed out
  auto run = [&](auto issue) -> bool {
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid == 0) {
      issue();
      umma_commit(mb);
      ++issued;
    }
    const bool ok = umma_mbar_wait(mb, phase, kUmmaWaitLimit);
    phase ^= 1u;
    if (__syncthreads_or(!ok)) return false;
    tc_fence_after();
    return true;
  };
  for (long long tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
    const long long row = tile * kUmmaRows + tid;
    float x[kMlpIn];
#pragma unroll
    for (int i = 0; i < kMlpIn; ++i) x[i] = row < n ? X[row * kMlpIn + i] : 0.0f;
    *reinterpret_cast<uint4*>(sA1 + umma_off(tid, 0, 16)) =
        make_uint4(bf16x2_of(x[0], x[1]), bf16x2_of(x[2], x[3]), bf16x2_of(x[4], x[5]), bf16x2_of(x[6], x[7]));
    if (!run([&] { umma_bf16(tbase, dA1, dB1, id32, 0u); })) { failed = true; break; }
    float d[32];
    tmem_ld32(lane_base, d);
    umma_store_hidden(sA2, tid, d, sbias);
    if (!run([&] {
          umma_bf16(tbase + 32, dA2[0], dB2[0], id32, 0u);
          umma_bf16(tbase + 32, dA2[1], dB2[1], id32, 1u);
        })) { failed = true; break; }
    tmem_ld32(lane_base + 32, d);
    umma_store_hidden(sA2, tid, d, sbias + 32);
    if (!run([&] {
          umma_bf16(tbase, dA2[0], dB3[0], id16, 0u);
          umma_bf16(tbase, dA2[1], dB3[1], id16, 1u);
        })) { failed = true; break; }
    const float o = tmem_ld1(lane_base) + sbias[64];
    if (row < n) out[row] = softplus_f(o);
    tc_fence_before();
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(err, 1);
      umma_mbar_wait(mb, (uint32_t)((issued - 1) & 1), kUmmaWaitLimit);  // the last commit
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tbase, kUmmaCols);
}

// ---- wall distance: jump flooding over the solid cells (Rong & Tan, 2006) ----------
// Each cell keeps the packed coordinates (10 bits each) of the nearest solid cell seen.
constexpr uint32_t kNoSeed = 0xffffffffu;
__device__ __forceinline__ uint32_t pack_xyz(int x, int y, int z) {
  return (uint32_t)x | ((uint32_t)y << 10) | ((uint32_t)z << 20);
}
__device__ __forceinline__ float seed_dist2(uint32_t s, int x, int y, int z) {
  const float dx = (float)((int)(s & 1023u) - x), dy = (float)((int)((s >> 10) & 1023u) - y),
              dz = (float)((int)((s >> 20) & 1023u) - z);
  return dx * dx + dy * dy + dz * dz;
}

__global__ void jfa_init_kernel(const uint8_t* __restrict__ flags, int nx, int ny, int nz, uint32_t* __restrict__ seed) {
  const long long N = (long long)nx * ny * nz;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const long long r = i / nx;
    seed[i] = flags[i] == CELL_SOLID ? pack_xyz(x, (int)(r % ny), (int)(r / ny)) : kNoSeed;
  }
}

__global__ void jfa_pass_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int nx, int ny, int nz,
                                int k) {
  const long long N = (long long)nx * ny * nz;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const long long r = i / nx;
    const int y = (int)(r % ny), z = (int)(r / ny);
    uint32_t best = in[i];
    float bd = best == kNoSeed ? 3.0e38f : seed_dist2(best, x, y, z);
    for (int dz = -k; dz <= k; dz += k)
      for (int dy = -k; dy <= k; dy += k)
        for (int dx = -k; dx <= k; dx += k) {
          const int xx = x + dx, yy = y + dy, zz = z + dz;
          if (xx < 0 || yy < 0 || zz < 0 || xx >= nx || yy >= ny || zz >= nz) continue;
          const uint32_t s = in[xx + (long long)nx * (yy + (long long)ny * zz)];
          if (s == kNoSeed) continue;
          const float d = seed_dist2(s, x, y, z);
          if (d < bd) {
            bd = d;
            best = s;
          }
        }
    out[i] = best;
  }
}

// Distances (cells) into a dense float array and, rounded and capped at 31, into
// bits 3..7 of the solver's class bytes.
__global__ void jfa_finish_kernel(const uint32_t* __restrict__ seed, int nx, int ny, int nz, float* __restrict__ dist,
                                  uint8_t* __restrict__ cls, int pitch) {
  const long long N = (long long)nx * ny * nz;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const long long r = i / nx;
    const int y = (int)(r % ny), z = (int)(r / ny);
    const uint32_t s = seed[i];
    const float d = s == kNoSeed ? 1.0e4f : sqrtf(seed_dist2(s, x, y, z));
    if (dist) dist[i] = d;
    if (cls) {
      const int q = d >= 31.0f ? 31 : (int)lrintf(d);
      uint8_t& c = cls[r * pitch + x];
      c = (uint8_t)((c & 7) | (q << 3));
    }
  }
}

// ---- training samples from a fine-grid flow -------------------------------------
// Coarse cell (X, Y, Z) covers fine cells (2X..2X+1, 2Y.., 2Z..).  Pass 1: box-filtered
// velocity, density and velocity products; cells with a solid child are invalid.
__global__ void sgs_filter_kernel(const float* __restrict__ ux, const float* __restrict__ uy,
                                  const float* __restrict__ uz, const float* __restrict__ rho,
                                  const uint8_t* __restrict__ fflags, int fx, int fy, int fz, int cx, int cy, int cz,
                                  float* __restrict__ ubar /*[Nc][4]*/, float* __restrict__ uu /*[Nc][6]*/) {
  const long long Nc = (long long)cx * cy * cz;
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < Nc; c += (long long)gridDim.x * blockDim.x) {
    const int X = (int)(c % cx);
    const long long R = c / cx;
    const int Y = (int)(R % cy), Z = (int)(R / cy);
    float su[3] = {0, 0, 0}, sr = 0.0f, sq[6] = {0, 0, 0, 0, 0, 0};
    bool ok = true;
    for (int dz = 0; dz < 2; ++dz)
      for (int dy = 0; dy < 2; ++dy)
        for (int dx = 0; dx < 2; ++dx) {
          const long long f = (2 * X + dx) + (long long)fx * ((2 * Y + dy) + (long long)fy * (2 * Z + dz));
          if (fflags[f] == CELL_SOLID) ok = false;
          const float a = ux[f], b = uy[f], d = uz[f];
          su[0] += a; su[1] += b; su[2] += d; sr += rho[f];
          sq[0] += a * a; sq[1] += b * b; sq[2] += d * d; sq[3] += a * b; sq[4] += a * d; sq[5] += b * d;
        }
    const float* qq = sq;
    ubar[c * 4 + 0] = su[0] * 0.125f;
    ubar[c * 4 + 1] = su[1] * 0.125f;
    ubar[c * 4 + 2] = su[2] * 0.125f;
    ubar[c * 4 + 3] = ok ? sr * 0.125f : -1.0f;  // density; -1 marks an invalid cell
    for (int k = 0; k < 6; ++k) uu[c * 6 + k] = qq[k] * 0.125f;
  }
}

// Pass 2: filtered strain rate (central differences), subgrid stress
// tau = (u u)~ - u~ u~ and the two terms of the least-squares eddy viscosity
// nu_t = -tau_d : S / (2 S : S): numerator and denominator per cell (0 where invalid);
// features as in mlp_features with the filtered strain rate.
__global__ void sgs_sample_kernel(const float* __restrict__ ubar, const float* __restrict__ uu,
                                  const uint8_t* __restrict__ ccls, int cpitch, int cx, int cy, int cz,
                                  float* __restrict__ Xo, float2* __restrict__ nd, uint8_t* __restrict__ valid) {
  const long long Nc = (long long)cx * cy * cz;
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < Nc; c += (long long)gridDim.x * blockDim.x) {
    const int X = (int)(c % cx);
    const long long R = c / cx;
    const int Y = (int)(R % cy), Z = (int)(R / cy);
    bool ok = X > 0 && Y > 0 && Z > 0 && X < cx - 1 && Y < cy - 1 && Z < cz - 1 && ubar[c * 4 + 3] > 0.0f;
    float g[3][3];  // g[a][b] = d u_a / d x_b
    const long long st[3] = {1, cx, (long long)cx * cy};
    for (int bdir = 0; bdir < 3 && ok; ++bdir) {
      const long long p = c + st[bdir], m = c - st[bdir];
      if (ubar[p * 4 + 3] <= 0.0f || ubar[m * 4 + 3] <= 0.0f) ok = false;
      for (int a = 0; a < 3; ++a) g[a][bdir] = 0.5f * (ubar[p * 4 + a] - ubar[m * 4 + a]);
    }
    valid[c] = ok ? 1 : 0;
    if (!ok) {
      nd[c] = make_float2(0.0f, 0.0f);
      continue;
    }
    const float sxx = g[0][0], syy = g[1][1], szz = g[2][2];
    const float sxy = 0.5f * (g[0][1] + g[1][0]), sxz = 0.5f * (g[0][2] + g[2][0]), syz = 0.5f * (g[1][2] + g[2][1]);
    const float ux = ubar[c * 4], uy = ubar[c * 4 + 1], uz = ubar[c * 4 + 2], r = ubar[c * 4 + 3];
    float t[6] = {uu[c * 6] - ux * ux, uu[c * 6 + 1] - uy * uy, uu[c * 6 + 2] - uz * uz,
                  uu[c * 6 + 3] - ux * uy, uu[c * 6 + 4] - ux * uz, uu[c * 6 + 5] - uy * uz};
    const float tr = (t[0] + t[1] + t[2]) * (1.0f / 3.0f);
    t[0] -= tr; t[1] -= tr; t[2] -= tr;
    const float ss = sxx * sxx + syy * syy + szz * szz + 2.0f * (sxy * sxy + sxz * sxz + syz * syz);
    const float ts = t[0] * sxx + t[1] * syy + t[2] * szz + 2.0f * (t[3] * sxy + t[4] * sxz + t[5] * syz);
    nd[c] = make_float2(-ts, 2.0f * ss);
    const float wd = (float)(ccls[R * cpitch + X] >> 3);
    float* xo = Xo + c * kMlpIn;
    xo[0] = 100.0f * sxx; xo[1] = 100.0f * syy; xo[2] = 100.0f * szz;
    xo[3] = 100.0f * sxy; xo[4] = 100.0f * sxz; xo[5] = 100.0f * syz;
    xo[6] = 100.0f * (r - 1.0f);
    xo[7] = wd * (1.0f / 16.0f);
  }
}

// Pass 3: the target nu_t / nu_0 of a valid cell: numerators and denominators summed
// over the valid cells of its (2 avg + 1)^3 neighbourhood, then divided and clipped to
// [min_ratio, max_ratio] (least-squares averaging, which keeps the sign information that a
// per-cell clip at zero would discard; min_ratio < 0 keeps backscatter in the targets, so
// that a regression onto a non-negative output learns the conditional mean rather than
// the mean of the clipped values, which lies above it).
__global__ void sgs_target_kernel(const float2* __restrict__ nd, const uint8_t* __restrict__ valid, int cx, int cy,
                                  int cz, int avg, float nu0, float min_ratio, float max_ratio,
                                  float* __restrict__ Yo) {
  const long long Nc = (long long)cx * cy * cz;
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < Nc; c += (long long)gridDim.x * blockDim.x) {
    if (!valid[c]) {
      Yo[c] = 0.0f;
      continue;
    }
    const int X = (int)(c % cx);
    const long long R = c / cx;
    const int Y = (int)(R % cy), Z = (int)(R / cy);
    float n = 0.0f, d = 0.0f;
    for (int dz = -avg; dz <= avg; ++dz)
      for (int dy = -avg; dy <= avg; ++dy)
        for (int dx = -avg; dx <= avg; ++dx) {
          const int xx = X + dx, yy = Y + dy, zz = Z + dz;
          if (xx < 0 || yy < 0 || zz < 0 || xx >= cx || yy >= cy || zz >= cz) continue;
          const float2 v = nd[xx + (long long)cx * (yy + (long long)cy * zz)];
          n += v.x;
          d += v.y;
        }
    float nut = d > 0.0f ? n / d : 0.0f;
    nut = fminf(fmaxf(nut, min_ratio * nu0), max_ratio * nu0);
    Yo[c] = nut / nu0;
  }
}

int sgs_fail(int code, const std::string& msg) {
  set_global_error(msg);
  return code;
}

// Device time of the last forward kernel run by aerosim_mlp_forward_tc / _umma.
double g_mlp_last_ms = 0.0;

// CUDA events around one kernel launch on the default stream.
struct KernelTimer {
  cudaEvent_t a = nullptr, b = nullptr;
  KernelTimer() {
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    cudaEventRecord(a);
  }
  double stop() {
    float ms = 0.0f;
    cudaEventRecord(b);
    cudaEventSynchronize(b);
    cudaEventElapsedTime(&ms, a, b);
    return ms;
  }
  ~KernelTimer() {
    cudaEventDestroy(a);
    cudaEventDestroy(b);
  }
};

#define SCU(x)                                                                                       \
  do {                                                                                               \
    cudaError_t e_ = (x);                                                                            \
    if (e_ != cudaSuccess) return sgs_fail(AEROSIM_ERR_CUDA, std::string(#x ": ") + cudaGetErrorString(e_)); \
  } while (0)

// RAII device buffer for the host-array entry points below.
struct DevBuf {
  void* p = nullptr;
  ~DevBuf() { cudaFree(p); }
  cudaError_t alloc(size_t bytes) { return cudaMalloc(&p, bytes ? bytes : 1); }
  template <class T> T* as() { return static_cast<T*>(p); }
};

// Device buffers of a training or gradient call, in one allocation: parameters, Adam
// moments, samples, the CTAs' partial sums and the losses.
constexpr int kMlpPad = (kMlpParams + 63) / 64 * 64;
struct TrainBufs {
  DevBuf mem;
  float *P = nullptr, *M = nullptr, *V = nullptr, *X = nullptr, *Y = nullptr, *partial = nullptr;
  double *loss_partial = nullptr, *loss = nullptr;
  int max_ctas = 1;
  cudaError_t alloc(int64_t n, int64_t batch, int64_t losses) {
    int dev = 0, sms = 1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmem);
    if (e != cudaSuccess) return e;
    const int64_t groups = (batch + kGradRows - 1) / kGradRows;
    max_ctas = (int)std::min<int64_t>(sms, (groups + kGradWarps - 1) / kGradWarps);
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t bx = up((size_t)n * kMlpIn * 4), by = up((size_t)n * 4), bp = up((size_t)max_ctas * kGradSlots * 4),
                 bl = up((size_t)max_ctas * 8), bL = up((size_t)losses * 8);
    e = mem.alloc(3 * kMlpPad * 4 + bx + by + bp + bl + bL);
    if (e != cudaSuccess) return e;
    char* c = mem.as<char>();
    P = reinterpret_cast<float*>(c);
    M = P + kMlpPad;
    V = M + kMlpPad;
    c += 3 * kMlpPad * 4;
    X = reinterpret_cast<float*>(c); c += bx;
    Y = reinterpret_cast<float*>(c); c += by;
    partial = reinterpret_cast<float*>(c); c += bp;
    loss_partial = reinterpret_cast<double*>(c); c += bl;
    loss = reinterpret_cast<double*>(c);
    return cudaSuccess;
  }
};

// Gradient of n samples and its use, on the default stream, each kernel a programmatic
// dependent of the one before it.
cudaError_t launch_train_step(const TrainBufs& t, const BatchRows& rows, int64_t n, float* G, const AdamState& st,
                              double* loss) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  const float inv_n = 1.0f / (float)n;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)t.max_ctas);
  cfg.blockDim = dim3(kGradWarps * 32);
  cfg.dynamicSmemBytes = kGradSmem;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, mlp_grad_kernel, (const float*)t.P, (const float*)t.X, (const float*)t.Y, rows,
                                     (long long)n, inv_n, t.partial, t.loss_partial);
  if (e != cudaSuccess) return e;
  cfg.gridDim = dim3(kGradCols);
  cfg.blockDim = dim3(kApplyThreads);
  cfg.dynamicSmemBytes = 0;
  return cudaLaunchKernelEx(&cfg, mlp_apply_kernel, (const float*)t.partial, (const double*)t.loss_partial, t.max_ctas,
                            inv_n, G, st, loss);
}

}  // namespace

// Jump-flood wall distance of a dense flag array (device), written as float distances
// (dist, may be null) and into bits 3..7 of the pitched class bytes (cls, may be null).
cudaError_t compute_wall_distance(const uint8_t* flags, int nx, int ny, int nz, float* dist, uint8_t* cls, int pitch,
                                  cudaStream_t s) {
  const long long N = (long long)nx * ny * nz;
  if (nx > 1024 || ny > 1024 || nz > 1024) return cudaErrorInvalidValue;
  uint32_t *a = nullptr, *b = nullptr;
  cudaError_t e = cudaMallocAsync(&a, N * sizeof(uint32_t), s);
  if (e == cudaSuccess) e = cudaMallocAsync(&b, N * sizeof(uint32_t), s);
  const int grid = (int)std::min<long long>((N + 255) / 256, 148 * 16);
  if (e == cudaSuccess) jfa_init_kernel<<<grid, 256, 0, s>>>(flags, nx, ny, nz, a);
  int k = 1;
  while (2 * k < std::max(nx, std::max(ny, nz))) k *= 2;
  for (; k >= 1 && e == cudaSuccess; k /= 2) {
    jfa_pass_kernel<<<grid, 256, 0, s>>>(a, b, nx, ny, nz, k);
    std::swap(a, b);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {  // one more unit pass removes most of the flood's errors (JFA+1)
    jfa_pass_kernel<<<grid, 256, 0, s>>>(a, b, nx, ny, nz, 1);
    std::swap(a, b);
    jfa_finish_kernel<<<grid, 256, 0, s>>>(a, nx, ny, nz, dist, cls, pitch);
    e = cudaGetLastError();
  }
  cudaFreeAsync(a, s);
  cudaFreeAsync(b, s);
  return e;
}

cudaError_t launch_sgs_samples(const float* ux, const float* uy, const float* uz, const float* rho,
                               const uint8_t* fflags, int fx, int fy, int fz, const uint8_t* ccls, int cpitch, int cx,
                               int cy, int cz, float nu0, float min_ratio, float max_ratio, int avg, float* X,
                               float* Y, uint8_t* valid, cudaStream_t s) {
  const long long Nc = (long long)cx * cy * cz;
  float *ubar = nullptr, *uu = nullptr;
  float2* nd = nullptr;
  cudaError_t e = cudaMallocAsync(&ubar, Nc * 4 * sizeof(float), s);
  if (e == cudaSuccess) e = cudaMallocAsync(&uu, Nc * 6 * sizeof(float), s);
  if (e == cudaSuccess) e = cudaMallocAsync(&nd, Nc * sizeof(float2), s);
  const int grid = (int)std::min<long long>((Nc + 255) / 256, 148 * 16);
  if (e == cudaSuccess) {
    sgs_filter_kernel<<<grid, 256, 0, s>>>(ux, uy, uz, rho, fflags, fx, fy, fz, cx, cy, cz, ubar, uu);
    sgs_sample_kernel<<<grid, 256, 0, s>>>(ubar, uu, ccls, cpitch, cx, cy, cz, X, nd, valid);
    sgs_target_kernel<<<grid, 256, 0, s>>>(nd, valid, cx, cy, cz, avg, nu0, min_ratio, max_ratio, Y);
    e = cudaGetLastError();
  }
  cudaFreeAsync(ubar, s);
  cudaFreeAsync(uu, s);
  cudaFreeAsync(nd, s);
  return e;
}

}  // namespace aerosim

using namespace aerosim;

extern "C" {

int aerosim_mlp_param_count(void) { return kMlpParams; }

int aerosim_mlp_forward(const float* params, const float* X, int64_t n, float* out) {
  if (!params || !X || !out || n < 0) return sgs_fail(AEROSIM_ERR_ARG, "mlp_forward: bad argument");
  if (n == 0) return AEROSIM_OK;
  DevBuf P, Xd, O;
  SCU(P.alloc(kMlpParams * 4));
  SCU(Xd.alloc((size_t)n * kMlpIn * 4));
  SCU(O.alloc((size_t)n * 4));
  SCU(cudaMemcpy(P.p, params, kMlpParams * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(Xd.p, X, (size_t)n * kMlpIn * 4, cudaMemcpyHostToDevice));
  mlp_forward_kernel<<<(unsigned)((n + 127) / 128), 128>>>(P.as<float>(), Xd.as<float>(), n, O.as<float>());
  SCU(cudaGetLastError());
  SCU(cudaMemcpy(out, O.p, (size_t)n * 4, cudaMemcpyDeviceToHost));
  return AEROSIM_OK;
}

int aerosim_mlp_forward_tc(const float* params, const float* X, int64_t n, float* out) {
  if (!params || !X || !out || n < 0) return sgs_fail(AEROSIM_ERR_ARG, "mlp_forward_tc: bad argument");
  if (n == 0) return AEROSIM_OK;
  std::vector<uint32_t> frag(kMlpFragWords * 32);
  std::vector<float> bias(kMlpBias);
  mlp_pack_fragments(params, frag.data(), bias.data());
  DevBuf F, B, Xd, O;
  SCU(F.alloc(frag.size() * 4));
  SCU(B.alloc(bias.size() * 4));
  SCU(Xd.alloc((size_t)n * kMlpIn * 4));
  SCU(O.alloc((size_t)n * 4));
  SCU(cudaMemcpy(F.p, frag.data(), frag.size() * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(B.p, bias.data(), bias.size() * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(Xd.p, X, (size_t)n * kMlpIn * 4, cudaMemcpyHostToDevice));
  {
    KernelTimer t;
    mlp_forward_tc_kernel<<<(unsigned)((n + 127) / 128), 128>>>(F.as<uint32_t>(), B.as<float>(), Xd.as<float>(), n,
                                                                O.as<float>());
    SCU(cudaGetLastError());
    g_mlp_last_ms = t.stop();
  }
  SCU(cudaMemcpy(out, O.p, (size_t)n * 4, cudaMemcpyDeviceToHost));
  return AEROSIM_OK;
}

int aerosim_mlp_forward_umma(const float* params, const float* X, int64_t n, float* out) {
  if (!params || !X || !out || n < 0) return sgs_fail(AEROSIM_ERR_ARG, "mlp_forward_umma: bad argument");
  if (n == 0) return AEROSIM_OK;
  std::vector<uint16_t> img(kUmmaBBytes / 2);
  std::vector<uint32_t> frag(kMlpFragWords * 32);
  std::vector<float> bias(kMlpBias);
  mlp_pack_umma(params, img.data());
  mlp_pack_fragments(params, frag.data(), bias.data());
  int dev = 0, sms = 0;
  SCU(cudaGetDevice(&dev));
  SCU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  DevBuf Bi, B, Xd, O, E;
  SCU(Bi.alloc(kUmmaBBytes));
  SCU(B.alloc(bias.size() * 4));
  SCU(Xd.alloc((size_t)n * kMlpIn * 4));
  SCU(O.alloc((size_t)n * 4));
  SCU(E.alloc(4));
  SCU(cudaMemcpy(Bi.p, img.data(), kUmmaBBytes, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(B.p, bias.data(), bias.size() * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(Xd.p, X, (size_t)n * kMlpIn * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemset(E.p, 0, 4));
  SCU(cudaFuncSetAttribute(mlp_forward_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kUmmaSmem));
  const long long tiles = (n + kUmmaRows - 1) / kUmmaRows;
  const unsigned grid = (unsigned)std::min<long long>(tiles, 8LL * sms);
  {
    KernelTimer t;
    mlp_forward_umma_kernel<<<grid, kUmmaRows, kUmmaSmem>>>(static_cast<const uint4*>(Bi.p), B.as<float>(),
                                                            Xd.as<float>(), n, O.as<float>(), E.as<int>());
    SCU(cudaGetLastError());
    g_mlp_last_ms = t.stop();
  }
  int e = 0;
  SCU(cudaMemcpy(&e, E.p, 4, cudaMemcpyDeviceToHost));
  if (e) return sgs_fail(AEROSIM_ERR_DEVICE, "mlp_forward_umma: tensor-core commit wait timed out");
  SCU(cudaMemcpy(out, O.p, (size_t)n * 4, cudaMemcpyDeviceToHost));
  return AEROSIM_OK;
}

int aerosim_mlp_last_timing(double* ms) {
  if (!ms) return sgs_fail(AEROSIM_ERR_ARG, "mlp_last_timing: bad argument");
  *ms = g_mlp_last_ms;
  return AEROSIM_OK;
}

int aerosim_mlp_gradients(const float* params, const float* X, const float* Y, int64_t n, float* grad,
                          double* loss) {
  if (!params || !X || !Y || !grad || !loss || n < 1) return sgs_fail(AEROSIM_ERR_ARG, "mlp_gradients: bad argument");
  TrainBufs t;
  SCU(t.alloc(n, n, 1));
  SCU(cudaMemcpy(t.P, params, kMlpParams * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(t.X, X, (size_t)n * kMlpIn * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(t.Y, Y, (size_t)n * 4, cudaMemcpyHostToDevice));
  AdamState st{};
  SCU(launch_train_step(t, BatchRows{0, 0, 0, 0}, n, t.M, st, t.loss));
  SCU(cudaMemcpy(grad, t.M, kMlpParams * 4, cudaMemcpyDeviceToHost));
  SCU(cudaMemcpy(loss, t.loss, 8, cudaMemcpyDeviceToHost));
  return AEROSIM_OK;
}

int aerosim_mlp_train(float* params, const float* X, const float* Y, int64_t n, int32_t iters, int32_t batch,
                      float lr, uint64_t seed, float* loss_curve) {
  if (!params || !X || !Y || n < 1 || iters < 0 || batch < 1 || !(lr > 0.0f))
    return sgs_fail(AEROSIM_ERR_ARG, "mlp_train: bad argument");
  TrainBufs t;
  SCU(t.alloc(n, batch, std::max(iters, 1)));
  SCU(cudaMemcpy(t.P, params, kMlpParams * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(t.X, X, (size_t)n * kMlpIn * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(t.Y, Y, (size_t)n * 4, cudaMemcpyHostToDevice));
  SCU(cudaMemsetAsync(t.M, 0, 2 * kMlpPad * 4));  // M and V
  AdamState st{t.P, t.M, t.V, lr, 1.0f, 1.0f};
  for (int it = 0; it < iters; ++it) {
    st.b1t *= 0.9f;
    st.b2t *= 0.999f;
    SCU(launch_train_step(t, BatchRows{seed, (unsigned long long)n, ~0ull / (unsigned long long)n, it}, batch, nullptr, st, t.loss + it));
  }
  SCU(cudaDeviceSynchronize());
  SCU(cudaMemcpy(params, t.P, kMlpParams * 4, cudaMemcpyDeviceToHost));
  if (loss_curve && iters > 0) {
    std::vector<double> l(iters);
    SCU(cudaMemcpy(l.data(), t.loss, (size_t)iters * 8, cudaMemcpyDeviceToHost));
    for (int i = 0; i < iters; ++i) loss_curve[i] = (float)l[i];
  }
  return AEROSIM_OK;
}

}  // extern "C"
