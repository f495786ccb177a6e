// dc_learned.cu -- the learned thin absorbing layer.
//
// A thin layer of L cells (L <= DC_GB300_MLP_DEPTHS) between the physical
// interior and the 4-cell halo replaces the wide sponge.  After every
// stencil pass, each of the layer's 4 outer cells -- those whose stencils
// reach into the zero halo -- gets a correction (dp, dq) predicted by a
// small MLP from the cells along its boundary normal (the inner L - 4 cells
// are updated by the stencil alone):
//
//   features  the cell and the 7 cells inward along the normal, p and q, at
//             t+1 (the stencil's output) and t: 8 x 2 x 2 = 32 values
//   scale     r = rms of the 32 features; the network sees x / r and its
//             output is multiplied by r (the correction is homogeneous of
//             degree 1 in the wavefield, like a linear absorbing condition)
//   network   32 -> 32 -> 32 -> 2, GELU (tanh form), BF16 weights and
//             activations, FP32 accumulation; the first hidden layer's bias
//             depends on the cell's depth in the layer (0 = next to the
//             interior).  Inference runs on the tensor cores (mma.sync
//             m16n8k16 BF16, activations kept in registers between layers);
//             training on CUDA cores.
//
// The normal of an edge or corner cell is the axis along which it lies
// deepest in the layer (lowest axis on ties).
//
// Training (teacher forcing): a wide simulation, whose margins keep every
// reflection out of the region of interest for the whole run, supplies the
// truth.  At a sampled step its fields (t and t-1) are cropped to the thin
// box (zero halo), stepped once by the thin simulation, and every layer cell
// yields a sample (features of the thin step) and a target (wide field at
// t+1 minus the thin step).  The loss is sum |r * y - target|^2 / sum r^2
// over a minibatch; gradients run through the BF16 roundings unchanged;
// Adam updates FP32 master weights.  Every kernel here is this project's own.
//
// The reference has no learned boundary; it absorbs with its random
// velocity boundary (src/boundary.c:7-104).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <string>
#include <vector>

#include "dc_internal.h"
#include "dc_ptx.cuh"

namespace dcg {
namespace {

constexpr int kIn = DC_GB300_MLP_IN, kHid = DC_GB300_MLP_HIDDEN, kOut = DC_GB300_MLP_OUT;
constexpr int kDepths = DC_GB300_MLP_DEPTHS;
constexpr int kStride = kIn + 1;  // sample row: 32 features + depth
constexpr int OFF_W1 = 0;                         // [kHid][kIn]
constexpr int OFF_B1 = OFF_W1 + kHid * kIn;       // [kDepths][kHid]
constexpr int OFF_W2 = OFF_B1 + kDepths * kHid;   // [kHid][kHid]
constexpr int OFF_B2 = OFF_W2 + kHid * kHid;      // [kHid]
constexpr int OFF_W3 = OFF_B2 + kHid;             // [kOut][kHid]
constexpr int OFF_B3 = OFF_W3 + kOut * kHid;      // [kOut]
constexpr int kParams = OFF_B3 + kOut;
static_assert(kParams == DC_GB300_MLP_PARAMS, "parameter count");
constexpr int kWin = 8;  // cells along the normal
constexpr int kCorrected = 4;  // outer layer cells corrected by the network

__device__ __forceinline__ bool is_weight(int p) {
  return (p >= OFF_W1 && p < OFF_B1) || (p >= OFF_W2 && p < OFF_B2) || (p >= OFF_W3 && p < OFF_B3);
}

__device__ __forceinline__ float bf16r(float v) {
  return __bfloat162float(__float2bfloat16_rn(v));
}

// GELU in its tanh form (Hendrycks & Gimpel 2016):
//   gelu(a) = a/2 (1 + tanh(c0 (a + c1 a^3))), c0 = sqrt(2/pi), c1 = 0.044715,
// with the hardware tanh (tanh.approx.f32, one MUFU operation), the same in
// training and inference.
constexpr float kGeluC0 = 0.7978845608028654f, kGeluC1 = 0.044715f;

__device__ __forceinline__ float tanh_hw(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// u = a (c0 + c0 c1 a^2); gelu = h + h tanh(u), h = a / 2.  The scalar and
// the packed (two values, FFMA2/FMUL2) forms round identically.
constexpr float kGeluC01 = kGeluC0 * kGeluC1;

__device__ __forceinline__ float gelu(float a) {
  const float u = fmaf(a * a, kGeluC01, kGeluC0) * a;
  const float h = 0.5f * a;
  return fmaf(h, tanh_hw(u), h);
}

__device__ __forceinline__ float2 gelu2(float2 a) {
  const float2 t = __ffma2_rn(__fmul2_rn(a, a), make_float2(kGeluC01, kGeluC01),
                              make_float2(kGeluC0, kGeluC0));
  const float2 u = __fmul2_rn(t, a);
  const float2 th = make_float2(tanh_hw(u.x), tanh_hw(u.y));
  const float2 h = __fmul2_rn(a, make_float2(0.5f, 0.5f));
  return __ffma2_rn(h, th, h);
}

__device__ __forceinline__ float gelu_grad(float a) {
  const float a2 = a * a;
  const float th = tanh_hw(fmaf(a2, kGeluC01, kGeluC0) * a);
  const float du = kGeluC0 * fmaf(3.0f * kGeluC1, a2, 1.0f);
  return 0.5f * (1.0f + th) + 0.5f * a * (1.0f - th * th) * du;
}

// ---------------------------------------------------------------------------
// Training: gradient of sum_i |r_i y_i - t_i|^2 over a set of samples.
// `sampled` = 0: samples [0, count); 1: `count` samples drawn with
// replacement from [0, n) by hashing `seed`.
//
// A pass of a CTA takes 128 samples; warp w computes the hidden units
// 4 (w / 2) .. + 3 of half of them, two neighbouring samples per lane: eight
// chains per thread over the inputs, fed by two vector loads from shared
// memory per input, and four chains over the samples in the weight gradients.
// A unit's value and a pass's share of a weight's gradient stay single
// chains, as when one thread took a whole sample (same bits).  What bounds
// the pass is latency and the shared-memory pipe (0.1 GFLOP per 8192
// samples): with one sample per thread each scheduler of 64 SMs had one warp
// (44 us); a quad of units and one sample per thread, 1024 threads, issued
// 32 k shared-memory wavefronts (24 us); a quad and four samples, 256
// threads, left two warps per scheduler (20 us).
constexpr int kTB = 128;           // samples per pass
constexpr int kTT = 512;           // threads
constexpr int kRow = kTB + 4;      // padded row: no bank conflicts along samples or units
constexpr int kU = 4, kS = 2;      // hidden units and samples per thread
static_assert(kIn == 32 && kHid == 32 && kTT * kU * kS == kTB * kHid && kTT == 32 * kDepths,
              "thread tiles; one depth of b1 per warp");

struct GradSmem {
  // [unit][sample]: normalised inputs, activations and deltas
  float xh[kIn * kRow], h1[kHid * kRow], h2[kHid * kRow], d1[kHid * kRow], d2[kHid * kRow];
  float w1t[kIn * kHid], w2t[kHid * kHid];  // [input][unit] (forward)
  float w2[kHid * kHid], w3[kOut * kHid];   // [unit][input] (backward)
  float b1[kDepths * kHid], b2[kHid];
  float dy[kOut * kTB], r[kTB];             // r: rms, 0 for silent or missing samples
  long long idx[kTB];
  int dep[kTB];
  float b3[kOut];
};

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

// a[m][i] += sum_k w[k][m] * x[k][i], k ascending: 8 chains.
__device__ __forceinline__ void chain32(const float *w, const float *x, float a[kU][kS]) {
#pragma unroll 8
  for (int k = 0; k < 32; ++k) {
    const float4 wk = *reinterpret_cast<const float4 *>(w + k * 32);
    const float2 xk = *reinterpret_cast<const float2 *>(x + k * kRow);
    const float wv[kU] = {wk.x, wk.y, wk.z, wk.w};
#pragma unroll
    for (int m = 0; m < kU; ++m) {
      a[m][0] = fmaf(wv[m], xk.x, a[m][0]);
      a[m][1] = fmaf(wv[m], xk.y, a[m][1]);
    }
  }
}

// g[o][j] += sum over the samples of d[row o][s] * x[row 16 j][s], s
// ascending: 4 chains.
__device__ __forceinline__ void outer128(const float *d, const float *x, float g[2][2]) {
  float s[2][2] = {};
#pragma unroll 4
  for (int q = 0; q < kTB; q += 4) {
    float4 dv[2], xv[2];
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      dv[o] = *reinterpret_cast<const float4 *>(d + o * kRow + q);
      xv[o] = *reinterpret_cast<const float4 *>(x + 16 * o * kRow + q);
    }
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        s[o][j] = fmaf(dv[o].x, xv[j].x, s[o][j]);
        s[o][j] = fmaf(dv[o].y, xv[j].y, s[o][j]);
        s[o][j] = fmaf(dv[o].z, xv[j].z, s[o][j]);
        s[o][j] = fmaf(dv[o].w, xv[j].w, s[o][j]);
      }
  }
#pragma unroll
  for (int o = 0; o < 2; ++o)
#pragma unroll
    for (int j = 0; j < 2; ++j) g[o][j] += s[o][j];
}

__global__ void __launch_bounds__(kTT) mlp_grad_kernel(const float *wc,
                                                       const float *__restrict__ xs,
                                                       const float *__restrict__ ts, long long n,
                                                       long long count, unsigned long long seed,
                                                       int sampled, float *grad, double *acc) {
  extern __shared__ __align__(16) unsigned char grad_smem[];
  GradSmem &sm = *reinterpret_cast<GradSmem *>(grad_smem);
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  auto stage = [&] {
    for (int i = t; i < kHid * kIn; i += kTT) {
      // (transposed: the reads are scattered over the 4 KB, the stores are not)
      const int k = i / kHid, o = i % kHid;
      sm.w1t[i] = wc[OFF_W1 + o * kIn + k];
      sm.w2t[i] = wc[OFF_W2 + o * kHid + k];
      sm.w2[i] = wc[OFF_W2 + i];
    }
    for (int i = t; i < kDepths * kHid; i += kTT) sm.b1[i] = wc[OFF_B1 + i];
    if (t < kOut * kHid) sm.w3[t] = wc[OFF_W3 + t];
    if (t < kHid) sm.b2[t] = wc[OFF_B2 + t];
    if (t < kOut) sm.b3[t] = wc[OFF_B3 + t];
  };
  bool staged = false;
  // gradients of this thread: units go, go + 1 x inputs gk, gk + 16 of W1
  // (warps 0-7) or W2 (8-15); unit `lane` at depth w of b1; W3 (warps 0, 1),
  // b2 (2) and b3 (3)
  const int go = 4 * (w & 7) + 2 * (lane >> 4), gk = lane & 15;
  float gW[2][2] = {}, gB1 = 0.f, gX = 0.f;
  double l_err = 0.0, l_w = 0.0;
  const int u0 = kU * (w >> 1), s0 = 64 * (w & 1) + kS * lane;  // this thread's units and samples
  for (long long base = static_cast<long long>(blockIdx.x) * kTB; base < count;
       base += static_cast<long long>(gridDim.x) * kTB) {
    if (t < kTB) {
      long long i = base + t;
      if (i >= count)
        i = -1;
      else if (sampled)
        i = static_cast<long long>(mix64(seed ^ (static_cast<unsigned long long>(i) * 0x2545F4914F6CDD1Dull)) % static_cast<unsigned long long>(n));
      sm.idx[t] = i;
      sm.dep[t] = i >= 0 ? min(max(static_cast<int>(xs[i * kStride + kIn]), 0), kDepths - 1) : 0;
    }
    __syncthreads();
    // eight sample rows per warp, transposed into [feature][sample]
    float x[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const long long i = sm.idx[8 * w + q];
      x[q] = i >= 0 ? xs[i * kStride + lane] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < 8; q += 4)
      *reinterpret_cast<float4 *>(sm.xh + lane * kRow + 8 * w + q) =
          make_float4(x[q], x[q + 1], x[q + 2], x[q + 3]);
    if (!staged) {  // the first rows come in while Adam updates the weights
      grid_dep_wait();
      grid_dep_launch();
      stage();
      staged = true;
    }
    __syncthreads();
    if (t < kTB) {
      float ss = 0.f;
#pragma unroll 8
      for (int k = 0; k < kIn; ++k) ss = fmaf(sm.xh[k * kRow + t], sm.xh[k * kRow + t], ss);
      sm.r[t] = sqrtf(ss * (1.0f / kIn));
    }
    __syncthreads();
    bool live[kS];  // silent samples contribute nothing
    {
      const float2 rv = *reinterpret_cast<const float2 *>(sm.r + s0);
      live[0] = rv.x > 0.f;
      live[1] = rv.y > 0.f;
      const float i0 = 1.0f / rv.x, i1 = 1.0f / rv.y;
#pragma unroll
      for (int m = 0; m < kU; ++m) {
        float2 *row = reinterpret_cast<float2 *>(sm.xh + (u0 + m) * kRow + s0);
        const float2 xv = *row;
        *row = make_float2(live[0] ? bf16r(xv.x * i0) : 0.f, live[1] ? bf16r(xv.y * i1) : 0.f);
      }
    }
    __syncthreads();
    // a layer's activations of this thread's tile, rounded, to `to`
    auto put = [&](float *to, const float a[kU][kS]) {
#pragma unroll
      for (int m = 0; m < kU; ++m)
        *reinterpret_cast<float2 *>(to + (u0 + m) * kRow + s0) = make_float2(
            live[0] ? bf16r(gelu(a[m][0])) : 0.f, live[1] ? bf16r(gelu(a[m][1])) : 0.f);
    };
    float a1[kU][kS], a2[kU][kS];
#pragma unroll
    for (int i = 0; i < kS; ++i) {
      const float4 bv = *reinterpret_cast<const float4 *>(sm.b1 + sm.dep[s0 + i] * kHid + u0);
      a1[0][i] = bv.x, a1[1][i] = bv.y, a1[2][i] = bv.z, a1[3][i] = bv.w;
    }
    chain32(sm.w1t + u0, sm.xh + s0, a1);
    put(sm.h1, a1);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < kU; ++m) a2[m][0] = a2[m][1] = sm.b2[u0 + m];
    chain32(sm.w2t + u0, sm.h1 + s0, a2);
    put(sm.h2, a2);
    __syncthreads();
    if (t < kOut * kTB) {  // output j of sample s
      const int j = t / kTB, s = t % kTB;
      const float r = sm.r[s];
      float d = 0.f;
      if (r > 0.f) {
        float a = sm.b3[j];
#pragma unroll 8
        for (int k = 0; k < kHid; ++k) a = fmaf(sm.w3[j * kHid + k], sm.h2[k * kRow + s], a);
        const float e = r * a - ts[sm.idx[s] * kOut + j];
        l_err += static_cast<double>(e) * e;
        if (j == 0) l_w += static_cast<double>(r) * r;
        d = 2.0f * r * e;
      }
      sm.dy[t] = d;
    }
    __syncthreads();
    {  // delta2 = (W3^T dy) * gelu'(a2); delta1 = (W2^T delta2) * gelu'(a1)
      const float2 e0 = *reinterpret_cast<const float2 *>(sm.dy + s0);
      const float2 e1 = *reinterpret_cast<const float2 *>(sm.dy + kTB + s0);
#pragma unroll
      for (int m = 0; m < kU; ++m) {
        const float w30 = sm.w3[u0 + m], w31 = sm.w3[kHid + u0 + m];
        *reinterpret_cast<float2 *>(sm.d2 + (u0 + m) * kRow + s0) = make_float2(
            live[0] ? fmaf(w31, e1.x, fmaf(w30, e0.x, 0.f)) * gelu_grad(a2[m][0]) : 0.f,
            live[1] ? fmaf(w31, e1.y, fmaf(w30, e0.y, 0.f)) * gelu_grad(a2[m][1]) : 0.f);
      }
    }
    __syncthreads();
    float dd[kU][kS] = {};
    chain32(sm.w2 + u0, sm.d2 + s0, dd);
#pragma unroll
    for (int m = 0; m < kU; ++m)
      *reinterpret_cast<float2 *>(sm.d1 + (u0 + m) * kRow + s0) =
          make_float2(live[0] ? dd[m][0] * gelu_grad(a1[m][0]) : 0.f,
                      live[1] ? dd[m][1] * gelu_grad(a1[m][1]) : 0.f);
    __syncthreads();
    // gradients: sums over the samples of this pass
    outer128((w < 8 ? sm.d1 : sm.d2) + go * kRow, (w < 8 ? sm.xh : sm.h1) + gk * kRow, gW);
    {
      float s1 = 0.f;
#pragma unroll 4
      for (int q = 0; q < kTB; q += 4) {
        const int4 dq = *reinterpret_cast<const int4 *>(sm.dep + q);
        const float4 av = *reinterpret_cast<const float4 *>(sm.d1 + lane * kRow + q);
        if (dq.x == w) s1 += av.x;
        if (dq.y == w) s1 += av.y;
        if (dq.z == w) s1 += av.z;
        if (dq.w == w) s1 += av.w;
      }
      gB1 += s1;
    }
    if (w < kOut + 2) {
      // W3: dy[j] . h2[unit]; b2: sum of delta2; b3: sum of dy
      const float *p = w < kOut ? sm.h2 + lane * kRow
                       : w == kOut ? sm.d2 + lane * kRow : sm.dy + (lane & (kOut - 1)) * kTB;
      float sx = 0.f;
#pragma unroll 4
      for (int q = 0; q < kTB; q += 4) {
        const float4 pv = *reinterpret_cast<const float4 *>(p + q);
        if (w < kOut) {
          const float4 ev = *reinterpret_cast<const float4 *>(sm.dy + w * kTB + q);
          sx = fmaf(ev.x, pv.x, sx);
          sx = fmaf(ev.y, pv.y, sx);
          sx = fmaf(ev.z, pv.z, sx);
          sx = fmaf(ev.w, pv.w, sx);
        } else {
          sx += pv.x;
          sx += pv.y;
          sx += pv.z;
          sx += pv.w;
        }
      }
      gX += sx;
    }
    __syncthreads();
  }
  {
    float *gw = grad + (w < 8 ? OFF_W1 : OFF_W2) + go * 32 + gk;
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
      for (int j = 0; j < 2; ++j) atomicAdd(&gw[o * 32 + 16 * j], gW[o][j]);
  }
  atomicAdd(&grad[OFF_B1 + t], gB1);
  if (w < kOut) atomicAdd(&grad[OFF_W3 + w * kHid + lane], gX);
  if (w == kOut) atomicAdd(&grad[OFF_B2 + lane], gX);
  if (w == kOut + 1 && lane < kOut) atomicAdd(&grad[OFF_B3 + lane], gX);
  // loss sums (the warps that computed outputs hold them)
  if (t < kOut * kTB) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      l_err += __shfl_down_sync(0xffffffffu, l_err, off);
      l_w += __shfl_down_sync(0xffffffffu, l_w, off);
    }
    if (lane == 0) {
      atomicAdd(&acc[0], l_err);
      if (t < kTB) atomicAdd(&acc[1], l_w);
    }
  }
}

// Adam step on the FP32 master weights with the gradient of the mean loss
// (grad / sum r^2); refreshes the compute copy (weights rounded to BF16),
// clears the gradient and the other step parity's loss sums, and records the
// loss.  64 threads per CTA: the FP64 division runs at a fiftieth of the FP32
// rate, so the parameters are spread over 42 SMs (done by the last CTA of the
// gradient kernel instead, the step took 20 us longer).
constexpr int kAdamT = 64;
__global__ void __launch_bounds__(kAdamT)
    mlp_adam_kernel(float *master, float *wc, float *m1, float *m2, float *grad,
                    const double *acc, double *next_acc, float lr, float b1, float b2, float eps, int step, float *loss_hist, int hist_index) {
  grid_dep_wait();
  grid_dep_launch();
  const int p = blockIdx.x * kAdamT + threadIdx.x;
  const double w = acc[1];
  if (p < kParams) {
    const float g = w > 0.0 ? static_cast<float>(grad[p] / w) : 0.0f;
    const float a = b1 * m1[p] + (1.0f - b1) * g;
    const float v = b2 * m2[p] + (1.0f - b2) * g * g;
    m1[p] = a;
    m2[p] = v;
    const float ah = a / (1.0f - powf(b1, static_cast<float>(step)));
    const float vh = v / (1.0f - powf(b2, static_cast<float>(step)));
    const float nw = master[p] - lr * ah / (sqrtf(vh) + eps);
    master[p] = nw;
    wc[p] = is_weight(p) ? bf16r(nw) : nw;
    grad[p] = 0.0f;
  }
  if (p == kParams) {  // a thread of the last CTA without a parameter
    next_acc[0] = next_acc[1] = 0.0;
    if (loss_hist) loss_hist[hist_index] = w > 0.0 ? static_cast<float>(acc[0] / w) : 0.0f;
  }
}
static_assert(kParams % kAdamT != 0, "the last CTA has a spare thread");

// Compute copy of a parameter vector.
__global__ void mlp_round_kernel(const float *master, float *wc) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < kParams) wc[p] = is_weight(p) ? bf16r(master[p]) : master[p];
}

// ---------------------------------------------------------------------------
// Layer cells: int4 {x, y, z, meta}, meta = axis | side << 2 | depth << 3
// (side 1 = the high end of the axis).

// The 32 features of cell c from the new (t+1) and current (t) pair
// buffers; returns the depth.
__device__ __forceinline__ int gather(const int4 c, const float2 *nw, const float2 *cur,
                                      long long pitch, long long plane, float x[kIn]) {
  const int axis = c.w & 3, side = (c.w >> 2) & 1, depth = c.w >> 3;
  const long long stride = axis == 0 ? 1 : axis == 1 ? pitch : plane;
  const long long step = side ? -stride : stride;  // inward
  long long g = static_cast<long long>(c.z) * plane + static_cast<long long>(c.y) * pitch + c.x;
#pragma unroll
  for (int k = 0; k < kWin; ++k) {
    const float2 a = nw[g], b = cur[g];
    x[k] = a.x;
    x[kWin + k] = a.y;
    x[2 * kWin + k] = b.x;
    x[3 * kWin + k] = b.y;
    g += step;
  }
  return depth;
}

// ---------------------------------------------------------------------------
// Inference on the tensor cores.  One warp evaluates 16 cells per pass with
// mma.sync.m16n8k16 (BF16 operands, FP32 accumulation).  Lane (g = lane/4,
// t = lane%4) holds rows g and g+8 -- two cells -- and, per cell, the
// features of window positions 2t and 2t+1: exactly its A-fragment elements
// of the first layer (feature order p(t+1)[0..7], q(t+1)[0..7], p(t)[0..7],
// q(t)[0..7]).  Each layer's accumulator fragments are the next layer's A
// fragments, so the activations never leave registers; the weights are
// loaded once per warp as B fragments.

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ void mma_bf16(float d[4], const uint32_t a[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// GELU of a layer's accumulator fragments, packed into the next layer's A
// fragments (k-chunk kk = n-tiles 2kk and 2kk+1).
__device__ __forceinline__ void gelu_to_a(const float acc[4][4], uint32_t a[2][4]) {
#pragma unroll
  for (int kk = 0; kk < 2; ++kk) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 g0 = gelu2(make_float2(acc[2 * kk + h][0], acc[2 * kk + h][1]));
      const float2 g1 = gelu2(make_float2(acc[2 * kk + h][2], acc[2 * kk + h][3]));
      a[kk][2 * h] = pack_bf16(g0.x, g0.y);
      a[kk][2 * h + 1] = pack_bf16(g1.x, g1.y);
    }
  }
}

// Feature sources: load(r, t, f) fills f = {p1[2t], p1[2t+1], q1[2t],
// q1[2t+1], p0[2t], p0[2t+1], q0[2t], q0[2t+1]} of cell / sample r (p1, q1
// at t+1, p0, q0 at t) and returns its depth.
struct RowSrc {  // sample rows [n][33]
  const float *rows;
  __device__ __forceinline__ int load(long long r, int t, float f[8]) const {
    const float *row = rows + r * kStride;
    f[0] = row[2 * t];
    f[1] = row[2 * t + 1];
    f[2] = row[kWin + 2 * t];
    f[3] = row[kWin + 2 * t + 1];
    f[4] = row[2 * kWin + 2 * t];
    f[5] = row[2 * kWin + 2 * t + 1];
    f[6] = row[3 * kWin + 2 * t];
    f[7] = row[3 * kWin + 2 * t + 1];
    return min(max(static_cast<int>(row[kIn]), 0), kDepths - 1);
  }
};

__device__ __forceinline__ int load_cell(int4 c, const float2 *nw, const float2 *cur,
                                         long long pitch, long long plane, int t, float f[8],
                                         float *rec) {
  const int axis = c.w & 3, side = (c.w >> 2) & 1, depth = (c.w >> 3) & 31;
  const long long stride = axis == 0 ? 1 : axis == 1 ? pitch : plane;
  const long long step = side ? -stride : stride;  // inward
  const long long g = static_cast<long long>(c.z) * plane + static_cast<long long>(c.y) * pitch +
                      c.x + step * (2 * t);
  const float2 a0 = nw[g], a1 = nw[g + step], b0 = cur[g], b1 = cur[g + step];
  f[0] = a0.x;
  f[1] = a1.x;
  f[2] = a0.y;
  f[3] = a1.y;
  f[4] = b0.x;
  f[5] = b1.x;
  f[6] = b0.y;
  f[7] = b1.y;
  if (rec) {  // rollout training: the sample row of this cell
    rec[2 * t] = f[0];
    rec[2 * t + 1] = f[1];
    rec[kWin + 2 * t] = f[2];
    rec[kWin + 2 * t + 1] = f[3];
    rec[2 * kWin + 2 * t] = f[4];
    rec[2 * kWin + 2 * t + 1] = f[5];
    rec[3 * kWin + 2 * t] = f[6];
    rec[3 * kWin + 2 * t + 1] = f[7];
    if (t == 0) rec[kIn] = static_cast<float>(depth);
  }
  return depth;
}

struct CellSrc {  // the layer cells of one simulation
  const int4 *cells;
  const float2 *nw, *cur;
  long long pitch, plane;
  float *rec;
  __device__ __forceinline__ int load(long long r, int t, float f[8]) const {
    return load_cell(cells[r], nw, cur, pitch, plane, t, f, rec ? rec + r * kStride : nullptr);
  }
};

// Entries of the in-step tables (face lines and edge cells): {offset low,
// offset high, inward stride, code}, made by layer_tables; code = depth of an
// edge cell | shot << 8.  (With coordinates the kernels spent a sixth of their
// instructions on 64-bit index products.)
__device__ __forceinline__ long long entry_offset(const int4 e) {
  return static_cast<long long>(static_cast<uint32_t>(e.x)) | static_cast<long long>(e.y) << 32;
}

struct LinePtr {
  float2 *nw;         // the entry's (outermost) cell in the new field
  const float2 *cur;  // ... in the current field
  int step;           // inward stride
};

struct SimEntries {  // table of one simulation
  const int4 *table;
  float2 *nw;
  const float2 *cur;
  __device__ __forceinline__ LinePtr at(const int4 e) const {
    const long long o = entry_offset(e);
    return LinePtr{nw + o, cur + o, e.z};
  }
};

struct BatchEntries {  // table over the shots of a batch
  const int4 *table;
  const LbShot *shots;
  int cur_buf;
  __device__ __forceinline__ LinePtr at(const int4 e) const {
    const LbShot &sh = shots[e.w >> 8];
    const long long o = entry_offset(e);
    return LinePtr{sh.pq[1 - cur_buf] + o, sh.pq[cur_buf] + o, e.z};
  }
};

template <class Entries>
struct EdgeSrc {  // edge cells: features of the cell's window
  Entries t;
  __device__ __forceinline__ int load(long long r, int q, float f[8]) const {
    const int4 e = t.table[r];
    const LinePtr p = t.at(e);
    const long long o = static_cast<long long>(2 * q) * p.step;
    const float2 *n = p.nw + o, *c = p.cur + o;
    const float2 a0 = n[0], a1 = n[p.step], b0 = c[0], b1 = c[p.step];
    f[0] = a0.x;
    f[1] = a1.x;
    f[2] = a0.y;
    f[3] = a1.y;
    f[4] = b0.x;
    f[5] = b1.x;
    f[6] = b0.y;
    f[7] = b1.y;
    return e.w & 0xff;
  }
};

// The weights' B fragments live in shared memory (one 8-byte entry per
// lane and 16 x 8 block, read with one LDS.64 per MMA), which keeps the
// kernels under 64 registers: eight 4-warp CTAs per SM hide the gathers'
// latency.
struct NetSmem {
  float b1[kDepths * kHid], b2[kHid], b3[kOut];
  uint2 w1[2][4][32], w2[2][4][32], w3[2][32];
};

// Stages the biases and the weights' B fragments; ends with __syncthreads.
__device__ __forceinline__ void stage_net(const float *__restrict__ wc, NetSmem &sm) {
  for (int i = threadIdx.x; i < kDepths * kHid; i += blockDim.x) sm.b1[i] = wc[OFF_B1 + i];
  if (threadIdx.x < kHid) sm.b2[threadIdx.x] = wc[OFF_B2 + threadIdx.x];
  if (threadIdx.x < kOut) sm.b3[threadIdx.x] = wc[OFF_B3 + threadIdx.x];
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if (threadIdx.x < 32) {
    // B fragments: B[k][n] = W[n][k] of each 16 x 8 (k x n) block
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      const int k0 = kk * 16 + 2 * t;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const float *r1 = wc + OFF_W1 + (nt * 8 + g) * kIn;
        const float *r2 = wc + OFF_W2 + (nt * 8 + g) * kHid;
        sm.w1[kk][nt][lane] = make_uint2(pack_bf16(r1[k0], r1[k0 + 1]),
                                         pack_bf16(r1[k0 + 8], r1[k0 + 9]));
        sm.w2[kk][nt][lane] = make_uint2(pack_bf16(r2[k0], r2[k0 + 1]),
                                         pack_bf16(r2[k0 + 8], r2[k0 + 9]));
      }
      const float *r3 = wc + OFF_W3 + min(g, kOut - 1) * kHid;
      sm.w3[kk][lane] = g < kOut ? make_uint2(pack_bf16(r3[k0], r3[k0 + 1]),
                                              pack_bf16(r3[k0 + 8], r3[k0 + 9]))
                                 : make_uint2(0u, 0u);
    }
  }
  __syncthreads();
}

// The network over the 16 rows of one warp pass: lane (g, t) brings the
// features f0 of row g and f1 of row g + 8 (window positions 2t, 2t + 1, in
// the order of the sample-row loader) and their depths.  Returns false,
// warp-uniformly, when all 16 rows are silent (no correction anywhere);
// otherwise the lanes with t == 0 hold the corrections r * y of row g in
// (rr0 * y[0], rr0 * y[1]) and of row g + 8 in (rr1 * y[2], rr1 * y[3]).
__device__ __forceinline__ bool net16(const NetSmem &sm, const float f0[8], const float f1[8],
                                      int d0, int d1, float &rr0, float &rr1, float y[4]) {
  const int lane = threadIdx.x & 31, t = lane & 3;
  // rms of each row's 32 features (spread over the 4 lanes of a quad)
  float s0 = 0.f, s1 = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    s0 = fmaf(f0[k], f0[k], s0);
    s1 = fmaf(f1[k], f1[k], s1);
  }
  s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
  s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
  s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
  s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
  if (__all_sync(0xffffffffu, s0 == 0.f && s1 == 0.f)) return false;
  rr0 = sqrtf(s0 * (1.0f / kIn));
  rr1 = sqrtf(s1 * (1.0f / kIn));
  const float i0 = rr0 > 0.f ? 1.0f / rr0 : 0.f, i1 = rr1 > 0.f ? 1.0f / rr1 : 0.f;
  uint32_t a[2][4];
#pragma unroll
  for (int kk = 0; kk < 2; ++kk) {
    a[kk][0] = pack_bf16(f0[4 * kk] * i0, f0[4 * kk + 1] * i0);
    a[kk][1] = pack_bf16(f1[4 * kk] * i1, f1[4 * kk + 1] * i1);
    a[kk][2] = pack_bf16(f0[4 * kk + 2] * i0, f0[4 * kk + 3] * i0);
    a[kk][3] = pack_bf16(f1[4 * kk + 2] * i1, f1[4 * kk + 3] * i1);
  }
  float acc[4][4];
  // layer 1 (bias per depth)
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const int c = nt * 8 + 2 * t;
    acc[nt][0] = sm.b1[d0 * kHid + c];
    acc[nt][1] = sm.b1[d0 * kHid + c + 1];
    acc[nt][2] = sm.b1[d1 * kHid + c];
    acc[nt][3] = sm.b1[d1 * kHid + c + 1];
    const uint2 b0 = sm.w1[0][nt][lane], b1 = sm.w1[1][nt][lane];
    mma_bf16(acc[nt], a[0], b0.x, b0.y);
    mma_bf16(acc[nt], a[1], b1.x, b1.y);
  }
  gelu_to_a(acc, a);
  // layer 2
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const int c = nt * 8 + 2 * t;
    acc[nt][0] = acc[nt][2] = sm.b2[c];
    acc[nt][1] = acc[nt][3] = sm.b2[c + 1];
    const uint2 b0 = sm.w2[0][nt][lane], b1 = sm.w2[1][nt][lane];
    mma_bf16(acc[nt], a[0], b0.x, b0.y);
    mma_bf16(acc[nt], a[1], b1.x, b1.y);
  }
  gelu_to_a(acc, a);
  // layer 3: outputs in columns 0 and 1, held by the lanes with t == 0
  y[0] = y[2] = t == 0 ? sm.b3[0] : 0.f;
  y[1] = y[3] = t == 0 ? sm.b3[1] : 0.f;
  const uint2 b0 = sm.w3[0][lane], b1 = sm.w3[1][lane];
  mma_bf16(y, a[0], b0.x, b0.y);
  mma_bf16(y, a[1], b1.x, b1.y);
  return true;
}

// The network over the 32 rows of two tiles: lane (g, t) brings the features
// f[q] of rows g (q = 0), g + 8 (1) of the first tile and g (2), g + 8 (3) of
// the second, all with this lane's first bias b1 (pairs of units 8 nt + 2t).
// Every weight fragment is loaded once for both tiles.  Returns a bit per
// tile that is not silent (0: nothing was computed); the lanes with t == 0
// then hold the corrections rr[q] * y[q].  Each tile's arithmetic is net16's.
__device__ __forceinline__ int net32(const NetSmem &sm, const float f[4][8], const float2 b1[4],
                                     const float2 b2[4], float rr[4], float2 y[4]) {
  const int lane = threadIdx.x & 31, t = lane & 3;
  float inv[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s = fmaf(f[q][k], f[q][k], s);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    rr[q] = s;
  }
  const int live = (__all_sync(0xffffffffu, rr[0] == 0.f && rr[1] == 0.f) ? 0 : 1) |
                   (__all_sync(0xffffffffu, rr[2] == 0.f && rr[3] == 0.f) ? 0 : 2);
  if (!live) return 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    rr[q] = sqrtf(rr[q] * (1.0f / kIn));
    inv[q] = rr[q] > 0.f ? 1.0f / rr[q] : 0.f;
  }
  uint32_t a[2][2][4];  // [tile][k chunk]
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      const float *f0 = f[2 * m], *f1 = f[2 * m + 1];
      const float i0 = inv[2 * m], i1 = inv[2 * m + 1];
      a[m][kk][0] = pack_bf16(f0[4 * kk] * i0, f0[4 * kk + 1] * i0);
      a[m][kk][1] = pack_bf16(f1[4 * kk] * i1, f1[4 * kk + 1] * i1);
      a[m][kk][2] = pack_bf16(f0[4 * kk + 2] * i0, f0[4 * kk + 3] * i0);
      a[m][kk][3] = pack_bf16(f1[4 * kk + 2] * i1, f1[4 * kk + 3] * i1);
    }
  float acc[2][4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const uint2 w0 = sm.w1[0][nt][lane], w1 = sm.w1[1][nt][lane];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      acc[m][nt][0] = acc[m][nt][2] = b1[nt].x;
      acc[m][nt][1] = acc[m][nt][3] = b1[nt].y;
      mma_bf16(acc[m][nt], a[m][0], w0.x, w0.y);
      mma_bf16(acc[m][nt], a[m][1], w1.x, w1.y);
    }
  }
  gelu_to_a(acc[0], a[0]);
  gelu_to_a(acc[1], a[1]);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const uint2 w0 = sm.w2[0][nt][lane], w1 = sm.w2[1][nt][lane];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      acc[m][nt][0] = acc[m][nt][2] = b2[nt].x;
      acc[m][nt][1] = acc[m][nt][3] = b2[nt].y;
      mma_bf16(acc[m][nt], a[m][0], w0.x, w0.y);
      mma_bf16(acc[m][nt], a[m][1], w1.x, w1.y);
    }
  }
  gelu_to_a(acc[0], a[0]);
  gelu_to_a(acc[1], a[1]);
  const uint2 w0 = sm.w3[0][lane], w1 = sm.w3[1][lane];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    float o[4];
    o[0] = o[2] = t == 0 ? sm.b3[0] : 0.f;
    o[1] = o[3] = t == 0 ? sm.b3[1] : 0.f;
    mma_bf16(o, a[m][0], w0.x, w0.y);
    mma_bf16(o, a[m][1], w1.x, w1.y);
    y[2 * m] = make_float2(o[0], o[1]);
    y[2 * m + 1] = make_float2(o[2], o[3]);
  }
  return live;
}

// One correction per cell or sample row, written to out (zeros for silent
// rows): the training-side and recorded-rollout evaluation.
template <class Src>
__global__ void __launch_bounds__(128, 8) lb_tc_kernel(const float *__restrict__ wc, Src src,
                                                       long long n, float2 *out) {
  __shared__ NetSmem sm;
  stage_net(wc, sm);
  grid_dep_wait();  // the fields of the launch before
  grid_dep_launch();
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  for (long long base = warp * 16; base < n; base += nwarps * 16) {
    const long long r0 = base + g, r1 = base + g + 8;
    float f0[8], f1[8];
    int d0 = 0, d1 = 0;
    if (r0 < n) {
      d0 = src.load(r0, t, f0);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) f0[k] = 0.f;
    }
    if (r1 < n) {
      d1 = src.load(r1, t, f1);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) f1[k] = 0.f;
    }
    float rr0 = 0.f, rr1 = 0.f, y[4];
    const bool live = net16(sm, f0, f1, d0, d1, rr0, rr1, y);
    if (t == 0) {
      if (r0 < n) out[r0] = live ? make_float2(rr0 * y[0], rr0 * y[1]) : make_float2(0.f, 0.f);
      if (r1 < n) out[r1] = live ? make_float2(rr1 * y[2], rr1 * y[3]) : make_float2(0.f, 0.f);
    }
  }
}

// ---------------------------------------------------------------------------
// Fused in-step correction of the face lines.  A face line is the kLine
// corrected cells of one boundary normal (outermost first) whose tangential
// coordinates lie far enough inside the other two axes' interiors that no
// other line's cell is in its windows and no other cell's window reaches it
// (layer_plan below); its kLine windows span kLineCells distinct cells.  A
// warp takes 16 lines, four of them to the 16 rows of an MMA tile: it gathers
// the 16 x kLineCells cells of both time levels once into shared memory,
// evaluates the network over two tiles at a time and stores the corrected
// cells.  Every value a warp reads was read before it writes, and no other
// warp touches its lines, so the result is bit-identical to the two-pass form
// (lb_tc_kernel then the add) while reading each cell once instead of up to
// 8 times.
//
// What bounds it: the shared-memory pipe, then the special-function pipe (32
// tanh per tile).  Sixteen lines per warp, because neighbours in the table
// are neighbours in x on four of the six faces: one gather instruction brings
// two 128-byte runs (with four lines eight 32-byte ones).  [line][cell] in
// shared memory and weight fragments shared by two tiles issue 70 wavefronts
// per tile where [cell][line] and a tile at a time issued 130 (82 % of the
// pipe); that costs registers, so four CTAs per SM instead of eight.
constexpr int kLine = kCorrected;               // corrected cells per line
constexpr int kLineCells = kLine + kWin - 1;    // cells the line's windows span
constexpr int kLineWarp = 16;                   // lines per warp pass
constexpr int kLineCtas = 4;                    // CTAs per SM
static_assert(kLine == 4 && kLineWarp == 16, "four lines to a 16-row tile, four tiles");

// Asynchronous 8-byte copy global -> shared (zero fill when !valid; gsrc
// must still be a mapped address).
__device__ __forceinline__ void cp_async8(void *sdst, const void *gsrc, bool valid) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(sdst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(gsrc),
               "r"(valid ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait0() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// Each warp keeps one pass's copies in flight while the network runs on the
// previous one: at the top of pass p it waits for pass p's cells and queues
// pass p + 1's, whose addresses it worked out during pass p - 1 from entries
// loaded during pass p - 2.  Nothing waits on a global load issued in the
// same pass.
template <class Entries>
__global__ void __launch_bounds__(128, kLineCtas)
    lb_line_kernel(const float *__restrict__ wc, Entries src, long long nlines, int layer) {
  __shared__ NetSmem sm;
  // per warp and buffer: [field][line][cell] (field 0 = new, 1 = current)
  __shared__ __align__(16) float2 sl[4][2][2][kLineWarp][kLineCells];
  stage_net(wc, sm);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, w = threadIdx.x >> 5;
  const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long stride = ((static_cast<long long>(gridDim.x) * blockDim.x) >> 5) * kLineWarp;
  // rows g and g + 8 of a tile: position j of lines g / 4 and g / 4 + 2
  const int j = g % kLine;
  const int depth = layer - 1 - j;
  const int ml = lane % kLineWarp, half = lane / kLineWarp;  // line and parity of cells copied
  float2 b1[4], b2[4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const int c = nt * 8 + 2 * t;
    b1[nt] = make_float2(sm.b1[depth * kHid + c], sm.b1[depth * kHid + c + 1]);
    b2[nt] = make_float2(sm.b2[c], sm.b2[c + 1]);
  }
  auto entry = [&](long long base) {  // (code -1: no line)
    return base + ml < nlines ? src.table[base + ml] : make_int4(0, 0, 0, -1);
  };
  auto pointers = [&](const int4 e) {
    return e.w >= 0 ? src.at(e) : LinePtr{nullptr, nullptr, 0};
  };
  auto fetch = [&](const LinePtr p, int buf) {
    const bool v = p.nw != nullptr;
    const float2 *dummy = reinterpret_cast<const float2 *>(wc);
    const float2 *n = (v ? p.nw : dummy) + half * p.step, *c = (v ? p.cur : dummy) + half * p.step;
    const long long two = 2ll * p.step;
#pragma unroll
    for (int k = 0; k < kLineCells; k += 2) {
      if (k + half < kLineCells) {
        cp_async8(&sl[w][buf][0][ml][k + half], n, v);
        cp_async8(&sl[w][buf][1][ml][k + half], c, v);
      }
      n += two;
      c += two;
    }
  };
  long long base = warp * kLineWarp;
  grid_dep_wait();  // the weights are staged while the stencil finishes
  grid_dep_launch();
  if (base >= nlines) return;  // (no CTA barrier below)
  LinePtr now = pointers(entry(base)), next = pointers(entry(base + stride));
  int4 after = entry(base + 2 * stride);
  fetch(now, 0);
  cp_async_commit();
  for (int buf = 0; base < nlines; base += stride, buf ^= 1) {
    cp_async_wait0();  // this pass's cells have landed
    __syncwarp();      // every lane has read the other buffer
    if (base + stride < nlines) fetch(next, buf ^ 1);
    cp_async_commit();
    const LinePtr third = pointers(after);
    after = entry(base + 3 * stride);
    float2(*ls)[kLineWarp][kLineCells] = sl[w][buf];
    int live = 0;  // a bit per tile
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      const int l0 = 8 * h + g / kLine, c0 = j + 2 * t;
      float f[4][8], rr[4];
      float2 y[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 *n = &ls[0][l0 + 2 * q][c0], *c = &ls[1][l0 + 2 * q][c0];
        const float2 a0 = n[0], a1 = n[1], e0 = c[0], e1 = c[1];
        f[q][0] = a0.x, f[q][1] = a1.x, f[q][2] = a0.y, f[q][3] = a1.y;
        f[q][4] = e0.x, f[q][5] = e1.x, f[q][6] = e0.y, f[q][7] = e1.y;
      }
      const int lv = net32(sm, f, b1, b2, rr, y);
      live |= lv << (2 * h);
      __syncwarp();  // every lane has its features
      if (t == 0) {
        // new value = stencil output + correction, rounded as the two-pass
        // form
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (lv & (1 << (q / 2))) {
            float2 &v = ls[0][l0 + 2 * q][j];
            v = make_float2(__fadd_rn(v.x, __fmul_rn(rr[q], y[q].x)),
                            __fadd_rn(v.y, __fmul_rn(rr[q], y[q].y)));
          }
      }
    }
    __syncwarp();
    // the corrected cells of the tiles that were evaluated
    if (now.nw && (live >> (ml / kLine)) & 1)
#pragma unroll
      for (int k = 0; k < kLine; k += 2)
        now.nw[static_cast<long long>(k + half) * now.step] = ls[0][ml][k + half];
    now = next;
    next = third;
  }
}

template <class Entries>
__global__ void lb_add_edge_kernel(Entries src, long long n, const float2 *corr) {
  grid_dep_wait();
  grid_dep_launch();
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float2 *p = src.at(src.table[i]).nw;
    const float2 d = corr[i], v = *p;
    *p = make_float2(v.x + d.x, v.y + d.y);
  }
}

__global__ void lb_add_kernel(const int4 *__restrict__ cells, long long n, float2 *nw,
                              const float2 *__restrict__ corr, long long pitch, long long plane) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int4 c = cells[i];
    const long long g = static_cast<long long>(c.z) * plane + static_cast<long long>(c.y) * pitch + c.x;
    const float2 d = corr[i], v = nw[g];
    nw[g] = make_float2(v.x + d.x, v.y + d.y);
  }
}

// Training samples of the thin box: features from its step and targets
// from the wide field (offset into the wide box).
__global__ void lb_sample_kernel(const int4 *__restrict__ cells, long long n, const float2 *nw,
                                 const float2 *cur, long long pitch, long long plane,
                                 const float2 *wide, long long wpitch, long long wplane, int ox,
                                 int oy, int oz, float *xs, float *ts) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int4 c = cells[i];
    float x[kIn];
    const int depth = gather(c, nw, cur, pitch, plane, x);
    float *row = xs + i * kStride;
#pragma unroll
    for (int k = 0; k < kIn; ++k) row[k] = x[k];
    row[kIn] = static_cast<float>(depth);
    const long long g = static_cast<long long>(c.z) * plane + static_cast<long long>(c.y) * pitch + c.x;
    const long long w = static_cast<long long>(c.z + oz) * wplane +
                        static_cast<long long>(c.y + oy) * wpitch + (c.x + ox);
    const float2 tv = wide[w], sv = nw[g];
    ts[i * kOut] = tv.x - sv.x;
    ts[i * kOut + 1] = tv.y - sv.y;
  }
}

// Rollout targets: wide field at t+1 minus the thin stencil's output, which
// is features 0 (p) and 8 (q) of each recorded row.
__global__ void lb_target_kernel(const int4 *__restrict__ cells, long long n,
                                 const float *__restrict__ rows, const float2 *wide,
                                 long long wpitch, long long wplane, int ox, int oy, int oz,
                                 float *ts) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int4 c = cells[i];
    const long long w = static_cast<long long>(c.z + oz) * wplane +
                        static_cast<long long>(c.y + oy) * wpitch + (c.x + ox);
    const float2 tv = wide[w];
    ts[i * kOut] = tv.x - rows[i * kStride];
    ts[i * kOut + 1] = tv.y - rows[i * kStride + kWin];
  }
}

// Thin box <- wide box at (ox, oy, oz), zero outside [4, s-4)^3.
__global__ void crop_kernel(float2 *dst, long long sx, long long sy, long long sz,
                            long long pitch, const float2 *src, long long wpitch,
                            long long wplane, int ox, int oy, int oz) {
  const long long n = sx * sy * sz;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long x = i % sx, y = (i / sx) % sy, z = i / (sx * sy);
    float2 v = make_float2(0.f, 0.f);
    if (x >= 4 && x < sx - 4 && y >= 4 && y < sy - 4 && z >= 4 && z < sz - 4)
      v = src[(z + oz) * wplane + (y + oy) * wpitch + (x + ox)];
    dst[(z * sy + y) * pitch + x] = v;
  }
}

// The face-line pass: at most one wave of its CTAs (each stages the weights
// once and loops over its passes; four warps of kLineWarp lines).
int line_grid(long long nl) {
  const long long per = 4 * kLineWarp;
  return static_cast<int>(
      std::max<long long>(1, std::min<long long>((nl + per - 1) / per, 152 * kLineCtas)));
}

int grid_for(long long n, int per_block) {
  return static_cast<int>(std::max<long long>(1, std::min<long long>((n + per_block - 1) / per_block, 152 * 16)));
}

}  // namespace

// ---------------------------------------------------------------------------
std::vector<int4> layer_cells(long long sx, long long sy, long long sz, int layer) {
  std::vector<int4> out;
  const long long s[3] = {sx, sy, sz};
  auto depth_on = [&](int a, long long c, int *side) -> int {
    const long long lo = 4 + layer, hi = s[a] - 4 - layer;
    if (c < lo) {
      *side = 0;
      return static_cast<int>(lo - 1 - c);
    }
    if (c >= hi) {
      *side = 1;
      return static_cast<int>(c - hi);
    }
    return -1;
  };
  for (long long z = 4; z < sz - 4; ++z)
    for (long long y = 4; y < sy - 4; ++y) {
      int sdz = 0, sdy = 0;
      const int dz = depth_on(2, z, &sdz), dy = depth_on(1, y, &sdy);
      const bool band = dz < 0 && dy < 0;  // only the two x slabs are in the layer
      for (long long x = 4; x < sx - 4; ++x) {
        if (band && x == 4 + layer) x = sx - 4 - layer;  // skip the interior
        int sdx = 0;
        const int dx = depth_on(0, x, &sdx);
        int axis = -1, depth = -1, side = 0;
        if (dx > depth) { axis = 0; depth = dx; side = sdx; }
        if (dy > depth) { axis = 1; depth = dy; side = sdy; }
        if (dz > depth) { axis = 2; depth = dz; side = sdz; }
        // only the outer cells, whose stencils reach into the halo, are
        // corrected; the inner ones are updated by the stencil alone
        if (axis < 0 || depth < layer - kCorrected) continue;
        out.push_back(make_int4(static_cast<int>(x), static_cast<int>(y), static_cast<int>(z),
                                axis | side << 2 | depth << 3));
      }
    }
  return out;
}

cudaError_t launch_lb_step(cudaStream_t st, const float *wc, const int4 *cells, long long n,
                           float2 *nw, const float2 *cur, long long pitch, long long plane,
                           float2 *corr, float *rec) {
  lb_tc_kernel<CellSrc><<<grid_for(n, 64), 128, 0, st>>>(
      wc, CellSrc{cells, nw, cur, pitch, plane, rec}, n, corr);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  lb_add_kernel<<<grid_for(n, 256), 256, 0, st>>>(cells, n, nw, corr, pitch, plane);
  return cudaGetLastError();
}

// Splits the corrected cells into face lines (entries for the outermost
// cell, meta = axis | side << 2) and the remaining edge cells (layer_cells
// entries).  The windows of the least deep corrected cells reach m cells
// past the layer into the interior; a line is a face line when both of its
// tangential coordinates lie at least m + 1 cells inside the other axes'
// interiors.  Then (a) every cell a face line reads has those tangential
// coordinates, so it is the line's own or an interior cell, and (b) no edge
// cell's window reaches a face line's cell: a window along the line's axis
// keeps the edge cell's tangential coordinates, and one along another axis
// stays within m cells of that axis' layer.  So the face lines and the edge
// cells can be corrected independently.
LayerPlan layer_plan(long long sx, long long sy, long long sz, int layer) {
  LayerPlan plan;
  const std::vector<int4> cells = layer_cells(sx, sy, sz, layer);
  if (layer < kCorrected) {
    plan.edge = cells;
    return plan;
  }
  const int m = std::max(0, kWin - 1 - (layer - kCorrected));
  const long long s[3] = {sx, sy, sz};
  auto inside = [&](int a, long long c) {
    return c >= 4 + layer + m && c < s[a] - 4 - layer - m;
  };
  for (const int4 &c : cells) {
    const int axis = c.w & 3, depth = (c.w >> 3) & 31;
    const long long p[3] = {c.x, c.y, c.z};
    const int a1 = (axis + 1) % 3, a2 = (axis + 2) % 3;
    if (!(inside(a1, p[a1]) && inside(a2, p[a2])))
      plan.edge.push_back(c);
    else if (depth == layer - 1)
      plan.lines.push_back(make_int4(c.x, c.y, c.z, c.w & 7));
  }
  return plan;
}

LayerTables layer_tables(long long sx, long long sy, long long sz, long long pitch, int layer,
                         int shot) {
  const LayerPlan plan = layer_plan(sx, sy, sz, layer);
  const long long plane = pitch * sy;
  auto pack = [&](const int4 &c, int code) {
    const long long off = c.z * plane + c.y * pitch + c.x;
    const int axis = c.w & 3, side = (c.w >> 2) & 1;
    const long long stride = axis == 0 ? 1 : axis == 1 ? pitch : plane;
    return make_int4(static_cast<int>(off & 0xffffffffll), static_cast<int>(off >> 32),
                     static_cast<int>(side ? -stride : stride), code | shot << 8);
  };
  LayerTables out;
  out.lines.reserve(plan.lines.size());
  out.edge.reserve(plan.edge.size());
  for (const int4 &c : plan.lines) out.lines.push_back(pack(c, 0));
  for (const int4 &c : plan.edge) out.edge.push_back(pack(c, (c.w >> 3) & 31));
  return out;
}

namespace {

// The face lines in place, then the edge cells through `corr`.
template <class Entries>
cudaError_t launch_entries(cudaStream_t st, const float *wc, int layer, Entries lines,
                           long long nl, Entries edge, long long ne, float2 *corr) {
  if (nl > 0) {
    const cudaError_t e = launch_dependent(lb_line_kernel<Entries>, dim3(line_grid(nl)), 128, 0, st,
                                           wc, lines, nl, layer);
    if (e != cudaSuccess) return e;
  }
  if (ne <= 0) return cudaSuccess;
  const cudaError_t e = launch_dependent(lb_tc_kernel<EdgeSrc<Entries>>, dim3(grid_for(ne, 64)),
                                         128, 0, st, wc, EdgeSrc<Entries>{edge}, ne, corr);
  if (e != cudaSuccess) return e;
  return launch_dependent(lb_add_edge_kernel<Entries>, dim3(grid_for(ne, 256)), 256, 0, st, edge,
                          ne, corr);
}

}  // namespace

cudaError_t launch_lb_fused(cudaStream_t st, const float *wc, int layer, const int4 *lines,
                            long long nl, const int4 *edge, long long ne, float2 *nw,
                            const float2 *cur, float2 *corr) {
  return launch_entries(st, wc, layer, SimEntries{lines, nw, cur}, nl, SimEntries{edge, nw, cur},
                        ne, corr);
}

cudaError_t launch_lb_batch_fused(cudaStream_t st, const float *wc, int layer, const int4 *lines,
                                  long long nl, const int4 *edge, long long ne,
                                  const LbShot *shots, int cur_buf, float2 *corr) {
  return launch_entries(st, wc, layer, BatchEntries{lines, shots, cur_buf}, nl,
                        BatchEntries{edge, shots, cur_buf}, ne, corr);
}

cudaError_t launch_lb_sample(cudaStream_t st, const int4 *cells, long long n, const float2 *nw,
                             const float2 *cur, long long pitch, long long plane,
                             const float2 *wide, long long wpitch, long long wplane,
                             const int off[3], float *xs, float *ts) {
  lb_sample_kernel<<<grid_for(n, 256), 256, 0, st>>>(cells, n, nw, cur, pitch, plane, wide,
                                                     wpitch, wplane, off[0], off[1], off[2], xs,
                                                     ts);
  return cudaGetLastError();
}

cudaError_t launch_lb_target(cudaStream_t st, const int4 *cells, long long n, const float *rows,
                             const float2 *wide, long long wpitch, long long wplane,
                             const int off[3], float *ts) {
  lb_target_kernel<<<grid_for(n, 256), 256, 0, st>>>(cells, n, rows, wide, wpitch, wplane,
                                                     off[0], off[1], off[2], ts);
  return cudaGetLastError();
}

cudaError_t launch_crop(cudaStream_t st, float2 *dst, long long sx, long long sy, long long sz,
                        long long pitch, const float2 *src, long long wpitch, long long wplane,
                        const int off[3]) {
  crop_kernel<<<grid_for(sx * sy * sz, 256), 256, 0, st>>>(dst, sx, sy, sz, pitch, src, wpitch,
                                                           wplane, off[0], off[1], off[2]);
  return cudaGetLastError();
}

}  // namespace dcg

// ===========================================================================
// C ABI
// ===========================================================================
struct dc_gb300_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  float *master = nullptr, *wc = nullptr, *m1 = nullptr, *m2 = nullptr, *grad = nullptr;
  double *acc = nullptr;  // (sum e^2, sum r^2) per step parity
  int adam_step = 0;
};

namespace {

int fail(int code, const std::string &msg) {
  dcg::set_error(msg);
  return code;
}

#define LB_TRY(call)                                                                 \
  do {                                                                               \
    const cudaError_t e_ = (call);                                                   \
    if (e_ != cudaSuccess)                                                           \
      return fail(DC_GB300_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

void release(dc_gb300_mlp *m) {
  cudaFree(m->master);
  cudaFree(m->wc);
  cudaFree(m->m1);
  cudaFree(m->m2);
  cudaFree(m->grad);
  cudaFree(m->acc);
  if (m->stream) cudaStreamDestroy(m->stream);
}

}  // namespace

extern "C" int dc_gb300_mlp_create(int device, dc_gb300_mlp **out) {
  if (!out) return fail(DC_GB300_ERR_ARG, "null argument");
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return fail(DC_GB300_ERR_DEVICE, "no CUDA device");
  int dev = device;
  if (dev < 0) LB_TRY(cudaGetDevice(&dev));
  if (dev >= ndev) return fail(DC_GB300_ERR_DEVICE, "device ordinal out of range");
  LB_TRY(cudaSetDevice(dev));
  auto *m = new dc_gb300_mlp();
  m->device = dev;
  const size_t pb = sizeof(float) * dcg::kParams;
  if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMalloc(&m->master, pb) != cudaSuccess || cudaMalloc(&m->wc, pb) != cudaSuccess ||
      cudaMalloc(&m->m1, pb) != cudaSuccess || cudaMalloc(&m->m2, pb) != cudaSuccess ||
      cudaMalloc(&m->grad, pb) != cudaSuccess ||
      cudaMalloc(&m->acc, 4 * sizeof(double)) != cudaSuccess) {
    release(m);
    delete m;
    return fail(DC_GB300_ERR_NOMEM, "MLP buffers");
  }
  cudaMemsetAsync(m->master, 0, pb, m->stream);
  cudaMemsetAsync(m->wc, 0, pb, m->stream);
  cudaMemsetAsync(m->m1, 0, pb, m->stream);
  cudaMemsetAsync(m->m2, 0, pb, m->stream);
  cudaMemsetAsync(m->grad, 0, pb, m->stream);
  cudaMemsetAsync(m->acc, 0, 2 * sizeof(double), m->stream);
  if (cudaStreamSynchronize(m->stream) != cudaSuccess) {
    release(m);
    delete m;
    return fail(DC_GB300_ERR_CUDA, "MLP set-up");
  }
  *out = m;
  return DC_GB300_OK;
}

extern "C" int dc_gb300_mlp_destroy(dc_gb300_mlp *m) {
  if (!m) return DC_GB300_OK;
  cudaSetDevice(m->device);
  release(m);
  delete m;
  return DC_GB300_OK;
}

extern "C" int dc_gb300_mlp_set_params(dc_gb300_mlp *m, const float *params) {
  if (!m || !params) return fail(DC_GB300_ERR_ARG, "null argument");
  LB_TRY(cudaSetDevice(m->device));
  const size_t pb = sizeof(float) * dcg::kParams;
  LB_TRY(cudaMemcpyAsync(m->master, params, pb, cudaMemcpyHostToDevice, m->stream));
  dcg::mlp_round_kernel<<<(dcg::kParams + 255) / 256, 256, 0, m->stream>>>(m->master, m->wc);
  LB_TRY(cudaGetLastError());
  LB_TRY(cudaMemsetAsync(m->m1, 0, pb, m->stream));
  LB_TRY(cudaMemsetAsync(m->m2, 0, pb, m->stream));
  LB_TRY(cudaMemsetAsync(m->grad, 0, pb, m->stream));
  LB_TRY(cudaStreamSynchronize(m->stream));
  m->adam_step = 0;
  return DC_GB300_OK;
}

extern "C" int dc_gb300_mlp_init(dc_gb300_mlp *m, unsigned int seed) {
  if (!m) return fail(DC_GB300_ERR_ARG, "null argument");
  std::vector<float> p(dcg::kParams, 0.0f);
  std::mt19937 rng(seed);
  auto fill = [&](int off, int rows, int cols, float gain) {
    const float sd = gain / std::sqrt(static_cast<float>(cols));
    std::normal_distribution<float> nd(0.0f, sd);
    for (int i = 0; i < rows * cols; ++i) p[off + i] = nd(rng);
  };
  fill(dcg::OFF_W1, dcg::kHid, dcg::kIn, 1.0f);
  fill(dcg::OFF_W2, dcg::kHid, dcg::kHid, 1.0f);
  fill(dcg::OFF_W3, dcg::kOut, dcg::kHid, 0.01f);  // corrections start near zero
  return dc_gb300_mlp_set_params(m, p.data());
}

extern "C" int dc_gb300_mlp_get_params(dc_gb300_mlp *m, float *params) {
  if (!m || !params) return fail(DC_GB300_ERR_ARG, "null argument");
  LB_TRY(cudaSetDevice(m->device));
  LB_TRY(cudaMemcpyAsync(params, m->master, sizeof(float) * dcg::kParams, cudaMemcpyDeviceToHost,
                         m->stream));
  LB_TRY(cudaStreamSynchronize(m->stream));
  return DC_GB300_OK;
}

extern "C" int dc_gb300_mlp_forward(dc_gb300_mlp *m, const float *samples, long long n,
                                    float *out) {
  if (!m || (n > 0 && (!samples || !out))) return fail(DC_GB300_ERR_ARG, "null argument");
  if (n <= 0) return DC_GB300_OK;
  LB_TRY(cudaSetDevice(m->device));
  dcg::lb_tc_kernel<dcg::RowSrc><<<dcg::grid_for(n, 64), 128, 0, m->stream>>>(
      m->wc, dcg::RowSrc{samples}, n, reinterpret_cast<float2 *>(out));
  LB_TRY(cudaGetLastError());
  LB_TRY(cudaStreamSynchronize(m->stream));
  return DC_GB300_OK;
}

extern "C" int dc_gb300_mlp_gradient(dc_gb300_mlp *m, const float *samples, const float *targets,
                                     long long n, float *grad, double *loss) {
  if (!m || !samples || !targets || !grad || n <= 0)
    return fail(DC_GB300_ERR_ARG, "invalid argument");
  LB_TRY(cudaSetDevice(m->device));
  LB_TRY(cudaFuncSetAttribute(dcg::mlp_grad_kernel,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(sizeof(dcg::GradSmem))));
  LB_TRY(cudaMemsetAsync(m->grad, 0, sizeof(float) * dcg::kParams, m->stream));
  LB_TRY(cudaMemsetAsync(m->acc, 0, 2 * sizeof(double), m->stream));
  dcg::mlp_grad_kernel<<<dcg::grid_for(n, dcg::kTB), dcg::kTT, sizeof(dcg::GradSmem), m->stream>>>(
      m->wc, samples, targets, n, n, 0ull, 0, m->grad, m->acc);
  LB_TRY(cudaGetLastError());
  double acc[2];
  LB_TRY(cudaMemcpyAsync(grad, m->grad, sizeof(float) * dcg::kParams, cudaMemcpyDeviceToHost,
                         m->stream));
  LB_TRY(cudaMemcpyAsync(acc, m->acc, sizeof(acc), cudaMemcpyDeviceToHost, m->stream));
  LB_TRY(cudaMemsetAsync(m->grad, 0, sizeof(float) * dcg::kParams, m->stream));
  LB_TRY(cudaStreamSynchronize(m->stream));
  if (loss) {
    loss[0] = acc[0];
    loss[1] = acc[1];
  }
  return DC_GB300_OK;
}

extern "C" int dc_gb300_mlp_train(dc_gb300_mlp *m, const float *samples, const float *targets,
                                  long long n, int steps, int batch, float lr,
                                  unsigned long long seed, float *loss_hist) {
  if (!m || !samples || !targets || n <= 0 || steps < 0 || batch < 1 || !(lr > 0))
    return fail(DC_GB300_ERR_ARG, "invalid argument");
  LB_TRY(cudaSetDevice(m->device));
  LB_TRY(cudaFuncSetAttribute(dcg::mlp_grad_kernel,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(sizeof(dcg::GradSmem))));
  float *d_hist = nullptr;
  if (loss_hist && steps > 0) LB_TRY(cudaMalloc(&d_hist, sizeof(float) * steps));
  LB_TRY(cudaMemsetAsync(m->grad, 0, sizeof(float) * dcg::kParams, m->stream));
  LB_TRY(cudaMemsetAsync(m->acc, 0, 4 * sizeof(double), m->stream));
  cudaError_t e = cudaSuccess;
  const int blocks = dcg::grid_for(batch, dcg::kTB);
  for (int s = 0; s < steps && e == cudaSuccess; ++s) {
    double *acc = m->acc + 2 * (s & 1), *next = m->acc + 2 * (1 - (s & 1));
    e = dcg::launch_dependent(dcg::mlp_grad_kernel, dim3(blocks), dcg::kTT, sizeof(dcg::GradSmem),
                              m->stream, m->wc, samples, targets, n, batch,
                              seed + 0x9E3779B97F4A7C15ull * (m->adam_step + 1), 1, m->grad, acc);
    if (e != cudaSuccess) break;
    ++m->adam_step;
    e = dcg::launch_dependent(dcg::mlp_adam_kernel,
                              dim3((dcg::kParams + dcg::kAdamT - 1) / dcg::kAdamT), dcg::kAdamT, 0,
                              m->stream, m->master, m->wc, m->m1, m->m2, m->grad, acc, next, lr,
                              0.9f, 0.999f, 1e-8f, m->adam_step, d_hist, s);
  }
  if (e == cudaSuccess && d_hist)
    e = cudaMemcpyAsync(loss_hist, d_hist, sizeof(float) * steps, cudaMemcpyDeviceToHost,
                        m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  cudaFree(d_hist);
  if (e != cudaSuccess) return fail(DC_GB300_ERR_CUDA, std::string("MLP training: ") + cudaGetErrorString(e));
  return DC_GB300_OK;
}

extern "C" long long dc_gb300_layer_cells(long sx, long sy, long sz, int layer, int *cells,
                                         long long cap) {
  if (layer < 1 || layer > DC_GB300_MLP_DEPTHS || sx < 2 * layer + 16 || sy < 2 * layer + 16 ||
      sz < 2 * layer + 16) {
    fail(DC_GB300_ERR_ARG, "invalid layer geometry");
    return -1;
  }
  const std::vector<int4> v = dcg::layer_cells(sx, sy, sz, layer);
  const long long n = static_cast<long long>(v.size());
  if (cells)
    for (long long i = 0; i < std::min(n, cap); ++i) {
      cells[4 * i] = v[i].x;
      cells[4 * i + 1] = v[i].y;
      cells[4 * i + 2] = v[i].z;
      cells[4 * i + 3] = v[i].w;
    }
  return n;
}

extern "C" int dc_gb300_layer_plan(long sx, long sy, long sz, int layer, int *lines,
                                   long long lines_cap, int *edge, long long edge_cap,
                                   long long *n_lines, long long *n_edge) {
  if (!n_lines || !n_edge) return fail(DC_GB300_ERR_ARG, "null count");
  if (layer < 1 || layer > DC_GB300_MLP_DEPTHS || sx < 2 * layer + 16 || sy < 2 * layer + 16 ||
      sz < 2 * layer + 16)
    return fail(DC_GB300_ERR_ARG, "invalid layer geometry");
  const dcg::LayerPlan p = dcg::layer_plan(sx, sy, sz, layer);
  auto put = [](const std::vector<int4> &v, int *out, long long cap) {
    if (!out) return;
    for (long long i = 0; i < std::min(static_cast<long long>(v.size()), cap); ++i) {
      out[4 * i] = v[i].x;
      out[4 * i + 1] = v[i].y;
      out[4 * i + 2] = v[i].z;
      out[4 * i + 3] = v[i].w;
    }
  };
  put(p.lines, lines, lines_cap);
  put(p.edge, edge, edge_cap);
  *n_lines = static_cast<long long>(p.lines.size());
  *n_edge = static_cast<long long>(p.edge.size());
  return DC_GB300_OK;
}

extern "C" const float *dc_gb300_mlp_device_params(const dc_gb300_mlp *m) {
  return m ? m->wc : nullptr;
}
