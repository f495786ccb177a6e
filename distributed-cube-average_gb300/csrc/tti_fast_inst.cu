// tti_fast_inst.cu -- the fast sm_103a Fletcher TTI time step: the kernels of
// one coefficient form (DC_FORM) and tile shape (DC_TX x DC_TY).  The build
// compiles this file once per combination, in parallel; tti_fast.cu picks one.
//
// One pass updates p and q (the coupled pseudo-acoustic TTI system of the
// reference, include/sample_compute.h:105-185) for every point of a box.
//
// Work decomposition: a CTA owns a 32 x TY column tile in (x, y) and sweeps
// a chunk of output planes along z.  It receives by TMA, a group of three
// planes per copy into one of two shared-memory stages:
//   * the (p, q) pairs of the leading planes k with a 4-cell halo in x and y
//     and the in-plane coefficient group (cxx, cyy, cxy, czz) of plane k,
//   * the other coefficients and the (pp, qp) tile of the output planes
//     z = k - 4.
// Each lane owns two x-adjacent columns and keeps, in registers, the (p, q)
// pairs of the last eight planes: the centre value, the x-derivative and the
// y-derivative.
// The cross derivatives are evaluated in their separable form: with the
// 8th-order first-derivative weights L1..L4 the reference's 64-point
// derCross (include/derivatives.h:56-91) has weights L_ab = L_a * L_b, so it
// equals D_a(D_b p):
//   d2/dxdy = D_x of a shared-memory plane of the y-derivative,
//   d2/dxdz = D_z of the x-derivative queue,
//   d2/dydz = D_z of the y-derivative queue.
// The in-plane part of H1 (cxx d2/dx2 + cyy d2/dy2 + cxy d2/dxdy), the
// in-plane Laplacian and czz of plane k wait four planes in registers until
// plane k is the output plane.
//
// What bounds it, and why this shape.  Next to HBM the shared-memory pipe and
// the instruction issue of the few resident warps count: with one column per
// lane (16 warps per SM, 114 registers, one barrier per plane) a 304^3 FP16
// step took 347 us at 70 % of the shared-memory wavefronts and 268
// instructions per 32 points, 107 of them addresses, branches and barriers.
//   * Two adjacent columns share their row's values: five 16-byte loads bring
//     ten pairs instead of eighteen 8-byte ones, and four the y-derivatives
//     around both: 89 -> 59 wavefronts per 32 points.  The queues of two
//     columns (up to 255 registers) leave 8 warps per SM.
//   * A warp owns two whole tile rows, so the y-derivative plane is exchanged
//     inside a warp and the CTA meets at a barrier once per group.  One copy
//     per array and group: a third of the TMA instructions, one wait.
//   * The unrolled body is one group (three planes) and the queues move by
//     three planes at its end.  Unrolled over the nine planes of a register
//     ring nothing moves, but the 50 KB body misses the instruction cache:
//     0.84 of 4.4 stall cycles per instruction, 286 against 264 us (six
//     planes: 282 us).
// 304^3 FP16 step 347 -> 264 us (ncu), 616^3 FP32 step 2.59 -> 2.19 ms (96 %
// of the measured copy bandwidth), 872 x 872 x 616 FP16 5.19 -> 3.79 ms;
// loading the next plane's values ahead of the output arithmetic ran out of
// registers (282 us).
//
// The sweep of one column tile is `sweep_column`; `fast_kernel` runs one
// tile per CTA over one box, `batch_kernel` runs CTAs over the tiles of many
// boxes (shots) cropped out of one shared medium.
// Rounding differs from the reference's direct sums (the exact kernel is
// bit-identical).
//
// p and q are processed as pairs with packed f32x2 arithmetic (FFMA2,
// FADD2, FMUL2): one instruction updates both fields.
//
// Medium forms (CoefForm): CF_F32 reads the grouped FP32 coefficients
// (40 B/point); CF_VV reads (vpz, vsv) with the reference CUDA backend's
// constant angles (8 B/point); CF_F16 / CF_BF16 read a 20 B/point copy in
// FP16 / BF16 (the mixed-precision form), converted to FP32 on load -- all
// arithmetic stays FP32.
//
// Compulsory DRAM traffic per point-update: read (pc,qc) 8 B, (pp,qp) 8 B and
// the medium, write (pp,qp) 8 B: 64 B (CF_F32), 32 B (CF_VV), 44 B (CF_F16,
// CF_BF16).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "dc_internal.h"
#include "dc_ptx.cuh"

namespace dcg {
namespace {

constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s per TMA wait

template <int V>
using Const = std::integral_constant<int, V>;


template <int CF>
struct CoefBytes {
  // bytes per point of each coefficient group: L (cxx, cyy, cxy, czz) is
  // read at the leading plane, O1 and O2 (the rest) at the output plane
  static constexpr int L = CF == CF_F32 ? 16 : CF == CF_VV ? 0 : 8;
  static constexpr int O1 = CF == CF_F32 ? 16 : 8;  // VV: (vpz, vsv)
  static constexpr int O2 = CF == CF_F32 ? 8 : CF == CF_VV ? 0 : 4;
};

template <int TX, int TY, int CF>
struct FastLayout {
  using CB = CoefBytes<CF>;
  static constexpr int HX = TX + 2 * kHalo;
  static constexpr int HY = TY + 2 * kHalo;
  static constexpr int NP = TX * TY;   // points of a tile plane
  static constexpr int NT = NP / 2;    // threads: two x-adjacent points each
  // Two stages, each a group of kGroup planes of every array: one is read
  // while the other is refilled.
  static constexpr int H_PLANE = HX * HY * 8;       // (p, q) pairs
  static constexpr int L_PLANE = NP * CB::L, O1_PLANE = NP * CB::O1, O2_PLANE = NP * CB::O2;
  static constexpr int OWN_PLANE = NP * 8;          // (pp, qp) pairs
  // FP16 form: the velocity bases of the tile's TY rows at the output plane
  static constexpr int VB_PLANE = CF == CF_F16 ? TY * 16 : 0;
  static constexpr int OFF_H = 0;
  static constexpr int OFF_L = kGroup * H_PLANE;
  static constexpr int OFF_O1 = OFF_L + kGroup * L_PLANE;
  static constexpr int OFF_O2 = OFF_O1 + kGroup * O1_PLANE;
  static constexpr int OFF_OWN = OFF_O2 + kGroup * O2_PLANE;
  static constexpr int OFF_VB = OFF_OWN + kGroup * OWN_PLANE;
  static constexpr int STAGE_BYTES = OFF_VB + kGroup * VB_PLANE;
  static constexpr int DY_BYTES = TY * HX * 8;      // y-derivative plane
  static constexpr int OFF_DY = 2 * STAGE_BYTES;    // 3 buffers
  static constexpr int OFF_BAR = OFF_DY + 3 * DY_BYTES;
  static constexpr int SMEM_BYTES = OFF_BAR + 2 * 8;
  static constexpr uint32_t TX_HALO = kGroup * H_PLANE;
  static constexpr uint32_t TX_LEAD = kGroup * L_PLANE;
  static constexpr uint32_t TX_OUT = kGroup * (O1_PLANE + O2_PLANE + OWN_PLANE + VB_PLANE);
  static_assert(H_PLANE % 128 == 0 && L_PLANE % 128 == 0 && O1_PLANE % 128 == 0 &&
                    O2_PLANE % 128 == 0 && VB_PLANE % 128 == 0 && DY_BYTES % 128 == 0,
                "every TMA destination is 128-byte aligned");
  static constexpr int ROWS = 64 / TX;  // tile rows of a warp (two points per lane)
  static_assert((TX == 32 || TX == 16) && TY % ROWS == 0, "a warp owns whole tile rows");
};

// Packed FP32 pair arithmetic (one instruction updates p and q).
__device__ __forceinline__ float2 bc(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  return __ffma2_rn(a, b, c);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

// Second derivative of a (p, q) pair with pre-scaled weights w[0..4]
// (K_i / da^2), summed as two independent chains.
__device__ __forceinline__ float2 d2(const float *w, float2 c, float2 m1, float2 p1,
                                     float2 m2, float2 p2, float2 m3, float2 p3,
                                     float2 m4, float2 p4) {
  const float2 s1 = add2(m1, p1), s2 = add2(m2, p2), s3 = add2(m3, p3), s4 = add2(m4, p4);
  float2 t0 = fma2(bc(w[1]), s1, mul2(bc(w[0]), c));
  const float2 t1 = fma2(bc(w[3]), s3, mul2(bc(w[2]), s2));
  t0 = fma2(bc(w[4]), s4, t0);
  return add2(t0, t1);
}

// First derivative of a (p, q) pair with weights w[0..3] (L_i / da).
__device__ __forceinline__ float2 d1(const float *w, float2 m1, float2 p1, float2 m2,
                                     float2 p2, float2 m3, float2 p3, float2 m4, float2 p4) {
  const float2 n = bc(-1.0f);
  const float2 e1 = fma2(n, m1, p1), e2 = fma2(n, m2, p2), e3 = fma2(n, m3, p3),
               e4 = fma2(n, m4, p4);
  const float2 t0 = fma2(bc(w[2]), e3, mul2(bc(w[0]), e1));
  const float2 t1 = fma2(bc(w[3]), e4, mul2(bc(w[1]), e2));
  return add2(t0, t1);
}

// With equal spacing on all axes the stencil uses the unscaled 8th-order
// weights (K_i for the second derivative, L_i for the first) as
// compile-time constants and applies 1/d^2 once, in dt2_iso: every term of
// the update is a second derivative, so the scale factors out of the sum.
constexpr float kK0 = -205.0f / 72.0f, kK1 = 8.0f / 5.0f, kK2 = -1.0f / 5.0f,
                kK3 = 8.0f / 315.0f, kK4 = -1.0f / 560.0f;
constexpr float kL1 = 4.0f / 5.0f, kL2 = -1.0f / 5.0f, kL3 = 4.0f / 105.0f,
                kL4 = -1.0f / 280.0f;

// Two forms of each derivative with the constant weights: two FMA chains
// summed at the end (shorter dependency chains), or one chain (one
// instruction fewer).  The FP16/BF16 sweeps use the second (with one column
// per lane it was 2 % faster: 64-shot FP16 batch 32.57 vs 33.19 ms); the
// FP32-medium sweep, nearer its memory bound, gained nothing and keeps the
// first.
template <bool CHAIN>
__device__ __forceinline__ float2 d2k(float2 c, float2 m1, float2 p1, float2 m2, float2 p2,
                                      float2 m3, float2 p3, float2 m4, float2 p4) {
  const float2 s1 = add2(m1, p1), s2 = add2(m2, p2), s3 = add2(m3, p3), s4 = add2(m4, p4);
  if (CHAIN) {
    float2 t = fma2(bc(kK1), s1, mul2(bc(kK0), c));
    t = fma2(bc(kK2), s2, t);
    t = fma2(bc(kK3), s3, t);
    return fma2(bc(kK4), s4, t);
  }
  float2 t0 = fma2(bc(kK1), s1, mul2(bc(kK0), c));
  const float2 t1 = fma2(bc(kK3), s3, mul2(bc(kK2), s2));
  t0 = fma2(bc(kK4), s4, t0);
  return add2(t0, t1);
}

template <bool CHAIN>
__device__ __forceinline__ float2 d1k(float2 m1, float2 p1, float2 m2, float2 p2, float2 m3,
                                      float2 p3, float2 m4, float2 p4) {
  const float2 n = bc(-1.0f);
  const float2 e1 = fma2(n, m1, p1), e2 = fma2(n, m2, p2), e3 = fma2(n, m3, p3),
               e4 = fma2(n, m4, p4);
  if (CHAIN) {
    float2 t = fma2(bc(kL2), e2, mul2(bc(kL1), e1));
    t = fma2(bc(kL3), e3, t);
    return fma2(bc(kL4), e4, t);
  }
  const float2 t0 = fma2(bc(kL3), e3, mul2(bc(kL1), e1));
  const float2 t1 = fma2(bc(kL4), e4, mul2(bc(kL2), e2));
  return add2(t0, t1);
}

// Second / first derivative with the runtime weights w, or with the
// unscaled constants when ISO.
template <bool ISO, bool CHAIN>
__device__ __forceinline__ float2 d2s(const float *w, float2 c, float2 m1, float2 p1, float2 m2,
                                      float2 p2, float2 m3, float2 p3, float2 m4, float2 p4) {
  return ISO ? d2k<CHAIN>(c, m1, p1, m2, p2, m3, p3, m4, p4)
             : d2(w, c, m1, p1, m2, p2, m3, p3, m4, p4);
}
template <bool ISO, bool CHAIN>
__device__ __forceinline__ float2 d1s(const float *w, float2 m1, float2 p1, float2 m2, float2 p2,
                                      float2 m3, float2 p3, float2 m4, float2 p4) {
  return ISO ? d1k<CHAIN>(m1, p1, m2, p2, m3, p3, m4, p4)
             : d1(w, m1, p1, m2, p2, m3, p3, m4, p4);
}

// Constant-angle factors of the reference CUDA backend
// (include/sample_compute.h:9-18).
constexpr float kCxx = 0.1459632909f, kCyy = 0.3540367091f, kCzz = 0.5f;
constexpr float kCxy = 0.4546487134f, kCyz = 0.8414709848f;
constexpr float kCxz = 0.5403023059f;
constexpr float kV2pxFactor = 1.48f, kV2pnFactor = 1.2f;

__device__ __forceinline__ float2 h2f(uint32_t v, bool bf16) {
  if (bf16) {  // bfloat16 -> float: the 16 bits are the float's high half
    return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
  }
  __half2 h;
  *reinterpret_cast<uint32_t *>(&h) = v;
  return __half22float2(h);
}

// Two 16-bit fixed-point values (low half first, each stored biased by
// 2^15) as exact floats: a byte permutation places each half in the low
// mantissa bits of 2^23, and one packed subtraction of 2^23 + 2^15 removes
// both offsets.  The values come out scaled by 2^15; the sweep unscales H1
// once (unscaling here instead costs the same and rounds differently where
// the products are subnormal, at the far fringe of a wave).
__device__ __forceinline__ float2 fx2f(uint32_t w) {
  const uint32_t lo = __byte_perm(w, 0x4b000000u, 0x7610);
  const uint32_t hi = __byte_perm(w, 0x4b000000u, 0x7632);
  return __fadd2_rn(make_float2(__uint_as_float(lo), __uint_as_float(hi)),
                    make_float2(-8421376.0f, -8421376.0f));
}

// Scale of the angle terms as the kernel reads them (1 / 2^15 for the
// fixed-point FP16 form, applied to H1).
template <int CF>
constexpr float kChUnscale = CF == CF_F16 ? 1.0f / 32768.0f : 1.0f;

// Shared-memory loads and stores at a 32-bit address plus a compile-time
// offset, so every access of the unrolled sweep is one instruction on a
// base register (through pointers the compiler recomputed addresses: a
// tenth of the instructions).
template <int OFF>
__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4 + %5];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ float2 lds2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2 + %3];" : "=f"(v.x), "=f"(v.y) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ uint4 lds4u(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4 + %5];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(a), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ uint2 lds2u(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2 + %3];" : "=r"(v.x), "=r"(v.y) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ void sts4(uint32_t a, float2 u, float2 v) {
  asm volatile("st.shared.v4.f32 [%0 + %1], {%2, %3, %4, %5};" ::"r"(a), "n"(OFF), "f"(u.x),
               "f"(u.y), "f"(v.x), "f"(v.y)
               : "memory");
}
template <int OFF>
__device__ __forceinline__ void sts2(uint32_t a, float2 u) {
  asm volatile("st.shared.v2.f32 [%0 + %1], {%2, %3};" ::"r"(a), "n"(OFF), "f"(u.x), "f"(u.y)
               : "memory");
}

// Two x-adjacent (p, q) pairs of a shared-memory row, one 16-byte load.
template <int OFF>
__device__ __forceinline__ void ld_pairs(uint32_t p, float2 &a, float2 &b) {
  const float4 v = lds4<OFF>(p);
  a = make_float2(v.x, v.y);
  b = make_float2(v.z, v.w);
}

// A thread's shared-memory addresses inside a stage: `t8` its points in an
// 8-byte group, `t4` in a 4-byte group, `t16` in a 16-byte group, `row` its
// row of velocity bases.
struct StageAddr {
  uint32_t halo, col, t8, t4, t16, row;
  __device__ __forceinline__ void shift(uint32_t by) {
    halo += by;
    col += by;
    t8 += by;
    t4 += by;
    t16 += by;
    row += by;
  }
};

// The 16-byte groups of a thread's two points.  Lanes 4-7 of every eight
// read the second point first (`t16` points at it): at the 32-byte stride of
// the lanes both loads are then free of bank conflicts (two-way otherwise).
template <int OFF>
__device__ __forceinline__ void ld_groups16(uint32_t t16, float4 out[2]) {
  const bool swap = threadIdx.x & 4;
  const float4 a = lds4<OFF>(t16), b = lds4<OFF>(t16 ^ 16u);
  out[0] = make_float4(swap ? b.x : a.x, swap ? b.y : a.y, swap ? b.z : a.z, swap ? b.w : a.w);
  out[1] = make_float4(swap ? a.x : b.x, swap ? a.y : b.y, swap ? a.z : b.z, swap ? a.w : b.w);
}

// (cxx, cyy, cxy, czz) of the thread's two points at the leading plane
// (group at offset OFF of the stage).
template <int CF, int OFF>
__device__ __forceinline__ void load_lead(const StageAddr &sa, float4 out[2]) {
  if (CF == CF_F32) {
    ld_groups16<OFF>(sa.t16, out);
  } else if (CF == CF_VV) {
    out[0] = out[1] = make_float4(kCxx, kCyy, kCxy, kCzz);
  } else {
    const uint4 v = lds4u<OFF>(sa.t8);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 a = CF == CF_F16 ? fx2f(w[2 * c]) : h2f(w[2 * c], true);
      const float2 b = CF == CF_F16 ? fx2f(w[2 * c + 1]) : h2f(w[2 * c + 1], true);
      out[c] = make_float4(a.x, a.y, b.x, b.y);
    }
  }
}

// (cxz, cyz, v2px, v2pz, v2sz, v2pn) of a point at the output plane.
struct OutMedium {
  float cxz, cyz, v2px, v2pz, v2sz, v2pn;
};

// Of the thread's two points; O1, O2, VB: the groups' offsets in the stage.
template <int CF, int O1, int O2, int VB>
__device__ __forceinline__ void load_out(const StageAddr &sa, OutMedium out[2]) {
  if (CF == CF_F32) {
    float4 g1[2];
    ld_groups16<O1>(sa.t16, g1);
    const float4 g2 = lds4<O2>(sa.t8);
    out[0] = OutMedium{g1[0].x, g1[0].y, g1[0].z, g1[0].w, g2.x, g2.y};
    out[1] = OutMedium{g1[1].x, g1[1].y, g1[1].z, g1[1].w, g2.z, g2.w};
  } else if (CF == CF_VV) {
    // include/sample_compute.h:51-54
    const float4 v = lds4<O1>(sa.t8);
    const float vp[2] = {v.x, v.z}, vs[2] = {v.y, v.w};
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float v2pz = vp[c] * vp[c];
      out[c] = OutMedium{kCxz, kCyz, v2pz * kV2pxFactor, v2pz, vs[c] * vs[c],
                         v2pz * kV2pnFactor};
    }
  } else {
    // FP16 form: the velocity bases of this lane's row (a broadcast read)
    const float4 vb = CF == CF_F16 ? lds4<VB>(sa.row) : make_float4(0.f, 0.f, 0.f, 0.f);
    const uint4 g1 = lds4u<O1>(sa.t8);
    const uint2 g2 = lds2u<O2>(sa.t4);
    const uint32_t w1[4] = {g1.x, g1.y, g1.z, g1.w}, w2[2] = {g2.x, g2.y};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (CF == CF_F16) {
        // fixed-point cxz, cyz (x 2^15); velocity v = b + b * d from the row's
        // bases vb and the FP16 ratios d
        const float2 a = fx2f(w1[2 * k]), b = h2f(w1[2 * k + 1], false), c = h2f(w2[k], false);
        out[k] = OutMedium{a.x, a.y, fmaf(vb.x, b.x, vb.x), fmaf(vb.y, b.y, vb.y),
                           fmaf(vb.z, c.x, vb.z), fmaf(vb.w, c.y, vb.w)};
      } else {
        const float2 a = h2f(w1[2 * k], true), b = h2f(w1[2 * k + 1], true), c = h2f(w2[k], true);
        out[k] = OutMedium{a.x, a.y, b.x, b.y, c.x, c.y};
      }
    }
  }
}

// Sweeps the column tile at (x0, y0) over the output planes [zb, ze) of the
// box in prm, with the CTA's shared memory `smem` (128-byte aligned).  The
// FD weights, dt2 and the energy output are read from `cw`, the parameters
// shared by every box of the launch (kept at fixed constant-bank offsets so
// they feed the arithmetic directly).
// Returns false if a TMA wait timed out: the error word is set and the
// copies in flight have been given a bounded chance to land.
template <int TX, int TY, int CF, bool SPONGE, bool ISO>
__device__ __forceinline__ bool sweep_column(const CUtensorMap *tm_cur,
                                             const CUtensorMap *tm_prev,
                                             const CUtensorMap *tm_l,
                                             const CUtensorMap *tm_o1,
                                             const CUtensorMap *tm_o2,
                                             const CUtensorMap *tm_vb, const StepParams &prm,
                                             const StepParams &cw, const int x0, const int y0, const int zb,
                                             const int ze, unsigned char *smem) {
  using Lay = FastLayout<TX, TY, CF>;
  using CB = CoefBytes<CF>;
  // Planes of the unrolled body: one group, or two in the vpz/vsv form, whose
  // planes are the shortest (its 408^3 step: 525 -> 516 us; half the queue
  // moves).  In the other forms two no longer fit the instruction cache
  // (FP16, 872 x 424 x 268: 30.1 -> 30.8 ms for 24 steps).
  constexpr int GROUP = kGroup, BODY = CF == CF_VV ? 2 * kGroup : kGroup;
  constexpr int HX = Lay::HX;
  constexpr int NT = Lay::NT;
  constexpr unsigned kAll = 0xffffffffu;
  // single-chain derivatives for the narrow-coefficient sweeps (see d2k)
  constexpr bool CHAIN = CF == CF_F16 || CF == CF_BF16;
  // equal spacing on all axes: one set of weights serves x, y and z
  const float *w2x = cw.w2x, *w1x = cw.w1x;
  const float *w2y = ISO ? cw.w2x : cw.w2y, *w1y = ISO ? cw.w1x : cw.w1y;
  const float *w2z = ISO ? cw.w2x : cw.w2z, *w1z = ISO ? cw.w1x : cw.w1z;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + Lay::OFF_BAR);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // a warp owns ROWS tile rows, a lane the points tx and tx + 1 of one
  constexpr int ROWS = Lay::ROWS;
  const int tx = 2 * (lane % (TX / 2)), ty = ROWS * warp + lane / (TX / 2);
  const int n_it = ze - zb + 2 * kHalo;
  const int gx = x0 + tx, gy = y0 + ty;
  const bool row_in = gy >= prm.y0 && gy < prm.y1;
  const bool act[2] = {row_in && gx >= prm.x0 && gx < prm.x1,
                       row_in && gx + 1 >= prm.x0 && gx + 1 < prm.x1};
  // medium coordinates of the tile
  const int mx0 = x0 + prm.mox, my0 = y0 + prm.moy;

  if (tid == 0) {
    for (int s = 0; s < 2; ++s) mbar_init(&bars[s], 1);
    mbar_init_fence();
    prefetch_tensormap(tm_cur);
    prefetch_tensormap(tm_prev);
    if (CB::L) prefetch_tensormap(tm_l);
    prefetch_tensormap(tm_o1);
    if (CB::O2) prefetch_tensormap(tm_o2);
    if (Lay::VB_PLANE) prefetch_tensormap(tm_vb);
  }
  __syncthreads();
  // Everything above ran while the previous grid of the stream was finishing;
  // its fields are read and overwritten from here on.  Only then may the next
  // one be brought in: one grid waits at a time.
  if (!prm.beside) grid_dep_wait();
  grid_dep_launch();

  // Producer: one elected thread fills stage s with the group of iterations
  // j .. j + GROUP - 1, one copy per array (planes past the array read
  // zeros, planes past the sweep are never used).
  auto issue = [&](int j, int s) {
    unsigned char *st = smem + s * Lay::STAGE_BYTES;
    const int k = zb - kHalo + j;
    const bool want_lead = CB::L > 0 && j + GROUP > kHalo && j < n_it - kHalo;
    const bool want_out = j + GROUP > 2 * kHalo;
    mbar_arrive_expect_tx(&bars[s], Lay::TX_HALO + (want_lead ? Lay::TX_LEAD : 0u) +
                                        (want_out ? Lay::TX_OUT : 0u));
    tma_load_3d(st + Lay::OFF_H, tm_cur, x0 - kHalo, y0 - kHalo, k, &bars[s]);
    // 16-byte groups are mapped as two 8-byte elements per point (x
    // coordinate 2 * x: one 512-byte row per tile row), 8- and 4-byte groups
    // as one element per point
    constexpr int XL = CB::L == 16 ? 2 : 1, XO = CB::O1 == 16 ? 2 : 1;
    if (want_lead) tma_load_3d(st + Lay::OFF_L, tm_l, XL * mx0, my0, k + prm.moz, &bars[s]);
    if (want_out) {
      const int z = k - kHalo;
      const int mz = z + prm.moz;
      tma_load_3d(st + Lay::OFF_O1, tm_o1, XO * mx0, my0, mz, &bars[s]);
      if (CB::O2) tma_load_3d(st + Lay::OFF_O2, tm_o2, mx0, my0, mz, &bars[s]);
      // FP16 form: rows my0 .. my0 + TY - 1 of the bases (two 8-byte
      // elements per row)
      if (Lay::VB_PLANE) tma_load_2d(st + Lay::OFF_VB, tm_vb, 2 * my0, mz, &bars[s]);
      tma_load_3d(st + Lay::OFF_OWN, tm_prev, x0, y0, z, &bars[s]);
    }
  };

  if (tid == 0) issue(0, 0);

  // Register queues of both columns.  cq, dxq, dyq: centre value, x- and
  // y-derivative of the last eight planes (oldest first) and of the body's
  // own; aq, bq, zq: in-plane part of H1, in-plane Laplacian and czz of the
  // last four and the body's own.  Moved down by BODY after every body.
  float2 cq[8 + BODY][2], dxq[8 + BODY][2], dyq[8 + BODY][2];
  float2 aq[kHalo + BODY][2], bq[kHalo + BODY][2];
  float zq[kHalo + BODY][2];
  float2 e_acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  bool bad = false;  // a wait of this thread timed out

  // inactive threads of edge tiles may sit past the array: no profile read
  float gxy[2] = {1.0f, 1.0f};
  if (SPONGE) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (act[c]) gxy[c] = prm.sponge[gx + c] * prm.sponge[prm.sponge_oy + gy];
  }
  // profile of the next output plane (gz[ze] exists: ze <= sz - 4)
  const float *gzp = SPONGE ? prm.sponge + prm.sponge_oz + (zb - 2 * kHalo) : nullptr;
  float gzv = SPONGE ? gzp[2 * kHalo] : 1.0f;
  // iteration of the next output plane where one of the two columns records
  // or injects something, relative to it0, and each column's next receiver
  constexpr int kNever = 1 << 30;
  int ev = kNever, rk[2] = {0, 0};
#pragma unroll
  for (int c = 0; c < 2; ++c)
    if (act[c]) {
      if (prm.rec_col) {
        const int2 e = prm.rec_col[gy * prm.col_stride + gx + c];
        rk[c] = e.x;
        while (rk[c] < e.x + e.y && prm.rec_z[rk[c]] < zb) ++rk[c];
        if (rk[c] < e.x + e.y) ev = min(ev, prm.rec_z[rk[c]]);
      }
      if (gx + c == prm.src_x && gy == prm.src_y && prm.src_z >= zb) ev = min(ev, prm.src_z);
    }
  ev += 2 * kHalo - zb;
  int am = (act[0] ? 1 : 0) | (act[1] ? 2 : 0);
  // shared-memory addresses: stage 0, and the thread's points in dy plane 0
  const uint32_t sbase = smem_u32(smem);
  StageAddr sa;
  sa.halo = sbase + Lay::OFF_H + 8 * ((ty + kHalo) * HX + tx + kHalo);
  // the halo column whose y-derivative this lane computes (four columns on
  // either side of the warp's rows; with two rows lanes 16-31 do the next
  // plane's)
  const int hrow = ROWS * warp + (lane >> 3) % ROWS;
  const int hcol = (lane & 7) < 4 ? (lane & 7) : TX + (lane & 7);
  const bool hnext = ROWS == 2 && lane >= 16;
  sa.col = sbase + Lay::OFF_H + 8 * ((hrow + kHalo) * HX + hcol) + (hnext ? Lay::H_PLANE : 0);
  sa.t8 = sbase + 8 * (ty * TX + tx);
  sa.t4 = sbase + 4 * (ty * TX + tx);
  sa.t16 = (sbase + 16 * (ty * TX + tx)) ^ ((tid & 4) ? 16u : 0u);
  sa.row = sbase + 16 * ty;
  const uint32_t dy = sbase + Lay::OFF_DY + 8 * (ty * HX + tx + kHalo);
  const uint32_t dycol =
      sbase + Lay::OFF_DY + 8 * (hrow * HX + hcol) + (hnext ? Lay::DY_BYTES : 0);
  // global position of the first point at the first output plane (advanced
  // by one plane per output; never dereferenced for inactive points)
  float2 *out = prm.prev + (static_cast<long long>(zb) * prm.plane +
                            static_cast<long long>(gy) * prm.pitch + gx);

  int sel = 1;        // stage of the current group
  uint32_t par = 1u;  // its mbarrier parity
  sa.shift(Lay::STAGE_BYTES);
  int it0 = 0;      // first iteration of the body
  int stop = n_it;  // a group boundary where a time-out was seen

  // Iteration it0 + u; false past the end of the sweep.
  auto plane = [&](auto U) __attribute__((always_inline)) {
    constexpr int u = decltype(U)::value;
    constexpr int g = u % GROUP;  // the plane inside its group
    constexpr int DY = g * Lay::DY_BYTES;
    if (it0 + u >= n_it) return false;  // CTA-uniform
    if (g == 0) {
      // Every warp has read the previous group: refill its stage with the
      // next one, then wait for the current one.
      if (__syncthreads_or(bad)) {
        stop = it0 + u;
        return false;
      }
      if (tid == 0 && it0 + u + GROUP < n_it) issue(it0 + u + GROUP, sel);
      sa.shift(sel ? -Lay::STAGE_BYTES : Lay::STAGE_BYTES);
      sel ^= 1;
      par ^= sel ^ 1;
      if (!mbar_wait_bounded(&bars[sel], par, kWaitLimitNs)) {
        // the warp goes on to the group's end, but writes no more outputs
        bad = true;
        am = 0;
        ev = kNever;
      }
    }

    // ---- leading plane k: centre, x/y second and first derivatives
    float2 xx[2], yy[2];
    {
      float2 w[10], v[8][2];  // row of the two points; their columns
      constexpr int H = Lay::OFF_H + g * Lay::H_PLANE;
      ld_pairs<H - 32>(sa.halo, w[0], w[1]);
      ld_pairs<H - 16>(sa.halo, w[2], w[3]);
      ld_pairs<H>(sa.halo, w[4], w[5]);
      ld_pairs<H + 16>(sa.halo, w[6], w[7]);
      ld_pairs<H + 32>(sa.halo, w[8], w[9]);
      ld_pairs<H - 32 * HX>(sa.halo, v[0][0], v[0][1]);
      ld_pairs<H - 24 * HX>(sa.halo, v[1][0], v[1][1]);
      ld_pairs<H - 16 * HX>(sa.halo, v[2][0], v[2][1]);
      ld_pairs<H - 8 * HX>(sa.halo, v[3][0], v[3][1]);
      ld_pairs<H + 8 * HX>(sa.halo, v[4][0], v[4][1]);
      ld_pairs<H + 16 * HX>(sa.halo, v[5][0], v[5][1]);
      ld_pairs<H + 24 * HX>(sa.halo, v[6][0], v[6][1]);
      ld_pairs<H + 32 * HX>(sa.halo, v[7][0], v[7][1]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float2 m = w[4 + c];
        cq[8 + u][c] = m;
        dyq[8 + u][c] = d1s<ISO, CHAIN>(w1y, v[3][c], v[4][c], v[2][c], v[5][c], v[1][c], v[6][c],
                                    v[0][c], v[7][c]);
        yy[c] = d2s<ISO, CHAIN>(w2y, m, v[3][c], v[4][c], v[2][c], v[5][c], v[1][c], v[6][c],
                                v[0][c], v[7][c]);
        xx[c] = d2s<ISO, CHAIN>(w2x, m, w[3 + c], w[5 + c], w[2 + c], w[6 + c], w[1 + c],
                                w[7 + c], w[c], w[8 + c]);
        dxq[8 + u][c] = d1s<ISO, CHAIN>(w1x, w[3 + c], w[5 + c], w[2 + c], w[6 + c], w[1 + c],
                                    w[7 + c], w[c], w[8 + c]);
      }
      sts4<DY>(dy, dyq[8 + u][0], dyq[8 + u][1]);
      // y-derivatives of the 4 + 4 halo columns (needed by d2/dxdy): with two
      // rows of this plane and the next one at once where the group holds both
      if (ROWS > 2 || (g % 2 == 0 && (g + 1 < GROUP || lane < 16)))
        sts2<DY>(dycol, d1s<ISO, CHAIN>(w1y, lds2<H - 8 * HX>(sa.col), lds2<H + 8 * HX>(sa.col),
                                        lds2<H - 16 * HX>(sa.col), lds2<H + 16 * HX>(sa.col),
                                        lds2<H - 24 * HX>(sa.col), lds2<H + 24 * HX>(sa.col),
                                        lds2<H - 32 * HX>(sa.col), lds2<H + 32 * HX>(sa.col)));
    }

    // ---- output plane z = k - 4
    if (it0 + u >= 2 * kHalo) {
      // queue slots of planes z-4 .. z+4
      constexpr int m4 = u, m3 = u + 1, m2 = u + 2, m1 = u + 3, z0 = u + 4, p1 = u + 5,
                    p2 = u + 6, p3 = u + 7, p4 = u + 8;
      OutMedium md[2];
      load_out<CF, Lay::OFF_O1 + g * Lay::O1_PLANE, Lay::OFF_O2 + g * Lay::O2_PLANE,
               Lay::OFF_VB + g * Lay::VB_PLANE>(sa, md);
      float2 pv[2], nv[2];
      ld_pairs<Lay::OFF_OWN + g * Lay::OWN_PLANE>(sa.t8, pv[0], pv[1]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float2 zz = d2s<ISO, CHAIN>(w2z, cq[z0][c], cq[m1][c], cq[p1][c], cq[m2][c],
                                          cq[p2][c], cq[m3][c], cq[p3][c], cq[m4][c], cq[p4][c]);
        const float2 xz = d1s<ISO, CHAIN>(w1z, dxq[m1][c], dxq[p1][c], dxq[m2][c], dxq[p2][c],
                                          dxq[m3][c], dxq[p3][c], dxq[m4][c], dxq[p4][c]);
        const float2 yz = d1s<ISO, CHAIN>(w1z, dyq[m1][c], dyq[p1][c], dyq[m2][c], dyq[p2][c],
                                          dyq[m3][c], dyq[p3][c], dyq[m4][c], dyq[p4][c]);
        // H1 = sum c * d2 over the six second derivatives; the Laplacian
        // (H1 + H2) = xx + yy + zz
        float2 h1 = fma2(bc(md[c].cyz), yz,
                         fma2(bc(md[c].cxz), xz, fma2(bc(zq[u][c]), zz, aq[u][c])));
        if (CF == CF_F16) h1 = mul2(h1, bc(kChUnscale<CF>));
        const float2 h2 = fma2(bc(-1.0f), h1, add2(bq[u][c], zz));
        const float rhsp =
            fmaf(md[c].v2sz, h1.x - h1.y, fmaf(md[c].v2pz, h1.y, md[c].v2px * h2.x));
        const float rhsq =
            fmaf(-md[c].v2sz, h2.x - h2.y, fmaf(md[c].v2pz, h1.y, md[c].v2pn * h2.x));
        const float2 rhs = make_float2(rhsp, rhsq);
        const float2 cc = add2(cq[z0][c], cq[z0][c]);  // 2 * current
        if (SPONGE) {
          const float g = gxy[c] * gzv;
          nv[c] = mul2(fma2(rhs, bc(ISO ? cw.dt2_iso : cw.dt2), fma2(bc(-g), pv[c], cc)), bc(g));
        } else {
          nv[c] = fma2(rhs, bc(ISO ? cw.dt2_iso : cw.dt2), fma2(bc(-1.0f), pv[c], cc));
        }
        // energy partials of both columns (inactive ones are dropped below)
        e_acc[c] = fma2(nv[c], nv[c], e_acc[c]);
      }
      if (SPONGE) gzv = gzp[u + 1];
      if (u != ev && am == 3) {  // gx is even: 16-byte aligned
        *reinterpret_cast<float4 *>(out) = make_float4(nv[0].x, nv[0].y, nv[1].x, nv[1].y);
      } else {
        if (u == ev) {  // a receiver and/or the source sits at these points
          const int z = zb + it0 + u - 2 * kHalo;
          const int step = *prm.d_step + prm.step_offset;
          ev = kNever;
#pragma unroll
          for (int c = 0; c < 2; ++c)
            if (am & (1 << c)) {
              if (prm.rec_col) {
                const int2 e = prm.rec_col[gy * prm.col_stride + gx + c];
                const int rend = e.x + e.y;
                while (rk[c] < rend && prm.rec_z[rk[c]] == z) {
                  if (step >= 0 && step < prm.trace_cap)
                    prm.traces[static_cast<long long>(step) * prm.nrec + prm.rec_r[rk[c]]] =
                        nv[c].x;
                  ++rk[c];
                }
                if (rk[c] < rend) ev = min(ev, prm.rec_z[rk[c]] - z + u);
              }
              if (gx + c == prm.src_x && gy == prm.src_y) {
                if (z == prm.src_z) {
                  const float sv = step + 1 < prm.src_count ? prm.src_table[step + 1] : 0.0f;
                  prm.src_pre[0] = nv[c].x;
                  prm.src_pre[1] = nv[c].y;
                  nv[c].x += sv;
                  nv[c].y += sv;
                } else if (prm.src_z > z) {
                  ev = min(ev, prm.src_z - z + u);
                }
              }
            }
        }
        if (am & 1) out[0] = nv[0];
        if (am & 2) out[1] = nv[1];
      }
      out += prm.plane;
    }

    // ---- in-plane part of H1 (A) and of the Laplacian (B) at plane k; they
    // wait in the queues for 4 planes.  The dy rows are the warp's own:
    // only its lanes have to have stored them.  (Before iteration 4 and in
    // the last four the slot is never read: whatever the stage holds will
    // do.)
    __syncwarp();
    {
      float2 e[10];  // y-derivatives of the row, x - 4 .. x + 5
      ld_pairs<DY - 32>(dy, e[0], e[1]);
      ld_pairs<DY - 16>(dy, e[2], e[3]);
      ld_pairs<DY + 16>(dy, e[6], e[7]);
      ld_pairs<DY + 32>(dy, e[8], e[9]);
      e[4] = dyq[8 + u][0];
      e[5] = dyq[8 + u][1];
      float4 lc[2];
      load_lead<CF, Lay::OFF_L + g * Lay::L_PLANE>(sa, lc);  // cxx, cyy, cxy, czz
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float2 xy = d1s<ISO, CHAIN>(w1x, e[3 + c], e[5 + c], e[2 + c], e[6 + c], e[1 + c],
                                          e[7 + c], e[c], e[8 + c]);
        aq[kHalo + u][c] = fma2(bc(lc[c].z), xy, fma2(bc(lc[c].y), yy[c], mul2(bc(lc[c].x), xx[c])));
        bq[kHalo + u][c] = add2(xx[c], yy[c]);
        zq[kHalo + u][c] = lc[c].w;
      }
    }
    return true;
  };
  while (plane(Const<0>{}) && plane(Const<1>{}) && plane(Const<2>{}) &&
         (BODY == 3 || (plane(Const<BODY == 3 ? 0 : 3>{}) && plane(Const<BODY == 3 ? 0 : 4>{}) &&
                        plane(Const<BODY == 3 ? 0 : 5>{})))) {
    it0 += BODY;
    ev -= BODY;
    if (SPONGE) gzp += BODY;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        cq[i][c] = cq[i + BODY][c];
        dxq[i][c] = dxq[i + BODY][c];
        dyq[i][c] = dyq[i + BODY][c];
      }
#pragma unroll
      for (int i = 0; i < kHalo; ++i) {
        aq[i][c] = aq[i + BODY][c];
        bq[i][c] = bq[i + BODY][c];
        zq[i][c] = zq[i + BODY][c];
      }
    }
  }
  if (__syncthreads_or(bad)) {
    // A TMA wait timed out: record it, give the copies still in flight a
    // bounded chance to land, and leave.
    if (tid == 0) {
      atomicOr(prm.err, kErrTimeout);
      const int last = (stop < n_it ? stop : n_it - 1) / GROUP;  // group issued last
      for (int j = max(0, last - 1); j <= last; ++j)
        mbar_wait_bounded(&bars[j & 1], static_cast<uint32_t>(j >> 1) & 1u, kWaitLimitNs);
    }
    return false;
  }
  if (cw.energy) {
    // CTA reduction of the float partials in double, one atomic per CTA.
    double e = 0.0;
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (act[c]) e += static_cast<double>(e_acc[c].x) + static_cast<double>(e_acc[c].y);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) e += __shfl_down_sync(kAll, e, off);
    double *red = reinterpret_cast<double *>(smem + Lay::OFF_DY);
    if (lane == 0) red[warp] = e;
    __syncthreads();
    if (tid == 0) {
      double tot = 0.0;
      for (int w = 0; w < NT / 32; ++w) tot += red[w];
      const int step = *prm.d_step + prm.step_offset;
      if (step >= 0 && step < cw.energy_cap) atomicAdd(&cw.energy[step], tot);
    }
  }
  // every copy of this column has landed and been read: release the
  // barriers so the CTA can initialise them again for its next column
  __syncthreads();
  if (tid == 0)
    for (int s = 0; s < 2; ++s) mbar_inval(&bars[s]);
  return true;
}

// CTAs per SM the register allocation must allow: two of 128 threads, one
// of 256 (up to 255 registers a thread).
template <int NT>
constexpr int kMinBlocks = NT <= 128 ? 2 : 1;

// No static shared memory in these kernels: the dynamic window starts at
// the CTA's shared base, so the 1024-byte alignment holds and every access
// is a shared-space access.  TMA destinations must be 128-byte aligned; the
// kernels refuse to run otherwise (CTA-uniform, before any copy is issued).

// One pass over a box: CTA (bx, by, bz) sweeps tile (bx, by), z-chunk bz.
template <int TX, int TY, int CF, bool SPONGE, bool ISO>
__global__ void __launch_bounds__(TX *TY / 2, kMinBlocks<TX * TY / 2>)
    fast_kernel(const __grid_constant__ CUtensorMap tm_cur,
                const __grid_constant__ CUtensorMap tm_prev,
                const __grid_constant__ CUtensorMap tm_l,
                const __grid_constant__ CUtensorMap tm_o1,
                const __grid_constant__ CUtensorMap tm_o2,
                const __grid_constant__ CUtensorMap tm_vb,
                const __grid_constant__ StepParams prm) {
  extern __shared__ __align__(1024) unsigned char smem[];
  if (smem_u32(smem) & 127u) {
    if (threadIdx.x == 0) atomicOr(prm.err, kErrAlign);
    grid_dep_wait();
    return;
  }
  const int x0 = prm.tile_x0 + static_cast<int>(blockIdx.x) * TX;
  const int y0 = prm.tile_y0 + static_cast<int>(blockIdx.y) * TY;
  const int zb = prm.z0 + static_cast<int>(blockIdx.z) * prm.zchunk;
  const int ze = min(zb + prm.zchunk, prm.z1);
  sweep_column<TX, TY, CF, SPONGE, ISO>(&tm_cur, &tm_prev, &tm_l, &tm_o1, &tm_o2, &tm_vb, prm,
                                        prm, x0, y0, zb, ze, smem);
  // beside another pass: done only when that one is, so that whoever waits for
  // this grid waits for all boxes of the step
  if (prm.beside) grid_dep_wait();
}

// One step of a batch of shots: one CTA per work item, or (LOOP) CTAs that
// stride over them.  The host's table gives an item's shot, tile and planes,
// so every index here is CTA-uniform.  Two kernels, because around the sweep a
// loop costs the compiled sweep 12 % more instructions (moves of the queues,
// addresses worked out again in every plane): eight FP16 shots, 97 M points,
// 0.964 ms per step with the loop, 0.925 without.
template <int TX, int TY, int CF, bool SPONGE, bool ISO, bool LOOP>
__global__ void __launch_bounds__(TX *TY / 2, kMinBlocks<TX * TY / 2>)
    batch_kernel(const __grid_constant__ BatchLaunch bl) {
  extern __shared__ __align__(1024) unsigned char smem[];
  if (smem_u32(smem) & 127u) {
    if (threadIdx.x == 0) atomicOr(bl.err, kErrAlign);
    return;
  }
  int slot = blockIdx.x;
  if (slot >= bl.n_items) return;
  do {
    const int4 item = bl.items[slot];
    const int s = item.x, zb = item.z, ze = item.w;
    const StepParams &prm = bl.shot[s];
    const int x0 = prm.tile_x0 + (item.y & 0xffff) * TX, y0 = prm.tile_y0 + (item.y >> 16) * TY;
    const CUtensorMap *m = bl.maps + 4 * s;
    // weights, dt2 and energy (none) are the same in every shot: read them
    // from shot 0 at fixed offsets
    if (!sweep_column<TX, TY, CF, SPONGE, ISO>(m + bl.cur_buf, m + 2 + (1 - bl.cur_buf),
                                               &bl.tm_l, &bl.tm_o1, &bl.tm_o2, &bl.tm_vb, prm,
                                               bl.shot[0], x0, y0, zb, ze, smem))
      return;
    slot += gridDim.x;
  } while (LOOP && slot < bl.n_items);
}

constexpr int kTX = DC_TX, kTY = DC_TY, kCF = DC_FORM;
using Lay = FastLayout<kTX, kTY, kCF>;

template <bool SPONGE, bool ISO>
cudaError_t launch_fast_t(const Sim *sim, const FastMaps &maps, const StepParams &prm,
                          int cur_buf, int prev_buf) {
  const int nx = prm.x1 - prm.tile_x0, ny = prm.y1 - prm.tile_y0;
  const int nz = prm.z1 - prm.z0;
  dim3 grid((nx + kTX - 1) / kTX, (ny + kTY - 1) / kTY, (nz + prm.zchunk - 1) / prm.zchunk);
  return launch_dependent(fast_kernel<kTX, kTY, kCF, SPONGE, ISO>, grid, Lay::NT, Lay::SMEM_BYTES,
                          sim->stream, maps.halo[cur_buf], maps.own[prev_buf], maps.c[0],
                          maps.c[1], maps.c[2], maps.c[3], prm);
}

cudaError_t launch_one(const Sim *sim, const FastMaps &maps, const StepParams &prm, int cur,
                       int prev) {
  const bool iso = sim->dx == sim->dy && sim->dy == sim->dz;
  if (prm.sponge)
    return iso ? launch_fast_t<true, true>(sim, maps, prm, cur, prev)
               : launch_fast_t<true, false>(sim, maps, prm, cur, prev);
  return iso ? launch_fast_t<false, true>(sim, maps, prm, cur, prev)
             : launch_fast_t<false, false>(sim, maps, prm, cur, prev);
}

template <typename K>
cudaError_t allow_smem(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              Lay::SMEM_BYTES);
}

cudaError_t attrs_one() {
  cudaError_t e = allow_smem(fast_kernel<kTX, kTY, kCF, false, false>);
  if (e == cudaSuccess) e = allow_smem(fast_kernel<kTX, kTY, kCF, false, true>);
  if (e == cudaSuccess) e = allow_smem(fast_kernel<kTX, kTY, kCF, true, false>);
  if (e == cudaSuccess) e = allow_smem(fast_kernel<kTX, kTY, kCF, true, true>);
  return e;
}

template <typename K>
int occupancy(K kernel) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, Lay::NT, Lay::SMEM_BYTES) !=
      cudaSuccess)
    return 0;
  return n;
}

// CTAs of the fast sweep one SM holds at once (the sponge, equal-spacing
// instance; the others differ by a few registers, well inside the limit).
int occ_one() { return occupancy(fast_kernel<kTX, kTY, kCF, true, true>); }

// Batch kernel variants: either spacing with the sponge; without it (all shots'
// profiles are 1, e.g. learned layers) equal spacing.
template <int CF>
struct BatchOps {
  template <bool LOOP>
  static cudaError_t attrs_loop() {
    cudaError_t e = allow_smem(batch_kernel<kTX, kTY, CF, true, false, LOOP>);
    if (e == cudaSuccess) e = allow_smem(batch_kernel<kTX, kTY, CF, true, true, LOOP>);
    if (e == cudaSuccess) e = allow_smem(batch_kernel<kTX, kTY, CF, false, true, LOOP>);
    return e;
  }

  static cudaError_t attrs() {
    const cudaError_t e = attrs_loop<false>();
    return e == cudaSuccess ? attrs_loop<true>() : e;
  }

  static int occ(bool iso, bool sponge) {
    if (iso && !sponge) return occupancy(batch_kernel<kTX, kTY, CF, false, true, true>);
    return iso ? occupancy(batch_kernel<kTX, kTY, CF, true, true, true>)
               : occupancy(batch_kernel<kTX, kTY, CF, true, false, true>);
  }

  template <bool LOOP>
  static cudaError_t launch_loop(cudaStream_t st, const BatchLaunch &bl, bool iso, bool sponge,
                                 int blocks) {
    auto go = [&](auto kernel) {
      return launch_dependent(kernel, dim3(blocks), Lay::NT, Lay::SMEM_BYTES, st, bl);
    };
    if (iso && !sponge) return go(batch_kernel<kTX, kTY, CF, false, true, LOOP>);
    return iso ? go(batch_kernel<kTX, kTY, CF, true, true, LOOP>)
               : go(batch_kernel<kTX, kTY, CF, true, false, LOOP>);
  }

  static cudaError_t launch(cudaStream_t st, const BatchLaunch &bl, bool iso, bool sponge,
                            bool loop, int blocks) {
    return loop ? launch_loop<true>(st, bl, iso, sponge, blocks)
                : launch_loop<false>(st, bl, iso, sponge, blocks);
  }
};

template <int TX, int CF>
FastOps make_ops() {
  FastOps ops = {attrs_one, occ_one, launch_one, nullptr, nullptr, nullptr};
  if constexpr (TX == 32 && CF != CF_VV) {  // what a batch runs
    using B = BatchOps<CF>;
    ops.batch_attrs = B::attrs;
    ops.batch_occupancy = B::occ;
    ops.launch_batch = B::launch;
  }
  return ops;
}

}  // namespace

template <>
const FastOps &fast_ops<DC_FORM, DC_TX, DC_TY>() {
  static const FastOps ops = make_ops<kTX, kCF>();
  return ops;
}

}  // namespace dcg
