// tti_exact.cu -- the bit-exact sm_103a Fletcher TTI time step.
//
// Same update as the fast kernel, but every floating-point operation is the
// reference's, in the reference's order, with explicit round-to-nearest
// intrinsics so that nothing is contracted into an FMA:
//   der2      include/derivatives.h:47-54   (9-point second derivative)
//   derCross  include/derivatives.h:56-91   (64-point direct cross sum)
//   update    include/sample_compute.h:106-185 (sample_compute) or
//             include/sample_compute.h:21-102  (sample_compute_optimized,
//             the vpz/vsv medium form with constant angles).
// Results are bit-identical to the reference's OpenMP path built without
// FMA contraction (and to its CUDA arithmetic executed the same way).
//
// Data path: a lane owns two x-adjacent columns and sweeps a chunk of z; a CTA
// covers 32 x 8 columns.  The stencil reads go through the read-only data
// cache as (p, q) pairs, so this kernel is bound by the L1's data pipe and its
// latency, not HBM (168 x 168 x 152: 75 % of the pipe's wavefronts, 5.6 of 8 stall
// cycles per instruction on its loads, issue 31 %, DRAM 1.3 TB/s): per two points
// the x-y and x-z terms read eight rows of ten pairs in five 16-byte loads each,
// the y-z term one 16-byte load per position (149 loads; one point per thread took
// 217 8-byte loads per point), and packed f32x2 operations round p and q as scalar
// ones do.  It is the parity anchor, not the throughput path.
#include "dc_internal.h"

namespace dcg {
namespace {

// Second-derivative weights K0..K4 and the cross weights L_a*L_b rounded
// once, in the order of include/derivatives.h:58-89.
__device__ __forceinline__ constexpr float kw(int k) {
  return k == 0 ? static_cast<float>(-205.0 / 72.0)
         : k == 1 ? static_cast<float>(8.0 / 5.0)
         : k == 2 ? static_cast<float>(-1.0 / 5.0)
         : k == 3 ? static_cast<float>(8.0 / 315.0)
                  : static_cast<float>(-1.0 / 560.0);
}
__device__ __forceinline__ constexpr double lw(int a) {
  return a == 1 ? 4.0 / 5.0 : a == 2 ? -1.0 / 5.0 : a == 3 ? 4.0 / 105.0 : -1.0 / 280.0;
}
__device__ __forceinline__ constexpr int pair_a(int g) {
  return g < 4 ? 1 : g < 7 ? 2 : g < 9 ? 3 : 4;
}
__device__ __forceinline__ constexpr int pair_b(int g) {
  return g < 4 ? g + 1 : g < 7 ? g - 2 : g < 9 ? g - 4 : 4;
}

struct H12 {
  float h1, h2;
};

// der2 (include/derivatives.h:47-54) and derCross (:56-91) of p and q
// together: one 8-byte load of a (p, q) pair feeds both fields, and each
// field's arithmetic is the reference's, term by term and in its order.
__device__ __forceinline__ float2 ldp(const float2 *__restrict__ f, long long i) {
  return __ldg(f + i);
}

__device__ __forceinline__ float2 der2_x2(const float2 *__restrict__ f, long long i, long long s,
                                          float inv) {
  const float2 c = ldp(f, i);
  float2 a = make_float2(__fmul_rn(kw(0), c.x), __fmul_rn(kw(0), c.y));
#pragma unroll
  for (int k = 1; k <= 4; ++k) {
    const float2 u = ldp(f, i + k * s), v = ldp(f, i - k * s);
    a.x = __fadd_rn(a.x, __fmul_rn(kw(k), __fadd_rn(u.x, v.x)));
    a.y = __fadd_rn(a.y, __fmul_rn(kw(k), __fadd_rn(u.y, v.y)));
  }
  return make_float2(__fmul_rn(a.x, inv), __fmul_rn(a.y, inv));
}

__device__ __forceinline__ float2 cross_x2(const float2 *__restrict__ f, long long i,
                                           long long s1, long long s2, float inv) {
  float2 total = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int g = 0; g < 10; ++g) {
    const long long a = pair_a(g), b = pair_b(g);
    const float2 v0 = ldp(f, i + a * s2 + b * s1), v1 = ldp(f, i + a * s2 - b * s1);
    const float2 v2 = ldp(f, i - a * s2 + b * s1), v3 = ldp(f, i - a * s2 - b * s1);
    float2 acc;
    acc.x = __fadd_rn(__fsub_rn(__fsub_rn(v0.x, v1.x), v2.x), v3.x);
    acc.y = __fadd_rn(__fsub_rn(__fsub_rn(v0.y, v1.y), v2.y), v3.y);
    if (a != b) {
      const float2 w0 = ldp(f, i + b * s2 + a * s1), w1 = ldp(f, i + b * s2 - a * s1);
      const float2 w2 = ldp(f, i - b * s2 + a * s1), w3 = ldp(f, i - b * s2 - a * s1);
      acc.x = __fadd_rn(__fsub_rn(__fsub_rn(__fadd_rn(acc.x, w0.x), w1.x), w2.x), w3.x);
      acc.y = __fadd_rn(__fsub_rn(__fsub_rn(__fadd_rn(acc.y, w0.y), w1.y), w2.y), w3.y);
    }
    const float w = static_cast<float>(lw(pair_a(g)) * lw(pair_b(g)));
    const float2 term = make_float2(__fmul_rn(w, acc.x), __fmul_rn(w, acc.y));
    total = g == 0 ? term
                   : make_float2(__fadd_rn(total.x, term.x), __fadd_rn(total.y, term.y));
  }
  return make_float2(__fmul_rn(total.x, inv), __fmul_rn(total.y, inv));
}

// h1 / h2 of p (.x) and q (.y) from pair-buffer strides (sX = 1).
__device__ __forceinline__ void hterms2(const float2 *__restrict__ f, long long i, long long sY,
                                        long long sZ, const StepParams &prm, float cxx,
                                        float cyy, float czz, float cxy, float cyz, float cxz,
                                        H12 *hp, H12 *hq) {
  const float2 fxx = der2_x2(f, i, 1, prm.dxxinv);
  const float2 fyy = der2_x2(f, i, sY, prm.dyyinv);
  const float2 fzz = der2_x2(f, i, sZ, prm.dzzinv);
  const float2 fxy = cross_x2(f, i, 1, sY, prm.dxyinv);
  const float2 fyz = cross_x2(f, i, sY, sZ, prm.dyzinv);
  const float2 fxz = cross_x2(f, i, 1, sZ, prm.dxzinv);
  const float xx[2] = {fxx.x, fxx.y}, yy[2] = {fyy.x, fyy.y}, zz[2] = {fzz.x, fzz.y};
  const float xy[2] = {fxy.x, fxy.y}, yz[2] = {fyz.x, fyz.y}, xz[2] = {fxz.x, fxz.y};
  H12 *out[2] = {hp, hq};
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    float h1 = __fmul_rn(cxx, xx[c]);
    h1 = __fadd_rn(h1, __fmul_rn(cyy, yy[c]));
    h1 = __fadd_rn(h1, __fmul_rn(czz, zz[c]));
    h1 = __fadd_rn(h1, __fmul_rn(cxy, xy[c]));
    h1 = __fadd_rn(h1, __fmul_rn(cxz, xz[c]));
    h1 = __fadd_rn(h1, __fmul_rn(cyz, yz[c]));
    out[c]->h1 = h1;
    out[c]->h2 = __fsub_rn(__fadd_rn(__fadd_rn(xx[c], yy[c]), zz[c]), h1);
  }
}


// ---- two x-adjacent points per lane ---------------------------------------
// (p, q) pairs in packed arithmetic: each half is the scalar operation of the
// same name.  a - b is fma(-1, b, a), which rounds once.  The compiler fuses a
// packed product into a packed addition that uses it, rounding modifiers or
// not (scalar ones it leaves alone), so a product is never an operand of
// add2: a + w b is written a - (-w) b, whose product is already the
// multiplicand of an FMA.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  return __ffma2_rn(make_float2(-1.0f, -1.0f), b, a);
}
__device__ __forceinline__ float2 mul2(float a, float2 b) {
  return __fmul2_rn(make_float2(a, a), b);
}

// The pairs at index i and i + 1 (i even).
__device__ __forceinline__ void ld_two(const float2 *__restrict__ f, long long i, float2 v[2]) {
  const float4 t = __ldg(reinterpret_cast<const float4 *>(f + i));
  v[0] = make_float2(t.x, t.y);
  v[1] = make_float2(t.z, t.w);
}

// Pairs x - 4 .. x + 5 of the row at index i (of the first point).
__device__ __forceinline__ void ld_row(const float2 *__restrict__ f, long long i, float2 w[10]) {
#pragma unroll
  for (int k = 0; k < 10; k += 2) ld_two(f, i - 4 + k, w + k);
}

// der2 (include/derivatives.h:47-54): c centre, u[k - 1] / v[k - 1] the
// values at +k / -k.
__device__ __forceinline__ float2 der2_pair(float2 c, const float2 u[4], const float2 v[4],
                                            float inv) {
  float2 a = mul2(kw(0), c);
#pragma unroll
  for (int k = 1; k <= 4; ++k) a = sub2(a, mul2(-kw(k), add2(u[k - 1], v[k - 1])));
  return mul2(inv, a);
}

// derCross (include/derivatives.h:56-91) from at(i2, i1): the pair at i2 steps
// along the second axis and i1 along the first.
template <class At>
__device__ __forceinline__ float2 cross_pair(At at, float inv) {
  float2 total = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int g = 0; g < 10; ++g) {
    const int a = pair_a(g), b = pair_b(g);
    float2 acc = add2(sub2(sub2(at(a, b), at(a, -b)), at(-a, b)), at(-a, -b));
    if (a != b)
      acc = add2(sub2(sub2(add2(acc, at(b, a)), at(b, -a)), at(-b, a)), at(-b, -a));
    const float w = static_cast<float>(lw(pair_a(g)) * lw(pair_b(g)));
    total = g == 0 ? mul2(w, acc) : sub2(total, mul2(-w, acc));
  }
  return mul2(inv, total);
}

// The six second derivatives of the two points at index i (even), (p, q)
// pairs: out[0..5] = xx, yy, zz, xy, yz, xz.
__device__ __forceinline__ void derivs_two(const float2 *__restrict__ f, long long i,
                                           long long sY, long long sZ, const StepParams &prm,
                                           float2 out[6][2], float2 centre[2]) {
  {
    float2 w[10];
    ld_row(f, i, w);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 u[4] = {w[5 + c], w[6 + c], w[7 + c], w[8 + c]};
      const float2 v[4] = {w[3 + c], w[2 + c], w[1 + c], w[c]};
      centre[c] = w[4 + c];
      out[0][c] = der2_pair(w[4 + c], u, v, prm.dxxinv);
    }
  }
#pragma unroll
  for (int ax = 0; ax < 2; ++ax) {  // rows along y, then along z
    const long long st = ax == 0 ? sY : sZ;
    float2 up[4][10], dn[4][10];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      ld_row(f, i + (k + 1) * st, up[k]);
      ld_row(f, i - (k + 1) * st, dn[k]);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 u[4] = {up[0][4 + c], up[1][4 + c], up[2][4 + c], up[3][4 + c]};
      const float2 v[4] = {dn[0][4 + c], dn[1][4 + c], dn[2][4 + c], dn[3][4 + c]};
      out[1 + ax][c] = der2_pair(centre[c], u, v, ax == 0 ? prm.dyyinv : prm.dzzinv);
      out[ax == 0 ? 3 : 5][c] = cross_pair(
          [&](int r, int x) { return r > 0 ? up[r - 1][4 + c + x] : dn[-r - 1][4 + c + x]; },
          ax == 0 ? prm.dxyinv : prm.dxzinv);
    }
  }
  // y-z: every position is used once per point, both points' values in one
  // load; group by group, so few are live
  float2 total[2];
#pragma unroll
  for (int g = 0; g < 10; ++g) {
    const int a = pair_a(g), b = pair_b(g);
    float2 v[8][2];
    ld_two(f, i + a * sZ + b * sY, v[0]);
    ld_two(f, i + a * sZ - b * sY, v[1]);
    ld_two(f, i - a * sZ + b * sY, v[2]);
    ld_two(f, i - a * sZ - b * sY, v[3]);
    if (a != b) {
      ld_two(f, i + b * sZ + a * sY, v[4]);
      ld_two(f, i + b * sZ - a * sY, v[5]);
      ld_two(f, i - b * sZ + a * sY, v[6]);
      ld_two(f, i - b * sZ - a * sY, v[7]);
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float2 acc = add2(sub2(sub2(v[0][c], v[1][c]), v[2][c]), v[3][c]);
      if (a != b) acc = add2(sub2(sub2(add2(acc, v[4][c]), v[5][c]), v[6][c]), v[7][c]);
      const float w = static_cast<float>(lw(pair_a(g)) * lw(pair_b(g)));
      total[c] = g == 0 ? mul2(w, acc) : sub2(total[c], mul2(-w, acc));
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) out[4][c] = mul2(prm.dyzinv, total[c]);
}

// The medium at index i.
struct PointMedium {
  float cxx, cyy, czz, cxy, cyz, cxz, v2px, v2pz, v2sz, v2pn;
};
template <int MEDIUM>
__device__ __forceinline__ PointMedium load_medium(const StepParams &prm, long long i) {
  if (MEDIUM == DC_GB300_MEDIUM_PRECOMP) {
    const long long n = prm.count;
    const float4 g0 = __ldg(reinterpret_cast<const float4 *>(prm.coef) + i);
    const float4 g1 = __ldg(reinterpret_cast<const float4 *>(prm.coef + 4 * n) + i);
    const float2 g2 = __ldg(reinterpret_cast<const float2 *>(prm.coef + 8 * n) + i);
    return PointMedium{g0.x, g0.y, g0.w, g0.z, g1.y, g1.x, g1.z, g1.w, g2.x, g2.y};
  }
  // include/sample_compute.h:9-18 and :51-54
  const float2 v = __ldg(reinterpret_cast<const float2 *>(prm.vv) + i);
  const float v2pz = __fmul_rn(v.x, v.x);
  return PointMedium{0.1459632909f, 0.3540367091f, 0.5f, 0.4546487134f, 0.8414709848f,
                     0.5403023059f, __fmul_rn(v2pz, 1.48f), v2pz, __fmul_rn(v.y, v.y),
                     __fmul_rn(v2pz, 1.2f)};
}

// New (p, q) of a point (include/sample_compute.h:106-185, in its order) from
// the derivatives d = xx, yy, zz, xy, yz, xz, the current and previous values
// and the sponge factor.
template <bool SPONGE>
__device__ __forceinline__ float2 update_point(const StepParams &prm, const PointMedium &m,
                                               const float2 d[6], float2 cv, float2 pv, float g) {
  // (scalar from here on: the derivatives are products)
  float h1[2], h2[2];
  const float xx[2] = {d[0].x, d[0].y}, yy[2] = {d[1].x, d[1].y}, zz[2] = {d[2].x, d[2].y};
  const float xy[2] = {d[3].x, d[3].y}, yz[2] = {d[4].x, d[4].y}, xz[2] = {d[5].x, d[5].y};
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    float h = __fmul_rn(m.cxx, xx[c]);
    h = __fadd_rn(h, __fmul_rn(m.cyy, yy[c]));
    h = __fadd_rn(h, __fmul_rn(m.czz, zz[c]));
    h = __fadd_rn(h, __fmul_rn(m.cxy, xy[c]));
    h = __fadd_rn(h, __fmul_rn(m.cxz, xz[c]));
    h = __fadd_rn(h, __fmul_rn(m.cyz, yz[c]));
    h1[c] = h;
    h2[c] = __fsub_rn(__fadd_rn(__fadd_rn(xx[c], yy[c]), zz[c]), h);
  }
  const float h1pmq = __fsub_rn(h1[0], h1[1]), h2pmq = __fsub_rn(h2[0], h2[1]);
  const float rhs[2] = {
      __fadd_rn(__fadd_rn(__fmul_rn(m.v2px, h2[0]), __fmul_rn(m.v2pz, h1[1])),
                __fmul_rn(m.v2sz, h1pmq)),
      __fsub_rn(__fadd_rn(__fmul_rn(m.v2pn, h2[0]), __fmul_rn(m.v2pz, h1[1])),
                __fmul_rn(m.v2sz, h2pmq))};
  const float cur[2] = {cv.x, cv.y}, prev[2] = {pv.x, pv.y};
  float out[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const float t = __fmul_rn(__fmul_rn(rhs[c], prm.dt), prm.dt);
    const float cc = __fmul_rn(2.0f, cur[c]);
    out[c] = SPONGE && g != 1.0f
                 ? __fmul_rn(__fadd_rn(__fsub_rn(cc, __fmul_rn(g, prev[c])), t), g)
                 : __fadd_rn(__fsub_rn(cc, prev[c]), t);  // the reference's own expression
  }
  return make_float2(out[0], out[1]);
}

// Tile of a CTA: 16 lanes of two columns x 8 rows.  Three CTAs per SM: the
// loads' latency is what is left to hide (168 x 168 x 152, 8 steps: 1.34 ms; without
// the bound two CTAs fit, 1.55 ms; four, with 128 registers for 168, 1.38; one point
// per thread 1.63).  Three spill 0 to 28 bytes a thread, four 4 to 36.
constexpr int kPairTX = 32, kPairTY = 8;

template <int MEDIUM, bool SPONGE>
__global__ void __launch_bounds__(kPairTX *kPairTY / 2, 3)
    exact_pair_kernel(const StepParams prm) {
  const int gx = (prm.x0 & ~1) + static_cast<int>(blockIdx.x) * kPairTX + 2 * (threadIdx.x & 15);
  const int gy = prm.y0 + static_cast<int>(blockIdx.y) * kPairTY + (threadIdx.x >> 4);
  const bool row = gy < prm.y1;
  const bool act[2] = {row && gx >= prm.x0 && gx < prm.x1, row && gx + 1 >= prm.x0 && gx + 1 < prm.x1};
  const int zb = prm.z0 + static_cast<int>(blockIdx.z) * prm.zchunk;
  const int ze = min(zb + prm.zchunk, prm.z1);
  const long long sY = prm.pitch, sZ = prm.plane;
  float e_acc[2] = {0.f, 0.f};
  int rk[2] = {0, 0}, rend[2] = {0, 0};  // receivers of the two columns
  if (prm.rec_col) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (act[c]) {
        const int2 e = prm.rec_col[gy * prm.col_stride + gx + c];
        rk[c] = e.x;
        rend[c] = e.x + e.y;
        while (rk[c] < rend[c] && prm.rec_z[rk[c]] < zb) ++rk[c];
      }
  }
  if (act[0] || act[1])
    for (int z = zb; z < ze; ++z) {
      const long long i = static_cast<long long>(z) * sZ + static_cast<long long>(gy) * sY + gx;
      float2 d[6][2], cv[2], nv[2];
      derivs_two(prm.cur, i, sY, sZ, prm, d, cv);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (!act[c]) continue;
        float g = 1.0f;
        if (SPONGE)
          g = __fmul_rn(__fmul_rn(prm.sponge[gx + c], prm.sponge[prm.sponge_oy + gy]),
                        prm.sponge[prm.sponge_oz + z]);
        const float2 dc[6] = {d[0][c], d[1][c], d[2][c], d[3][c], d[4][c], d[5][c]};
        nv[c] = update_point<SPONGE>(prm, load_medium<MEDIUM>(prm, i + c), dc, cv[c],
                                     prm.prev[i + c], g);
        if (prm.energy) e_acc[c] = fmaf(nv[c].x, nv[c].x, fmaf(nv[c].y, nv[c].y, e_acc[c]));
        if (rk[c] < rend[c] && prm.rec_z[rk[c]] == z) {
          const int step = *prm.d_step + prm.step_offset;
          do {
            if (step >= 0 && step < prm.trace_cap)
              prm.traces[static_cast<long long>(step) * prm.nrec + prm.rec_r[rk[c]]] = nv[c].x;
            ++rk[c];
          } while (rk[c] < rend[c] && prm.rec_z[rk[c]] == z);
        }
        if (gx + c == prm.src_x && gy == prm.src_y && z == prm.src_z) {
          const int step = *prm.d_step + prm.step_offset;
          const float sv = step + 1 < prm.src_count ? prm.src_table[step + 1] : 0.0f;
          prm.src_pre[0] = nv[c].x;
          prm.src_pre[1] = nv[c].y;
          nv[c] = add2(nv[c], make_float2(sv, sv));
        }
        prm.prev[i + c] = nv[c];
      }
    }
  if (prm.energy) {
    double e = static_cast<double>(e_acc[0]) + static_cast<double>(e_acc[1]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) e += __shfl_down_sync(0xffffffffu, e, off);
    if ((threadIdx.x & 31) == 0) {
      const int step = *prm.d_step + prm.step_offset;
      if (step >= 0 && step < prm.energy_cap) atomicAdd(&prm.energy[step], e);
    }
  }
}

// ---- one point per thread: buffers whose pairs are not 16-byte aligned ------
template <int MEDIUM, bool SPONGE>
__global__ void __launch_bounds__(128)
    exact_kernel(const StepParams prm) {
  const int gx = prm.x0 + static_cast<int>(blockIdx.x * 32 + threadIdx.x);
  const int gy = prm.y0 + static_cast<int>(blockIdx.y * 4 + threadIdx.y);
  if (gx >= prm.x1 || gy >= prm.y1) return;
  const int zb = prm.z0 + static_cast<int>(blockIdx.z) * prm.zchunk;
  const int ze = min(zb + prm.zchunk, prm.z1);
  const long long sY = prm.pitch, sZ = prm.plane;
  float e_acc = 0.f;
  int rk = 0, rend = 0, rnext = -1;  // receivers of this column
  if (prm.rec_col) {
    const int2 e = prm.rec_col[gy * prm.col_stride + gx];
    rk = e.x;
    rend = e.x + e.y;
    while (rk < rend && prm.rec_z[rk] < zb) ++rk;
    rnext = rk < rend ? prm.rec_z[rk] : -1;
  }
  for (int z = zb; z < ze; ++z) {
    const long long i = static_cast<long long>(z) * sZ +
                        static_cast<long long>(gy) * sY + gx;
    float cxx, cyy, czz, cxy, cyz, cxz, v2px, v2pz, v2sz, v2pn;
    if (MEDIUM == DC_GB300_MEDIUM_PRECOMP) {
      const long long n = prm.count;
      const float4 g0 = __ldg(reinterpret_cast<const float4 *>(prm.coef) + i);
      const float4 g1 = __ldg(reinterpret_cast<const float4 *>(prm.coef + 4 * n) + i);
      const float2 g2 = __ldg(reinterpret_cast<const float2 *>(prm.coef + 8 * n) + i);
      cxx = g0.x;
      cyy = g0.y;
      cxy = g0.z;
      czz = g0.w;
      cxz = g1.x;
      cyz = g1.y;
      v2px = g1.z;
      v2pz = g1.w;
      v2sz = g2.x;
      v2pn = g2.y;
    } else {
      // include/sample_compute.h:9-18 and :51-54
      const float2 v = __ldg(reinterpret_cast<const float2 *>(prm.vv) + i);
      const float vp = v.x, vs = v.y;
      cxx = 0.1459632909f;
      cyy = 0.3540367091f;
      czz = 0.5f;
      cxy = 0.4546487134f;
      cyz = 0.8414709848f;
      cxz = 0.5403023059f;
      v2pz = __fmul_rn(vp, vp);
      v2sz = __fmul_rn(vs, vs);
      v2px = __fmul_rn(v2pz, 1.48f);
      v2pn = __fmul_rn(v2pz, 1.2f);
    }
    H12 hp, hq;
    hterms2(prm.cur, i, sY, sZ, prm, cxx, cyy, czz, cxy, cyz, cxz, &hp, &hq);
    const float h1pmq = __fsub_rn(hp.h1, hq.h1);
    const float h2pmq = __fsub_rn(hp.h2, hq.h2);
    const float rhsp = __fadd_rn(
        __fadd_rn(__fmul_rn(v2px, hp.h2), __fmul_rn(v2pz, hq.h1)),
        __fmul_rn(v2sz, h1pmq));
    const float rhsq = __fsub_rn(
        __fadd_rn(__fmul_rn(v2pn, hp.h2), __fmul_rn(v2pz, hq.h1)),
        __fmul_rn(v2sz, h2pmq));
    const float2 cv = prm.cur[i];
    const float pc = cv.x, qc = cv.y;
    const float2 pv = prm.prev[i];
    const float ppo = pv.x, qpo = pv.y;
    const float tp = __fmul_rn(__fmul_rn(rhsp, prm.dt), prm.dt);
    const float tq = __fmul_rn(__fmul_rn(rhsq, prm.dt), prm.dt);
    float np, nq;
    if (SPONGE) {
      const float g = __fmul_rn(__fmul_rn(prm.sponge[gx], prm.sponge[prm.sponge_oy + gy]),
                                prm.sponge[prm.sponge_oz + z]);
      np = __fmul_rn(__fadd_rn(__fsub_rn(__fmul_rn(2.0f, pc), __fmul_rn(g, ppo)), tp), g);
      nq = __fmul_rn(__fadd_rn(__fsub_rn(__fmul_rn(2.0f, qc), __fmul_rn(g, qpo)), tq), g);
      if (g == 1.0f) {  // interior: the reference's own expression
        np = __fadd_rn(__fsub_rn(__fmul_rn(2.0f, pc), ppo), tp);
        nq = __fadd_rn(__fsub_rn(__fmul_rn(2.0f, qc), qpo), tq);
      }
    } else {
      np = __fadd_rn(__fsub_rn(__fmul_rn(2.0f, pc), ppo), tp);
      nq = __fadd_rn(__fsub_rn(__fmul_rn(2.0f, qc), qpo), tq);
    }
    if (prm.energy) e_acc = fmaf(np, np, fmaf(nq, nq, e_acc));
    if (z == rnext) {
      const int step = *prm.d_step + prm.step_offset;
      do {
        if (step >= 0 && step < prm.trace_cap)
          prm.traces[static_cast<long long>(step) * prm.nrec + prm.rec_r[rk]] = np;
        ++rk;
      } while (rk < rend && prm.rec_z[rk] == z);
      rnext = rk < rend ? prm.rec_z[rk] : -1;
    }
    if (gx == prm.src_x && gy == prm.src_y && z == prm.src_z) {
      const int step = *prm.d_step + prm.step_offset;
      const float sv = step + 1 < prm.src_count ? prm.src_table[step + 1] : 0.0f;
      prm.src_pre[0] = np;
      prm.src_pre[1] = nq;
      np = __fadd_rn(np, sv);
      nq = __fadd_rn(nq, sv);
    }
    prm.prev[i] = make_float2(np, nq);
  }
  if (prm.energy) {
    double e = static_cast<double>(e_acc);
    // threads of a CTA that returned early contribute nothing; reduce
    // within the warp of the active ones
    const unsigned mask = __activemask();
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double o = __shfl_down_sync(mask, e, off);
      if ((threadIdx.x + off) < 32 && ((mask >> (threadIdx.x + off)) & 1u)) e += o;
    }
    if (threadIdx.x == 0) {
      const int step = *prm.d_step + prm.step_offset;
      if (step >= 0 && step < prm.energy_cap) atomicAdd(&prm.energy[step], e);
    }
  }
}

template <int MEDIUM, bool SPONGE>
cudaError_t launch_exact_t(Sim *sim, const StepParams &prm) {
  const int ny = prm.y1 - prm.y0, nz = prm.z1 - prm.z0;
  const int chunks = (nz + prm.zchunk - 1) / prm.zchunk;
  // pitch and plane are multiples of four pairs; a caller's own buffers need
  // only be aligned to one pair
  const auto base = reinterpret_cast<uintptr_t>(prm.cur);
  if (base % 16 == 0) {
    const int nx = prm.x1 - (prm.x0 & ~1);
    dim3 grid((nx + kPairTX - 1) / kPairTX, (ny + kPairTY - 1) / kPairTY, chunks);
    exact_pair_kernel<MEDIUM, SPONGE><<<grid, kPairTX * kPairTY / 2, 0, sim->stream>>>(prm);
  } else {
    const int nx = prm.x1 - prm.x0;
    dim3 grid((nx + 31) / 32, (ny + 3) / 4, chunks);
    exact_kernel<MEDIUM, SPONGE><<<grid, dim3(32, 4), 0, sim->stream>>>(prm);
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_exact(Sim *sim, const StepParams &prm) {
  const bool sp = prm.sponge != nullptr;
  if (sim->medium == DC_GB300_MEDIUM_PRECOMP)
    return sp ? launch_exact_t<DC_GB300_MEDIUM_PRECOMP, true>(sim, prm)
              : launch_exact_t<DC_GB300_MEDIUM_PRECOMP, false>(sim, prm);
  return sp ? launch_exact_t<DC_GB300_MEDIUM_VPZ_VSV, true>(sim, prm)
            : launch_exact_t<DC_GB300_MEDIUM_VPZ_VSV, false>(sim, prm);
}

}  // namespace dcg
