// tti_fast.cu -- host side of the fast stencil: tile and z-chunk choice,
// tensor maps, and the dispatch to the kernels of tti_fast_inst.cu.
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "dc_internal.h"

namespace dcg {
namespace {

constexpr int kTX = kFastTX;

// The kernels of a coefficient form and tile height (8 or 16 rows of 32), and
// of its strips.
template <int FORM>
const FastOps &ops_of(int ty) {
  return ty == 16 ? fast_ops<FORM, kTX, 16>() : fast_ops<FORM, kTX, 8>();
}
const FastOps &ops_for(int form, int ty) {
  switch (form) {
    case CF_VV: return ops_of<CF_VV>(ty);
    case CF_F16: return ops_of<CF_F16>(ty);
    case CF_BF16: return ops_of<CF_BF16>(ty);
    default: return ops_of<CF_F32>(ty);
  }
}
const FastOps &strip_ops(int form) {
  switch (form) {
    case CF_VV: return fast_ops<CF_VV, kStripTX, kStripTY>();
    case CF_F16: return fast_ops<CF_F16, kStripTX, kStripTY>();
    case CF_BF16: return fast_ops<CF_BF16, kStripTX, kStripTY>();
    default: return fast_ops<CF_F32, kStripTX, kStripTY>();
  }
}

// 32 x 8 tiles (two CTAs of 128 threads per SM): with 32 x 16 and one CTA of
// 256 threads per SM nothing runs while the CTA waits at its barrier or fills
// its queues (616^3 FP32 step 2.19 vs 2.31 ms, 872 x 872 x 616 FP16 3.79 vs
// 4.35, 408^3 vpz/vsv 0.54 vs 0.62, 104^3 shot 2.3 vs 3.2 ms).  DC_GB300_FAST_TY=16 selects 32 x 16.
int chosen_ty() {
  const char *e = std::getenv("DC_GB300_FAST_TY");
  const int v = e ? std::atoi(e) : 0;
  return v == 16 ? 16 : 8;
}

long long div_up(long long a, long long b) { return (a + b - 1) / b; }

// CTAs of the fast sweep resident on the device at once.
long long slots_of(const Sim *sim) { return sim->fast_slots > 0 ? sim->fast_slots : 2 * 152; }

// Whether the last nx % 32 columns of a pass go to a launch of 16 x 16 tiles
// beside the one of 32 x 8 tiles: when they fit 16 columns, where a 32-column
// tile would compute more padding than points.  Per step without / with: 240 x
// 222 x 251 BF16 (8 of 232 columns left over) 114 / 110 us, 408^3 vpz/vsv (16 of
// 400) 541 / 525 us.  The FP32 ten-coefficient form waits for HBM, not for the
// padding's arithmetic (307 x 291 x 299: 255 / 262 us), and a box that does not
// give every SM a CTA takes as long as one CTA, however many there are: neither
// has a second launch.  A single narrow column (the x faces of the seven-box
// loop) is one launch of 16 x 16 tiles in every form.
bool has_strip(const Sim *sim, long long nx, long long ny) {
  const long long rest = nx % kTX;
  if (sim->maps_ty != 8 || rest < 1 || rest > kStripTX) return false;
  return nx < kTX || (sim->coef_form != CF_F32 &&
                      div_up(nx, kTX) * div_up(ny, 8) > slots_of(sim) / 2);
}

// CTAs per chunk of a pass.
long long tiles_of(long long nx, long long ny, int ty, bool strip) {
  if (strip) return nx / kTX * div_up(ny, ty) + div_up(ny, kStripTY);
  return std::max(1ll, div_up(nx, kTX)) * std::max(1ll, div_up(ny, ty));
}

}  // namespace

// z-chunk of a pass: a CTA sweeping zc output planes streams zc + 8 leading
// planes (the 8-plane warm-up of the z queues), and the CTAs run in waves of
// `fast_slots`, a partly filled last wave taking about as long as a full
// one.  So the pass costs ~ ceil(tiles * chunks / slots) * (zc + 8) plane
// sweeps; the chunk count minimising it is taken, the smaller on ties.
// Chunks of at least 32 planes (and at most 8) are always considered, within
// 1.2 % of the fastest of 1..8 on cubes of 200^3 to 616^3.  Shorter ones, down
// to kMinChunk planes, only while every SM gets one CTA at most: there the
// step takes as long as one CTA's sweep, and the warm-up planes cost nothing
// that was in use, not even when three simulations share the GPU.  Per step
// alone / of three at once, FP32: 56^3 28.2 -> 7.2 / 9.6 -> 3.5 us, 72^3 19.8
// -> 8.9 / 6.8 -> 4.6, 104^3 19.9 -> 16.1 / 10.4 -> 9.9; past one CTA per SM
// the second figure grows (104^3 with 8 chunks: 14.3 / 11.6).
// The energy log sums FP32 partials per column and chunk: with it on, only
// the long chunks are considered, so that its values stay as they were.
// DC_GB300_FAST_ZCHUNKS=<n> forces n chunks.
constexpr long long kLongChunk = 32, kMinChunk = 4;

FastShape fast_shape(const Sim *sim, long long nx, long long ny, long long nz) {
  const int ty = sim->maps_ty ? sim->maps_ty : chosen_ty();
  if (nz < 1) return FastShape{kTX, ty, 1};
  const long long tiles = tiles_of(nx, ny, ty, !sim->d_energy && has_strip(sim, nx, ny));
  const long long slots = slots_of(sim);
  const long long one_each = slots / 2;  // two CTAs fit an SM
  long long best_zc = nz, best_cost = -1;
  for (long long c = 1; c <= nz; ++c) {
    const long long zc = (nz + c - 1) / c;
    const long long chunks = (nz + zc - 1) / zc;
    if (c > 1 && (c > 8 || zc < kLongChunk) &&
        (zc < kMinChunk || sim->d_energy || tiles * chunks > one_each))
      break;
    const long long cost = (tiles * chunks + slots - 1) / slots * (zc + 8);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best_zc = zc;
    }
  }
  if (const char *e = std::getenv("DC_GB300_FAST_ZCHUNKS")) {
    const long long c = std::max(1, std::atoi(e));
    best_zc = (nz + c - 1) / c;
  }
  return FastShape{kTX, ty, static_cast<int>(best_zc)};
}

int fast_default_ty() { return chosen_ty(); }

bool fast_encode_pair_maps(const float2 *buf, long long sx, long long sy, long long sz,
                           long long pitch, int tx, int ty, CUtensorMap *halo, CUtensorMap *own,
                           std::string *err) {
  const uint32_t w = static_cast<uint32_t>(tx);
  const uint64_t dims3[3] = {static_cast<uint64_t>(sx), static_cast<uint64_t>(sy),
                             static_cast<uint64_t>(sz)};
  // (p, q) pair buffers: 8-byte elements
  const uint64_t str8[2] = {static_cast<uint64_t>(pitch) * 8,
                            static_cast<uint64_t>(pitch * sy) * 8};
  const uint32_t box_halo[3] = {w + 8, static_cast<uint32_t>(ty) + 8, kGroup};
  const uint32_t box_tile[3] = {w, static_cast<uint32_t>(ty), kGroup};
  const auto U64 = CU_TENSOR_MAP_DATA_TYPE_UINT64;
  return encode_tiled(halo, buf, 3, dims3, str8, box_halo, err, U64) &&
         encode_tiled(own, buf, 3, dims3, str8, box_tile, err, U64);
}

bool fast_encode_medium_maps(int form, const float *coef, const void *coef16, const float *vv,
                             const float4 *vbase, long long sx, long long sy, long long sz,
                             long long pitch, long long count, int tx, int ty,
                             CUtensorMap out[4], std::string *err) {
  const uint32_t w = static_cast<uint32_t>(tx);
  const uint64_t X = sx, Y = sy, Z = sz, P = pitch, PL = pitch * sy;
  const uint64_t dims3[3] = {X, Y, Z};
  const uint64_t str8[2] = {P * 8, PL * 8};
  const uint64_t str4[2] = {P * 4, PL * 4};
  const uint32_t box_tile[3] = {w, static_cast<uint32_t>(ty), kGroup};
  // 16-byte coefficient groups: two 8-byte elements per point, so a tile
  // row is one 512-byte box row (a box whose innermost extent is a single
  // 16-byte group makes the copy engine walk 32 x TY rows of 16 bytes)
  const uint64_t dims16[3] = {2 * X, Y, Z};
  const uint64_t str16[2] = {P * 16, PL * 16};
  const uint32_t box16[3] = {2 * w, static_cast<uint32_t>(ty), kGroup};
  const auto U64 = CU_TENSOR_MAP_DATA_TYPE_UINT64, U32 = CU_TENSOR_MAP_DATA_TYPE_UINT32;
  const long long cnt = count;
  // out[0] = L (cxx, cyy, cxy, czz), out[1] = O1, out[2] = O2, out[3] = the
  // FP16 form's row bases
  bool ok = false;
  switch (form) {
    case CF_F32: {
      const char *c = reinterpret_cast<const char *>(coef);
      ok = encode_tiled(&out[0], c, 3, dims16, str16, box16, err, U64) &&
           encode_tiled(&out[1], c + cnt * 16, 3, dims16, str16, box16, err, U64) &&
           encode_tiled(&out[2], c + cnt * 32, 3, dims3, str8, box_tile, err, U64);
      break;
    }
    case CF_VV:
      ok = encode_tiled(&out[1], vv, 3, dims3, str8, box_tile, err, U64);
      out[0] = out[2] = out[1];  // unused
      break;
    default: {  // CF_F16, CF_BF16: 8-byte L, 8-byte O1, 4-byte O2
      const char *h = static_cast<const char *>(coef16);
      ok = encode_tiled(&out[0], h, 3, dims3, str8, box_tile, err, U64) &&
           encode_tiled(&out[1], h + cnt * 8, 3, dims3, str8, box_tile, err, U64) &&
           encode_tiled(&out[2], h + cnt * 16, 3, dims3, str4, box_tile, err, U32);
    }
  }
  if (!ok) return false;
  if (form != CF_F16) {
    out[3] = out[2];  // unused
    return true;
  }
  // row bases: [sz][sy] float4 as a 2-D tensor of 8-byte elements, x = 2 y
  const uint64_t dims_vb[2] = {2 * Y, Z};
  const uint64_t str_vb[1] = {Y * 16};
  const uint32_t box_vb[2] = {2 * static_cast<uint32_t>(ty), kGroup};
  return encode_tiled(&out[3], vbase, 2, dims_vb, str_vb, box_vb, err, U64);
}

bool fast_encode_maps(Sim *sim, std::string *err) {
  // dynamic shared memory above 48 KB must be enabled per kernel and device
  // (done here, before any stream capture)
  const int kTY = chosen_ty();
  cudaError_t ae = ops_for(sim->coef_form, kTY).attrs();
  if (ae == cudaSuccess) ae = strip_ops(sim->coef_form).attrs();
  if (ae != cudaSuccess) {
    *err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(ae);
    return false;
  }
  auto encode = [&](FastMaps &m, int tx, int ty) {
    for (int b = 0; b < 2; ++b)
      if (!fast_encode_pair_maps(sim->pq[b], sim->sx, sim->sy, sim->sz, sim->pitch, tx, ty,
                                 &m.halo[b], &m.own[b], err))
        return false;
    return fast_encode_medium_maps(sim->coef_form, sim->coef, sim->coef16, sim->vv, sim->vbase,
                                   sim->sx, sim->sy, sim->sz, sim->pitch, sim->count, tx, ty, m.c,
                                   err);
  };
  if (!encode(sim->maps, kTX, kTY) || !encode(sim->strip_maps, kStripTX, kStripTY)) return false;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, sim->device) != cudaSuccess)
    sms = 0;
  const int per_sm = ops_for(sim->coef_form, kTY).occupancy();
  sim->fast_slots = sms > 0 && per_sm > 0 ? sms * per_sm : 0;
  cudaGetLastError();  // a failed occupancy query leaves the fallback slot count
  sim->maps_ty = kTY;
  return true;
}

bool fast_tile_rows_valid(int ty) { return ty == 8 || ty == 16; }

cudaError_t batch_prepare(int ty, int form) { return ops_for(form, ty).batch_attrs(); }

int batch_blocks_per_sm(int ty, int form, bool iso, bool sponge) {
  return ops_for(form, ty).batch_occupancy(iso, sponge);
}

cudaError_t launch_batch(cudaStream_t st, const BatchLaunch &bl, int ty, int form, bool iso,
                         bool sponge, bool loop, int blocks) {
  return ops_for(form, ty).launch_batch(st, bl, iso, sponge, loop, blocks);
}

int fast_launches(const Sim *sim, long long nx, long long ny) {
  return has_strip(sim, nx, ny) && nx >= kTX ? 2 : 1;
}

cudaError_t launch_fast(Sim *sim, const StepParams &prm, int cur_buf, int prev_buf) {
  const FastOps &ops = ops_for(sim->coef_form, sim->maps_ty);
  const long long nx = prm.x1 - prm.tile_x0, ny = prm.y1 - prm.tile_y0;
  if (!has_strip(sim, nx, ny)) return ops.launch(sim, sim->maps, prm, cur_buf, prev_buf);
  // the strip first: its few CTAs start with the first wave of the others,
  // which share no point with it
  const int cut = prm.tile_x0 + static_cast<int>(nx / kTX * kTX);
  StepParams p = prm;
  p.tile_x0 = cut;
  p.x0 = std::max(prm.x0, cut);
  const cudaError_t e =
      strip_ops(sim->coef_form).launch(sim, sim->strip_maps, p, cur_buf, prev_buf);
  if (e != cudaSuccess || cut == prm.tile_x0) return e;
  p = prm;
  p.x1 = cut;
  p.beside = 1;
  return ops.launch(sim, sim->maps, p, cur_buf, prev_buf);
}

}  // namespace dcg
