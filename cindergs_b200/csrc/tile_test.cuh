// The pieces of the ellipse-vs-tile test (ellipse_intersects_tile_gpu,
// render/kernels/binning.rs:37-96), every product and sum rounded separately
// in the reference's operand order: the splat's tile box and the pixel centres,
// which the projection, the entry binning and the screen-block lists share, and
// the column and row terms of a tile with their divisions, for the entry
// binning.
#pragma once
#include "kernels.h"

namespace cgs {

struct SplatBox {
  bool valid;
  uint32_t x0, x1, y0, y1;
  float mu_x, mu_y, ca, cb, cc, alpha;
};

__device__ __forceinline__ uint32_t tile_coord(float v, int32_t hi, float inv_tile) {
  // clamp(floor(v / tile) as i32, 0, hi) with Rust's saturating cast; the
  // tile size is a power of two, so v * (1 / tile) is the exact quotient.
  const float f = floorf(__fmul_rn(v, inv_tile));
  int32_t i = __float2int_rz(f);  // saturates, NaN -> 0
  i = i < 0 ? 0 : (i > hi ? hi : i);
  return (uint32_t)i;
}

// Box of splat s; Args holds recs, tiles_x, tiles_y, tile_w_log2, tile_h_log2.
template <class Args>
__device__ __forceinline__ SplatBox load_box(const Args& a, uint32_t s, uint32_t active) {
  SplatBox b;
  b.valid = false;
  b.x0 = b.x1 = b.y0 = b.y1 = 0;
  b.mu_x = b.mu_y = b.ca = b.cb = b.cc = b.alpha = 0.0f;
  if (s >= active || a.tiles_x == 0 || a.tiles_y == 0) return b;
  const float4 cc4 = a.recs[s].cc;
  const uint32_t p = __float_as_uint(cc4.w);
  if (p == 0u) return b;
  const float4 geo = a.recs[s].geo;
  const float ext_x = (float)(p & 0xFFFFu), ext_y = (float)((p >> 16) & 0xFFFFu);
  b.mu_x = geo.x;
  b.mu_y = geo.y;
  b.ca = geo.z;
  b.cb = geo.w;
  b.cc = cc4.x;
  b.alpha = cc4.y;
  const int32_t mx = (int32_t)a.tiles_x - 1, my = (int32_t)a.tiles_y - 1;
  const float itw = __uint_as_float((127u - a.tile_w_log2) << 23);  // 2^-lw
  const float ith = __uint_as_float((127u - a.tile_h_log2) << 23);
  b.x0 = tile_coord(__fsub_rn(b.mu_x, ext_x), mx, itw);
  b.x1 = tile_coord(__fadd_rn(b.mu_x, ext_x), mx, itw);
  b.y0 = tile_coord(__fsub_rn(b.mu_y, ext_y), my, ith);
  b.y1 = tile_coord(__fadd_rn(b.mu_y, ext_y), my, ith);
  // ellipse_intersects_tile_gpu returns false for every tile when alpha < 1/255.
  b.valid = !(b.alpha < (1.0f / 255.0f));
  return b;
}

// (float)v + 0.5f for v < 2^22, exactly: 2^23 + v is exact in binary32 and
// the subtraction of 2^23 - 0.5 is exact (Sterbenz), so the result equals the
// reference's integer-to-float conversion plus one half without a conversion.
__device__ __forceinline__ float pixel_center(uint32_t v) {
  return __fsub_rn(__int_as_float(0x4B000000u | v), 8388607.5f);
}

// n / d correctly rounded to binary32, for d > 0, from y = RN64(1 / d) (one
// binary64 reciprocal per splat instead of a binary32 division per tile).
// The binary64 product n * y is within 2^-52 (relative) of n / d. A quotient
// of two binary32 numbers is never closer than 2^-49 (relative) to a midpoint
// of two binary32 neighbours in the normal range: if n / d = m (1 + e) with m
// a midpoint, m = M 2^k with M odd and M >= 2^24, then n - d m is a nonzero
// multiple of 2^k ulp(d) -- an odd factor of M >= 2^24 cannot divide a 24-bit
// significand -- so |e| >= 2^-49. Hence n * y and n / d round to the same
// binary32 value. Results below 2^-125 in magnitude, where the binary32 grid
// is finer relative to the value than that argument assumes, use the binary32
// division itself; zero stays a signed zero.
static __device__ __noinline__ float div_ieee(float n, float d) { return __fdiv_rn(n, d); }

__device__ __forceinline__ float div_rcp64(float n, float d, double y) {
  const double q = __dmul_rn((double)n, y);
  float r = __double2float_rn(q);
  // a call, so that the compiler cannot turn the rare case into a division
  // on every lane
  if (q != 0.0 && fabs(q) < 0x1p-125) r = div_ieee(n, d);
  return r;
}

// Column terms of a splat's tile column tx (the parts of the test that depend
// on the column alone): x edges, the y minimiser at the column's nearest x
// (before its clamp to the row), a x_near^2.
__device__ __forceinline__ float4 col_terms(uint32_t tx, uint32_t lw, uint32_t wm1, const float4 geo,
                                            const float4 con, const double2 rcp) {
  const uint32_t xs = tx << lw;
  const float dx0 = __fsub_rn(pixel_center(xs), geo.x);
  const float dx1 = __fsub_rn(pixel_center(min(xs + ((1u << lw) - 1u), wm1)), geo.x);
  const float x_near = clampf(0.0f, dx0, dx1);
  return make_float4(dx0, dx1, div_rcp64(__fmul_rn(geo.z, x_near), con.w, rcp.x),
                     __fmul_rn(__fmul_rn(con.x, x_near), x_near));
}

// Row terms of tile row ty: y edges, the x minimiser at the row's nearest y
// (before its clamp to the column), c y_near^2.
__device__ __forceinline__ float4 row_terms(uint32_t ty, uint32_t lh, uint32_t hm1, const float4 geo,
                                            const float4 con, const double2 rcp) {
  const uint32_t ys = ty << lh;
  const float dy0 = __fsub_rn(pixel_center(ys), geo.y);
  const float dy1 = __fsub_rn(pixel_center(min(ys + ((1u << lh) - 1u), hm1)), geo.y);
  const float y_near = clampf(0.0f, dy0, dy1);
  return make_float4(dy0, dy1, div_rcp64(__fmul_rn(geo.z, y_near), con.z, rcp.y),
                     __fmul_rn(__fmul_rn(con.y, y_near), y_near));
}

}  // namespace cgs
