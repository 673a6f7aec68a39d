// The tile columns of a screen block's row that a splat's ellipse reaches,
// without testing them one by one (host and device).
//
// The tile test (ellipse_intersects_tile_gpu, render/kernels/binning.rs:37-96)
// compares the minimum of Q = a x^2 + 2 b x y + c y^2 over the tile's pixel
// centres' box (relative to the splat's centre) with a limit: the minimum of a
// convex form with its centre outside the box lies on the box's edges nearest
// to the centre, the two the test evaluates. Along a row of tiles, y in
// [y0, y1], a tile column [x0, x1] therefore passes exactly when it meets
// [xl, xr], the x-extent of {Q <= lim} in the strip: xr = (-b y + sqrt(a lim -
// (a c - b^2) y^2)) / a at the y of the strip nearest to that of the ellipse's
// rightmost point, xl alike. In binary32 both the test's Q and these ends carry
// errors, so a column counts as inside only if it meets the interval shrunk by
// a margin, as outside only if it misses the widened one, and in between the
// test itself decides.
//
// The margin: with kappa = a c / (a c - b^2), at Q = lim the three terms of Q
// sum to at most 4 kappa lim in magnitude, so the test's Q is within 16 kappa
// 2^-24 lim of the exact one; det = a c - b^2 is within 2 kappa 2^-24 of its
// value and a lim - det y^2 within 5 kappa 2^-24 a lim. All are changes of lim
// by less than kappa 1.4e-6 of it; eta = 4e-6 kappa is used. A change of s = a
// lim - det y^2 by d = eta a lim moves its root by at most min(d / sqrt(s),
// sqrt(d)) (doubled below, which also covers the root's approximation), and
// `eps` covers the rounding of the ends' last operations. Conics with kappa
// above 10^4 or out of the range of these bounds are left to the test.
#pragma once
#include <math.h>
#include <stdint.h>

#ifdef __CUDACC__
#define CGS_SPAN_HD __host__ __device__ __forceinline__
#else
#define CGS_SPAN_HD static inline
#endif

namespace cgs {

CGS_SPAN_HD float span_rsqrt(float x) {
#ifdef __CUDA_ARCH__
  return rsqrtf(x);
#elif defined(CGS_SPAN_RSQRT)
  return CGS_SPAN_RSQRT(x);  // a test's root with the device function's error
#else
  return 1.0f / sqrtf(x);
#endif
}
CGS_SPAN_HD int span_int(float v) {  // nearest integer, |v| < 2^22
  union {
    float f;
    int i;
  } u;
  u.f = v + 12582912.0f;
  return u.i - 0x4B400000;
}

// Per splat and block: what the rows share.
struct SplatSpan {
  float b, ia, alim, det, yx, ymax, d, eps, dx00, dx10, xlast, itw;
  bool ok;  // the bounds hold; otherwise every tile is tested
};

// (a, b, c) the conic, lim the test's limit; dx00, dx10 the block's first
// column's edges and xlast the last pixel column, relative to the centre; tw
// the tile width.
CGS_SPAN_HD SplatSpan splat_span(float a, float b, float c, float lim, float dx00, float dx10,
                                 float xlast, float tw) {
  SplatSpan s;
  const float ac = a * c;
  s.det = ac - b * b;
  s.ok = a > 1e-9f && c > 1e-9f && a < 1e6f && c < 1e6f && s.det * 1e4f > ac && lim >= 1e-5f &&
         lim < 100.0f && fabsf(dx00) < 1e5f;
  const float rd = span_rsqrt(s.det);      // 1 / sqrt(det)
  const float kappa = ac * rd * rd;
  const float eta = 4e-6f * kappa;
  const float rl = lim * span_rsqrt(lim);  // sqrt(lim)
  const float ra = span_rsqrt(a), rc = span_rsqrt(c);
  const float xmax = rl * rd * (c * rc);   // sqrt(lim c / det)
  s.b = b;
  s.ia = ra * ra;
  s.alim = a * lim;
  s.yx = -b * (rc * rc) * xmax;
  s.eps = 4e-6f * (xmax + fabsf(dx00) + 256.0f);
  s.ymax = rl * rd * (a * ra) * (1.0f + eta) + s.eps;
  s.d = eta * s.alim;
  s.dx00 = dx00;
  s.dx10 = dx10;
  s.xlast = xlast;
  s.itw = 1.0f / tw;
  return s;
}

// Columns [0, 7] of the row whose pixel centres lie in [y0, y1] (relative to
// the centre): `in` those that pass for sure, `out` those that may.
CGS_SPAN_HD void row_span(const SplatSpan& s, float y0, float y1, uint32_t& in, uint32_t& out) {
  const float lo = fmaxf(y0, -s.ymax), hi = fminf(y1, s.ymax);
  in = out = 0u;
  const float yr = fminf(fmaxf(s.yx, lo), hi), yl = fminf(fmaxf(-s.yx, lo), hi);
  const float sr = fmaxf(s.alim - s.det * (yr * yr), 0.0f);
  const float sl = fmaxf(s.alim - s.det * (yl * yl), 0.0f);
  const float rr = span_rsqrt(fmaxf(sr, s.d)), rl = span_rsqrt(fmaxf(sl, s.d));
  const float xr = (sr * rr - s.b * yr) * s.ia, mr = 2.0f * s.d * rr * s.ia + s.eps;
  const float xl = (-s.b * yl - sl * rl) * s.ia, ml = 2.0f * s.d * rl * s.ia + s.eps;
  const float ur = (xr - s.dx00) * s.itw, er = mr * s.itw;  // columns <= floor(ur)
  const float ul = (xl - s.dx10) * s.itw, el = ml * s.itw;  // columns >= ceil(ul)
  // bounded so that the conversions stay in range; floor and ceil as the
  // nearest integer of +- 1/2 (the margins are larger than a tie)
  const int hi_o = span_int(fminf(fmaxf(ur + er - 0.5f, -1.0f), 7.0f));
  const int hi_i = span_int(fminf(fmaxf(ur - er - 0.5f, -1.0f), 7.0f));
  const int lo_o = span_int(fminf(fmaxf(ul - el + 0.5f, 0.0f), 8.0f));
  const int lo_i = span_int(fminf(fmaxf(ul + el + 0.5f, 0.0f), 8.0f));
  if (lo > hi) return;
  if (xl - ml <= s.xlast) out = ((2u << (hi_o + 1)) >> 1) - 1u & ~((1u << lo_o) - 1u);
  // (a strip that barely reaches the ellipse has no interval to be sure of)
  if (xl + ml <= s.xlast && xl + ml <= xr - mr)
    in = ((2u << (hi_i + 1)) >> 1) - 1u & ~((1u << lo_i) - 1u);
}

}  // namespace cgs
