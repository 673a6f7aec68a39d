// tile_span.h against the tile test, tile by tile, on random splats: prints
// the number of tiles it decides wrongly, the tiles it leaves to the test and
// the rows looked at. Arguments: splats, seed.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "tile_span.h"

static uint64_t state;
static double uniform() {
  uint64_t z = (state += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return ((z ^ (z >> 31)) >> 11) * (1.0 / 9007199254740992.0);
}
static float clamp(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }

// ellipse_intersects_tile_gpu (render/kernels/binning.rs:37-96), float32
static bool tile_test(float a, float b, float c, float lim, float x0, float x1, float y0, float y1) {
  const float xn = clamp(0.0f, x0, x1), yn = clamp(0.0f, y0, y1);
  const float y = clamp((-b * xn) / fmaxf(c, 1e-12f), y0, y1);
  const float q1 = ((a * xn) * xn + ((2.0f * b) * xn) * y) + (c * y) * y;
  const float x = clamp((-b * yn) / fmaxf(a, 1e-12f), x0, x1);
  const float q2 = ((a * x) * x + ((2.0f * b) * x) * yn) + (c * yn) * yn;
  return fminf(q1, q2) <= lim;
}

int main(int, char** av) {
  const long splats = atol(av[1]);
  state = strtoull(av[2], nullptr, 10) * 7919 + 1;
  long wrong = 0, open = 0, rows = 0, tests = 0;
  for (long i = 0; i < splats; ++i) {
    // round, long, axis-aligned and diagonal splats, some at whole and half pixels
    const double s1 = exp(uniform() * 7.0 - 0.6);
    double s2 = exp(uniform() * (uniform() < 0.3 ? 7.0 : 2.5) - 0.6), th = uniform() * 6.2831853;
    if (uniform() < 0.1) s2 = s1 * (0.999 + 0.002 * uniform());
    if (uniform() < 0.1) th = 0.0;
    if (uniform() < 0.02) th = 0.7853981634;
    const double cs = cos(th), sn = sin(th);
    const float xx = (float)(s1 * s1 * cs * cs + s2 * s2 * sn * sn + 0.3);
    const float yy = (float)(s1 * s1 * sn * sn + s2 * s2 * cs * cs + 0.3);
    const float xy = (float)((s1 * s1 - s2 * s2) * cs * sn);
    const float det = xx * yy - xy * xy;
    if (!(det > 1e-6f)) continue;
    const float inv = 1.0f / det, a = yy * inv, b = -xy * inv, c = xx * inv;
    const float alpha = (float)(uniform() < 0.1 ? 0.00393 + 1e-4 * uniform() : uniform());
    const float qmax = clamp(2.0f * logf(255.0f * alpha), 0.0f, 8.0f), lim = qmax + 1e-4f;
    const int tw = uniform() < 0.3 ? 8 : (uniform() < 0.5 ? 32 : 16), tall = tw == 8 ? 8 : 16;
    const int W = (int)(1 + uniform() * 7680), H = (int)(1 + uniform() * 4320);
    float mx = (float)(uniform() * (W + 200) - 100), my = (float)(uniform() * (H + 200) - 100);
    if (uniform() < 0.05) mx = floorf(mx) + 0.5f;
    if (uniform() < 0.05) my = floorf(my);
    const float cut = sqrtf(qmax);
    const float ex = clamp(ceilf(cut * sqrtf(xx)), 1.0f, 1024.0f);
    const float ey = clamp(ceilf(cut * sqrtf(yy)), 1.0f, 1024.0f);
    const int tx_n = (W + tw - 1) / tw, ty_n = (H + tall - 1) / tall;
    auto tile = [](float v, int n, int t) { return std::min(std::max((int)floorf(v / t), 0), n - 1); };
    const int x0 = tile(mx - ex, tx_n, tw), x1 = tile(mx + ex, tx_n, tw);
    const int y0 = tile(my - ey, ty_n, tall), y1 = tile(my + ey, ty_n, tall);
    const int bx = x0 / 8 + (int)(uniform() * (x1 / 8 - x0 / 8 + 1));
    const int by = y0 / 4 + (int)(uniform() * (y1 / 4 - y0 / 4 + 1));
    const float px0 = (float)(bx * 8 * tw) + 0.5f, xl = (float)W - 0.5f, yl = (float)H - 0.5f;
    const cgs::SplatSpan s = cgs::splat_span(a, b, c, lim, px0 - mx, (px0 + (tw - 1.0f)) - mx, xl - mx,
                                             (float)tw);
    if (!s.ok) continue;
    for (int r = 0; r < 4; ++r) {
      const int ty = by * 4 + r;
      if (ty < y0 || ty > y1) continue;
      const float p = (float)(ty * tall) + 0.5f;
      const float dy0 = p - my, dy1 = fminf(p + (tall - 1.0f), yl) - my;
      uint32_t in, out;
      cgs::row_span(s, dy0, dy1, in, out);
      ++rows;
      for (int k = 0; k < 8; ++k) {
        const int tx = bx * 8 + k;
        if (tx < x0 || tx > x1) continue;
        const float q = (float)(tx * tw) + 0.5f;
        const bool hit = tile_test(a, b, c, lim, q - mx, fminf(q + (tw - 1.0f), xl) - mx, dy0, dy1);
        const bool i_ = (in >> k) & 1u, o_ = (out >> k) & 1u;
        ++tests;
        wrong += (i_ && !hit) || (!o_ && hit) || (i_ && !o_);
        open += o_ && !i_;
      }
    }
  }
  printf("%ld %ld %ld %ld\n", wrong, open, rows, tests);
  return 0;
}
