// tile_span_check.cpp with roots that are off as the device's are: rsqrtf is
// within 2 units in the last place, here up to 4 either way, by the bits of the
// argument.
#include <cmath>
#include <cstdint>
#include <cstring>

static float off_rsqrt(float x) {
  const float r = (float)(1.0 / std::sqrt((double)x));
  uint32_t b, a;
  std::memcpy(&b, &r, 4);
  std::memcpy(&a, &x, 4);
  if (!(r > 1e-30f) || !(r < 1e30f)) return r;
  b += (a * 2654435761u >> 16) % 9u;
  b -= 4u;
  float o;
  std::memcpy(&o, &b, 4);
  return o;
}
#define CGS_SPAN_RSQRT off_rsqrt
#include "tile_span_check.cpp"
