// s2d_host_checks.h -- checks of host fields before they are stored on the device.  Whole-range
// scans without early exits, so that the compiler vectorises them.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cstring>

namespace s2d {

// whether every float's exponent says finite
__attribute__((optimize("O3"))) inline bool all_finite(const float* v, size_t count) {
  uint32_t bad = 0;
  for (size_t i = 0; i < count; ++i) {
    uint32_t u;
    std::memcpy(&u, v + i, sizeof(u));
    bad |= (u & 0x7f800000u) == 0x7f800000u;
  }
  return bad == 0;
}
// whether every float is +-0
__attribute__((optimize("O3"))) inline bool all_zero(const float* v, size_t count) {
  uint32_t bits = 0;
  for (size_t i = 0; i < count; ++i) {
    uint32_t u;
    std::memcpy(&u, v + i, sizeof(u));
    bits |= u & 0x7fffffffu;
  }
  return bits == 0;
}
// whether a (prefix of a) complex n x n spectrum, `count` floats of it, is zero outside the
// dealias band
inline bool band_limited(const float* w, size_t count, int n) {
  auto zero = [&](size_t lo, size_t hi) {
    if (hi > count) hi = count;
    return lo >= hi || all_zero(w + lo, hi - lo);
  };
  for (int r = 0; r < n; ++r) {
    const size_t row = (size_t)2 * n * r;
    const bool in = r <= n / 3 || r >= n - n / 3;
    if (!zero(row + (in ? 2 * (size_t)(n / 3 + 1) : 0), row + (in ? 2 * (size_t)(n - n / 3) : 2 * (size_t)n))) return false;
  }
  return true;
}

}  // namespace s2d
