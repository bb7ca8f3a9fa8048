// Sphere test of the energy flux without a square root per mode.  Plain C++.
#pragma once
#include <cmath>

namespace ts {

// The largest x with sqrt(x) <= R, so that |K| <= R is K^2 <= x.  Every radius but NaN (which
// compares false either way) ends: no mode lies inside a negative radius, all inside an infinite
// one; for the others R * R is a few roundings from x (the largest finite double where it
// overflows).
inline double k2_limit(double R) {
  if (R < 0) return -1.0;
  if (std::isinf(R)) return R;
  double x = R * R;
  while (sqrt(x) > R) x = nextafter(x, 0.0);
  while (sqrt(nextafter(x, HUGE_VAL)) <= R) x = nextafter(x, HUGE_VAL);
  return x;
}

}  // namespace ts
