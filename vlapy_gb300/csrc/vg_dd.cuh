// Double-double arithmetic of the host tables, by exact products (fma) and two-sums
#pragma once

#include <cmath>

namespace vg {

struct dd {
  double h, l;
};
inline dd dd_norm(double a, double b) {
  const double s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}
inline dd dd_mul(dd a, dd b) {
  const double p = a.h * b.h;
  return dd_norm(p, std::fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
inline dd dd_add(dd a, dd b) {
  const dd s = dd_norm(a.h, b.h);
  return dd_norm(s.h, s.l + (a.l + b.l));
}
// a / b, b a double
inline dd dd_div(dd a, double b) {
  const double q = a.h / b;
  return dd_norm(q, (std::fma(-q, b, a.h) + a.l) / b);
}

}  // namespace vg
