// Host build of recip_div.h for tests/test_recip_div_host.py.
#include <cstdint>
#include "recip_div.h"
// Returns the number of pairs whose checked quotient or reciprocal is not the IEEE one; *used
// counts the pairs that passed the checks.
extern "C" int64_t recip_div_check(const double *a, const double *b, int64_t n, int64_t *used) {
  int64_t bad = 0;
  *used = 0;
  for (int64_t i = 0; i < n; i++) {
    if (!div_b_ok(b[i]) || !div_a_ok(a[i])) continue;
    ++*used;
    const double y = div_recip(b[i]);
    bad += oco_d2u(y) != oco_d2u(1.0 / b[i]);
    bad += oco_d2u(div_quot(a[i], b[i], y)) != oco_d2u(a[i] / b[i]);
  }
  return bad;
}
extern "C" int recip_div_accepts(double a, double b) { return div_b_ok(b) & div_a_ok(a); }
