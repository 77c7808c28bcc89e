// Host build of oco_log_nb for tests/test_ocomath_nb.py.
#include "ocomath.h"
// Mismatches of oco_log_nb with oco_log over n arguments where it returns 1; *used counts those.
extern "C" int64_t log_nb_check(const double *x, int64_t n, int64_t *used) {
  int64_t bad = 0;
  *used = 0;
  for (int64_t i = 0; i < n; i++) {
    double r;
    if (!oco_log_nb(x[i], &r)) continue;
    ++*used;
    bad += oco_d2u(r) != oco_d2u(oco_log(x[i]));
  }
  return bad;
}
