// The stopping rule of the resident solve as a bound on ||r||^2 (host and device).
#ifndef FREHD_CG_LIMIT_H
#define FREHD_CG_LIMIT_H

#include <cmath>

#ifdef __CUDACC__
#define FREHD_HD __host__ __device__
#else
#define FREHD_HD
#endif

namespace frehd {

// The stopping rule (rtc.c:53: ||r|| < eps ||b||, or 1 + ||r|| = 1 for b = 0) as a
// bound on ||r||^2: the largest double whose root meets it (-1: none does), so that
// no iteration takes a root and every decision is the rule's own.  The bound lies
// within a few doubles of where the search starts, unless no root meets the rule:
// that is answered first (a negative eps would have searched all doubles below c^2).
FREHD_HD inline double res_limit(double bnorm, double eps) {
  const double c = eps * bnorm;
  if (bnorm != 0.0 && !(c > 0.0)) return -1.0;
  auto holds = [&](double rr) {
    const double rn = sqrt(rr);
    return rn < c || (bnorm == 0.0 && 1.0 + rn == 1.0);
  };
  double t = bnorm == 0.0 ? 0x1p-106 : c * c;
  while (holds(t)) t = nextafter(t, HUGE_VAL);
  while (t > 0.0 && !holds(t)) t = nextafter(t, 0.0);
  return holds(t) ? t : -1.0;
}

}  // namespace frehd

#endif
