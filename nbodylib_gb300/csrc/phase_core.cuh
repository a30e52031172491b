// The phase-space distances in the reference's rounding.
#pragma once
#include "nbk_build.h"

namespace nbk {
namespace {

// PhaseDistSqd (DistFunc.h:41-49): ((((dx^2 + dy^2) + dz^2) + dvx^2) + dvy^2) + dvz^2.
__device__ __forceinline__ double phase_d2(const double x[6], const P4& p, const V4& v) {
  double a = dsub(x[0], p.x), b = dsub(x[1], p.y), c = dsub(x[2], p.z);
  double e = dsub(x[3], v.x), f = dsub(x[4], v.y), g = dsub(x[5], v.z);
  double s = dadd(dmul(a, a), dmul(b, b));
  s = dadd(s, dmul(c, c));
  s = dadd(s, dmul(e, e));
  s = dadd(s, dmul(f, f));
  return dadd(s, dmul(g, g));
}
// MetricDistSqd (DistFunc.h:58-65): total += (metric[i] * d) * d from 0, dimension order.
__device__ __forceinline__ double metric_d2(const double x[6], const P4& p, const V4& v,
                                            const double m[6]) {
  const double y[6] = {p.x, p.y, p.z, v.x, v.y, v.z};
  double total = 0.0;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    double d = dsub(x[k], y[k]);
    total = dadd(total, dmul(dmul(m[k], d), d));
  }
  return total;
}

}  // namespace
}  // namespace nbk
