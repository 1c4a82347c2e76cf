// Device helpers shared by the plane kernels.
#pragma once
#include "asg_internal.h"

// ---------------------------------------------------------------------------
// stability test and plane skip (uniform across a cluster)
// ---------------------------------------------------------------------------
ASG_DEV bool xy_should_skip(const XYParams& p) {
  if (*((volatile const unsigned*)p.status) != 0u) return true;
  if (p.check_stability) {
    const float m = __uint_as_float(*p.max_cur);
    const bool nan = (m != m) || isinf(m);
    const bool bad = nan || (p.stab_coef * (double)m > p.stab_thr);
    if (bad) {
      if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        if (atomicCAS(p.status, 0u, (unsigned)(nan ? -ASG_ERR_NAN : -ASG_ERR_STABILITY)) == 0u)
          *p.status_step = *p.step;
      }
      return true;
    }
  }
  return false;
}

ASG_DEV bool is_dc_or_nyq(int f, int nT) { return f == 0 || 2 * f == nT; }
