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

// Engquist-Majda correction of `cur` at edge coordinate i of n (weight w)
ASG_DEV float2 edge_correct(float2 prev, float2 cur, float2 next, int i, int n, float w, float cf,
                            float st, float inv2d, float invd) {
  float2 d;
  if (i == 0) d = cscale(csub(next, cur), invd);
  else if (i == n - 1) d = cscale(csub(cur, prev), invd);
  else d = cscale(csub(next, prev), inv2d);
  const float2 cd = make_float2(cf * d.y, -cf * d.x);
  const float2 P = (i < n / 2) ? make_float2(0.5f * (cur.x + cd.x), 0.5f * (cur.y + cd.y))
                               : make_float2(0.5f * (cur.x - cd.x), 0.5f * (cur.y - cd.y));
  return make_float2(cur.x - st * w * P.x, cur.y - st * w * P.y);
}

constexpr size_t LINE_SMEM = 72 * 1024;  // shared memory of a block at most

template <class K>
inline int line_smem_attr(K kern, bool* done) {
  if (*done) return ASG_OK;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LINE_SMEM) !=
      cudaSuccess)
    return ASG_ERR_CUDA;
  *done = true;
  return ASG_OK;
}
