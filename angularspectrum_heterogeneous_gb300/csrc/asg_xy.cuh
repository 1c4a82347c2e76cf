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

// ---------------------------------------------------------------------------
// (x, y, omega) epilogue on rows [0, R) of a plane held in shared memory.
// Row r is global x = x0 + r; element (r, y) at base[r*RS + POS(y)].
// halo_lo / halo_hi: rows x0-1 and x0+R (null at the global edges).
// PART: 0 all of it, bins 0 and nT/2 made real first; otherwise without that, 1 what acts
// along x (it commutes with the y transform), 2 what acts along y and the screens.
// ---------------------------------------------------------------------------
struct PosIdentity {
  ASG_DEV static int pos(int s) { return s; }
};

template <class POS, int PART = 0>
ASG_DEV void epilogue(const XYParams& p, int plane, int f, float2* base, int RS, int R, int x0,
                      const float2* halo_lo, const float2* halo_hi) {
  const int X = p.X, Y = p.Y;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const bool realify = PART == 0 && is_dc_or_nyq(f, p.nT);
  // Re() after the attenuation inverse (irfft between reference steps)
  if (realify) {
    for (int i = tid; i < R * Y; i += nthr) {
      const int r = i / Y, y = i - (i / Y) * Y;
      base[r * RS + POS::pos(y)].y = 0.f;
    }
    __syncthreads();
  }
  if (p.epi & EPI_FREQW) {
    const float e = p.fw_exp[plane];
    for (int i = tid; i < R * Y; i += nthr) {
      const int r = i / Y, y = i - (i / Y) * Y;
      const float lx = PART == 2 ? 0.f : p.fw_lx[x0 + r], ly = PART == 1 ? 0.f : p.fw_ly[y];
      const float g = exp2f(e * (lx + ly));
      float2& v = base[r * RS + POS::pos(y)];
      v = cscale(v, g);
    }
    __syncthreads();
  }
  if (p.epi & EPI_SUPERABS) {
    const float c = p.sa_coef[plane];  // coeff = -i c
    const float s = p.sa_strength;
    // ---- x edges: one thread per y walks the rows, keeping the originals ----
    for (int y = tid; PART != 2 && y < Y; y += nthr) {
      const int py = POS::pos(y);
      float2 prev = halo_lo ? halo_lo[py] : make_float2(0.f, 0.f);
      float2 cur = base[py];
      for (int r = 0; r < R; ++r) {
        const int x = x0 + r;
        float2 next = (r + 1 < R) ? base[(r + 1) * RS + py]
                                  : (halo_hi ? halo_hi[py] : make_float2(0.f, 0.f));
        const float w = p.sa_wx[x];
        if (w != 0.f) {
          float2 d;
          if (x == 0) d = cscale(csub(next, cur), p.sa_invdx);
          else if (x == X - 1) d = cscale(csub(cur, prev), p.sa_invdx);
          else d = cscale(csub(next, prev), p.sa_inv2dx);
          // coeff * d = -i c d = (c d.y, -c d.x)
          const float2 cd = make_float2(c * d.y, -c * d.x);
          const bool lo = x < X / 2;
          const float2 P = lo ? make_float2(0.5f * (cur.x + cd.x), 0.5f * (cur.y + cd.y))
                              : make_float2(0.5f * (cur.x - cd.x), 0.5f * (cur.y - cd.y));
          base[r * RS + py] = make_float2(cur.x - s * w * P.x, cur.y - s * w * P.y);
        }
        prev = cur;
        cur = next;
      }
    }
    __syncthreads();
    // ---- y edges on the x-corrected values: one warp per row, 32 y at a
    //      time; neighbours come from shuffles, the chunk borders from the
    //      original values kept before they are overwritten ----
    const int lane = tid & 31, warp = tid >> 5, nw = nthr >> 5;
    for (int r = warp; PART != 1 && r < R; r += nw) {
      float2* row = base + r * RS;
      float2 prev_last = make_float2(0.f, 0.f);  // original value at y0-1
      for (int y0 = 0; y0 < Y; y0 += 32) {
        const int y = y0 + lane;
        const float2 cur = (y < Y) ? row[POS::pos(y)] : make_float2(0.f, 0.f);
        float2 left, right;
        left.x = __shfl_up_sync(0xffffffffu, cur.x, 1);
        left.y = __shfl_up_sync(0xffffffffu, cur.y, 1);
        right.x = __shfl_down_sync(0xffffffffu, cur.x, 1);
        right.y = __shfl_down_sync(0xffffffffu, cur.y, 1);
        if (lane == 0) left = prev_last;
        if (lane == 31 && y + 1 < Y) right = row[POS::pos(y + 1)];
        float2 res = cur;
        if (y < Y) {
          const float w = p.sa_wy[y];
          if (w != 0.f) {
            float2 d;
            if (y == 0) d = cscale(csub(right, cur), p.sa_invdy);
            else if (y == Y - 1) d = cscale(csub(cur, left), p.sa_invdy);
            else d = cscale(csub(right, left), p.sa_inv2dy);
            const float2 cd = make_float2(c * d.y, -c * d.x);
            const bool lo = y < Y / 2;
            const float2 P = lo ? make_float2(0.5f * (cur.x + cd.x), 0.5f * (cur.y + cd.y))
                                : make_float2(0.5f * (cur.x - cd.x), 0.5f * (cur.y - cd.y));
            res = make_float2(cur.x - s * w * P.x, cur.y - s * w * P.y);
          }
          if (realify) res.y = 0.f;
        }
        prev_last.x = __shfl_sync(0xffffffffu, cur.x, 31);
        prev_last.y = __shfl_sync(0xffffffffu, cur.y, 31);
        __syncwarp();
        if (y < Y) row[POS::pos(y)] = res;
        __syncwarp();
      }
    }
    __syncthreads();
  }
  for (int k = 0; PART != 1 && k < p.nscreens; ++k) {
    const float fs = p.screen_fscale[plane];
    const ScreenDev sc = p.screens[k];
    for (int i = tid; i < R * Y; i += nthr) {
      const int r = i / Y, y = i - (i / Y) * Y;
      const size_t g = (size_t)(x0 + r) * Y + y;
      float sn, cs;
      sincosf(sc.phase[g] * fs, &sn, &cs);
      float2 v = cmul(base[r * RS + POS::pos(y)], make_float2(cs, -sn));
      if (sc.amp != nullptr) {
        const float a = fminf(fmaxf(sc.amp[g], 1e-6f), 1.0f);
        v = cscale(v, exp2f(fs * log2f(a)));
      }
      if (realify) v.y = 0.f;
      base[r * RS + POS::pos(y)] = v;
    }
    __syncthreads();
  }
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
