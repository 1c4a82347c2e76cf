// Small planes of any size in one launch per stage: a block holds a plane in shared
// memory and runs the transforms along y and x, the multiplier, the inverse transforms and
// the (x, y, omega) epilogue on it.
//
// Bounded by latency, the data being a few KB: launches, barriers, dependent loads and
// above all instruction fetch, since each pass over a plane is short and its code cold.
// Row, column and row pass of such a plane cost three launches, 21 to 25 us per stage
// however small it is; for 65 planes one block each takes 10 to 14 up to 32 x 32, 18 for
// 48 x 48 (16 x 16: 12 with 65 planes, 14 with 1025).  Hence small radices (a DFT of 12 or
// 16 points per thread took 14 to 16 us), one copy of a pass's code for both axes and sums
// over odd primes spread over the block's threads where these are enough (17 x 17 22 -> 15
// us), else rolled.
//
// A line is transformed in its own slots: a pass of radix r on sublines of m samples takes
// the samples b + (m / r) a to their DFT's bins ka at b + (m / r) ka, times W_m^(b ka), and
// leaves sublines of m / r.  The inverse takes the passes back.  All factors are two floats
// (see asg_lines.cuh).
//
// Reference semantics: see asg_xykernel.cu.
#include <algorithm>

#include "asg_internal.h"
#include "asg_lines.cuh"
#include "asg_xy.cuh"

ASG_DEFINE_LINE_ROOT_UPLOADER(asg_roots_upload_xyplane)

namespace {

constexpr int PLANE_NT = 256;

// The lines of an axis: line l at base + l ls, its sample j es further per step.
struct Lines {
  float2* base;
  int count, ls, es;
};

// One pass of radix R, a thread per DFT, lanes along the lines.
template <int R, bool INV>
ASG_DEV void pass_small(const Lines& L, const PlaneAxis& ax, int m) {
  const int mp = m / R, ts = ax.n / m, st = mp * L.es;
  for (int it = threadIdx.x; it < L.count * (ax.n / R); it += blockDim.x) {
    const int j = it / L.count, l = it - j * L.count, sub = j / mp, b = j - sub * mp;
    float2* s = L.base + l * L.ls + (sub * m + b) * L.es;
    float2 v[R];
#pragma unroll
    for (int a = 0; a < R; ++a) v[a] = s[a * st];
    if (INV && mp > 1) {
#pragma unroll
      for (int a = 1; a < R; ++a) v[a] = mulc_f4(v[a], __ldg(ax.tw + ts * b * a));
    }
    ldft<R, INV>(v);
    if (!INV && mp > 1) {
#pragma unroll
      for (int a = 1; a < R; ++a) v[a] = mul_f4(v[a], __ldg(ax.tw + ts * b * a));
    }
#pragma unroll
    for (int a = 0; a < R; ++a) s[a * st] = v[a];
  }
  __syncthreads();
}

// The same for a larger odd prime R, by the sums of ldft in a loop over the bins (unrolled, the
// code of 17 points takes longer to fetch than to run).
template <int R, bool INV>
ASG_DEV void pass_prime(const Lines& L, const PlaneAxis& ax, int m) {
  constexpr int H = (R - 1) / 2;
  const int mp = m / R, ts = ax.n / m, st = mp * L.es;
  for (int it = threadIdx.x; it < L.count * (ax.n / R); it += blockDim.x) {
    const int j = it / L.count, l = it - j * L.count, sub = j / mp, b = j - sub * mp;
    float2* s = L.base + l * L.ls + (sub * m + b) * L.es;
    const float2 v0 = s[0];
    float2 t[H], d[H], x0 = v0;
#pragma unroll
    for (int a = 1; a <= H; ++a) {
      float2 u = s[a * st], w = s[(R - a) * st];
      if (INV && mp > 1) {
        u = mulc_f4(u, __ldg(ax.tw + ts * b * a));
        w = mulc_f4(w, __ldg(ax.tw + ts * b * (R - a)));
      }
      t[a - 1] = cadd(u, w);
      d[a - 1] = csub(u, w);
      x0 = cadd(x0, t[a - 1]);
    }
    s[0] = x0;
#pragma unroll 1
    for (int k = 1; k <= H; ++k) {
      float2 r = make_float2(0.f, 0.f), q = r;
      int e = 0;
#pragma unroll
      for (int a = 0; a < H; ++a) {  // the roots' low parts first (see ldft)
        e = e + k < R ? e + k : e + k - R;
        const float4 w = c_roots[R * (R - 1) / 2 + e];
        r = make_float2(fmaf(t[a].x, w.z, r.x), fmaf(t[a].y, w.z, r.y));
        q = make_float2(fmaf(d[a].x, w.w, q.x), fmaf(d[a].y, w.w, q.y));
      }
      e = 0;
#pragma unroll
      for (int a = 0; a < H; ++a) {
        e = e + k < R ? e + k : e + k - R;
        const float4 w = c_roots[R * (R - 1) / 2 + e];
        r = make_float2(fmaf(t[a].x, w.x, r.x), fmaf(t[a].y, w.x, r.y));
        q = make_float2(fmaf(d[a].x, w.y, q.x), fmaf(d[a].y, w.y, q.y));
      }
      r = cadd(r, v0);
      const float2 iq = make_float2(-q.y, q.x);
      float2 x = INV ? csub(r, iq) : cadd(r, iq), y = INV ? cadd(r, iq) : csub(r, iq);
      if (!INV && mp > 1) {
        x = mul_f4(x, __ldg(ax.tw + ts * b * k));
        y = mul_f4(y, __ldg(ax.tw + ts * b * (R - k)));
      }
      s[k * st] = x;
      s[(R - k) * st] = y;
    }
  }
  __syncthreads();
}

// The same, a thread per DFT and pair of bins k, R - k (k = 0: the plain sum), for a block with a
// thread for each: all inputs are read before any bin is written.  A rolled sum leaves most of
// a small plane's threads idle (17 x 17 18 -> 15 us per stage, 11 x 11 17 -> 13).
template <bool INV>
ASG_DEV void pass_spread(const Lines& L, const PlaneAxis& ax, int R, int m) {
  const int H = (R - 1) / 2, mp = m / R, ts = ax.n / m, st = mp * L.es;
  const int rs = ax.n / R;  // exp(-2 pi i e / R) at tw[e rs]
  const int dfts = L.count * rs, k = threadIdx.x / dfts, it = threadIdx.x - k * dfts;
  const bool on = k <= H, turn = mp > 1;
  const int j = it / L.count, l = it - j * L.count, sub = j / mp, b = j - sub * mp;
  float2* s = L.base + l * L.ls + (sub * m + b) * L.es;
  float2 x, y;
  if (on) {
    const float2 v0 = s[0];
    float2 r = make_float2(0.f, 0.f), q = r;
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {  // the roots' low parts first (see ldft)
      if (part == 1 && k == 0) r = v0;
      int e = 0;
#pragma unroll 4
      for (int a = 1; a <= H; ++a) {
        float2 u = s[a * st], w = s[(R - a) * st];
        if (INV && turn) {
          u = mulc_f4(u, __ldg(ax.tw + ts * b * a));
          w = mulc_f4(w, __ldg(ax.tw + ts * b * (R - a)));
        }
        e = e + k < R ? e + k : e + k - R;
        const float4 f = __ldg(ax.tw + e * rs);
        const float c = part ? f.x : f.z, sn = part ? f.y : f.w;
        const float2 t = cadd(u, w), d = csub(u, w);
        r = make_float2(fmaf(t.x, c, r.x), fmaf(t.y, c, r.y));
        q = make_float2(fmaf(d.x, sn, q.x), fmaf(d.y, sn, q.y));
      }
    }
    if (k > 0) r = cadd(r, v0);
    const float2 iq = make_float2(-q.y, q.x);
    x = INV ? csub(r, iq) : cadd(r, iq);
    y = INV ? cadd(r, iq) : csub(r, iq);
    if (!INV && turn && k > 0) {
      x = mul_f4(x, __ldg(ax.tw + ts * b * k));
      y = mul_f4(y, __ldg(ax.tw + ts * b * (R - k)));
    }
  }
  __syncthreads();
  if (on) {
    s[k * st] = x;
    if (k > 0) s[(R - k) * st] = y;
  }
  __syncthreads();
}

// All passes of an axis (not inlined: the second axis finds the code fetched).
template <bool INV>
__device__ __noinline__ void plane_passes(Lines L, PlaneAxis ax) {
  int np = 0;
  while ((ax.radices >> (8 * np)) & 255) ++np;
  int m = INV ? 1 : ax.n;
#pragma unroll 1
  for (int i = 0; i < np; ++i) {
    const int r = (int)(ax.radices >> (8 * (INV ? np - 1 - i : i))) & 255;
    if (INV) m *= r;
    const int spread = r > 9 ? asg_plane_spread(r, ax.n, L.count) : 0;
    if (spread > 0 && spread <= (int)blockDim.x) {
      pass_spread<INV>(L, ax, r, m);
    } else switch (r) {
      case 2: pass_small<2, INV>(L, ax, m); break;
      case 3: pass_small<3, INV>(L, ax, m); break;
      case 4: pass_small<4, INV>(L, ax, m); break;
      case 5: pass_small<5, INV>(L, ax, m); break;
      case 6: pass_small<6, INV>(L, ax, m); break;
      case 7: pass_small<7, INV>(L, ax, m); break;
      case 8: pass_small<8, INV>(L, ax, m); break;
      case 9: pass_small<9, INV>(L, ax, m); break;
      case 11: pass_prime<11, INV>(L, ax, m); break;
      case 13: pass_prime<13, INV>(L, ax, m); break;
      case 17: pass_prime<17, INV>(L, ax, m); break;
      default: break;
    }
    if (!INV) m /= r;
  }
}

__global__ void __launch_bounds__(PLANE_NT, 3) xy_plane(XYParams p, PlaneAxis axx, PlaneAxis axy,
                                                     int RS) {
  pdl_wait();
  if (xy_should_skip(p)) return;
  extern __shared__ float4 smraw[];
  float2* P = reinterpret_cast<float2*>(smraw);  // sample (x, y) at x RS + y, RS odd
  __shared__ float red[2][PLANE_NT / 32];
  const int X = p.X, Y = p.Y, tid = threadIdx.x, NT = blockDim.x;
  const int plane = blockIdx.x, f = p.f_of_plane[plane];
  float2* g = p.spec + (size_t)plane * X * Y;
  if (p.zero_dc_nyq && is_dc_or_nyq(f, p.nT)) {
    for (int i = tid; i < X * Y; i += NT) g[i] = make_float2(0.f, 0.f);
    return;
  }
  // fn(i, x, y) over the plane
  const int dx = NT / Y, dy = NT - dx * Y;
  auto samples = [&](auto fn) {
#pragma unroll 4
    for (int i = tid, x = tid / Y, y = tid - x * Y; i < X * Y; i += NT) {
      fn(i, x, y);
      x += dx;
      y += dy;
      if (y >= Y) {
        y -= Y;
        ++x;
      }
    }
  };
  const Lines rows = {P, X, RS, 1}, cols = {P, Y, 1, RS};
  samples([&](int i, int x, int y) { P[x * RS + y] = g[i]; });
  __syncthreads();
  plane_passes<false>(rows, axy);
  plane_passes<false>(cols, axx);
  if (p.power_only) {
    const float* obl = p.obl_table + (size_t)plane * p.ncx * p.ncy;
    float psum = 0.f, pden = 0.f;
    samples([&](int, int x, int y) {
      const float o = __ldg(obl + __ldg(p.cls_x + x) * p.ncy + __ldg(p.cls_y + y));
      const float2 v = P[x * RS + y];
      const float q = v.x * v.x + v.y * v.y;
      psum = fmaf(q, o, psum);
      pden += (o > 0.f) ? q : 0.f;
    });
    psum = warp_sum(psum);
    pden = warp_sum(pden);
    if ((tid & 31) == 0) {
      red[0][tid >> 5] = psum;
      red[1][tid >> 5] = pden;
    }
    __syncthreads();
    if (tid == 0) {
      double a = 0.0, b = 0.0;
      for (int w = 0; w < NT / 32; ++w) {
        a += (double)red[0][w];
        b += (double)red[1][w];
      }
      atomicAdd(p.power_acc, a);
      atomicAdd(p.power_acc + 1, b);
    }
    return;
  }
  const float2* tab = p.table ? p.table + (size_t)plane * p.ncx * p.ncy : nullptr;
  const float nrm = 1.0f / ((float)X * (float)Y);
  samples([&](int, int x, int y) {
    float2& v = P[x * RS + y];
    v = tab != nullptr ? cmul(v, __ldg(tab + __ldg(p.cls_x + x) * p.ncy + __ldg(p.cls_y + y)))
                       : cscale(v, nrm);
  });
  __syncthreads();
  plane_passes<true>(cols, axx);
  // as in the line passes: along x before the inverse y transform, and the Nyquist plane,
  // whose Re() precedes the corrections, at the end
  const bool epi = p.epi != 0 || p.nscreens > 0, nyq = 2 * f == p.nT;
  if (epi && !nyq) epilogue<PosIdentity, 1>(p, plane, f, P, RS, X, 0, nullptr, nullptr);
  plane_passes<true>(rows, axy);
  if (epi && !nyq) epilogue<PosIdentity, 2>(p, plane, f, P, RS, X, 0, nullptr, nullptr);
  if (epi && nyq) epilogue<PosIdentity>(p, plane, f, P, RS, X, 0, nullptr, nullptr);
  samples([&](int i, int x, int y) { g[i] = P[x * RS + y]; });
}

}  // namespace

int asg_launch_xy_plane(const XYParams& p, const PlaneAxis& axx, const PlaneAxis& axy,
                        cudaStream_t st) {
  const int RS = p.Y | 1;
  const size_t smem = (size_t)p.X * RS * sizeof(float2);
  if (axx.n != p.X || axy.n != p.Y || smem > ASG_PLANE_MAX_SMEM) return ASG_ERR_SHAPE;
  // about four samples per thread, a DFT of radix 4; passes of odd primes spread over more;
  // no more threads than let all planes be resident
  int nt = std::max(32, (p.X * p.Y / 4 + 31) / 32 * 32);
  auto spread = [&](const PlaneAxis& ax, int lines) {
    for (unsigned long long r = ax.radices; r != 0; r >>= 8)
      if ((r & 255) > 9)
        nt = std::max(nt, (asg_plane_spread((int)(r & 255), ax.n, lines) + 31) / 32 * 32);
  };
  spread(axx, p.Y);
  spread(axy, p.X);
  nt = std::min(nt, asg_plane_threads(p.nplanes));
  return asg_launch_pdl(p.pdl != 0, xy_plane, dim3(p.nplanes), dim3(nt), smem, st, p, axx, axy, RS);
}
