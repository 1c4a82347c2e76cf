// Plane passes for any nX, nY up to 1024: per rfft bin the forward 2-D FFT, the
// per-mode multiplier and the inverse 2-D FFT as three passes over the planes
// in HBM, each a line transform of any length (asg_lines.cuh):
//   rows      forward y transform, in place (a block takes rows of any planes);
//   columns   forward x transform, multiplier, inverse x transform: in the chirp
//             form the closing chirp of the first and the opening chirp of the
//             second cancel, so the multiplier is applied in registers between
//             step A^-1 and step A;
//   rows      inverse y transform.
// The (x, y, omega) epilogue of a closing stage is fused as in the closing plane
// kernel (asg_xyl2.cu): what acts along x (damping factor, Engquist-Majda x
// edges) commutes with the y transform and runs in the column pass, what acts
// along y (damping factor, y edges) and the screens in the last row pass.  The
// Nyquist plane, whose Re() precedes the corrections, is left without epilogue
// (p.skip_plane) and goes through the epilogue pass.
//
// Against one CTA per plane (small planes, 51 CTAs for 101 samples) or Stockham
// lines with direct sums over prime factors, per stage: 257 x 257 x 601 12.6 ->
// 1.05 ms, 81 x 81 x 101 94-112 -> 31-37 us, 51 x 51 x 401 72 -> 44 us,
// 200 x 180 x 400 580-640 -> 430-520 us (5 x 5 x 1001, three launches for one:
// 15 -> 19 us).
//
// Reference semantics: see asg_xykernel.cu.
#include "asg_internal.h"
#include "asg_lines.cuh"
#include "asg_xy.cuh"

ASG_DEFINE_ROOT_UPLOADER_HL(asg_roots_upload_xylines)

namespace {

template <int M, bool DIRECT>
constexpr int line_min_blocks() {  // blocks of 128 threads per SM (register DFTs, as in asg_tpairs.cu)
  return M >= 2048 ? 2 : (M >= 1536 || (!DIRECT && FastPlan<M>::N2 >= 32)) ? 3 : 4;
}

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
// y transforms.  L rows per block of 128 threads, so that the N1 tasks of step B
// fill it; the rows of all planes are one sequence (X rows each).
// ---------------------------------------------------------------------------
template <int M>
struct RowShape {
  using PL = FastPlan<M>;
  static constexpr int L = 128 / PL::N1;
  // lines 8 complex apart modulo 16: lanes crossing from a line to the next
  // (8-slot sublines, 4-task lines) meet no bank twice
  static constexpr int LS = LineStride<PL, 2>::value;
};

template <int M, bool DIRECT, bool INV>
__global__ void __launch_bounds__(128, line_min_blocks<M, DIRECT>())
    xy_rows(XYParams p, LineAxis ax, float2* dst) {
  using PL = FastPlan<M>;
  constexpr int N1 = PL::N1, N2 = PL::N2, NT = 128, L = RowShape<M>::L, LS = RowShape<M>::LS;
  constexpr int NA = DIRECT ? N1 : N1 / 2;
  if (xy_should_skip(p)) return;
  extern __shared__ float4 smraw[];
  float2* lines = reinterpret_cast<float2*>(smraw);
  const int tid = threadIdx.x;
  const int X = p.X, Y = DIRECT ? M : ax.n;
  const int total = p.nplanes * X;
  const int g0 = blockIdx.x * L, nr = min(L, total - g0);
  const bool epi = INV && (p.epi != 0 || p.nscreens > 0);
  auto zero_row = [&](int l) {
    return p.zero_dc_nyq && is_dc_or_nyq(p.f_of_plane[(g0 + l) / X], p.nT);
  };
  const float2* src = p.spec + (size_t)g0 * Y;
  float2* out = dst + (size_t)g0 * Y;

  if constexpr (!DIRECT) {
    for (int it = tid; it < nr * N2; it += NT) {
      const int l = it / N2, b = it - l * N2;
      const float2* row = src + (size_t)l * Y;
      float2 v[N1];
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const int y = b + N2 * a;
        v[a] = make_float2(0.f, 0.f);
        if (y < Y) {
          const float4 w = __ldg(ax.ch + y);
          v[a] = INV ? mulc_f4(row[y], w) : mul_f4(row[y], w);
        }
      }
      chirp_stepA<PL>(lines + l * LS, b, v, ax.tw);
    }
    __syncthreads();
    for (int it = tid; it < nr * N1; it += NT) {
      const int l = it / N1, ka = it - l * N1;
      chirp_stepB<PL, INV>(lines + l * LS, ka, ax.bt);
    }
    __syncthreads();
  } else if constexpr (INV) {
    // bins ka + N1 kb of the row -> step B^-1
    for (int it = tid; it < nr * N1; it += NT) {
      const int l = it / N1, ka = it - l * N1;
      const float2* row = src + (size_t)l * Y;
      float2 v[N2];
#pragma unroll
      for (int kb = 0; kb < N2; ++kb) v[kb] = row[ka + N1 * kb];
      dft<N2, true, true>(v);
      run_store<PL>(lines + l * LS, ka, v);
    }
    __syncthreads();
  } else {
    for (int it = tid; it < nr * N2; it += NT) {
      const int l = it / N2, b = it - l * N2;
      const float2* row = src + (size_t)l * Y;
      float2 v[N1];
#pragma unroll
      for (int a = 0; a < N1; ++a) v[a] = row[b + N2 * a];
      direct_stepA<PL>(lines + l * LS, b, v, ax.tw);
    }
    __syncthreads();
    for (int it = tid; it < nr * N1; it += NT) {
      const int l = it / N1, ka = it - l * N1;
      float2* row = out + (size_t)l * Y;
      float2 v[N2];
      run_load<PL>(lines + l * LS, ka, v);
      dft<N2, false, true>(v);
#pragma unroll
      for (int kb = 0; kb < N2; ++kb) row[ka + N1 * kb] = v[kb];
    }
    return;
  }
  // last step A^-1: outputs b + N2 a
  for (int it = tid; it < nr * N2; it += NT) {
    const int l = it / N2, b = it - l * N2;
    float2* line = lines + l * LS;
    float2* row = out + (size_t)l * Y;
    const bool zero = zero_row(l);
    float2 v[N1];
    chirp_stepA_inv<PL>(line, b, v, ax.tw);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int y = b + N2 * a;
      if (y >= Y) continue;
      float2 r = v[a];
      if constexpr (!DIRECT) {
        const float4 w = __ldg(ax.ch + y);
        r = INV ? mulc_f4(r, w) : mul_f4(r, w);
      }
      if (INV && zero) r = make_float2(0.f, 0.f);
      if (epi) line[PL::pos(y)] = r;  // this task's own slots
      else row[y] = r;
    }
  }
  if (!epi) return;
  __syncthreads();
  // ---- along y: damping factor, Engquist-Majda edges; screens ----
  const bool fw = (p.epi & EPI_FREQW) != 0, sa = (p.epi & EPI_SUPERABS) != 0;
  for (int i = tid; i < nr * Y; i += NT) {
    const int l = i / Y, y = i - l * Y;
    const int plane = (g0 + l) / X, x = g0 + l - plane * X;
    const float2* line = lines + l * LS;
    float2 r = line[PL::pos(y)];
    if (plane != p.skip_plane) {
      const float e = fw ? p.fw_exp[plane] : 0.f;
      auto damped = [&](int j) {
        const float2 v = line[PL::pos(j)];
        return fw ? cscale(v, exp2f(e * p.fw_ly[j])) : v;
      };
      if (fw) r = cscale(r, exp2f(e * p.fw_ly[y]));
      const float w = sa ? p.sa_wy[y] : 0.f;
      if (w != 0.f)
        r = edge_correct(y > 0 ? damped(y - 1) : r, r, y + 1 < Y ? damped(y + 1) : r, y, Y, w,
                         p.sa_coef[plane], p.sa_strength, p.sa_inv2dy, p.sa_invdy);
      for (int k = 0; k < p.nscreens; ++k) {
        const float fs = p.screen_fscale[plane];
        const ScreenDev sc = p.screens[k];
        const size_t g = (size_t)x * Y + y;
        float sn, cs;
        sincosf(sc.phase[g] * fs, &sn, &cs);
        r = cmul(r, make_float2(cs, -sn));
        if (sc.amp != nullptr) {
          const float a = fminf(fmaxf(sc.amp[g], 1e-6f), 1.0f);
          r = cscale(r, exp2f(fs * log2f(a)));
        }
      }
    }
    out[(size_t)l * Y + y] = r;
  }
}

// ---------------------------------------------------------------------------
// x transforms.  A block takes C y-columns of one plane (64-byte runs of each
// row); lanes run along the columns, then along the sublines.
// ---------------------------------------------------------------------------
template <int M>
struct ColShape {
  using PL = FastPlan<M>;
  static constexpr int C = M >= 1536 ? 4 : 8;
  static constexpr int TASKS = C * (PL::N1 > PL::N2 ? PL::N1 : PL::N2);
  static constexpr int NT = TASKS > 256 ? 128 : (TASKS + 31) / 32 * 32;
  static constexpr int LS = LineStride<PL, C>::value;
};
template <int M, bool DIRECT>
constexpr int col_min_blocks() {  // the same registers per thread as in the row pass
  constexpr int n = line_min_blocks<M, DIRECT>() * 128 / ColShape<M>::NT;
  return n > 0 ? n : 1;
}

template <int M, bool DIRECT>
__global__ void __launch_bounds__(ColShape<M>::NT, col_min_blocks<M, DIRECT>())
    xy_cols(XYParams p, LineAxis ax, float2* buf) {
  using PL = FastPlan<M>;
  using SH = ColShape<M>;
  constexpr int N1 = PL::N1, N2 = PL::N2, NT = SH::NT, C = SH::C, LS = SH::LS;
  constexpr int NA = DIRECT ? N1 : N1 / 2;
  if (xy_should_skip(p)) return;
  extern __shared__ float4 smraw[];
  float2* lines = reinterpret_cast<float2*>(smraw);
  __shared__ float red[2][8];
  const int tid = threadIdx.x;
  const int X = DIRECT ? M : ax.n, Y = p.Y;
  const int plane = blockIdx.y, y0 = blockIdx.x * C, nc = min(C, Y - y0);
  if (p.zero_dc_nyq && is_dc_or_nyq(p.f_of_plane[plane], p.nT)) return;  // the last row pass zeroes
  float2* g = buf + (size_t)plane * X * Y + y0;
  const float2* tab = p.table ? p.table + (size_t)plane * p.ncx * p.ncy : nullptr;
  const float* obl = p.power_only ? p.obl_table + (size_t)plane * p.ncx * p.ncy : nullptr;
  const float nrm = 1.0f / ((float)X * (float)Y);
  float psum = 0.f, pden = 0.f;
  // the multiplier (or the power sums) of mode (x, column c)
  auto mode = [&](float2 v, int x, int c) {
    const int ti = p.cls_x[x] * p.ncy + p.cls_y[y0 + c];
    if (obl != nullptr) {
      const float o = obl[ti], P = v.x * v.x + v.y * v.y;
      psum = fmaf(P, o, psum);
      pden += (o > 0.f) ? P : 0.f;
      return v;
    }
    return tab != nullptr ? cmul(v, tab[ti]) : cscale(v, nrm);
  };

  for (int it = tid; it < C * N2; it += NT) {
    const int c = it % C, b = it / C;
    float2 v[N1];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int x = b + N2 * a;
      v[a] = make_float2(0.f, 0.f);
      if (x < X && c < nc) {
        v[a] = g[(size_t)x * Y + c];
        if constexpr (!DIRECT) v[a] = mul_f4(v[a], __ldg(ax.ch + x));
      }
    }
    if constexpr (DIRECT) direct_stepA<PL>(lines + c * LS, b, v, ax.tw);
    else chirp_stepA<PL>(lines + c * LS, b, v, ax.tw);
  }
  __syncthreads();
  if constexpr (DIRECT) {
    for (int it = tid; it < C * N1; it += NT) {
      const int c = it / N1, ka = it - c * N1;
      if (c >= nc) continue;
      float2* line = lines + c * LS;
      float2 v[N2];
      run_load<PL>(line, ka, v);
      dft<N2, false, true>(v);
#pragma unroll
      for (int kb = 0; kb < N2; ++kb) v[kb] = mode(v[kb], ka + N1 * kb, c);
      if (obl != nullptr) continue;
      dft<N2, true, true>(v);
      run_store<PL>(line, ka, v);
    }
  } else {
    for (int it = tid; it < C * N1; it += NT) {
      const int c = it / N1, ka = it - c * N1;
      chirp_stepB<PL, false>(lines + c * LS, ka, ax.bt);
    }
    __syncthreads();
    for (int it = tid; it < C * N2; it += NT) {
      const int c = it % C, b = it / C;
      if (c >= nc) continue;
      float2* line = lines + c * LS;
      float2 v[N1];
      chirp_stepA_inv<PL>(line, b, v, ax.tw);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const int x = b + N2 * a;
        v[a] = x < X ? mode(v[a], x, c) : make_float2(0.f, 0.f);
      }
      if (obl != nullptr) continue;
      chirp_stepA<PL>(line, b, v, ax.tw);
    }
  }
  if (p.power_only) {
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
  __syncthreads();
  if constexpr (!DIRECT) {
    for (int it = tid; it < C * N1; it += NT) {
      const int c = it / N1, ka = it - c * N1;
      chirp_stepB<PL, true>(lines + c * LS, ka, ax.bt);
    }
    __syncthreads();
  }
  const bool epi = p.epi != 0 && plane != p.skip_plane;
  const bool fw = epi && (p.epi & EPI_FREQW) != 0, sa = epi && (p.epi & EPI_SUPERABS) != 0;
  const float e = fw ? p.fw_exp[plane] : 0.f;
  for (int it = tid; it < C * N2; it += NT) {
    const int c = it % C, b = it / C;
    if (c >= nc) continue;
    float2* line = lines + c * LS;
    float2 v[N1];
    chirp_stepA_inv<PL>(line, b, v, ax.tw);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int x = b + N2 * a;
      if (x >= X) continue;
      float2 r = v[a];
      if constexpr (!DIRECT) r = mulc_f4(r, __ldg(ax.ch + x));
      if (fw) r = cscale(r, exp2f(e * p.fw_lx[x]));
      if (sa) line[PL::pos(x)] = r;  // this task's own slots
      else g[(size_t)x * Y + c] = r;
    }
  }
  if (!sa) return;
  __syncthreads();
  // Engquist-Majda x edges on the damped values
  const float cf = p.sa_coef[plane], st = p.sa_strength;
  for (int i = tid; i < X * C; i += NT) {
    const int c = i % C, x = i / C;
    if (c >= nc) continue;
    const float2* line = lines + c * LS;
    float2 r = line[PL::pos(x)];
    const float w = p.sa_wx[x];
    if (w != 0.f)
      r = edge_correct(x > 0 ? line[PL::pos(x - 1)] : r, r,
                       x + 1 < X ? line[PL::pos(x + 1)] : r, x, X, w, cf, st, p.sa_inv2dx,
                       p.sa_invdx);
    g[(size_t)x * Y + c] = r;
  }
}

template <class K>
int smem_attr(K kern, size_t smem, bool* done) {
  if (*done) return ASG_OK;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return ASG_ERR_CUDA;
  *done = true;
  return ASG_OK;
}

template <int M, bool DIRECT>
int launch_rows(const XYParams& p, const LineAxis& ax, float2* dst, bool inverse, cudaStream_t st) {
  using SH = RowShape<M>;
  const size_t smem = (size_t)SH::L * SH::LS * sizeof(float2);
  static bool done[2][ASG_MAX_DEVICES] = {};
  const int dev = asg_device_slot();
  const int s = inverse ? smem_attr(xy_rows<M, DIRECT, true>, smem, &done[1][dev])
                        : smem_attr(xy_rows<M, DIRECT, false>, smem, &done[0][dev]);
  if (s != ASG_OK) return s;
  const int grid = (p.nplanes * p.X + SH::L - 1) / SH::L;
  if (inverse) xy_rows<M, DIRECT, true><<<grid, 128, smem, st>>>(p, ax, dst);
  else xy_rows<M, DIRECT, false><<<grid, 128, smem, st>>>(p, ax, dst);
  return cudaPeekAtLastError() == cudaSuccess ? ASG_OK : ASG_ERR_CUDA;
}

template <int M, bool DIRECT>
int launch_cols(const XYParams& p, const LineAxis& ax, float2* buf, cudaStream_t st) {
  using SH = ColShape<M>;
  const size_t smem = (size_t)SH::C * SH::LS * sizeof(float2);
  static bool done[ASG_MAX_DEVICES] = {};
  const int s = smem_attr(xy_cols<M, DIRECT>, smem, &done[asg_device_slot()]);
  if (s != ASG_OK) return s;
  xy_cols<M, DIRECT><<<dim3((p.Y + SH::C - 1) / SH::C, p.nplanes), SH::NT, smem, st>>>(p, ax, buf);
  return cudaPeekAtLastError() == cudaSuccess ? ASG_OK : ASG_ERR_CUDA;
}

#define ASG_LINE_SIZES(F, direct)                                                            \
  case 32: return F<32, direct>(ARGS);                                                      \
  case 64: return F<64, direct>(ARGS);                                                      \
  case 96: return F<96, direct>(ARGS);                                                      \
  case 128: return F<128, direct>(ARGS);                                                    \
  case 192: return F<192, direct>(ARGS);                                                    \
  case 256: return F<256, direct>(ARGS);                                                    \
  case 384: return F<384, direct>(ARGS);                                                    \
  case 512: return F<512, direct>(ARGS);                                                    \
  case 576: return F<576, direct>(ARGS);                                                    \
  case 768: return F<768, direct>(ARGS);                                                    \
  case 1024: return F<1024, direct>(ARGS);

int rows(const XYParams& p, const LineAxis& ax, float2* dst, bool inverse, cudaStream_t st) {
#define ARGS p, ax, dst, inverse, st
  if (ax.direct) {
    switch (ax.m) {
      ASG_LINE_SIZES(launch_rows, true)
      default: return ASG_ERR_SHAPE;
    }
  }
  switch (ax.m) {
    ASG_LINE_SIZES(launch_rows, false)
    case 1536: return launch_rows<1536, false>(ARGS);
    case 2048: return launch_rows<2048, false>(ARGS);
    default: return ASG_ERR_SHAPE;
  }
#undef ARGS
}

int cols(const XYParams& p, const LineAxis& ax, float2* buf, cudaStream_t st) {
#define ARGS p, ax, buf, st
  if (ax.direct) {
    switch (ax.m) {
      ASG_LINE_SIZES(launch_cols, true)
      default: return ASG_ERR_SHAPE;
    }
  }
  switch (ax.m) {
    ASG_LINE_SIZES(launch_cols, false)
    case 1536: return launch_cols<1536, false>(ARGS);
    case 2048: return launch_cols<2048, false>(ARGS);
    default: return ASG_ERR_SHAPE;
  }
#undef ARGS
}

}  // namespace

int asg_launch_xy_lines(const XYParams& p, const LineAxis& axx, const LineAxis& axy,
                        cudaStream_t st) {
  if (axx.n != p.X || axy.n != p.Y) return ASG_ERR_SHAPE;
  // the power sums leave the spectrum as it is
  if (p.power_only) {
    if (p.spec_tmp == nullptr) return ASG_ERR_STATE;
    const int s = rows(p, axy, p.spec_tmp, false, st);
    return s != ASG_OK ? s : cols(p, axx, p.spec_tmp, st);
  }
  int s = rows(p, axy, p.spec, false, st);
  if (s == ASG_OK) s = cols(p, axx, p.spec, st);
  if (s == ASG_OK) s = rows(p, axy, p.spec, true, st);
  return s;
}
