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
// Against one CTA per plane or Stockham lines with direct sums over prime factors, per
// stage: 257 x 257 x 601 12.6 -> 1.03 ms, 81 x 81 x 101 94-112 -> 27-33 us, 200 x 180 x 400
// 580-640 -> 135-218 us.  Small planes run in one launch (asg_xyplane.cu).
//
// Reference semantics: see asg_xykernel.cu.
#include "asg_internal.h"
#include "asg_lines.cuh"
#include "asg_xy.cuh"

ASG_DEFINE_LINE_ROOT_UPLOADER(asg_roots_upload_xyrows)

namespace {

// ---------------------------------------------------------------------------
// y transforms.  L rows per block; the rows of all planes are one sequence (X
// rows each).
// ---------------------------------------------------------------------------
template <class PL, bool INV>
__global__ void __launch_bounds__(LineBlock<PL::BIG>::NT, LineBlock<PL::BIG>::MB)
    xy_rows(XYParams p, LineAxis ax, float2* dst, int L, int LS) {
  pdl_wait();
  if (xy_should_skip(p)) return;
  extern __shared__ float4 smraw[];
  float2* lines = reinterpret_cast<float2*>(smraw);
  const int tid = threadIdx.x, NT = blockDim.x;
  constexpr bool DIRECT = PL::DIRECT;
  constexpr int S2 = PL::S2;
  const int X = p.X, Y = ax.n, n1 = PL::n1(ax), n2 = PL::n2(ax);
  const int total = p.nplanes * X;
  const int g0 = blockIdx.x * L, nr = min(L, total - g0);
  const bool epi = INV && (p.epi != 0 || p.nscreens > 0);
  // columns that the epilogue leaves as they are go straight out (all are staged: the
  // bands' edges need their neighbours)
  const int ey0 = p.nscreens > 0 ? Y : p.ey0, ey1 = p.nscreens > 0 ? Y : p.ey1;
  auto zero_row = [&](int l) {
    return p.zero_dc_nyq && is_dc_or_nyq(p.f_of_plane[(g0 + l) / X], p.nT);
  };
  const float2* src = p.spec + (size_t)g0 * Y;
  float2* out = dst + (size_t)g0 * Y;

  if constexpr (!DIRECT) {
    PL::with_n1(ax, [&](auto R) {
      constexpr int N1 = decltype(R)::v;
      for (int it = tid; it < nr * n2; it += NT) {
        const int l = PL::div2(ax, it), b = it - l * n2;
        const float2* row = src + (size_t)l * Y;
        float2 v[N1];
#pragma unroll
        for (int a = 0; a < N1 / 2; ++a) {
          const int y = b + n2 * a;
          v[a] = y < Y ? chirp_mul(row[y], ax.ch + y, INV) : make_float2(0.f, 0.f);
        }
        line_stepA<PL, N1>(lines + l * LS, b, v, ax);
      }
    });
    __syncthreads();
    PL::with_n2(ax, [&](auto R) {
      for (int it = tid; it < nr * n1; it += NT) {
        const int l = PL::div1(ax, it), ka = it - l * n1;
        chirp_stepB<PL, decltype(R)::v>(lines + l * LS + ka * S2, ka, ax, INV);
      }
    });
  } else if constexpr (INV) {
    // bins ka + n1 kb of the row -> step B^-1
    PL::with_n2(ax, [&](auto R) {
      constexpr int N2 = decltype(R)::v;
      for (int it = tid; it < nr * n1; it += NT) {
        const int l = PL::div1(ax, it), ka = it - l * n1;
        const float2* row = src + (size_t)l * Y;
        float2* run = lines + l * LS + ka * S2;
        float2 v[N2];
#pragma unroll
        for (int kb = 0; kb < N2; ++kb) v[kb] = row[ka + n1 * kb];
        ldft<N2, true>(v);
        run_store<N2>(run, v);
      }
    });
  } else {
    PL::with_n1(ax, [&](auto R) {
      constexpr int N1 = decltype(R)::v;
      for (int it = tid; it < nr * n2; it += NT) {
        const int l = PL::div2(ax, it), b = it - l * n2;
        const float2* row = src + (size_t)l * Y;
        float2 v[N1];
#pragma unroll
        for (int a = 0; a < N1; ++a) v[a] = row[b + n2 * a];
        line_stepA<PL, N1>(lines + l * LS, b, v, ax);
      }
    });
    __syncthreads();
    PL::with_n2(ax, [&](auto R) {
      constexpr int N2 = decltype(R)::v;
      for (int it = tid; it < nr * n1; it += NT) {
        const int l = PL::div1(ax, it), ka = it - l * n1;
        float2* row = out + (size_t)l * Y;
        const float2* run = lines + l * LS + ka * S2;
        float2 v[N2];
        run_load<N2>(run, v);
        ldft<N2, false>(v);
#pragma unroll
        for (int kb = 0; kb < N2; ++kb) row[ka + n1 * kb] = v[kb];
      }
    });
    return;
  }
  __syncthreads();
  // last step A^-1: outputs b + n2 a
  PL::with_n1(ax, [&](auto R) {
    constexpr int N1 = decltype(R)::v, NA = DIRECT ? N1 : N1 / 2;
    for (int it = tid; it < nr * n2; it += NT) {
      const int l = PL::div2(ax, it), b = it - l * n2;
      float2* line = lines + l * LS;
      float2* row = out + (size_t)l * Y;
      const bool zero = INV && zero_row(l);
      float2 v[N1];
      line_stepA_inv<PL, N1>(line, b, v, ax);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const int y = b + n2 * a;
        if (!DIRECT && y >= Y) continue;
        float2 r = v[a];
        if constexpr (!DIRECT) r = chirp_mul(r, ax.ch + y, INV);
        if (zero) r = make_float2(0.f, 0.f);
        if (epi) line[b + S2 * a] = r;  // this task's own slots
        if (!epi || (y >= ey0 && y < ey1)) row[y] = r;
      }
    }
  });
  if (!epi) return;
  __syncthreads();
  // ---- along y: damping factor, Engquist-Majda edges; screens (a warp per row) ----
  const bool fw = (p.epi & EPI_FREQW) != 0, sa = (p.epi & EPI_SUPERABS) != 0;
  for (int l = tid >> 5; l < nr; l += NT >> 5) {
    const int plane = (g0 + l) / X, x = g0 + l - plane * X;
    const float2* line = lines + l * LS;
    const bool row_epi = plane != p.skip_plane;
    const float e = fw && row_epi ? p.fw_exp[plane] : 0.f;
    const float cf = sa && row_epi ? p.sa_coef[plane] : 0.f;
    const float fs = p.nscreens > 0 ? p.screen_fscale[plane] : 0.f;
    auto damped = [&](int j) {
      const float2 v = line[line_pos<PL>(ax, j)];
      const float g = fw ? p.fw_ly[j] : 0.f;  // 0 inside the boundary bands: factor 1
      return g != 0.f ? cscale(v, exp2f(e * g)) : v;
    };
    const int nb = ey0 + Y - ey1;
#pragma unroll 2
    for (int k = tid & 31; k < nb; k += 32) {
      const int y = k < ey0 ? k : k - ey0 + ey1;
      float2 r;
      if (row_epi) {
        r = damped(y);
        const float w = sa ? p.sa_wy[y] : 0.f;
        if (w != 0.f)
          r = edge_correct(y > 0 ? damped(y - 1) : r, r, y + 1 < Y ? damped(y + 1) : r, y, Y, w,
                           cf, p.sa_strength, p.sa_inv2dy, p.sa_invdy);
        for (int q = 0; q < p.nscreens; ++q) {
          const ScreenDev sc = p.screens[q];
          const size_t g = (size_t)x * Y + y;
          float sn, cs;
          sincosf(sc.phase[g] * fs, &sn, &cs);
          r = cmul(r, make_float2(cs, -sn));
          if (sc.amp != nullptr) {
            const float a = fminf(fmaxf(sc.amp[g], 1e-6f), 1.0f);
            r = cscale(r, exp2f(fs * log2f(a)));
          }
        }
      } else {
        r = line[line_pos<PL>(ax, y)];
      }
      out[(size_t)l * Y + y] = r;
    }
  }
}

template <class PL>
int launch_rows(const XYParams& p, const LineAxis& ax, float2* dst, bool inverse, cudaStream_t st) {
  // rows per block: what fills it, while four blocks' shared memory fits an SM;
  // lines 8 complex apart modulo 16 (lanes crossing from a line of short sublines to
  // the next)
  const int tasks = line_tasks(ax), LS = line_stride(ax, 2);
  int L = (LineBlock<PL::BIG>::NT + tasks - 1) / tasks;
  if (L * tasks > LineBlock<PL::BIG>::NT && L > 1) --L;
  while (L > 1 && (size_t)L * LS * sizeof(float2) > 48 * 1024) --L;
  const int total = p.nplanes * p.X;
  while (L > 1 && total / L < 4 * asg_sm_count()) --L;
  const size_t smem = (size_t)L * LS * sizeof(float2);
  static bool done[2][ASG_MAX_DEVICES] = {};
  const int dev = asg_device_slot();
  const int s = inverse ? line_smem_attr(xy_rows<PL, true>, &done[1][dev])
                        : line_smem_attr(xy_rows<PL, false>, &done[0][dev]);
  if (s != ASG_OK) return s;
  const int grid = (total + L - 1) / L, nt = line_threads(L * tasks, LineBlock<PL::BIG>::NT);
  return asg_launch_pdl(p.pdl != 0, inverse ? xy_rows<PL, true> : xy_rows<PL, false>, dim3(grid),
                        dim3(nt), smem, st, p, ax, dst, L, LS);
}

}  // namespace

int asg_launch_xy_rows(const XYParams& p, const LineAxis& ax, float2* dst, bool inverse, cudaStream_t st) {
  if (ax.direct)
    return ax.rm == 16 ? launch_rows<DirectPlan<16>>(p, ax, dst, inverse, st)
         : ax.rm == 24 ? launch_rows<DirectPlan<24>>(p, ax, dst, inverse, st)
                       : launch_rows<DirectPlan<32>>(p, ax, dst, inverse, st);
#define F(a, b) \
  if (ax.n1 == a && ax.n2 == b) return launch_rows<ChirpPlan<a, b>>(p, ax, dst, inverse, st);
  ASG_CHIRP_SIZES(F)
#undef F
  return ASG_ERR_SHAPE;
}

int asg_launch_xy_lines(const XYParams& p, const LineAxis& axx, const LineAxis& axy,
                        cudaStream_t st) {
  if (axx.n != p.X || axy.n != p.Y) return ASG_ERR_SHAPE;
  // the power sums leave the spectrum as it is
  if (p.power_only) {
    if (p.spec_tmp == nullptr) return ASG_ERR_STATE;
    const int s = asg_launch_xy_rows(p, axy, p.spec_tmp, false, st);
    return s != ASG_OK ? s : asg_launch_xy_cols(p, axx, p.spec_tmp, st);
  }
  int s = asg_launch_xy_rows(p, axy, p.spec, false, st);
  if (s == ASG_OK) s = asg_launch_xy_cols(p, axx, p.spec, st);
  if (s == ASG_OK) s = asg_launch_xy_rows(p, axy, p.spec, true, st);
  return s;
}
