// Column passes of the any-size planes: forward x transform, multiplier, inverse x
// transform and what the closing epilogue does along x (see asg_xyrows.cu).
#include "asg_internal.h"
#include "asg_lines.cuh"
#include "asg_xy.cuh"

ASG_DEFINE_LINE_ROOT_UPLOADER(asg_roots_upload_xycols)

namespace {

// ---------------------------------------------------------------------------
// x transforms.  A block takes C = 2^lc y-columns of one plane; lanes run along the columns, then along the sublines.
// ---------------------------------------------------------------------------
// threads of a block at most and blocks per SM (so 112 or 168 registers up to radix 24: a
// chirp variant holds both convolutions' code): eight columns' tasks in one round there
// (two rounds of 96 threads: 257 x 257 x 601 610 us against 555)
template <class PL>
struct ColBlock {
  static constexpr int NT = PL::BIG <= 24 ? 192 : LineBlock<PL::BIG>::NT;
  static constexpr int MB = PL::BIG > 24 ? LineBlock<PL::BIG>::MB : PL::DIRECT || PL::BIG <= 16 ? 3 : 2;
};

template <class PL>
__global__ void __launch_bounds__(ColBlock<PL>::NT, ColBlock<PL>::MB)
    xy_cols(XYParams p, LineAxis ax, float2* buf, int lc, int LS) {
  pdl_wait();
  if (xy_should_skip(p)) return;
  extern __shared__ float4 smraw[];
  float2* lines = reinterpret_cast<float2*>(smraw);
  __shared__ float red[2][8];
  const int tid = threadIdx.x, NT = blockDim.x, C = 1 << lc;
  constexpr bool DIRECT = PL::DIRECT;
  constexpr int S2 = PL::S2;
  const int X = ax.n, Y = p.Y, n1 = PL::n1(ax), n2 = PL::n2(ax);
  const int plane = blockIdx.y, y0 = blockIdx.x * C, nc = min(C, Y - y0);
  if (p.zero_dc_nyq && is_dc_or_nyq(p.f_of_plane[plane], p.nT)) return;  // the last row pass zeroes
  float2* g = buf + (size_t)plane * X * Y + y0;
  const float2* tab = p.table ? p.table + (size_t)plane * p.ncx * p.ncy : nullptr;
  const float* obl = p.power_only ? p.obl_table + (size_t)plane * p.ncx * p.ncy : nullptr;
  const float nrm = 1.0f / ((float)X * (float)Y);
  float psum = 0.f, pden = 0.f;
  // the multiplier (or the power sums) of mode (x, column of class cy)
  auto mode = [&](float2 v, int x, int cy) {
    const int ti = __ldg(p.cls_x + x) * p.ncy + cy;
    if (obl != nullptr) {
      const float o = __ldg(obl + ti), P = v.x * v.x + v.y * v.y;
      psum = fmaf(P, o, psum);
      pden += (o > 0.f) ? P : 0.f;
      return v;
    }
    return tab != nullptr ? cmul(v, __ldg(tab + ti)) : cscale(v, nrm);
  };

  PL::with_n1(ax, [&](auto R) {
    constexpr int N1 = decltype(R)::v, NA = DIRECT ? N1 : N1 / 2;
    for (int it = tid; it < C * n2; it += NT) {
      const int c = it & (C - 1), b = it >> lc;
      float2 v[N1];
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const int x = b + n2 * a;
        v[a] = make_float2(0.f, 0.f);
        if ((DIRECT || x < X) && c < nc) {
          v[a] = g[(size_t)x * Y + c];
          if constexpr (!DIRECT) v[a] = chirp_mul(v[a], ax.ch + x, false);
        }
      }
      line_stepA<PL, N1>(lines + c * LS, b, v, ax);
    }
  });
  __syncthreads();
  if constexpr (DIRECT) {
    PL::with_n2(ax, [&](auto R) {
      constexpr int N2 = decltype(R)::v;
      // lanes along the columns: neighbouring entries of a table row
      for (int it = tid; it < C * n1; it += NT) {
        const int c = it & (C - 1), ka = it >> lc;
        if (c >= nc) continue;
        const int cy = p.cls_y[y0 + c];
        float2* run = lines + c * LS + ka * S2;
        float2 v[N2];
        run_load<N2>(run, v);
        ldft<N2, false>(v);
#pragma unroll
        for (int kb = 0; kb < N2; ++kb) v[kb] = mode(v[kb], ka + n1 * kb, cy);
        if (obl != nullptr) continue;
        ldft<N2, true>(v);
        run_store<N2>(run, v);
      }
    });
  } else {
    // forward, then inverse convolution (one copy of the code for both)
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      PL::with_n2(ax, [&](auto R) {
        for (int it = tid; it < C * n1; it += NT) {
          const int c = PL::div1(ax, it), ka = it - c * n1;
          chirp_stepB<PL, decltype(R)::v>(lines + c * LS + ka * S2, ka, ax, dir == 1);
        }
      });
      if (dir == 1) break;
      __syncthreads();
      PL::with_n1(ax, [&](auto R) {
        constexpr int N1 = decltype(R)::v;
        for (int it = tid; it < C * n2; it += NT) {
          const int c = it & (C - 1), b = it >> lc;
          if (c >= nc) continue;
          const int cy = p.cls_y[y0 + c];
          float2* line = lines + c * LS;
          float2 v[N1];
          line_stepA_inv<PL, N1>(line, b, v, ax);
#pragma unroll
          for (int a = 0; a < N1 / 2; ++a) line[b + S2 * a] = v[a];
          // (through this task's own slots, a few at a time: N1/2 table entries and
          // their addresses at once spill)
#pragma unroll 4
          for (int a = 0; a < N1 / 2; ++a) {
            const int x = b + n2 * a;
            float2& s = line[b + S2 * a];
            s = x < X ? mode(s, x, cy) : make_float2(0.f, 0.f);
          }
          if (obl != nullptr) continue;
#pragma unroll
          for (int a = 0; a < N1 / 2; ++a) v[a] = line[b + S2 * a];
          line_stepA<PL, N1>(line, b, v, ax);
        }
      });
      if (obl != nullptr) break;
      __syncthreads();
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
  const bool epi = p.epi != 0 && plane != p.skip_plane;
  const bool fw = epi && (p.epi & EPI_FREQW) != 0, sa = epi && (p.epi & EPI_SUPERABS) != 0;
  const float e = fw ? p.fw_exp[plane] : 0.f;
  PL::with_n1(ax, [&](auto R) {
    constexpr int N1 = decltype(R)::v, NA = DIRECT ? N1 : N1 / 2;
    for (int it = tid; it < C * n2; it += NT) {
      const int c = it & (C - 1), b = it >> lc;
      if (c >= nc) continue;
      float2* line = lines + c * LS;
      float2 v[N1];
      line_stepA_inv<PL, N1>(line, b, v, ax);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const int x = b + n2 * a;
        if (!DIRECT && x >= X) continue;
        float2 r = v[a];
        if constexpr (!DIRECT) r = chirp_mul(r, ax.ch + x, true);
        if (fw) {
          const float l = p.fw_lx[x];  // 0 inside the boundary bands: factor 1
          if (l != 0.f) r = cscale(r, exp2f(e * l));
        }
        if (sa) line[b + S2 * a] = r;  // this task's own slots
        if (!sa || (x >= p.ex0 && x < p.ex1)) g[(size_t)x * Y + c] = r;
      }
    }
  });
  if (!sa) return;
  __syncthreads();
  // Engquist-Majda x edges on the damped values of the bands
  const float cf = p.sa_coef[plane], st = p.sa_strength;
  for (int i = tid; i < (p.ex0 + X - p.ex1) * C; i += NT) {
    const int c = i & (C - 1), k = i >> lc, x = k < p.ex0 ? k : k - p.ex0 + p.ex1;
    if (c >= nc) continue;
    const float2* line = lines + c * LS;
    float2 r = line[line_pos<PL>(ax, x)];
    const float w = p.sa_wx[x];
    if (w != 0.f)
      r = edge_correct(x > 0 ? line[line_pos<PL>(ax, x - 1)] : r, r,
                       x + 1 < X ? line[line_pos<PL>(ax, x + 1)] : r, x, X, w, cf, st, p.sa_inv2dx,
                       p.sa_invdx);
    g[(size_t)x * Y + c] = r;
  }
}

template <class PL>
int launch_cols(const XYParams& p, const LineAxis& ax, float2* buf, cudaStream_t st) {
  // eight columns (64-byte runs), more where they do not fill a block of 128 threads
  const int tasks = line_tasks(ax);
  int lc = 3;
  // no lanes without a column: 381 x 2 x 128 176 -> 103 us per step, 700 x 4 x 512 178 -> 109
  while (lc > 0 && (1 << (lc - 1)) >= p.Y) --lc;
  while (lc > 0 && ((size_t)line_stride(ax, 1 << lc) * sizeof(float2) << lc) > LINE_SMEM) --lc;
  while (lc >= 3 && lc < 5 && (tasks << lc) < 128 && (1 << lc) < p.Y &&
         ((size_t)line_stride(ax, 2 << lc) * sizeof(float2) << (lc + 1)) <= LINE_SMEM &&
         p.nplanes * ((p.Y + (2 << lc) - 1) >> (lc + 1)) >= 8 * asg_sm_count())
    ++lc;
  const int C = 1 << lc, LS = line_stride(ax, C);
  const size_t smem = (size_t)C * LS * sizeof(float2);
  static bool done[ASG_MAX_DEVICES] = {};
  const int s = line_smem_attr(xy_cols<PL>, &done[asg_device_slot()]);
  if (s != ASG_OK) return s;
  return asg_launch_pdl(p.pdl != 0, xy_cols<PL>, dim3((p.Y + C - 1) / C, p.nplanes),
                        dim3(line_threads(C * tasks, ColBlock<PL>::NT)), smem, st, p, ax, buf,
                        lc, LS);
}

}  // namespace

int asg_launch_xy_cols(const XYParams& p, const LineAxis& ax, float2* buf, cudaStream_t st) {
  if (ax.direct)
    return ax.rm == 16 ? launch_cols<DirectPlan<16>>(p, ax, buf, st)
         : ax.rm == 24 ? launch_cols<DirectPlan<24>>(p, ax, buf, st)
                       : launch_cols<DirectPlan<32>>(p, ax, buf, st);
#define F(a, b) \
  if (ax.n1 == a && ax.n2 == b) return launch_cols<ChirpPlan<a, b>>(p, ax, buf, st);
  ASG_CHIRP_SIZES(F)
#undef F
  return ASG_ERR_SHAPE;
}
