// t-column kernel for any nT (and any nX, nY): per (x, y) column the inverse
// real FFT along t, the column phase (taper, Burgers step, sources,
// accumulators) and the forward real FFT along t.  Two neighbouring columns
// c, c+1 travel as one complex line u_c + i u_{c+1}: their spectra separate by
// symmetry, so a pair costs one complex transform of length nT each way
// (asg_lines.cuh: direct where the length splits into two radices, a chirp
// convolution for every other length).  Planes are in natural bin order.
//
// A block of 4 warps holds P pairs (a power of two up to 32).  Bounded by instruction
// issue and its latencies (five blocks per SM by registers, 40 to 55 % of the issue slots):
// register DFTs, their exchanges through shared memory, instruction fetch.  Per pass, against
// mixed-radix Stockham lines with direct sums over the prime factors:
// 257 x 257 x 601 27-30 -> 0.9 ms (its HBM traffic alone: 0.05 ms),
// 51 x 51 x 401 620-640 -> 40-47 us, 200 x 180 x 400 780-930 -> 90-160 us,
// 81 x 81 x 101 100 -> 23-31 us, 5 x 5 x 1001 120 -> 46 us.
//
// Also here: the Burgers step alone on real columns (no transforms).
//
// Reference semantics: see asg_tkernel.cu and asg_column.cuh.
#include "asg_internal.h"
#include "asg_column.cuh"
#include "asg_lines.cuh"

ASG_DEFINE_LINE_ROOT_UPLOADER(asg_roots_upload_tp)

namespace {

// real samples of one column of a pair: the real or imaginary parts of a padded
// line in natural order
template <class PL>
struct PairColumn {
  float* base;  // the line's floats + 0 (column c) or 1 (column c + 1)
  const LineAxis& ax;
  ASG_DEV float get(int t) const { return base[2 * line_pos<PL>(ax, t)]; }
  ASG_DEV void set(int t, float v) const { base[2 * line_pos<PL>(ax, t)] = v; }
};

// the largest |u| of a block's columns into max_next (NaN if one is not finite)
ASG_DEV void block_max_next(float am, const ColumnOps& op) {
  __shared__ float red_max[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (lane == 0) red_max[warp] = am;
  __syncthreads();
  if (tid == 0) {
    float m = 0.f;
    bool bad = false;
    for (int w = 0; w < (int)blockDim.x / 32; ++w) {
      const float v = red_max[w];
      bad |= (v != v);
      m = fmaxf(m, v);
    }
    if (bad) m = __uint_as_float(0x7fc00000u);
    stats_block_done(op, m, gridDim.x);
  }
}

template <class PL>
__global__ void __launch_bounds__(LineBlock<PL::BIG>::NT, LineBlock<PL::BIG>::MB)
    tk_pairs(TParams p, LineAxis ax, int lp, int LS) {
  pdl_wait();
  if (*p.status != 0) return;
  constexpr bool DIRECT = PL::DIRECT;
  constexpr int S2 = PL::S2;
  const int n = ax.n, n1 = PL::n1(ax), n2 = PL::n2(ax), NT = blockDim.x, NW = NT / 32;
  const int P = 1 << lp;
  const int F = n / 2 + 1;
  extern __shared__ float4 smraw[];
  float2* lines = reinterpret_cast<float2*>(smraw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ncols = p.ncols;
  const int c0 = blockIdx.x * 2 * P;
  // position of bin k of a line's spectrum: direct plans keep bin ka + n1 kb at slot
  // kb + S2 ka
  auto posk = [&](int k) {
    if (!DIRECT) return line_pos<PL>(ax, k);
    const int kb = PL::div1(ax, k);
    return kb + S2 * (k - kb * n1);
  };
  float am = 0.f;

  // dir 0: spectrum -> samples and the column work; dir 1: samples -> spectrum
#pragma unroll 1
  for (int dir = p.in_real ? 1 : 0; dir < 2; ++dir) {
    if (dir == 0) {
      // Z = S_c + i S_{c+1} on all bins from the halves f <= n/2 of both columns
      // (imaginary parts of bins 0 and n/2 dropped, as irfft does)
#pragma unroll 4
      for (int it = tid; it < F * P; it += NT) {
        const int q = it & (P - 1), f = it >> lp;
        const int c = c0 + 2 * q;
        const float2* s = p.spec + (size_t)f * ncols + c;
        const float2 a = c < ncols ? s[0] : make_float2(0.f, 0.f);
        const float2 b = c + 1 < ncols ? s[1] : make_float2(0.f, 0.f);
        float2* line = lines + q * LS;
        if (f == 0 || 2 * f == n) {
          line[posk(f)] = make_float2(a.x, b.x);
        } else {
          line[posk(f)] = make_float2(a.x - b.y, a.y + b.x);
          line[posk(n - f)] = make_float2(a.x + b.y, b.x - a.y);
        }
      }
      __syncthreads();
    } else if (p.in_real) {
      for (int cc = warp; cc < 2 * P; cc += NW) {
        PairColumn<PL> col{reinterpret_cast<float*>(lines + (cc >> 1) * LS) + (cc & 1), ax};
        const int c = c0 + cc;
        const float* src = p.real_in + (size_t)c * n;
        for (int t = lane; t < n; t += 32) col.set(t, c < ncols ? src[t] : 0.f);
      }
      __syncthreads();
    }
    if (dir == 1) {
      // ---- column work: a warp per column ----
#pragma unroll 1
      for (int cc = warp; cc < 2 * P; cc += NW) {
        const int c = c0 + cc;
        if (c >= ncols) continue;
        PairColumn<PL> col{reinterpret_cast<float*>(lines + (cc >> 1) * LS) + (cc & 1), ax};
        const float a = column_phase<0>(col, c, n, p.op, p.stats != 0);
        am = (a != a || am != am) ? __uint_as_float(0x7fc00000u) : fmaxf(am, a);
        if (p.write_real) {
          float* dst = p.real_out + (size_t)c * n;
          for (int t = lane; t < n; t += 32) dst[t] = col.get(t);
        }
      }
      if (p.stats) block_max_next(am, p.op);
      if (!p.do_r2c) return;
      __syncthreads();
    }
    const bool inv = dir == 0;
    if constexpr (!DIRECT) {
      PL::with_n1(ax, [&](auto R) {
        constexpr int N1 = decltype(R)::v;
        for (int it = tid; it < P * n2; it += NT) {
          const int q = it & (P - 1), b = it >> lp;
          float2* line = lines + q * LS;
          float2 v[N1];
#pragma unroll
          for (int a = 0; a < N1 / 2; ++a) {
            const int k = b + n2 * a;
            v[a] = k < n ? chirp_mul(line[b + S2 * a], ax.ch + k, inv) : make_float2(0.f, 0.f);
          }
          line_stepA<PL, N1>(line, b, v, ax);
        }
      });
      __syncthreads();
      PL::with_n2(ax, [&](auto R) {
        for (int it = tid; it < P * n1; it += NT) {
          const int q = PL::div1(ax, it), ka = it - q * n1;
          chirp_stepB<PL, decltype(R)::v>(lines + q * LS + ka * S2, ka, ax, inv);
        }
      });
      __syncthreads();
      const float sh = inv ? ax.inv_hi : 1.f, sl = inv ? ax.inv_lo : 0.f;
      PL::with_n1(ax, [&](auto R) {
        constexpr int N1 = decltype(R)::v;
        for (int it = tid; it < P * n2; it += NT) {
          const int q = it & (P - 1), b = it >> lp;
          float2* line = lines + q * LS;
          float2 v[N1];
          line_stepA_inv<PL, N1>(line, b, v, ax);
#pragma unroll
          for (int a = 0; a < N1 / 2; ++a) {
            const int k = b + n2 * a;
            if (k < n) line[b + S2 * a] = scale_hl(chirp_mul(v[a], ax.ch + k, inv), sh, sl);
          }
        }
      });
    } else if (inv) {
      PL::with_n2(ax, [&](auto R) {
        constexpr int N2 = decltype(R)::v;
        for (int it = tid; it < P * n1; it += NT) {
          const int q = PL::div1(ax, it), ka = it - q * n1;
          float2* run = lines + q * LS + ka * S2;
          float2 v[N2];
          run_load<N2>(run, v);
          ldft<N2, true>(v);
          run_store<N2>(run, v);
        }
      });
      __syncthreads();
      PL::with_n1(ax, [&](auto R) {
        constexpr int N1 = decltype(R)::v;
        for (int it = tid; it < P * n2; it += NT) {
          const int q = it & (P - 1), b = it >> lp;
          float2* line = lines + q * LS;
          float2 v[N1];
          line_stepA_inv<PL, N1>(line, b, v, ax);
#pragma unroll
          for (int a = 0; a < N1; ++a) line[b + S2 * a] = scale_hl(v[a], ax.inv_hi, ax.inv_lo);
        }
      });
    } else {
      PL::with_n1(ax, [&](auto R) {
        constexpr int N1 = decltype(R)::v;
        for (int it = tid; it < P * n2; it += NT) {
          const int q = it & (P - 1), b = it >> lp;
          float2* line = lines + q * LS;
          float2 v[N1];
#pragma unroll
          for (int a = 0; a < N1; ++a) v[a] = line[b + S2 * a];
          line_stepA<PL, N1>(line, b, v, ax);
        }
      });
      __syncthreads();
      PL::with_n2(ax, [&](auto R) {
        constexpr int N2 = decltype(R)::v;
        for (int it = tid; it < P * n1; it += NT) {
          const int q = PL::div1(ax, it), ka = it - q * n1;
          float2* run = lines + q * LS + ka * S2;
          float2 v[N2];
          run_load<N2>(run, v);
          ldft<N2, false>(v);
          run_store<N2>(run, v);
        }
      });
    }
    __syncthreads();
  }

  float2* so = p.spec_out ? p.spec_out : p.spec;
#pragma unroll 4
  for (int it = tid; it < F * P; it += NT) {
    const int q = it & (P - 1), f = it >> lp;
    const int c = c0 + 2 * q;
    const float2* line = lines + q * LS;
    const float2 zk = line[posk(f)], zm = line[posk(f == 0 ? 0 : n - f)];
    // S_c = (z_k + conj z_{n-k}) / 2, S_{c+1} = -i (z_k - conj z_{n-k}) / 2
    float2* s = so + (size_t)f * ncols + c;
    if (c < ncols) s[0] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
    if (c + 1 < ncols) s[1] = make_float2(0.5f * (zk.y + zm.y), 0.5f * (zm.x - zk.x));
  }
}

// The Burgers step alone on real columns: a warp per column, the column in
// shared memory (CH < 0: the KT sub-steps in registers, see column_phase).
template <int CH>
__global__ void __launch_bounds__(256) k_flux_columns(TParams p) {
  if (*p.status != 0) return;
  extern __shared__ float smcol[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * (blockDim.x >> 5) + warp, nT = p.nT;
  if (c >= p.ncols) return;
  PlainColumn col{smcol + warp * nT};
  const float* src = p.real_in + (size_t)c * nT;
#pragma unroll 4
  for (int t = lane; t < nT; t += 32) col.set(t, src[t]);
  __syncwarp();
  column_phase<CH>(col, c, nT, p.op, false);
  float* dst = p.real_out + (size_t)c * nT;
#pragma unroll 4
  for (int t = lane; t < nT; t += 32) dst[t] = col.get(t);
}

template <class PL>
int launch_pairs(const TParams& p, const LineAxis& ax, cudaStream_t st) {
  // pairs per block: what fills it, at least 4 (64-byte runs in HBM), while 72 KB
  // hold them and the grid does not leave the GPU idle (two blocks for each SM)
  const int npairs = (p.ncols + 1) / 2, tasks = line_tasks(ax);
  int lp = 0;
  while (lp < 5 && (lp < 2 || (tasks << lp) < LineBlock<PL::BIG>::NT)) {
    const int k = lp + 1;
    if (((size_t)line_stride(ax, 1 << k) * sizeof(float2) << k) > 72 * 1024) break;
    if ((npairs >> k) < 2 * asg_sm_count()) break;
    lp = k;
  }
  const int P = 1 << lp, LS = line_stride(ax, P);
  const size_t smem = (size_t)P * LS * sizeof(float2);
  // (four warps even where the steps have fewer tasks: the column work, the loads)
  const int nt = LineBlock<PL::BIG>::NT;
  static bool attr_done[ASG_MAX_DEVICES] = {};
  const int dev = asg_device_slot();
  if (!attr_done[dev]) {
    if (cudaFuncSetAttribute(tk_pairs<PL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             72 * 1024) != cudaSuccess)
      return ASG_ERR_CUDA;
    attr_done[dev] = true;
  }
  return asg_launch_pdl(p.pdl != 0, tk_pairs<PL>, dim3((npairs + P - 1) / P), dim3(nt), smem, st, p,
                        ax, lp, LS);
}

}  // namespace

int asg_launch_t_pairs(const TParams& p, const LineAxis& ax, cudaStream_t st) {
  if (ax.n != p.nT) return ASG_ERR_SHAPE;
  if (ax.direct)
    return ax.rm == 16 ? launch_pairs<DirectPlan<16>>(p, ax, st)
         : ax.rm == 24 ? launch_pairs<DirectPlan<24>>(p, ax, st)
         : ax.rm == 32 ? launch_pairs<DirectPlan<32>>(p, ax, st)
                       : launch_pairs<DirectPlan<64>>(p, ax, st);
#define F(a, b) \
  if (ax.n1 == a && ax.n2 == b) return launch_pairs<ChirpPlan<a, b>>(p, ax, st);
  ASG_CHIRP_SIZES(F)
  F(64, 64)
#undef F
  return ASG_ERR_SHAPE;
}

template <int CH>
static int launch_flux(const TParams& p, cudaStream_t st) {
  if (CH < 0 && p.nT > -32 * CH) {
    if constexpr (CH < 0) return launch_flux<(CH > -8 ? CH - 1 : 0)>(p, st);
  }
  // 8 columns per block while they fit the default 48 KB
  int warps = 8;
  while (warps > 1 && (size_t)warps * p.nT * sizeof(float) > 48 * 1024) warps /= 2;
  k_flux_columns<CH><<<(p.ncols + warps - 1) / warps, 32 * warps,
                       (size_t)warps * p.nT * sizeof(float), st>>>(p);
  return cudaPeekAtLastError() == cudaSuccess ? ASG_OK : ASG_ERR_CUDA;
}
int asg_launch_flux_columns(const TParams& p, cudaStream_t st) {
  // KT columns up to 256 samples in registers (8 samples per lane; beyond, the registers of a
  // run leave too few warps per SM); Rusanov steps have none to keep (10000 x 224 12.7 us,
  // 14.5 in that variant)
  return p.op.flux == FLUX_KT_MC || p.op.flux == FLUX_KT_MINMOD ? launch_flux<-1>(p, st)
                                                                : launch_flux<0>(p, st);
}
