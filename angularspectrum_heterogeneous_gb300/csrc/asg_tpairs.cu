// t-column kernel for any nT (and any nX, nY): per (x, y) column the inverse
// real FFT along t, the column phase (taper, Burgers step, sources,
// accumulators) and the forward real FFT along t.  Two neighbouring columns
// c, c+1 travel as one complex line u_c + i u_{c+1}: their spectra separate by
// symmetry, so a pair costs one complex transform of length nT each way
// (asg_lines.cuh: direct for the four-step sizes, a chirp convolution for every
// other length).  Planes are in natural bin order.
//
// A block of 4 warps holds P pairs (a power of two up to 8).  Bounded by the
// register DFTs and their exchanges through shared memory.  Per pass, against
// mixed-radix Stockham lines with direct sums over the prime factors:
// 257 x 257 x 601 27-30 -> 0.89-0.94 ms (its HBM traffic alone: 0.05 ms),
// 51 x 51 x 401 620-640 -> 31-38 us, 200 x 180 x 400 780-930 -> 240-330 us,
// 81 x 81 x 101 100 -> 20-24 us, 5 x 5 x 1001 120 -> 45 us.
//
// Also here: the Burgers step alone on real columns (no transforms).
//
// Reference semantics: see asg_tkernel.cu and asg_column.cuh.
#include "asg_internal.h"
#include "asg_column.cuh"
#include "asg_lines.cuh"

ASG_DEFINE_ROOT_UPLOADER_HL(asg_roots_upload_tp)

namespace {

// real samples of one column of a pair: the real or imaginary parts of a padded
// line in natural order
template <int N2>
struct PairColumn {
  float* base;  // the line's floats + 0 (column c) or 1 (column c + 1)
  ASG_DEV int idx(int t) const { return 2 * (t + 2 * (t / N2)); }
  ASG_DEV float get(int t) const { return base[idx(t)]; }
  ASG_DEV void set(int t, float v) const { base[idx(t)] = v; }
};

// the largest |u| of a block's columns into max_next (NaN if one is not finite)
template <int NW>
ASG_DEV void block_max_next(float am, unsigned* max_next) {
  __shared__ float red_max[NW];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (lane == 0) red_max[warp] = am;
  __syncthreads();
  if (tid == 0) {
    float m = 0.f;
    bool bad = false;
    for (int w = 0; w < NW; ++w) {
      const float v = red_max[w];
      bad |= (v != v);
      m = fmaxf(m, v);
    }
    if (bad) m = __uint_as_float(0x7fc00000u);
    atomicMax(max_next, float_as_ordered(m));
  }
}

// Blocks of 128 threads per SM: the registers of the longest in-register DFT (a
// 32-point one with the chirp's spectrum spills at four blocks).
template <int M, bool DIRECT>
constexpr int pair_min_blocks() {
  return FastPlan<M>::N2 >= 64 ? 2 : FastPlan<M>::N2 >= (DIRECT ? 48 : 32) ? 3 : 4;
}

template <int M, bool DIRECT>
__global__ void __launch_bounds__(128, pair_min_blocks<M, DIRECT>())
    tk_pairs(TParams p, LineAxis ax, int lp, int LS) {
  if (*p.status != 0) return;
  using PL = FastPlan<M>;
  constexpr int N1 = PL::N1, N2 = PL::N2, NT = 128, NW = NT / 32;
  constexpr int NA = DIRECT ? N1 : N1 / 2;  // step A inputs that can be non-zero
  const int n = DIRECT ? M : ax.n;
  const int P = 1 << lp;
  const int F = n / 2 + 1;
  extern __shared__ float4 smraw[];
  float2* lines = reinterpret_cast<float2*>(smraw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ncols = p.ncols;
  const int c0 = blockIdx.x * 2 * P;
  // position of bin k of a line's spectrum (direct plans: four-step slot order)
  auto posk = [](int k) { return DIRECT ? PL::pos(PL::slot_of_freq(k)) : PL::pos(k); };

  if (p.in_real) {
    for (int cc = warp; cc < 2 * P; cc += NW) {
      PairColumn<N2> col{reinterpret_cast<float*>(lines + (cc >> 1) * LS) + (cc & 1)};
      const int c = c0 + cc;
      const float* src = p.real_in + (size_t)c * n;
      for (int t = lane; t < n; t += 32) col.set(t, c < ncols ? src[t] : 0.f);
    }
    __syncthreads();
  } else {
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
    if constexpr (!DIRECT) {
      for (int it = tid; it < P * N2; it += NT) {
        const int q = it & (P - 1), b = it >> lp;
        float2* line = lines + q * LS;
        float2 v[N1];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          const int k = b + N2 * a;
          v[a] = k < n ? mulc_f4(line[PL::pos(k)], __ldg(ax.ch + k)) : make_float2(0.f, 0.f);
        }
        chirp_stepA<PL>(line, b, v, ax.tw);
      }
      __syncthreads();
      for (int it = tid; it < P * N1; it += NT) {
        const int q = it / N1, ka = it - q * N1;
        chirp_stepB<PL, true>(lines + q * LS, ka, ax.bt);
      }
      __syncthreads();
      for (int it = tid; it < P * N2; it += NT) {
        const int q = it & (P - 1), b = it >> lp;
        float2* line = lines + q * LS;
        float2 v[N1];
        chirp_stepA_inv<PL>(line, b, v, ax.tw);
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          const int t = b + N2 * a;
          if (t < n) line[PL::pos(t)] = scale_hl(mulc_f4(v[a], __ldg(ax.ch + t)), ax.inv_hi, ax.inv_lo);
        }
      }
    } else {
      for (int it = tid; it < P * N1; it += NT) {
        const int q = it / N1, ka = it - q * N1;
        float2* line = lines + q * LS;
        float2 v[N2];
        run_load<PL>(line, ka, v);
        dft<N2, true, true>(v);
        run_store<PL>(line, ka, v);
      }
      __syncthreads();
      for (int it = tid; it < P * N2; it += NT) {
        const int q = it & (P - 1), b = it >> lp;
        float2* line = lines + q * LS;
        float2 v[N1];
        chirp_stepA_inv<PL>(line, b, v, ax.tw);
#pragma unroll
        for (int a = 0; a < N1; ++a) line[PL::pos(b + N2 * a)] = scale_hl(v[a], ax.inv_hi, ax.inv_lo);
      }
    }
    __syncthreads();
  }

  // ---- column work: a warp per column ----
  float am = 0.f;
#pragma unroll 1
  for (int cc = warp; cc < 2 * P; cc += NW) {
    const int c = c0 + cc;
    if (c >= ncols) continue;
    PairColumn<N2> col{reinterpret_cast<float*>(lines + (cc >> 1) * LS) + (cc & 1)};
    const float a = column_phase<0>(col, c, n, p.op, p.stats != 0);
    am = (a != a || am != am) ? __uint_as_float(0x7fc00000u) : fmaxf(am, a);
    if (p.write_real) {
      float* dst = p.real_out + (size_t)c * n;
      for (int t = lane; t < n; t += 32) dst[t] = col.get(t);
    }
  }
  if (p.stats) block_max_next<NW>(am, p.op.max_next);
  if (!p.do_r2c) return;
  __syncthreads();

  // ---- forward transform of the pairs, split into the two columns' bins ----
  for (int it = tid; it < P * N2; it += NT) {
    const int q = it & (P - 1), b = it >> lp;
    float2* line = lines + q * LS;
    float2 v[N1];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      const int t = b + N2 * a;
      if constexpr (DIRECT) v[a] = line[PL::pos(t)];
      else v[a] = t < n ? mul_f4(line[PL::pos(t)], __ldg(ax.ch + t)) : make_float2(0.f, 0.f);
    }
    if constexpr (DIRECT) direct_stepA<PL>(line, b, v, ax.tw);
    else chirp_stepA<PL>(line, b, v, ax.tw);
  }
  __syncthreads();
  for (int it = tid; it < P * N1; it += NT) {
    const int q = it / N1, ka = it - q * N1;
    float2* line = lines + q * LS;
    if constexpr (DIRECT) {
      float2 v[N2];
      run_load<PL>(line, ka, v);
      dft<N2, false, true>(v);
      run_store<PL>(line, ka, v);
    } else {
      chirp_stepB<PL, false>(line, ka, ax.bt);
    }
  }
  __syncthreads();
  if constexpr (!DIRECT) {
    for (int it = tid; it < P * N2; it += NT) {
      const int q = it & (P - 1), b = it >> lp;
      float2* line = lines + q * LS;
      float2 v[N1];
      chirp_stepA_inv<PL>(line, b, v, ax.tw);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const int k = b + N2 * a;
        if (k < n) line[PL::pos(k)] = mul_f4(v[a], __ldg(ax.ch + k));
      }
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
// shared memory.
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
  column_phase<0>(col, c, nT, p.op, false);
  float* dst = p.real_out + (size_t)c * nT;
#pragma unroll 4
  for (int t = lane; t < nT; t += 32) dst[t] = col.get(t);
}

template <int M, bool DIRECT>
int launch_pairs(const TParams& p, const LineAxis& ax, cudaStream_t st) {
  using PL = FastPlan<M>;
  // pairs per block: as many as 72 KB hold, fewer while the grid leaves the GPU
  // idle (two blocks for each of its 152 SMs)
  const int npairs = (p.ncols + 1) / 2;
  int lp = 3;
  while (lp > 0 && ((size_t)line_stride(PL::PADDED, 1 << lp) * sizeof(float2) << lp) > 72 * 1024)
    --lp;
  while (lp > 0 && (npairs >> lp) < 2 * 152) --lp;
  const int P = 1 << lp, LS = line_stride(PL::PADDED, P);
  const size_t smem = (size_t)P * LS * sizeof(float2);
  static bool attr_done[ASG_MAX_DEVICES] = {};
  const int dev = asg_device_slot();
  if (!attr_done[dev]) {
    if (cudaFuncSetAttribute(tk_pairs<M, DIRECT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             72 * 1024) != cudaSuccess)
      return ASG_ERR_CUDA;
    attr_done[dev] = true;
  }
  tk_pairs<M, DIRECT><<<(npairs + P - 1) / P, 128, smem, st>>>(p, ax, lp, LS);
  return cudaPeekAtLastError() == cudaSuccess ? ASG_OK : ASG_ERR_CUDA;
}

}  // namespace

int asg_launch_t_pairs(const TParams& p, const LineAxis& ax, cudaStream_t st) {
  if (ax.n != p.nT) return ASG_ERR_SHAPE;
  if (ax.direct) {
    switch (ax.m) {
      case 32: return launch_pairs<32, true>(p, ax, st);
      case 64: return launch_pairs<64, true>(p, ax, st);
      case 96: return launch_pairs<96, true>(p, ax, st);
      case 128: return launch_pairs<128, true>(p, ax, st);
      case 192: return launch_pairs<192, true>(p, ax, st);
      case 256: return launch_pairs<256, true>(p, ax, st);
      case 384: return launch_pairs<384, true>(p, ax, st);
      case 512: return launch_pairs<512, true>(p, ax, st);
      case 576: return launch_pairs<576, true>(p, ax, st);
      case 768: return launch_pairs<768, true>(p, ax, st);
      case 1024: return launch_pairs<1024, true>(p, ax, st);
      case 1536: return launch_pairs<1536, true>(p, ax, st);
      case 2048: return launch_pairs<2048, true>(p, ax, st);
      default: return ASG_ERR_SHAPE;
    }
  }
  switch (ax.m) {
    case 32: return launch_pairs<32, false>(p, ax, st);
    case 64: return launch_pairs<64, false>(p, ax, st);
    case 96: return launch_pairs<96, false>(p, ax, st);
    case 128: return launch_pairs<128, false>(p, ax, st);
    case 192: return launch_pairs<192, false>(p, ax, st);
    case 256: return launch_pairs<256, false>(p, ax, st);
    case 384: return launch_pairs<384, false>(p, ax, st);
    case 512: return launch_pairs<512, false>(p, ax, st);
    case 576: return launch_pairs<576, false>(p, ax, st);
    case 768: return launch_pairs<768, false>(p, ax, st);
    case 1024: return launch_pairs<1024, false>(p, ax, st);
    case 1536: return launch_pairs<1536, false>(p, ax, st);
    case 2048: return launch_pairs<2048, false>(p, ax, st);
    case 4096: return launch_pairs<4096, false>(p, ax, st);
    default: return ASG_ERR_SHAPE;
  }
}

int asg_launch_flux_columns(const TParams& p, cudaStream_t st) {
  // 8 columns per block while they fit the default 48 KB
  int warps = 8;
  while (warps > 1 && (size_t)warps * p.nT * sizeof(float) > 48 * 1024) warps /= 2;
  k_flux_columns<<<(p.ncols + warps - 1) / warps, 32 * warps,
                   (size_t)warps * p.nT * sizeof(float), st>>>(p);
  return cudaPeekAtLastError() == cudaSuccess ? ASG_OK : ASG_ERR_CUDA;
}
