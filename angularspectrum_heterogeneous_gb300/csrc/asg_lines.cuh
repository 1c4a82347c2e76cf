// Line transforms of any length in shared memory.
//
// A length that the four-step plans cover (FastPlan: 2^a and 3 2^a sizes) is
// transformed directly.  Every other length n, prime ones included, runs as a
// chirp convolution (Bluestein): with w_j = exp(-i pi j^2 / n),
//   X[k] = w_k sum_j (x[j] w_j) conj(w_{k-j}),
// a circular convolution of length M >= 2 n - 1 with M a four-step size.  The
// convolution's forward transform, the product with the transformed chirp and
// the inverse transform take two exchanges through shared memory:
//   step A     DFT_N1 of the chirped inputs, twiddles            -> shared
//   step B     DFT_N2, times the chirp's spectrum, inverse DFT_N2 -> shared
//   step A^-1  twiddles, inverse DFT_N1, times w_k
// n <= M/2, so the upper half of step A's inputs is zero and the upper half of
// step A^-1's outputs is not needed; both DFT_N1 skip that half.
// The inverse transform uses the conjugates of both tables (the chirp is even,
// so the spectrum of its conjugate is the conjugate of its spectrum).
//
// Every factor (chirp, its spectrum, twiddles, the constants of the register DFTs) is
// kept as two floats: rounded to one, the same relative errors of 3e-8 return at
// every step of a march and add up, which the direct sums of this length never
// did.  20 forward/inverse pairs of 101 samples: error 2.4e-6 with single
// factors, 7.5e-7 with double ones, 1.6e-6 for the direct sum.
//
// Against the direct sum over a prime length this is O(log n) instead of O(n)
// per sample: a column pass over 257 x 257 x 601 takes 0.89 ms instead of 27 ms.
#pragma once
#include "asg_common.cuh"

// Device tables of one axis (built in FP64 on the host, see line_axis()).
struct LineAxis {
  int n;              // line length
  int m;              // transform length: n when direct, else the convolution length
  int direct;
  float inv_hi, inv_lo;  // 1/n as two floats (one would scale every inverse transform alike)
  // factors as (hi.re, hi.im, lo.re, lo.im)
  const float4* ch;   // [n] w_j (chirp axes)
  const float4* bt;   // [m] spectrum of conj(w), bins in natural order, 1/m folded in
  const float4* tw;   // [m] W_m^(b ka) at index ka N2 + b: lanes along b read it coalesced
};

ASG_DEV float2 mul_f4(float2 a, float4 w) {
  return cmul_hl(a, make_float2(w.x, w.y), make_float2(w.z, w.w));
}
ASG_DEV float2 mulc_f4(float2 a, float4 w) {
  return cmulc_hl(a, make_float2(w.x, w.y), make_float2(w.z, w.w));
}

ASG_DEV float2 scale_hl(float2 a, float hi, float lo) {
  return make_float2(fmaf(a.x, hi, a.x * lo), fmaf(a.y, hi, a.y * lo));
}

// Forward DFT of N values whose upper half is zero (v[N/2..] need not be set).
template <int N>
ASG_DEV void dft_fwd_lo(float2 (&v)[N]) {
  if constexpr (N == 4) {
    const float2 a = v[0], b = v[1], c = mul_mi<false>(b);
    v[0] = cadd(a, b);
    v[1] = cadd(a, c);
    v[2] = csub(a, b);
    v[3] = csub(a, c);
  } else {
    constexpr int P = DftSplit<N>::P, Q = DftSplit<N>::Q;
    static_assert(P == 4 || P == 8, "half-empty DFT");
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      float2 t[P];
      if constexpr (P == 4) {
        const float2 a = v[q], b = v[Q + q], c = mul_mi<false>(b);
        t[0] = cadd(a, b);
        t[1] = cadd(a, c);
        t[2] = csub(a, b);
        t[3] = csub(a, c);
      } else {
        // DFT_8 of (a0..a3, 0, 0, 0, 0): even bins DFT_4(a), odd bins DFT_4(a W_8^p)
        float2 e[4], o[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          e[p] = v[Q * p + q];
          o[p] = twiddle_mul<8, false, true>(e[p], p);
        }
        dft<4, false, true>(e);
        dft<4, false, true>(o);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          t[2 * p] = e[p];
          t[2 * p + 1] = o[p];
        }
      }
#pragma unroll
      for (int ka = 0; ka < P; ++ka) v[Q * ka + q] = twiddle_mul<N, false, true>(t[ka], q * ka);
    }
    float2 o[N];
#pragma unroll
    for (int ka = 0; ka < P; ++ka) {
      float2 t[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) t[q] = v[Q * ka + q];
      dft<Q, false, true>(t);
#pragma unroll
      for (int kb = 0; kb < Q; ++kb) o[ka + P * kb] = t[kb];
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = o[i];
  }
}

// --- chirp convolution -------------------------------------------------------
// step A of subline b: v[a] = input b + N2 a for a < N1/2 (chirped, zero past n)
template <class PL>
ASG_DEV void chirp_stepA(float2* line, int b, float2 (&v)[PL::N1], const float4* __restrict__ tw) {
  dft_fwd_lo<PL::N1>(v);
  line[PL::pos(b)] = v[0];
#pragma unroll
  for (int ka = 1; ka < PL::N1; ++ka)
    line[PL::pos(b + PL::N2 * ka)] = mul_f4(v[ka], __ldg(tw + ka * PL::N2 + b));
}

template <class PL, bool INV>
ASG_DEV void chirp_stepB(float2* line, int ka, const float4* __restrict__ bt) {
  float2 v[PL::N2];
  float4* p = reinterpret_cast<float4*>(line + ka * (PL::N2 + 2));
#pragma unroll
  for (int b = 0; b < PL::N2 / 2; ++b) {
    const float4 q = p[b];
    v[2 * b] = make_float2(q.x, q.y);
    v[2 * b + 1] = make_float2(q.z, q.w);
  }
  dft<PL::N2, false, true>(v);
#pragma unroll
  for (int kb = 0; kb < PL::N2; ++kb) {
    const float4 w = __ldg(bt + ka + PL::N1 * kb);
    v[kb] = INV ? mulc_f4(v[kb], w) : mul_f4(v[kb], w);
  }
  dft<PL::N2, true, true>(v);
#pragma unroll
  for (int b = 0; b < PL::N2 / 2; ++b)
    p[b] = make_float4(v[2 * b].x, v[2 * b].y, v[2 * b + 1].x, v[2 * b + 1].y);
}

// step A^-1 of subline b: v[a], a < N1/2, are the outputs b + N2 a before the
// final chirp (the upper half is not formed: nothing reads it)
template <class PL>
ASG_DEV void chirp_stepA_inv(const float2* line, int b, float2 (&v)[PL::N1],
                             const float4* __restrict__ tw) {
  v[0] = line[PL::pos(b)];
#pragma unroll
  for (int ka = 1; ka < PL::N1; ++ka)
    v[ka] = mulc_f4(line[PL::pos(b + PL::N2 * ka)], __ldg(tw + ka * PL::N2 + b));
  dft<PL::N1, true, true>(v);
}

// --- direct four-step transforms with the axis' twiddle layout -----------------
// forward: step A from registers (v[a] = input b + N2 a), then step B leaves
// bin ka + N1 kb in v[kb] of task ka; inverse: step B^-1 from registers (bin
// ka + N1 kb in v[kb]), then step A^-1 leaves output b + N2 a in v[a].
template <class PL>
ASG_DEV void direct_stepA(float2* line, int b, float2 (&v)[PL::N1], const float4* __restrict__ tw) {
  dft<PL::N1, false, true>(v);
  line[PL::pos(b)] = v[0];
#pragma unroll
  for (int ka = 1; ka < PL::N1; ++ka)
    line[PL::pos(b + PL::N2 * ka)] = mul_f4(v[ka], __ldg(tw + ka * PL::N2 + b));
}
template <class PL>
ASG_DEV void run_load(const float2* line, int ka, float2 (&v)[PL::N2]) {
  const float4* p = reinterpret_cast<const float4*>(line + ka * (PL::N2 + 2));
#pragma unroll
  for (int b = 0; b < PL::N2 / 2; ++b) {
    const float4 q = p[b];
    v[2 * b] = make_float2(q.x, q.y);
    v[2 * b + 1] = make_float2(q.z, q.w);
  }
}
template <class PL>
ASG_DEV void run_store(float2* line, int ka, const float2 (&v)[PL::N2]) {
  float4* p = reinterpret_cast<float4*>(line + ka * (PL::N2 + 2));
#pragma unroll
  for (int b = 0; b < PL::N2 / 2; ++b)
    p[b] = make_float4(v[2 * b].x, v[2 * b].y, v[2 * b + 1].x, v[2 * b + 1].y);
}

// Padded line stride (complex) for lanes running over CL lines first: lines
// start 16 / CL complex apart modulo the 16 of one 128-byte wavefront, so 16
// lanes over CL lines and 16 / CL neighbouring slots meet no bank twice.  Even
// (float4 runs): CL <= 8.
template <class PL, int CL>
struct LineStride {
  static constexpr int R = CL >= 16 ? 2 : 16 / CL;
  static constexpr int value = PL::PADDED + ((R - PL::PADDED % 16) % 16 + 16) % 16;
};
inline int line_stride(int padded, int cl) {
  const int r = cl >= 8 ? 2 : 16 / cl;
  return padded + ((r - padded % 16) % 16 + 16) % 16;
}
