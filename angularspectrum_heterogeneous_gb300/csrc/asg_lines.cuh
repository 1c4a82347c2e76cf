// Line transforms of any length in shared memory, n = n1 n2: step A takes a DFT of
// n1 points in registers, step B one of n2.
//
// A length whose two factors are among the radices below (primes up to 17
// included, as direct sums over the half-sized symmetric and antisymmetric parts)
// is transformed directly (200 x 180 x 400 as 10 x 20, 12 x 15 and 20 x 20: 0.81 ms per
// step against 2.2 ms as chirp convolutions).  Every other length runs as a chirp convolution
// (Bluestein): with w_j = exp(-i pi j^2 / n),
//   X[k] = w_k sum_j (x[j] w_j) conj(w_{k-j}),
// a circular convolution of length m >= 2 n - 1, m a product of two radices.
// The convolution's forward transform, the product with the transformed chirp
// and the inverse transform take two exchanges through shared memory:
//   step A     DFT_n1 of the chirped inputs, twiddles            -> shared
//   step B     DFT_n2, times the chirp's spectrum, inverse DFT_n2 -> shared
//   step A^-1  twiddles, inverse DFT_n1, times w_k
// n <= m/2, so the upper half of step A's inputs is zero and the upper half of
// step A^-1's outputs is not needed; both DFT_n1 skip that half.
// The inverse transform uses the conjugates of both tables (the chirp is even,
// so the spectrum of its conjugate is the conjugate of its spectrum).
//
// Every factor (chirp, its spectrum, twiddles, the constants of the register DFTs) is
// kept as two floats: rounded to one, the same relative errors of 3e-8 return at
// every step of a march and add up.  20 forward/inverse pairs
// of 101 samples: error 2.4e-6 with single factors, 7.5e-7 with double ones,
// 1.6e-6 for the direct sum.
//
// Against Stockham lines with direct sums over a prime length this is O(log n)
// instead of O(n) per sample: a column pass over 257 x 257 x 601 takes 0.9 ms
// instead of 27 ms.
#pragma once
#include "asg_common.cuh"

// Block of a kernel variant whose largest radix is BIG: threads at most, blocks per SM (so
// 96, 128 or 255 registers; a few values spill in the largest).  Small blocks: their
// load, exchange and barrier phases overlap each other's (224-thread blocks, two per
// SM: 257 x 257 x 601 rows 20 % slower; one block less per SM: 200 x 180 x 400 10 %).
template <int BIG>
struct LineBlock {
  static constexpr int NT = 128;
  static constexpr int MB = BIG <= 24 ? 5 : BIG <= 48 ? 4 : 2;
};
// Device tables of one axis (built in FP64 on the host, see line_axis()).
struct LineAxis {
  int n;              // line length
  int m;              // transform length n1 n2: n when direct, else the convolution length
  int direct;
  int n1, n2;
  int s2;             // shared-memory stride of a subline (plan constant, PL::S2)
  int rm;             // direct variant: the larger of n1, n2 rounded up to 16, 24, 32 or 64
  unsigned mg1, mg2;  // ceil(2^20 / n1), ceil(2^20 / n2): exact quotients below 16384
  float inv_hi, inv_lo;  // 1/n as two floats (one would scale every inverse transform alike)
  // factors as (hi.re, hi.im, lo.re, lo.im)
  const float4* ch;   // [n] w_j (chirp axes)
  const float4* bt;   // [m] spectrum of conj(w), bins in natural order, 1/m folded in
  const float4* tw;   // W_m^(b ka) at index ka PL::TWS + b: lanes along b read it coalesced
};
__host__ __device__ inline int div_magic(int i, unsigned mg) { return (int)(((unsigned)i * mg) >> 20); }

// a * (hi + lo), and a * conj(hi + lo): a factor known to FP64 as the sum of two
// floats, the product rounded to FP32
ASG_DEV float2 cmul_hl(float2 a, float2 hi, float2 lo) {
  const float tx = fmaf(a.x, lo.x, -a.y * lo.y), ty = fmaf(a.x, lo.y, a.y * lo.x);
  return make_float2(fmaf(a.x, hi.x, fmaf(-a.y, hi.y, tx)), fmaf(a.x, hi.y, fmaf(a.y, hi.x, ty)));
}
ASG_DEV float2 mul_f4(float2 a, float4 w) {
  return cmul_hl(a, make_float2(w.x, w.y), make_float2(w.z, w.w));
}
ASG_DEV float2 mulc_f4(float2 a, float4 w) {
  return cmul_hl(a, make_float2(w.x, -w.y), make_float2(w.z, -w.w));
}
ASG_DEV float2 scale_hl(float2 a, float hi, float lo) {
  return make_float2(fmaf(a.x, hi, a.x * lo), fmaf(a.y, hi, a.y * lo));
}

// exp(-2 pi i j / N) for N <= 64 at index N (N - 1) / 2 + j, as two floats
constexpr int LINE_ROOTS = 64 * 65 / 2;
static __constant__ float4 c_roots[LINE_ROOTS];
#define ASG_DEFINE_LINE_ROOT_UPLOADER(name)                                                   \
  int name(const float4* r) {                                                                  \
    return cudaMemcpyToSymbol(c_roots, r, sizeof(float4) * LINE_ROOTS) == cudaSuccess ? 0 : -1; \
  }

// v * W_N^j (forward) or W_N^-j
template <int N, bool INV>
ASG_DEV float2 root_mul(float2 v, int j) {
  const int e = j % N;
  if (e == 0) return v;
  if (4 * e == N) return mul_mi<INV>(v);
  if (2 * e == N) return make_float2(-v.x, -v.y);
  if (4 * e == 3 * N) return mul_mi<!INV>(v);
  const float4 w = c_roots[N * (N - 1) / 2 + e];
  return INV ? mulc_f4(v, w) : mul_f4(v, w);
}

constexpr int radix_split(int n) {  // first factor of the register DFT's recursion
  return n % 4 == 0 && n > 4 ? (n % 8 == 0 && n >= 64 ? 8 : 4)
         : n % 2 == 0 ? 2 : n % 3 == 0 ? 3 : n % 5 == 0 ? 5 : n % 7 == 0 ? 7 : n;
}

// DFT of N values in registers, natural order in and out, unnormalised
template <int N, bool INV>
ASG_DEV void ldft(float2 (&v)[N]) {
  if constexpr (N == 1) {
    return;
  } else if constexpr (N == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (N == 4) {
    const float2 a = v[0], b = v[1], c = v[2], d = v[3];
    const float2 s0 = cadd(a, c), d0 = csub(a, c);
    const float2 s1 = cadd(b, d), d1 = mul_mi<INV>(csub(b, d));
    v[0] = cadd(s0, s1);
    v[2] = csub(s0, s1);
    v[1] = cadd(d0, d1);
    v[3] = csub(d0, d1);
  } else if constexpr (radix_split(N) == N) {
    // odd prime: X[m], X[N-m] = (v0 + sum_k t_k cos) -/+ i sum_k d_k sin over the sums
    // and differences t_k, d_k of v[k], v[N-k]
    constexpr int H = (N - 1) / 2;
    const float2 v0 = v[0];
    float2 t[H], d[H], x0 = v0;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      t[k - 1] = cadd(v[k], v[N - k]);
      d[k - 1] = csub(v[k], v[N - k]);
      x0 = cadd(x0, t[k - 1]);
    }
    v[0] = x0;
#pragma unroll
    for (int m = 1; m <= H; ++m) {
      // the low parts first: they survive only inside the rounding of a product (added to
      // v0 or to a rounded sum they are below half an ulp and lost: 159 x 159 x 139, 16 steps,
      // field error 1.95e-6 so, 1.07e-6 this way)
      float2 r = make_float2(0.f, 0.f), s = r;
#pragma unroll
      for (int k = 1; k <= H; ++k) {
        const float4 w = c_roots[N * (N - 1) / 2 + (k * m) % N];  // cos, -sin
        r = make_float2(fmaf(t[k - 1].x, w.z, r.x), fmaf(t[k - 1].y, w.z, r.y));
        s = make_float2(fmaf(d[k - 1].x, w.w, s.x), fmaf(d[k - 1].y, w.w, s.y));
      }
#pragma unroll
      for (int k = 1; k <= H; ++k) {
        const float4 w = c_roots[N * (N - 1) / 2 + (k * m) % N];
        r = make_float2(fmaf(t[k - 1].x, w.x, r.x), fmaf(t[k - 1].y, w.x, r.y));
        s = make_float2(fmaf(d[k - 1].x, w.y, s.x), fmaf(d[k - 1].y, w.y, s.y));
      }
      r = cadd(r, v0);
      // forward: X[m] = r + i s (s carries -sin), X[N-m] = r - i s
      const float2 is = make_float2(-s.y, s.x);
      v[m] = INV ? csub(r, is) : cadd(r, is);
      v[N - m] = INV ? cadd(r, is) : csub(r, is);
    }
  } else {
    constexpr int P = radix_split(N), Q = N / P;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      float2 t[P];
#pragma unroll
      for (int p = 0; p < P; ++p) t[p] = v[Q * p + q];
      ldft<P, INV>(t);
#pragma unroll
      for (int ka = 0; ka < P; ++ka) v[Q * ka + q] = root_mul<N, INV>(t[ka], q * ka);
    }
    float2 o[N];
#pragma unroll
    for (int ka = 0; ka < P; ++ka) {
      float2 t[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) t[q] = v[Q * ka + q];
      ldft<Q, INV>(t);
#pragma unroll
      for (int kb = 0; kb < Q; ++kb) o[ka + P * kb] = t[kb];
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = o[i];
  }
}

// Forward DFT of N values (a multiple of 4) whose upper half is zero (v[N/2..] need
// not be set).
template <int N>
ASG_DEV void ldft_lo(float2 (&v)[N]) {
  if constexpr (N == 4) {
    const float2 a = v[0], b = v[1], c = mul_mi<false>(b);
    v[0] = cadd(a, b);
    v[1] = cadd(a, c);
    v[2] = csub(a, b);
    v[3] = csub(a, c);
  } else {
    constexpr int P = radix_split(N), Q = N / P;
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
          o[p] = root_mul<8, false>(e[p], p);
        }
        ldft<4, false>(e);
        ldft<4, false>(o);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          t[2 * p] = e[p];
          t[2 * p + 1] = o[p];
        }
      }
#pragma unroll
      for (int ka = 0; ka < P; ++ka) v[Q * ka + q] = root_mul<N, false>(t[ka], q * ka);
    }
    float2 o[N];
#pragma unroll
    for (int ka = 0; ka < P; ++ka) {
      float2 t[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) t[q] = v[Q * ka + q];
      ldft<Q, false>(t);
#pragma unroll
      for (int kb = 0; kb < Q; ++kb) o[ka + P * kb] = t[kb];
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = o[i];
  }
}

// ---------------------------------------------------------------------------
// Plans.  Sublines are S2 complex apart in shared memory, even with S2 / 2 odd: a
// step's strided 8-byte accesses and the 16-byte accesses of a run meet no bank
// twice, and with S2 and the twiddle stride TWS known to the compiler every
// access of a step is an immediate offset from one address (run-time strides
// cost an integer multiply each: the chirp passes of 257 x 257 x 601 took 1.3-1.5 times as long).
//
// ChirpPlan: the convolution length's factors, compile-time.
// DirectPlan: any n1, n2 among the radices of a variant, the code of a radix picked
// by a switch that is uniform over the block: f(Radix<R>).
// The host's plan picks from the same lists (line_axis()).
// ---------------------------------------------------------------------------
template <int R>
struct Radix {
  static constexpr int v = R;
};

template <int N1, int N2>
struct ChirpPlan {
  static constexpr bool DIRECT = false;
  static constexpr int BIG = N1 > N2 ? N1 : N2, S2 = N2 + 2, TWS = N2;
  static_assert(N1 % 4 == 0 && N2 % 4 == 0 && (S2 / 2) % 2 == 1, "chirp radices");
  ASG_DEV static constexpr int n1(const LineAxis&) { return N1; }
  ASG_DEV static constexpr int n2(const LineAxis&) { return N2; }
  ASG_DEV static int div1(const LineAxis&, int i) { return i / N1; }
  ASG_DEV static int div2(const LineAxis&, int i) { return i / N2; }
  template <class F>
  ASG_DEV static void with_n1(const LineAxis&, F f) { f(Radix<N1>{}); }
  template <class F>
  ASG_DEV static void with_n2(const LineAxis&, F f) { f(Radix<N2>{}); }
};

// Radices of the direct variant RM: all up to 18 and the 7-smooth ones up to RM, 32 at
// most; the variant for lengths above 1024 (RM = 64) has some from 27 to 64.
constexpr bool line_radix(int rm, int r) {
  if (rm == 64)
    return r == 27 || r == 28 || r == 30 || r == 32 || r == 36 || r == 40 || r == 48 || r == 64;
  return r >= 1 && r <= rm &&
         (r <= 18 || r == 20 || r == 21 || r == 24 || r == 25 || r == 27 || r == 28 || r == 30 ||
          r == 32);
}
// Operations per value of a register DFT of r points, roughly: a direct sum over a
// prime, a radix-4 split as two stages of 2.
constexpr int radix_cost(int r) {
  int c = 0;
  while (r % 4 == 0) { c += 4; r /= 4; }
  for (int q = 2; r > 1; ++q)
    while (r % q == 0) { c += q; r /= q; }
  return c;
}
// Direct lines: for each length the cheapest pair n1 <= n2 of radices (0: none), its
// variant, and which radices a variant meets as n1 or as n2.  The kernels hold the code
// of those only.
constexpr int LINE_DIRECT_MAX = 2048;
struct LineDirect {
  unsigned char n1[LINE_DIRECT_MAX + 1], n2[LINE_DIRECT_MAX + 1], rm[LINE_DIRECT_MAX + 1];
  bool used[2][65][65];  // [n1, n2][variant][radix]
};
constexpr LineDirect make_line_direct() {
  LineDirect d{};
  int best[LINE_DIRECT_MAX + 1] = {};
  for (int a = 1; a <= 64; ++a)
    for (int b = a; b <= 64 && a * b <= LINE_DIRECT_MAX; ++b) {
      const int n = a * b;
      if (!line_radix(n > 1024 ? 64 : 32, a) || !line_radix(n > 1024 ? 64 : 32, b)) continue;
      // the larger variants hold fewer warps per SM; an exchange costs about as much as a
      // radix-4 stage
      const int c = radix_cost(a) + radix_cost(b) + (a > 1 ? 3 : 0) + (b - a) / 4 +
                    (n > 1024 ? 8 : b > 16 ? 4 : 0);
      if (best[n] != 0 && c >= best[n]) continue;
      best[n] = c;
      d.n1[n] = (unsigned char)a;
      d.n2[n] = (unsigned char)b;
      d.rm[n] = (unsigned char)(n > 1024 ? 64 : b <= 16 ? 16 : b <= 24 ? 24 : 32);
    }
  for (int n = 1; n <= LINE_DIRECT_MAX; ++n)
    if (d.n1[n] != 0) d.used[0][d.rm[n]][d.n1[n]] = d.used[1][d.rm[n]][d.n2[n]] = true;
  return d;
}
constexpr LineDirect LINE_DIRECT = make_line_direct();

template <int RM>
struct DirectPlan {
  static constexpr bool DIRECT = true;
  static constexpr int BIG = RM, S2 = RM + 2, TWS = RM;
  ASG_DEV static int n1(const LineAxis& ax) { return ax.n1; }
  ASG_DEV static int n2(const LineAxis& ax) { return ax.n2; }
  ASG_DEV static int div1(const LineAxis& ax, int i) { return div_magic(i, ax.mg1); }
  ASG_DEV static int div2(const LineAxis& ax, int i) { return div_magic(i, ax.mg2); }
  // f(Radix<R>) of the radix R that a line has as n1 (POS 0) or n2 (POS 1)
  template <int POS, class F>
  ASG_DEV static void with_radix(int r, F f) {
#define R_(R) \
  case R:     \
    if constexpr (LINE_DIRECT.used[POS][RM][R]) f(Radix<R>{}); \
    break;
    switch (r) {
      R_(1) R_(2) R_(3) R_(4) R_(5) R_(6) R_(7) R_(8) R_(9) R_(10) R_(11) R_(12) R_(13) R_(14)
      R_(15) R_(16) R_(17) R_(18) R_(20) R_(21) R_(24) R_(25) R_(27) R_(28) R_(30) R_(32)
      R_(36) R_(40) R_(48) R_(64) default: break;
    }
#undef R_
  }
  template <class F>
  ASG_DEV static void with_n1(const LineAxis& ax, F f) { with_radix<0>(ax.n1, f); }
  template <class F>
  ASG_DEV static void with_n2(const LineAxis& ax, F f) { with_radix<1>(ax.n2, f); }
};

// position of natural index j in a line
template <class PL>
ASG_DEV int line_pos(const LineAxis& ax, int j) {
  return j + PL::div2(ax, j) * (PL::S2 - PL::n2(ax));
}

// --- the steps on one subline -------------------------------------------------
// step A: v[a] = input b + n2 a (a < n1/2 in the chirp form) -> twiddled bins
template <class PL, int N1>
ASG_DEV void line_stepA(float2* line, int b, float2 (&v)[N1], const LineAxis& ax) {
  if constexpr (PL::DIRECT) ldft<N1, false>(v);
  else ldft_lo<N1>(v);
  line[b] = v[0];
  const float4* tw = ax.tw + b;
#pragma unroll
  for (int ka = 1; ka < N1; ++ka)
    line[b + PL::S2 * ka] = mul_f4(v[ka], __ldg(tw + ka * PL::TWS));
}
// step A^-1: v[a] = output b + n2 a (of the chirp form the lower half is used)
template <class PL, int N1>
ASG_DEV void line_stepA_inv(const float2* line, int b, float2 (&v)[N1], const LineAxis& ax) {
  v[0] = line[b];
  const float4* tw = ax.tw + b;
#pragma unroll
  for (int ka = 1; ka < N1; ++ka)
    v[ka] = mulc_f4(line[b + PL::S2 * ka], __ldg(tw + ka * PL::TWS));
  ldft<N1, true>(v);
}
// a run of N2 values of one subline (16-byte accesses)
template <int N2>
ASG_DEV void run_load(const float2* run, float2 (&v)[N2]) {
#pragma unroll
  for (int b = 0; b + 1 < N2; b += 2) {
    const float4 q = *reinterpret_cast<const float4*>(run + b);
    v[b] = make_float2(q.x, q.y);
    v[b + 1] = make_float2(q.z, q.w);
  }
  if constexpr (N2 % 2 == 1) v[N2 - 1] = run[N2 - 1];
}
template <int N2>
ASG_DEV void run_store(float2* run, const float2 (&v)[N2]) {
#pragma unroll
  for (int b = 0; b + 1 < N2; b += 2)
    *reinterpret_cast<float4*>(run + b) = make_float4(v[b].x, v[b].y, v[b + 1].x, v[b + 1].y);
  if constexpr (N2 % 2 == 1) run[N2 - 1] = v[N2 - 1];
}
// step B of the chirp form: DFT_n2, the chirp's spectrum (conj: of the inverse
// transform), inverse DFT_n2, in place
template <class PL, int N2>
ASG_DEV void chirp_stepB(float2* run, int ka, const LineAxis& ax, bool conj) {
  float2 v[N2];
  run_load<N2>(run, v);
  ldft<N2, false>(v);
  const float4* bt = ax.bt + ka;
  const float sg = conj ? -1.f : 1.f;
#pragma unroll
  for (int kb = 0; kb < N2; ++kb) {
    float4 w = __ldg(bt + PL::n1(ax) * kb);
    w.y *= sg;
    w.w *= sg;
    v[kb] = mul_f4(v[kb], w);
  }
  ldft<N2, true>(v);
  run_store<N2>(run, v);
}
// chirp factor at `ch`, conjugated for the inverse transform
ASG_DEV float2 chirp_mul(float2 v, const float4* ch, bool conj) {
  float4 w = __ldg(ch);
  if (conj) {
    w.y = -w.y;
    w.w = -w.w;
  }
  return mul_f4(v, w);
}

// Line stride (complex) of a block whose lanes run over cl lines first (a power of two):
// lines start 16 / cl complex apart modulo the 16 of one 128-byte wavefront, so
// 16 lanes over cl lines and 16 / cl neighbouring slots meet no bank twice.
inline int line_stride(const LineAxis& ax, int cl) {
  const int len = ax.n1 * ax.s2, r = cl >= 8 ? 2 : 16 / cl;  // even: runs are 16-byte aligned
  return len + ((r - len % 16) % 16 + 16) % 16;
}
// threads of a block with `tasks` tasks per step: as few rounds as the variant's
// largest block allows, no larger than they need
inline int line_threads(int tasks, int nt_max) {
  const int rounds = (tasks + nt_max - 1) / nt_max;
  const int t = ((tasks + rounds - 1) / rounds + 31) / 32 * 32;
  return t < 32 ? 32 : t;
}
// tasks per line of the step with the larger radix (the other step has more, smaller ones):
// a block takes as many lines as these need to fill it
inline int line_tasks(const LineAxis& ax) { return ax.n1 < ax.n2 ? ax.n1 : ax.n2; }

// Factors of the chirp convolutions: each length at most 1.5 times the one before, from
// 128 on 1.33 times.  F(n1, n2)
#define ASG_CHIRP_SIZES(F)                                                               \
  F(4, 12) F(8, 8) F(8, 12) F(8, 16) F(8, 20) F(12, 16) F(16, 16) F(16, 20)     \
  F(16, 24) F(16, 32) F(24, 24) F(20, 32) F(24, 32) F(32, 32) F(32, 40) F(32, 48) F(32, 64)
