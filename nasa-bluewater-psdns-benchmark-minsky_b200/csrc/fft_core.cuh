// fft_core.cuh -- batched 1-D complex FFT of lines held in shared memory.
//
// Replaces the FFTW 1-D transforms the reference plans in PSDNS/epfftw.f
// (plan4_p1/plan4_p3 along y, plan2_kx/plan2_xk along z, plan3_p2c/plan1_p2b
// along x).  Unnormalised forward transform X_k = sum_j x_j exp(-2 pi i jk/N);
// INV: the backward one, with conjugate twiddles in the same passes (K1 and K2;
// the x chain, whose pairs of real lines come conjugated, transforms forward both
// ways).
//
// Algorithm: Stockham auto-sort with mixed register radices.  A line of N
// points is split into passes of radix R_p (product = N).  In every pass each
// thread owns E/R_p butterflies of radix R_p whose operands it holds in
// registers; the radix-R kernels are unrolled at compile time.  Between passes
// data goes through shared memory in place: all operands are read, the threads of
// the line synchronise, then all results are written.  Element i of a line lives at
// padl(i), which keeps the strided writes of the first pass from serialising
// on one bank.
//
// What bounds the transforms inside the kernels is the number of instructions
// issued, not the FMA pipe (with scalar arithmetic and the twiddles multiplied
// onto the operands the x chain issued 0.59 per cycle and scheduler at 40% of that
// pipe; in this form 0.61, in a quarter fewer instructions: 914 -> 690 million a
// launch at 512^3 FP32), so the arithmetic is arranged for few instructions:
//  * Complex sums, and the sums of a twiddled butterfly, are packed FP32 pair
//    instructions (add, subtract, fma of (re, im)): one issue slot instead of
//    two, with the rounding of the scalar forms.
//  * A butterfly e +- w o with w = c (1 - i T), T = tan, is u = o (1 - i T)
//    (two scalar fma) and e +- c u (two packed fma): 4 instructions instead of
//    8.  Each component is rounded twice instead of three times.  (The form of
//    Linzer and Feig, Math. Comp. 60, 1993, and Goedecker, SIAM J. Sci. Comput.
//    18, 1997, for fused multiply-add machines.)
//  * The inter-pass twiddles are not applied to the operands before a radix-R
//    kernel but inside its butterflies, stage by stage, where a twiddle costs
//    nothing beyond the table load: a radix-R pass needs R/2 pairs (c, T) per
//    thread, one of each pair of twiddles that differ by a quarter turn.
#pragma once
#include <cmath>
#include <type_traits>
#include <cuda_runtime.h>
#include <stdint.h>

namespace psdns {

template <typename T> struct V2;
template <> struct V2<float> { using type = float2; };
template <> struct V2<double> { using type = double2; };
template <typename T> using C2 = typename V2<T>::type;

template <typename C> struct ElemOf;
template <> struct ElemOf<float2> { using type = float; };
template <> struct ElemOf<double2> { using type = double; };

template <typename C>
__host__ __device__ __forceinline__ C cmk(typename ElemOf<C>::type a, typename ElemOf<C>::type b) {
  C r; r.x = a; r.y = b; return r;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return cmk<C>(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return cmk<C>(a.x - b.x, a.y - b.y); }
// e + c u for real c
__device__ __forceinline__ double2 cfma(double c, double2 u, double2 e) {
  return make_double2(fma(c, u.x, e.x), fma(c, u.y, e.y));
}
#ifdef __CUDA_ARCH__
// the packed FP32 forms (sm_100a)
template <> __device__ __forceinline__ float2 cadd<float2>(float2 a, float2 b) { return __fadd2_rn(a, b); }
template <> __device__ __forceinline__ float2 csub<float2>(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
__device__ __forceinline__ float2 cfma(float c, float2 u, float2 e) { return __ffma2_rn(make_float2(c, c), u, e); }
#else
__device__ __forceinline__ float2 cfma(float c, float2 u, float2 e) {
  return make_float2(fmaf(c, u.x, e.x), fmaf(c, u.y, e.y));
}
#endif
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
  return cmk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename C> __device__ __forceinline__ C cconj(C a) { return cmk<C>(a.x, -a.y); }
template <typename C> __device__ __forceinline__ C cscale(typename ElemOf<C>::type s, C a) {
  return cmk<C>(s * a.x, s * a.y);
}
// multiply by -i (forward quarter turn)
template <typename C> __device__ __forceinline__ C cmul_mi(C a) { return cmk<C>(a.y, -a.x); }
// multiply by +i
template <typename C> __device__ __forceinline__ C cmul_pi(C a) { return cmk<C>(-a.y, a.x); }

// ---------------------------------------------------------------------------
// Compile-time cos/sin of 2*pi*k/R (Taylor series on a quadrant-reduced
// argument |phi| <= pi/4; exact to double rounding for the radices used).
// ---------------------------------------------------------------------------
__host__ __device__ constexpr double ct_sin_small(double x) {
  double x2 = x * x, term = x, sum = x;
  for (int n = 1; n < 14; n++) { term = -term * x2 / double((2 * n) * (2 * n + 1)); sum += term; }
  return sum;
}
__host__ __device__ constexpr double ct_cos_small(double x) {
  double x2 = x * x, term = 1.0, sum = 1.0;
  for (int n = 1; n < 14; n++) { term = -term * x2 / double((2 * n - 1) * (2 * n)); sum += term; }
  return sum;
}
// returns cos(2 pi k / R) (which = 0) or sin(2 pi k / R) (which = 1)
__host__ __device__ constexpr double ct_trig(int k, int R, int which) {
  int m = ((k % R) + R) % R;
  // 4m/R = q + f with q the nearest quadrant, |f| <= 1/2
  long num = 4L * m;            // angle = (num / R) * (pi/2)
  long q = (2 * num + R) / (2 * R);   // round(num / R)
  double f = double(num - q * R) / double(R);   // in [-1/2, 1/2]
  double phi = f * 1.57079632679489661923;
  double c = ct_cos_small(phi), s = ct_sin_small(phi);
  int qq = int(q % 4);
  double cc = 0, ss = 0;
  if (qq == 0) { cc = c; ss = s; }
  else if (qq == 1) { cc = -s; ss = c; }
  else if (qq == 2) { cc = -c; ss = -s; }
  else { cc = s; ss = -c; }
  return which == 0 ? cc : ss;
}

// multiply o by W_R^K = exp(-2 pi i K / R) with compile-time constants
template <int K, int R, typename C>
__device__ __forceinline__ C tw_const(C o) {
  using T = typename ElemOf<C>::type;
  constexpr int k = ((K % R) + R) % R;
  if constexpr (k == 0) {
    return o;
  } else if constexpr (4 * k == R) {
    return cmul_mi(o);
  } else if constexpr (2 * k == R) {
    return cmk<C>(-o.x, -o.y);
  } else if constexpr (4 * k == 3 * R) {
    return cmul_pi(o);
  } else if constexpr (8 * k == R) {
    constexpr T h = T(0.70710678118654752440);
    return cmk<C>((o.x + o.y) * h, (o.y - o.x) * h);
  } else if constexpr (8 * k == 3 * R) {
    constexpr T h = T(0.70710678118654752440);
    return cmk<C>((o.y - o.x) * h, -(o.x + o.y) * h);
  } else {
    constexpr T cr = T(ct_trig(k, R, 0));
    constexpr T ci = T(-ct_trig(k, R, 1));
    return cmk<C>(o.x * cr - o.y * ci, o.x * ci + o.y * cr);
  }
}

// In-register DFT of R points v[0], v[S], ..., v[(R-1)S] (natural order in
// and out), forward sign (INV: backward).  Radix-2 decimation in time,
// radix-4 and radix-3 leaves.
// ---------------------------------------------------------------------------
template <int R, int S, bool INV = false, typename C> __device__ __forceinline__ void dft_s(C* v);

// p = e + w o, m = e - w o with w = c (1 - i T) (INV: its conjugate), turned
// by a further -i (INV: +i) if QUARTER
template <bool INV, bool QUARTER, typename C>
__device__ __forceinline__ void bfly(C e, C o, typename ElemOf<C>::type c, typename ElemOf<C>::type T, C& p, C& m) {
  C u;
  if constexpr (!INV && !QUARTER) u = cmk<C>(fma(T, o.y, o.x), fma(-T, o.x, o.y));
  else if constexpr (INV && !QUARTER) u = cmk<C>(fma(-T, o.y, o.x), fma(T, o.x, o.y));
  else if constexpr (!INV) u = cmk<C>(fma(-T, o.x, o.y), fma(-T, o.y, -o.x));
  else u = cmk<C>(fma(-T, o.x, -o.y), fma(-T, o.y, o.x));
  p = cfma(c, u, e);
  m = cfma(-c, u, e);
}

// p = e -+ i o, m = e +- i o (upper signs: forward); the swapped components
// make scalar sums the shorter form
template <bool INV, typename C>
__device__ __forceinline__ void bfly_quarter(C e, C o, C& p, C& m) {
  const C a = cmk<C>(e.x + o.y, e.y - o.x), b = cmk<C>(e.x - o.y, e.y + o.x);
  p = INV ? b : a;
  m = INV ? a : b;
}

// butterfly K of a radix-R combine step: p, m = e +- W_R^K o, 0 <= K < R/2
template <int K, int R, bool INV, typename C>
__device__ __forceinline__ void bfly_const(C e, C o, C& p, C& m) {
  using T = typename ElemOf<C>::type;
  if constexpr (K == 0) {
    p = cadd(e, o);
    m = csub(e, o);
  } else if constexpr (4 * K == R) {
    bfly_quarter<INV>(e, o, p, m);
  } else {
    constexpr bool Q = 4 * K > R;
    // angle of the twiddle after the quarter turn: 2 pi j / (4 R) in (0, pi/2)
    constexpr int j = 4 * K - (Q ? R : 0);
    bfly<INV, Q>(e, o, T(ct_trig(j, 4 * R, 0)), T(ct_trig(j, 4 * R, 1) / ct_trig(j, 4 * R, 0)), p, m);
  }
}

template <int K, int R, int S, bool INV, typename C>
__device__ __forceinline__ void dit2_combine(C* v, C* tmp) {
  if constexpr (K < R / 2) {
    bfly_const<K, R, INV>(v[2 * S * K], v[S + 2 * S * K], tmp[K], tmp[K + R / 2]);
    dit2_combine<K + 1, R, S, INV>(v, tmp);
  }
}

template <int K, int R, int S, bool INV, typename C>
__device__ __forceinline__ void dit3_combine(C* v, C* tmp) {
  using T = typename ElemOf<C>::type;
  if constexpr (K < R / 3) {
    constexpr int M = R / 3;
    C a = v[3 * S * K];
    C b = tw_const<INV ? -K : K, R>(v[S + 3 * S * K]);
    C c = tw_const<INV ? -2 * K : 2 * K, R>(v[2 * S + 3 * S * K]);
    // radix-3 butterfly, W3 = exp(-+2 pi i/3) = (-1/2, -+sqrt(3)/2)
    constexpr T h = INV ? T(-0.86602540378443864676) : T(0.86602540378443864676);
    C s = cadd(b, c), d = csub(b, c);
    C m = cmk<C>(a.x - T(0.5) * s.x, a.y - T(0.5) * s.y);
    C r = cmk<C>(h * d.y, -h * d.x);   // -+i*sqrt(3)/2 * d
    tmp[K] = cadd(a, s);
    tmp[K + M] = cadd(m, r);
    tmp[K + 2 * M] = csub(m, r);
    dit3_combine<K + 1, R, S, INV>(v, tmp);
  }
}

template <int R, int S, bool INV, typename C>
__device__ __forceinline__ void dft_s(C* v) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    C a = v[0], b = v[S];
    v[0] = cadd(a, b);
    v[S] = csub(a, b);
  } else if constexpr (R == 4) {
    C a = v[0], b = v[S], c = v[2 * S], d = v[3 * S];
    C t0 = cadd(a, c), t1 = csub(a, c), t2 = cadd(b, d), t3 = csub(b, d);
    v[0] = cadd(t0, t2);
    v[2 * S] = csub(t0, t2);
    bfly_quarter<INV>(t1, t3, v[S], v[3 * S]);
  } else if constexpr (R % 4 == 0 || R % 2 == 0 && R % 3 != 0) {
    dft_s<R / 2, 2 * S, INV>(v);
    dft_s<R / 2, 2 * S, INV>(v + S);
    C tmp[R];
    dit2_combine<0, R, S, INV>(v, tmp);
#pragma unroll
    for (int k = 0; k < R; k++) v[S * k] = tmp[k];
  } else if constexpr (R % 3 == 0) {
    dft_s<R / 3, 3 * S, INV>(v);
    dft_s<R / 3, 3 * S, INV>(v + S);
    dft_s<R / 3, 3 * S, INV>(v + 2 * S);
    C tmp[R];
    dit3_combine<0, R, S, INV>(v, tmp);
#pragma unroll
    for (int k = 0; k < R; k++) v[S * k] = tmp[k];
  } else {
    static_assert(R % 2 == 0 || R % 3 == 0, "unsupported radix");
  }
}

// Twiddled DFT of a pass p >= 1: v[q] <- sum_r v[r] W_(NS R)^(r (k + NS q)),
// R a power of two, natural order in and out.  Decimation in time: the
// combine step of radix rho = 2, 4, .., R multiplies its odd half by
// W_(NS rho)^(k + NS q'), q' < rho/2, of which q' and q' + rho/4 differ by a
// quarter turn.  tw[row * NS] holds this thread's (c, T): row 0 for rho = 2,
// row rho/4 + q' for rho >= 4 (q' < rho/4); see build_twiddles.
template <int R, int NS, bool INV, typename C>
__device__ __forceinline__ void dft_tw(C* v, const C* __restrict__ tw) {
  static_assert(R >= 2 && (R & (R - 1)) == 0, "power-of-two radix");
  constexpr int LOG = R == 2 ? 1 : R == 4 ? 2 : R == 8 ? 3 : R == 16 ? 4 : R == 32 ? 5 : 6;
  C a[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    int j = 0;
#pragma unroll
    for (int b = 0; b < LOG; b++) j |= ((i >> b) & 1) << (LOG - 1 - b);
    a[i] = v[j];
  }
  {
    // k = NS/2 turns by a quarter, whose tangent does not exist: its pair is
    // marked by c = 2 and holds T = 1/2, and w = c (0 - i T).  The other tangents
    // are at most N / 2 pi, and an operand that much below the type's largest
    // value still passes.  (A tangent of 2^40 for the quarter would lose that much
    // of the range; the selects cost 0.8% of a step at 1024^3 FP32, less at the
    // other sizes.  Multiplying by 0 or 1 instead took the same in FP32, but 9%
    // of K2 at 512^3 FP64.)
    const C w = tw[0];
    const bool quarter = w.x > 1;
#pragma unroll
    for (int b = 0; b < R; b += 2) {
      const C o = a[b + 1], so = quarter ? cmk<C>(0, 0) : o;
      const C u = INV ? cmk<C>(fma(-w.y, o.y, so.x), fma(w.y, o.x, so.y))
                      : cmk<C>(fma(w.y, o.y, so.x), fma(-w.y, o.x, so.y));
      a[b + 1] = cfma(-w.x, u, a[b]);
      a[b] = cfma(w.x, u, a[b]);
    }
  }
#pragma unroll
  for (int l = 2; l <= LOG; l++) {
    const int rho = 1 << l;
#pragma unroll
    for (int q = 0; q < rho / 4; q++) {
      const C w = tw[(rho / 4 + q) * NS];
#pragma unroll
      for (int b = q; b < R; b += rho) {
        bfly<INV, false>(a[b], a[b + rho / 2], w.x, w.y, a[b], a[b + rho / 2]);
        bfly<INV, true>(a[b + rho / 4], a[b + 3 * rho / 4], w.x, w.y, a[b + rho / 4], a[b + 3 * rho / 4]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < R; i++) v[i] = a[i];
}

// ---------------------------------------------------------------------------
// Pass plans.  N = R0 * R1 [* R2]; E = max radix (operands per thread),
// P = N / E threads per line.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int ilog2c(int n) { int k = 0; while ((1 << k) < n) k++; return k; }

__host__ __device__ constexpr bool is_pow2(int n) { return n > 0 && (n & (n - 1)) == 0; }
__host__ __device__ constexpr int plan_npass(int N, bool dbl) {
  return is_pow2(N) ? ((ilog2c(N) <= 3) ? 1 : ((dbl && ilog2c(N) >= 9) ? 3 : 2)) : 2;
}
__host__ __device__ constexpr int plan_rad(int N, bool dbl, int p) {
  if (is_pow2(N)) {
    const int K = ilog2c(N), np = plan_npass(N, dbl);
    if (np == 1) return p == 0 ? N : 1;
    if (np == 2) return p == 0 ? (1 << (K / 2)) : (p == 1 ? (1 << (K - K / 2)) : 1);
    const int a = (K + 2) / 3, b = (K - a + 1) / 2, c = K - a - b;
    return p == 0 ? (1 << a) : (p == 1 ? (1 << b) : (p == 2 ? (1 << c) : 1));
  }
  if (N == 48) return p == 0 ? 12 : (p == 1 ? 4 : 1);
  if (N == 96) return p == 0 ? 12 : (p == 1 ? 8 : 1);
  return 1;
}
__host__ __device__ constexpr int gcd_i(int a, int b) { return b == 0 ? a : gcd_i(b, a % b); }
// operands per thread: a multiple of every radix (their lcm), so that each
// pass gives every thread whole butterflies
__host__ __device__ constexpr int plan_e(int N, bool dbl) {
  int e = 1;
  for (int p = 0; p < 3; p++) { int r = plan_rad(N, dbl, p); e = e / gcd_i(e, r) * r; }
  return e;
}
__host__ __device__ constexpr int plan_ns(int N, bool dbl, int p) {
  int s = 1; for (int i = 0; i < p; i++) s *= plan_rad(N, dbl, i); return s;
}
// (c, T) pairs of pass p >= 1: R/2 rows of NS (dft_tw)
__host__ __device__ constexpr int plan_twsz(int N, bool dbl, int p) {
  return plan_rad(N, dbl, p) / 2 * plan_ns(N, dbl, p);
}
__host__ __device__ constexpr int plan_twoff(int N, bool dbl, int p) {
  int o = 0; for (int i = 1; i < p; i++) o += plan_twsz(N, dbl, i); return o;
}

template <typename T, int N> struct FFTPlan {
  static constexpr bool DBL = sizeof(T) == 8;
  static_assert(is_pow2(N) || N == 48 || N == 96, "N must be a power of two, 48 or 96");
  static constexpr int NPASS = plan_npass(N, DBL);
  static constexpr int rad(int p) { return plan_rad(N, DBL, p); }
  static constexpr int E = plan_e(N, DBL);
  static constexpr int P = N / E;   // threads per line
  static_assert(P * E == N, "operands per thread must divide the line");
  static constexpr int ns(int p) { return plan_ns(N, DBL, p); }
  static constexpr int twoff(int p) { return plan_twoff(N, DBL, p); }
  static constexpr int TWSIZE = plan_twoff(N, DBL, plan_npass(N, DBL)) > 0 ? plan_twoff(N, DBL, plan_npass(N, DBL)) : 1;
};

// Shared-memory place of element i of a line: i + i/R0 for a power-of-two
// first radix R0 (i + i/32 otherwise).  Pass 0 writes with a stride of R0
// between threads, which then becomes R0 + 1: no two threads of a phase meet
// on a bank (with i/32 for every plan the 16-point first passes of n = 256 and
// 512 met two by two, the 8-point ones of FP64 n = 512 four by four).
__host__ __device__ constexpr int pad_shift(int N, bool dbl) {
  return is_pow2(plan_rad(N, dbl, 0)) ? ilog2c(plan_rad(N, dbl, 0)) : 5;
}
template <typename C, int N>
__host__ __device__ __forceinline__ constexpr int padl(int i) {
  return i + (i >> pad_shift(N, sizeof(C) == 16));
}
// elements from one line to the next: N and its padding, rounded up to
// residue M modulo 16 (FP32) or 8 (FP64), the banks of one phase.  4 (8 for
// eight threads a line) keeps the lines that share a phase apart in every
// pass; see the kernels for other residues.
__host__ __device__ constexpr int line_stride(int N, bool dbl, int M) {
  const int mod = dbl ? 8 : 16;
  int l = N + (N >> pad_shift(N, dbl));
  while (l % mod != M % mod) l++;
  return l;
}
template <typename T, int N> struct LS {
  static constexpr bool DBL = sizeof(T) == 8;
  static constexpr int value = line_stride(N, DBL, !DBL && N / plan_e(N, DBL) == 8 ? 8 : 4);
};

// Barrier among the threads that share a line.  A warp barrier where lines
// live inside warps; where a line is P / 32 whole warps, the named barrier of
// the line's group (1 + its index in the block, at most 15 groups), so that the
// lines of a block do not wait for one another.
template <int P>
__device__ __forceinline__ void line_sync() {
  if constexpr (P <= 32 && (32 % P) == 0) {
    __syncwarp();
  } else if constexpr (P % 32 == 0) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / P), "n"(P) : "memory");
  } else {
    __syncthreads();
  }
}

// Operands of butterfly set q of thread t in one Stockham pass: read from the
// line, twiddled, transformed in registers (v[q R .. q R + R - 1]).
template <typename C, int N, int R, int NS, int E, int P, bool INV = false>
__device__ __forceinline__ void pass_butterflies(const C* line, int t, const C* __restrict__ twp, C* v) {
  constexpr int NB = E / R;
#pragma unroll
  for (int q = 0; q < NB; q++) {
    const int j = t + q * P;
#pragma unroll
    for (int r = 0; r < R; r++) v[q * R + r] = line[padl<C, N>(j + r * (N / R))];
    if constexpr (NS > 1)
      dft_tw<R, NS, INV>(v + q * R, twp + j % NS);
    else
      dft_s<R, 1, INV>(v + q * R);
  }
}

// One Stockham pass over nlines lines (rounds of LPR lines).
template <typename C, int N, int R, int NS, int E, int P, int THREADS, bool INV = false>
__device__ __forceinline__ void fft_pass(C* buf, int nlines, int ls, const C* __restrict__ twp) {
  constexpr int LPR = THREADS / P;
  constexpr int NB = E / R;   // butterflies per thread
  static_assert(NB * R == E && NB * P * R == N, "a pass must give every thread whole butterflies");
  const int tid = threadIdx.x;
  const int lr = tid / P, t = tid % P;
  for (int l0 = 0; l0 < nlines; l0 += LPR) {
    const int l = l0 + lr;
    const bool act = (lr < LPR) && (l < nlines);
    C v[E];
    C* line = buf + (size_t)l * ls;
    if (act) pass_butterflies<C, N, R, NS, E, P, INV>(line, t, twp, v);
    line_sync<P>();
    if (act) {
#pragma unroll
      for (int q = 0; q < NB; q++) {
        const int j = t + q * P;
        const int k = j % NS;
        const int base = (j / NS) * NS * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) line[padl<C, N>(base + r * NS)] = v[q * R + r];
      }
    }
    line_sync<P>();
  }
}

template <typename T, int N, int THREADS, int PASS, bool INV = false>
__device__ __forceinline__ void fft_passes(C2<T>* buf, int nlines, int ls, const C2<T>* tw) {
  using PL = FFTPlan<T, N>;
  if constexpr (PASS < PL::NPASS) {
    constexpr int R = PL::rad(PASS);
    constexpr int NS = PL::ns(PASS);
    fft_pass<C2<T>, N, R, NS, PL::E, PL::P, THREADS, INV>(buf, nlines, ls, tw + PL::twoff(PASS));
    fft_passes<T, N, THREADS, PASS + 1, INV>(buf, nlines, ls, tw);
  }
}

// Forward FFT of nlines lines in shared memory (line l at buf + l*ls,
// element i at padl(i)); tw = shared twiddle table of FFTPlan<T,N>.
// Must be called by all THREADS threads of the block (contains barriers).
template <typename T, int N, int THREADS>
__device__ __forceinline__ void fft_lines(C2<T>* buf, int nlines, int ls, const C2<T>* tw) {
  static_assert(THREADS % FFTPlan<T, N>::P == 0, "THREADS must be a multiple of threads per line");
  fft_passes<T, N, THREADS, 0>(buf, nlines, ls, tw);
  // results are read by other warps afterwards
  __syncthreads();
}

// Pass 0 of the plan with operands that the caller supplies from registers:
// s = begin(l) describes line l, fetch(s, i) loads its element i (typically
// a predicated global load) and fix(s, i, raw) turns the raw value into the
// operand (shift, mask, derivative ...).  A thread issues the fetches of all
// its operands before the first fix, so that its loads are in flight
// together whatever branches fix takes.  Pass 0 has no twiddles; its output
// goes to the line in shared memory, so the staging copy of the input (a
// shared-memory write and read per element) disappears.
template <typename T, int N, int THREADS, bool INV = false, typename Begin, typename Fetch, typename Fix>
__device__ __forceinline__ void fft_pass0_load(C2<T>* buf, int nlines, int ls, Begin begin, Fetch fetch, Fix fix) {
  using C = C2<T>;
  using PL = FFTPlan<T, N>;
  constexpr int R = PL::rad(0), E = PL::E, P = PL::P;
  constexpr int LPR = THREADS / P;
  constexpr int NB = E / R;
  const int lr = threadIdx.x / P, t = threadIdx.x % P;
  for (int l0 = 0; l0 < nlines; l0 += LPR) {
    const int l = l0 + lr;
    if (l < nlines) {
      const auto s = begin(l);
      C v[E];
#pragma unroll
      for (int q = 0; q < NB; q++)
#pragma unroll
        for (int r = 0; r < R; r++) v[q * R + r] = fetch(s, t + q * P + r * (N / R));
#pragma unroll
      for (int q = 0; q < NB; q++)
#pragma unroll
        for (int r = 0; r < R; r++) v[q * R + r] = fix(s, t + q * P + r * (N / R), v[q * R + r]);
      C* line = buf + (size_t)l * ls;
#pragma unroll
      for (int q = 0; q < NB; q++) {
        const int j = t + q * P;
        dft_s<R, 1, INV>(v + q * R);
#pragma unroll
        for (int r = 0; r < R; r++) line[padl<C, N>(j * R + r)] = v[q * R + r];
      }
    }
  }
}

// fft_lines with pass 0 fed by fft_pass0_load; waits for the caller's
// cp.async twiddle copies before the passes that use them.
template <typename T, int N, int THREADS, bool INV = false, typename Begin, typename Fetch, typename Fix>
__device__ __forceinline__ void fft_lines_load(C2<T>* buf, int nlines, int ls, const C2<T>* tw, Begin begin,
                                               Fetch fetch, Fix fix) {
  static_assert(THREADS % FFTPlan<T, N>::P == 0, "THREADS must be a multiple of threads per line");
  fft_pass0_load<T, N, THREADS, INV>(buf, nlines, ls, begin, fetch, fix);
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  fft_passes<T, N, THREADS, 1, INV>(buf, nlines, ls, tw);
  __syncthreads();
}

template <typename T, int N, int THREADS, int PASS, int LAST, bool INV = false>
__device__ __forceinline__ void fft_passes_until(C2<T>* buf, int nlines, int ls, const C2<T>* tw) {
  using PL = FFTPlan<T, N>;
  if constexpr (PASS < LAST) {
    constexpr int R = PL::rad(PASS);
    constexpr int NS = PL::ns(PASS);
    fft_pass<C2<T>, N, R, NS, PL::E, PL::P, THREADS, INV>(buf, nlines, ls, tw + PL::twoff(PASS));
    fft_passes_until<T, N, THREADS, PASS + 1, LAST, INV>(buf, nlines, ls, tw);
  }
}

// ---------------------------------------------------------------------------
// Panels: PW lines of N points interleaved in rows of 16-byte slots, the
// layout of the z-pencils in global memory and, unchanged, of the z transforms
// in shared memory.  Row rho holds the entries z = rho ZS .. of every line (ZS =
// 2 entries of an FP32 line make a slot, 1 of an FP64 line); line x sits in
// slot x ^ sw(rho).  A panel is contiguous in global memory (64 KB at n =
// 1024), so a block copies it whole, and the x chain, which takes one slot of
// every line, reads and writes whole rows (128 bytes in FP32).  The rotation of
// the slots by sw(rho) spreads consecutive z of one line over all banks.
//
// A line is transformed in place, in its own slots: natural order (nat) at
// the ends, and between passes the order i ^ ((i / R0) & M) (xch), which makes
// the strided writes of a pass conflict-free like the padding of padl.  Both
// are linear over bitwise xor for N = 2^k, so an address is a thread's own part
// xor a constant, and the constant's bits above the permuted ones go into the
// instruction's immediate offset.
// ---------------------------------------------------------------------------
// SLOT1: the y transforms' panel of one slot a row (two FP32 columns side by
// side, one FP64 column), 16 N bytes; the columns of a slot swap with bit 3 of
// the row for the same reason.
template <typename T_, int N_, bool SLOT1 = false> struct Panel {
  using T = T_;
  static constexpr int N = N_;
  using C = C2<T>;
  using PL = FFTPlan<T, N>;
  static constexpr bool DBL = sizeof(T) == 8, POW2 = is_pow2(N);
  static constexpr int ZS = SLOT1 || DBL ? 1 : 2, PW = SLOT1 ? (DBL ? 1 : 2) : (DBL ? 4 : 8);
  static constexpr unsigned LX = SLOT1 ? 8 : 16;   // line x: xor LX x (SLOT1: FP32 only)
  static constexpr int ROW = PW * ZS;            // complex elements of a row
  static constexpr int ELEMS = N * PW;           // of a panel
  static constexpr unsigned BYTES = ELEMS * sizeof(C);
  static constexpr unsigned LOW = SLOT1 ? 255 : DBL ? 511 : 1023;   // bytes that the orders permute within
  static constexpr int S = POW2 ? ilog2c(PL::rad(0)) : 0;
  static constexpr unsigned M = !POW2 ? 0 : (PL::rad(0) < (DBL ? 8 : 16) ? PL::rad(0) : (DBL ? 8 : 16)) - 1;
  static_assert(N % ZS == 0 && BYTES % (LOW + 1) == 0, "panels keep the alignment that xor addressing needs");
  __host__ __device__ static constexpr unsigned sw(unsigned rho) {
    return SLOT1 ? (DBL ? 0 : (rho >> 3) & 1) : DBL ? (rho >> 1) & 3 : rho & 7;
  }
  // byte offset of element i of line 0 (line x: xor LX x)
  template <bool XCH> __host__ __device__ static constexpr unsigned off(unsigned i) {
    if (XCH) i ^= (i >> S) & M;
    const unsigned rho = i / ZS;
    return rho * (ROW * sizeof(C)) + sw(rho) * LX + (i % ZS) * sizeof(C);
  }
  // byte offset of element a + B of the line at byte offset o (panel offset + LX
  // x), oa = o ^ off(a); the bits of a and B are disjoint for N = 2^k
  template <bool XCH, unsigned B>
  __host__ __device__ __forceinline__ static constexpr unsigned addr(unsigned oa, unsigned o, unsigned a) {
    if constexpr (POW2) {
      constexpr unsigned c = off<XCH>(B);
      return (oa ^ (c & LOW)) + (c & ~LOW);
    } else {
      return (o & ~127u) + (off<XCH>(a + B) ^ (o & 127));
    }
  }
  template <bool XCH, unsigned B>
  __device__ __forceinline__ static C& at(unsigned char* smem, unsigned oa, unsigned o, unsigned a) {
    return *reinterpret_cast<C*>(smem + addr<XCH, B>(oa, o, a));
  }
};

template <typename PA, bool XCH, int R, int STEP, int r = 0>
__device__ __forceinline__ void panel_read(unsigned char* smem, unsigned oa, unsigned o, unsigned a,
                                           typename PA::C* v) {
  if constexpr (r < R) {
    v[r] = PA::template at<XCH, (unsigned)r * STEP>(smem, oa, o, a);
    panel_read<PA, XCH, R, STEP, r + 1>(smem, oa, o, a, v);
  }
}
template <typename PA, bool XCH, int R, int STEP, int r = 0>
__device__ __forceinline__ void panel_write(unsigned char* smem, unsigned oa, unsigned o, unsigned a,
                                            const typename PA::C* v) {
  if constexpr (r < R) {
    PA::template at<XCH, (unsigned)r * STEP>(smem, oa, o, a) = v[r];
    panel_write<PA, XCH, R, STEP, r + 1>(smem, oa, o, a, v);
  }
}

// elements t + q P + r (N / R) of a line, natural order (r < R, q < E / R)
template <typename PA, int R>
__device__ __forceinline__ void panel_load(unsigned char* smem, unsigned o, int t, typename PA::C* v) {
  using PL = typename PA::PL;
#pragma unroll
  for (int q = 0; q < PL::E / R; q++) {
    const unsigned a = t + q * PL::P;
    panel_read<PA, false, R, PA::N / R>(smem, o ^ PA::template off<false>(a), o, a, v + q * R);
  }
}
template <typename PA, int R>
__device__ __forceinline__ void panel_store(unsigned char* smem, unsigned o, int t, const typename PA::C* v) {
  using PL = typename PA::PL;
#pragma unroll
  for (int q = 0; q < PL::E / R; q++) {
    const unsigned a = t + q * PL::P;
    panel_write<PA, false, R, PA::N / R>(smem, o ^ PA::template off<false>(a), o, a, v + q * R);
  }
}

// Transform of one line by its group of P threads, exchanging through the
// line's own slots.  v: the operands of pass 0 (element t + q P + r (N / R0) in
// v[q R0 + r]) in, the outputs of the last pass (element t + q P + r NS in
// v[q R + r]) out; afterwards every slot of the line has been read.  Called by
// whole warps.
template <typename PA, bool INV>
__device__ __forceinline__ void panel_fft(unsigned char* smem, unsigned o, int t, const typename PA::C* tw,
                                          typename PA::C* v) {
  using PL = typename PA::PL;
  static_assert(PL::NPASS >= 2, "load and store passes must differ");
  constexpr int N = PA::N, E = PL::E, P = PL::P, R0 = PL::rad(0);
#pragma unroll
  for (int q = 0; q < E / R0; q++) dft_s<R0, 1, INV>(v + q * R0);
#pragma unroll
  for (int q = 0; q < E / R0; q++) {
    const unsigned a = (t + q * P) * R0;
    panel_write<PA, true, R0, 1>(smem, o ^ PA::template off<true>(a), o, a, v + q * R0);
  }
  line_sync<P>();
  if constexpr (PL::NPASS == 3) {
    constexpr int R = PL::rad(1), NS = PL::ns(1);
#pragma unroll
    for (int q = 0; q < E / R; q++) {
      const unsigned a = t + q * P;
      panel_read<PA, true, R, N / R>(smem, o ^ PA::template off<true>(a), o, a, v + q * R);
    }
    line_sync<P>();
#pragma unroll
    for (int q = 0; q < E / R; q++) {
      const int j = t + q * P;
      dft_tw<R, NS, INV>(v + q * R, tw + PL::twoff(1) + j % NS);
      const unsigned a = (j / NS) * NS * R + j % NS;
      panel_write<PA, true, R, NS>(smem, o ^ PA::template off<true>(a), o, a, v + q * R);
    }
    line_sync<P>();
  }
  constexpr int LAST = PL::NPASS - 1, R = PL::rad(LAST), NS = PL::ns(LAST);
#pragma unroll
  for (int q = 0; q < E / R; q++) {
    const unsigned a = t + q * P;
    panel_read<PA, true, R, N / R>(smem, o ^ PA::template off<true>(a), o, a, v + q * R);
  }
  line_sync<P>();
#pragma unroll
  for (int q = 0; q < E / R; q++) dft_tw<R, NS, INV>(v + q * R, tw + PL::twoff(LAST) + (t + q * P) % NS);
}

// Host: build the twiddle table of FFTPlan<T,N>: for every pass p >= 1 the
// pairs (c, T) = (cos, tan) of the angle 2 pi (k + NS q') / (NS rho) of
// dft_tw's combine steps, [row][k] with k < NS; the angle pi/2 (rho = 2,
// k = NS/2) as the pair (2, 1/2) that dft_tw knows it by.
template <typename T, int N>
void build_twiddles(C2<T>* out) {
  using PL = FFTPlan<T, N>;
  auto pair = [](long num, long den) {   // angle 2 pi num / den in [0, pi)
    if (4 * num == den) return cmk<C2<T>>(T(2), T(0.5));
    const long double ang = 2.0L * 3.14159265358979323846264338327950288L * (long double)num / (long double)den;
    return cmk<C2<T>>((T)cosl(ang), (T)(sinl(ang) / cosl(ang)));
  };
  for (int p = 1; p < PL::NPASS; p++) {
    const int R = PL::rad(p), NS = PL::ns(p), off = PL::twoff(p);
    for (int rho = 2; rho <= R; rho *= 2)
      for (int q = 0; q < (rho == 2 ? 1 : rho / 4); q++) {
        C2<T>* row = out + off + (rho == 2 ? 0 : rho / 4 + q) * NS;
        for (int k = 0; k < NS; k++) row[k] = pair(k + (long)NS * q, (long)NS * rho);
      }
  }
}

}  // namespace psdns
