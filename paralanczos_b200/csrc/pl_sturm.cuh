// pl_sturm.cuh -- FP64 Sturm-count bisection on the Lanczos tridiagonal.
//
// Replaces the reference's serial one-lane TQLRAT (ParaLanczos.cu:32-189, called
// at ParaLanczos.cu:1461).  The count of eigenvalues of T below x is the number of
// sign changes of the leading principal minors of T - xI (continuant form,
// division-free, with power-of-two rescaling every 8 or 16 rows).  The reference's
// own Sturm sketch, EIGVALS_BELOW (ParaLanczos.cu:519-552), is unused and skips
// alpha[1]; this is new code.  The CPU restatement is orc_sturm_count in
// oracle/pl_oracle.c.
#pragma once
#include <cuda_runtime.h>

namespace pl {

// Power-of-two rescaling of the last two minors by the larger one's exponent
// (where p1 vanishes it is p0's): exact, keeps signs and ratios.  (Without a
// branch: a taken-or-not one costs as much as ten rows.)
__device__ __forceinline__ void sturm_rescale(double& p0, double& p1) {
  constexpr int ONE = 1 << 20;  // an exponent of 1 in a high word
  const int f = max(__double2hiint(p0) & 2047 * ONE, __double2hiint(p1) & 2047 * ONE);
  const double s = __hiloint2double(2046 * ONE - min(f, 2045 * ONE), 0);  // 2^(1023 - f / ONE)
  p0 *= s;
  p1 *= s;
}

// N rows of the minors' recurrence, p_i = (alpha_i - x) p_{i-1} - beta_i^2 p_{i-2},
// behind p1 = p_{i-1} and p0 = p_{i-2}; FIRST: rows 0 .. N - 1, whose first two
// need no products with p_{-1} = 0 and p_0 = 1.
template <int N, bool FIRST>
__device__ __forceinline__ void sturm_minors(const double2* t, double x, double& p0, double& p1, double* p) {
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const double d = t[u].x - x;
    if (FIRST && u == 0) {
      p[u] = d;
    } else if (FIRST && u == 1) {
      p[u] = fma(d, p[0], -t[u].y);
    } else {
      const double pm1 = u == 0 ? p1 : p[u > 0 ? u - 1 : 0];
      const double pm2 = u == 0 ? p0 : (u == 1 ? p1 : p[u > 1 ? u - 2 : 0]);
      p[u] = fma(d, pm1, -t[u].y * pm2);
    }
  }
  p0 = N > 1 ? p[N > 1 ? N - 2 : 0] : (FIRST ? 1.0 : p1);
  p1 = p[N - 1];
}

// N rows at once.  The signs are looked at only when the N minors are done (the
// empty asm holds that work behind them): an integer use of a minor right
// behind it stalls the chain.
template <int N, bool FIRST>
__device__ __forceinline__ void sturm_rows(const double2* t, double x, double& p0, double& p1, unsigned& sp,
                                           int& cnt) {
  static_assert(N == 4 || N == 8 || N == 12 || N == 16, "rows per block");
  double p[N];
  sturm_minors<N, FIRST>(t, x, p0, p1, p);
#pragma unroll
  for (int u = N - 4; u >= 0; u -= 4)
    asm volatile("" : "+d"(p[u]), "+d"(p[u + 1]), "+d"(p[u + 2]), "+d"(p[u + 3]));
  unsigned m = sp;  // signs, the newest in bit 0
#pragma unroll
  for (int u = 0; u < N; ++u) m = __funnelshift_l((unsigned)__double2hiint(p[u]), m, 1);
  cnt += __popc((m ^ (m >> 1)) & ((1u << N) - 1u));
  sp = m & 1u;
}

// A decoupled row above the spectrum: no sign change at any x in it.  The
// engines whose T is counted many times over fill k up to a multiple of 4 with
// such rows (fro: Frobenius norm of A_S; 2^-290: above the couplings of 2^-300
// that a decoupled block stores, all that a zero matrix has), so that the counts
// have no odd rows at the end (one at a time they cost 60 to 100 cycles each).
__device__ __forceinline__ double2 sturm_pad_row(double fro) { return make_double2(4.0 * fro + 0x1p-290, 0.0); }

// N rows from row i on for each x, rescaled every RES rows (0: never).
template <int N, int E, bool FIRST, int RES>
__device__ __forceinline__ void sturm_block(const double2* __restrict__ ab, int stride, int i, const double (&x)[E],
                                            double (&p0)[E], double (&p1)[E], unsigned (&sp)[E], int (&cnt)[E]) {
  double2 t[N];
#pragma unroll
  for (int u = 0; u < N; ++u) t[u] = ab[(size_t)(i + u) * stride];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    if (RES > 0 && !FIRST && (i & (RES - 1)) == 0) sturm_rescale(p0[e], p1[e]);
    sturm_rows<N, FIRST>(t, x[e], p0[e], p1[e], sp[e], cnt[e]);
  }
}

// Numbers of eigenvalues of T strictly below x[0 .. E-1].  Element i of T at
// ab[i * stride] = {alpha_i, beta_i^2}, beta_0^2 = 0, beta_i^2 > 0 for i >= 1 (a
// decoupled block stores 2^-600, so two consecutive minors cannot both
// vanish).  Sign changes of the leading principal minors p_{-1} = 0, p_0 = 1,
// ...; a minor that is exactly zero counts as positive, which gives the right
// count because its neighbours then have opposite signs.  Rows go in blocks of
// U, the last ones in a block of 12, 8 or 4 and one at a time, each block loaded
// before its recurrence; 25 to 30 cycles a row where loads and signs in the chain
// took 42 (one warp, B200).  E > 1 shares the loads and runs E chains side by
// side.  The minors are rescaled every RES rows, single rows among them: a run
// of 16 rows stays within FP64 for matrices of scale 2^-59 to 2^57 or so, a run
// of 19 (three single rows behind 16) did so only from 2^-52 to 2^53.
template <int U, int E, int RES = 16>
__device__ __forceinline__ void sturm_counts(const double2* __restrict__ ab, int stride, int k,
                                             const double (&x)[E], int (&cnt)[E]) {
  double p0[E], p1[E];
  unsigned sp[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    p0[e] = 0.0;
    p1[e] = 1.0;
    sp[e] = 0u;
    cnt[e] = 0;
  }
  int i = 0;
  if (k >= U) {
    sturm_block<U, E, true, RES>(ab, stride, 0, x, p0, p1, sp, cnt);
    for (i = U; i + U <= k; i += U) sturm_block<U, E, false, RES>(ab, stride, i, x, p0, p1, sp, cnt);
  }
  const int r = k - i;
  if (U > 8 && r >= 12) {
    sturm_block<(U > 8 ? 12 : 4), E, false, RES>(ab, stride, i, x, p0, p1, sp, cnt);
    i += 12;
  } else if (U > 8 && r >= 8) {
    sturm_block<8, E, false, RES>(ab, stride, i, x, p0, p1, sp, cnt);
    i += 8;
  } else if (r >= 4) {
    sturm_block<4, E, false, RES>(ab, stride, i, x, p0, p1, sp, cnt);
    i += 4;
  }
  for (; i < k; ++i) {
    const double2 t = ab[(size_t)i * stride];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (RES > 0 && i > 0 && (i & (RES - 1)) == 0) sturm_rescale(p0[e], p1[e]);
      const double p2 = fma(t.x - x[e], p1[e], i > 0 ? -t.y * p0[e] : 0.0);
      const unsigned s2 = (unsigned)__double2hiint(p2) >> 31;
      cnt[e] += (int)(s2 ^ sp[e]);
      sp[e] = s2;
      p0[e] = p1[e];
      p1[e] = p2;
    }
  }
}

template <int U, int RES = 16>
__device__ __forceinline__ int sturm_count_strided(const double2* __restrict__ ab, int stride, int k,
                                                   double x) {
  const double xs[1] = {x};
  int cnt[1];
  sturm_counts<U, 1, RES>(ab, stride, k, xs, cnt);
  return cnt[0];
}

// T of any length k (the engines for k > 128 do not fill it up), rescaled every
// 8 rows: a few rounds a set, so the wider range costs nothing that shows.
__device__ __forceinline__ int sturm_count(const double2* __restrict__ ab, int k, double x) {
  return sturm_count_strided<8, 8>(ab, 1, k, x);
}

// The same count a row at a time, in few registers: for the kernels of many
// threads a set, where the blocks' registers cost more than the chain (plain
// form, k = 64: 3.80e6 sets/s, 2.98e6 with blocks of 8).
__device__ __forceinline__ int sturm_count_lean(const double2* __restrict__ ab, int k, double x) {
  double p0 = 1.0, p1 = ab[0].x - x;
  unsigned sp = (unsigned)__double2hiint(p1) >> 31;
  int cnt = (int)sp;
  auto row = [&](const double2 t) {
    const double p2 = fma(t.x - x, p1, -t.y * p0);
    const unsigned s2 = (unsigned)__double2hiint(p2) >> 31;
    cnt += (int)(s2 ^ sp);
    sp = s2;
    p0 = p1;
    p1 = p2;
  };
  int i = 1;
  for (; i + 16 <= k; i += 16) {
#pragma unroll
    for (int u = 0; u < 16; ++u) row(ab[i + u]);
    sturm_rescale(p0, p1);
  }
  for (; i < k; ++i) row(ab[i]);
  return cnt;
}

// Termination width for an interval whose ends have magnitude up to `mag`.
// 2^-34 (6e-11) of the spectrum's scale: far below the FP32 Lanczos error.
__device__ __forceinline__ double bisect_tol(double lo, double hi) {
  return 0x1p-34 * fmax(fabs(lo), fabs(hi)) + 1e-300;
}

// Rounds of bisection needed to shrink [lo, hi] below tol: the smallest r with
// (hi - lo) 2^-r <= tol, read off the exponents and mantissas (halving in a loop
// took 1,000 cycles).
__device__ __forceinline__ int bisect_rounds(double lo, double hi) {
  const double w = hi - lo;
  const double tol = bisect_tol(lo, hi);  // >= 1e-300: normal
  if (!(w > tol)) return 0;
  const long long bw = __double_as_longlong(w), bt = __double_as_longlong(tol);
  const long long mant = (1LL << 52) - 1;
  const int r = (int)((bw >> 52) - (bt >> 52)) + ((bw & mant) > (bt & mant) ? 1 : 0);
  return r < 200 ? r : 200;
}

// Rounds of (G+1)-way multisection needed to shrink [lo, hi] below tol.
__device__ __forceinline__ int multisect_rounds(double lo, double hi, int G) {
  double w = hi - lo, tol = bisect_tol(lo, hi);
  int r = 0;
  while (w > tol && r < 80) {
    w /= (double)(G + 1);
    ++r;
  }
  return r;
}

// lambda_min and lambda_max by (G+1)-way multisection.  Called by the 2G lanes
// [base, base+2G) of one warp (mask covers exactly them): lanes base..base+G-1
// bracket lambda_min, lanes base+G..base+2G-1 bracket lambda_max, each lane
// evaluating one Sturm count per round.  All callers get both results.
__device__ __forceinline__ void multisect_extremes(const double2* __restrict__ ab, int k,
                                                   double lo, double hi, int G, int base,
                                                   unsigned mask, double& lmin, double& lmax) {
  const int lane = (threadIdx.x & 31) - base;
  const bool isMax = lane >= G;
  const int gi = isMax ? lane - G : lane;
  const int target = isMax ? k : 1;
  const unsigned gm = (G >= 32) ? 0xffffffffu : ((1u << G) - 1u);
  const int shift = base + (isMax ? G : 0);
  const int R = multisect_rounds(lo, hi, G);
  double a = lo, b = hi;
  for (int r = 0; r < R; ++r) {
    const double step = (b - a) / (double)(G + 1);
    const double x = a + step * (double)(gi + 1);
    const bool pass = sturm_count_lean(ab, k, x) >= target;
    const unsigned bal = __ballot_sync(mask, pass);
    const unsigned mine = (bal >> shift) & gm;
    const int f = mine ? (__ffs(mine) - 1) : G;  // first sub-lane whose point passed
    const double na = (f > 0) ? a + step * (double)f : a;
    const double nb = (f < G) ? a + step * (double)(f + 1) : b;
    a = na;
    b = nb;
  }
  const double res = 0.5 * (a + b);
  lmin = __shfl_sync(mask, res, base);
  lmax = __shfl_sync(mask, res, base + G);
}

// One extreme by (G+1)-way multisection with the G = 32 lanes of one warp:
// the smallest x with count(x) >= target (target 1: lambda_min; k: lambda_max).
template <bool LEAN = false>
__device__ __forceinline__ double multisect_warp(const double2* __restrict__ ab, int k, double lo,
                                                 double hi, int target) {
  constexpr int G = 32;
  const int gi = threadIdx.x & 31;
  const int R = multisect_rounds(lo, hi, G);
  double a = lo, b = hi;
  for (int r = 0; r < R; ++r) {
    const double step = (b - a) / (double)(G + 1);
    const double x = a + step * (double)(gi + 1);
    const unsigned bal = __ballot_sync(0xffffffffu, (LEAN ? sturm_count_lean(ab, k, x) : sturm_count(ab, k, x)) >= target);
    const int f = bal ? (__ffs(bal) - 1) : G;
    const double na = (f > 0) ? a + step * (double)f : a;
    const double nb = (f < G) ? a + step * (double)(f + 1) : b;
    a = na;
    b = nb;
  }
  return 0.5 * (a + b);
}

// Eigenvalues number m, m + step, ... (E of them, 0-based, ascending; numbers
// >= k are left alone) by R rounds of plain bisection, side by side.
template <int U, int E, int RES = 16>
__device__ __forceinline__ void bisect_indices(const double2* __restrict__ ab, int k, int m, int step,
                                               double lo, double hi, int R, double (&lam)[E]) {
  double a[E], b[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    a[e] = lo;
    b[e] = hi;
  }
  for (int r = 0; r < R; ++r) {
    double x[E];
    int cnt[E];
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = 0.5 * (a[e] + b[e]);
    sturm_counts<U, E, RES>(ab, 1, k, x, cnt);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (cnt[e] >= m + e * step + 1) b[e] = x[e]; else a[e] = x[e];
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) lam[e] = 0.5 * (a[e] + b[e]);
}

// Eigenvalue number m (m = 0 .. k - 1 on as many threads: counts in few registers).
__device__ __forceinline__ double bisect_index(const double2* __restrict__ ab, int k, int m,
                                               double lo, double hi, int R) {
  for (int r = 0; r < R; ++r) {
    const double x = 0.5 * (lo + hi);
    if (sturm_count_lean(ab, k, x) >= m + 1) hi = x; else lo = x;
  }
  return 0.5 * (lo + hi);
}

}  // namespace pl
