// pl_queue.cuh -- deferred, batched extraction of lambda_min / lambda_max.
//
// Bisection inside the Lanczos group (several lanes per extreme, multisection)
// spends most Sturm counts on points that carry little information.  Instead a
// group queues the tridiagonals T of its last Q = NT/2 sets in a per-group slice
// of a global scratch buffer (L2-resident: Q * KB * 16 bytes per group) and then
// bisects them all at once, with one thread per extreme when the queue is full:
// plain bisection, one bit per Sturm count, every lane doing distinct useful work.
//
// Buffer layout: T[i][slot] (double2 {alpha_i, beta_i^2}), the slots of all groups
// of a warp side by side, so the lanes of a warp reading element i of their slots
// touch contiguous memory (four groups' slots apart took four lines an element).
#pragma once
#include "pl_common.cuh"
#include "pl_sturm.cuh"
#include "pl_engine.cuh"

namespace pl {

// double2 between elements i and i + 1 of a slot.
template <int NT>
constexpr int kQueueStride = NT < 32 ? 16 : NT / 2;

// Slots of group gic in the queue buffer of its CTA.
template <int KB, int NT>
__device__ __forceinline__ double2* queue_slots(double2* cta, int gic) {
  constexpr int GPW = NT < 32 ? 32 / NT : 1, Q = NT / 2;
  return cta + (size_t)(gic / GPW * GPW) * (Q * KB) + gic % GPW * Q;
}

struct QueueMeta {
  long long set;
  int k;
  int status;
};

// Bisection of the queued sets.  The group's NT threads share the 2 * nslots
// extremes evenly, L (a power of two, at most 16) threads each: thread t has
// extreme e = t / L, slot e / 2, lambda_min (e even) or lambda_max.  One round
// is D = log2(L) levels of plain bisection at once: the L threads count at the
// 2^D - 1 midpoints that those levels can reach and take the interval of the
// last one on the way, so the result is plain bisection's, in 1 / D of the
// rounds.  A full queue has L = 1 (every thread an extreme of its own, D = 1);
// a queue of few sets, as in a call of few, would otherwise leave most threads
// idle through some 36 serial rounds (one set of k = 32: 36,600 -> 12,000
// cycles).  Groups of less than a warp always have L = 1: what the rounds save
// their sub-warp shuffles cost (about 80 cycles each).  last: the T of the last
// queued set, still in shared memory (a queue of one set reads it there;
// nullptr: no).  Every thread of the group must call it (mask: its lanes of the
// warp).
template <int KB, int NT>
__device__ __forceinline__ void queue_bisect(const double2* __restrict__ T, int nslots,
                                             const QueueMeta* __restrict__ meta, int t, const SetOutputs& out,
                                             unsigned mask, const double2* last) {
  int L = 1, D = 1;
  if constexpr (NT >= 32) {
    if (NT / (2 * nslots) >= 4) {
      L = 4;
      D = 2;
      while (L < 16 && NT / (2 * nslots) >= 2 * L) {
        L *= 2;
        ++D;
      }
    }
  }
  const int e = t / L, sub = t % L, slot = e >> 1;
  const bool active = slot < nslots;
  int k = 0, status = 0;
  long long set = -1;
  double a = 0.0, b = 0.0;
  const double2* ab = T + (active ? slot : 0);
  int stride = kQueueStride<NT>;
  if (NT >= 32 && nslots == 1 && last) {
    ab = last;
    stride = 1;
  }
  [[maybe_unused]] double2 tr[KB <= 16 ? KB : 1];
  if (active) {
    k = meta[slot].k;
    status = meta[slot].status;
    set = meta[slot].set;
    if constexpr (KB == 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) tr[i] = ab[(size_t)i * stride];
    }
  }
  const bool solve = active && !(status & SET_NONFINITE);
  int R = 0;  // levels until the interval is below the tolerance
  {
    double lo = 1e300, hi = -1e300;
    if (solve && L == 1) {
      double bprev = 0.0;
#pragma unroll 4
      for (int i = 0; i < k; ++i) {
        const double al = ab[(size_t)i * stride].x;
        const double bnext = i + 1 < k ? sqrt(ab[(size_t)(i + 1) * stride].y) : 0.0;
        lo = fmin(lo, al - (bprev + bnext));
        hi = fmax(hi, al + (bprev + bnext));
        bprev = bnext;
      }
    } else if (solve) {
      for (int i = sub; i < k; i += L) {
        const double rad = (i > 0 ? sqrt(ab[(size_t)i * stride].y) : 0.0) +
                           (i + 1 < k ? sqrt(ab[(size_t)(i + 1) * stride].y) : 0.0);
        const double al = ab[(size_t)i * stride].x;
        lo = fmin(lo, al - rad);
        hi = fmax(hi, al + rad);
      }
    }
    for (int o = L / 2; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(mask, lo, o));
      hi = fmax(hi, __shfl_xor_sync(mask, hi, o));
    }
    if (solve) {
      const double pad = 0x1p-51 * fmax(fabs(lo), fabs(hi)) + 1e-300;
      a = lo - pad;
      b = hi + pad;
      R = bisect_rounds(a, b);
    }
  }
  const int target = (e & 1) ? k : 1;
  auto count = [&](double x) -> int {
    if constexpr (KB <= 16) {
      // all rows loaded at fixed offsets (KB = 8: once, into registers), no
      // branch but one: 1,160 -> 710 cycles a round of four k = 16 sets on a full
      // SM, where the loads' wavefronts and the instruction issue bound it
      double p0 = 0.0, p1 = 1.0;
      unsigned sp = 0;
      int cnt = 0;
      if constexpr (KB == 16) {
#pragma unroll
        for (int i = 0; i < 16; ++i) tr[i] = ab[(size_t)i * kQueueStride<NT>];
      }
      if (k <= KB - 4)
        sturm_rows<KB - 4, true>(tr, x, p0, p1, sp, cnt);
      else
        sturm_rows<KB, true>(tr, x, p0, p1, sp, cnt);
      return cnt;
    } else {
      // (blocks of 16 need 96 registers: the kernels with more than 128)
      return sturm_count_strided<(KB == 32 ? 8 : 16)>(ab, stride, (k + 3) & ~3, x);
    }
  };
  if (L == 1) {
    for (int r = 0; r < R; ++r) {
      const double x = 0.5 * (a + b);
      if (count(x) >= target) b = x; else a = x;
    }
  } else {
    const int first = (threadIdx.x & 31) / L * L;
    const int node = sub + 1 < L ? sub + 1 : 1;  // this thread's midpoint in the tree below [a, b]
    const int Rw = __reduce_max_sync(0xffffffffu, R);  // rounds of the warp (its slots may differ)
    for (int r = 0; r < Rw; r += D) {
      double xa = a, xb = b, x = 0.5 * (a + b);
      for (int bit = 30 - __clz(node); bit >= 0; --bit) {
        if ((node >> bit) & 1) xa = x; else xb = x;
        x = 0.5 * (xa + xb);
      }
      const bool p = r < R && count(x) >= target;
      const unsigned pass = __ballot_sync(0xffffffffu, p) >> first << 1;
      const int levels = R - r < D ? R - r : D;
      int m = 1;
      for (int d = 1; d < levels; ++d) m = 2 * m + (((pass >> m) & 1u) ? 0 : 1);
      // the interval below the last midpoint on the way
      const double na = __shfl_sync(0xffffffffu, p ? xa : x, first + m - 1);
      const double nb = __shfl_sync(0xffffffffu, p ? x : xb, first + m - 1);
      if (levels > 0) {
        a = na;
        b = nb;
      }
    }
  }
  const double lam = 0.5 * (a + b);
  // the other extreme of the same set is L threads on
  const double other = __shfl_xor_sync(mask, lam, L);
  if (active && (t & (2 * L - 1)) == 0) {
    if (status & SET_NONFINITE) {
      write_failed(out, set, 0, 0, status);
    } else {
      if (out.lmin) out.lmin[set] = lam;
      if (out.lmax) out.lmax[set] = other;
      if (out.delta) out.delta[set] = fmax(1.0 - lam, other - 1.0);
      if (out.err) out.err[set] = status;
    }
  }
}

}  // namespace pl
