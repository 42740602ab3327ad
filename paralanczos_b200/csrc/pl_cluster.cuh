// pl_cluster.cuh -- large-k per-set Lanczos on a thread-block cluster.
//
// For 128 < k <= 512 the per-set state (A_S and the projector P, 2 k^2 floats:
// 512 KB at k = 256, 2 MB at k = 512) does not fit one SM.  A cluster of CS
// CTAs (one per SM) holds one set: CTA c owns rows [c R, c R + R), R = KB/CS,
// with its rows of A_S in tensor memory (pl_tmem.cuh) and its rows of P in
// registers.  Same recurrence as pl_engine.cuh (three-term
// step, w = P w~, P -= v v^T fused with the next matvec, FP32 vectors, FP64
// alpha/beta).  Per step the CTAs exchange, through distributed shared memory:
// their FP64 partials of alpha and ||w||^2 (one per warp; every warp adds all
// of them in the same order, so the scalars are bitwise identical cluster-wide
// and every branch is cluster-uniform), and their rows of y = A v and w
// (written into every peer's broadcast buffers).
//
// What bounds it is the latency of the two exchanges of a step, so they are
// built to be short: each lane that holds a finished row sum writes it into
// the peers with st.async, whose bytes the receiving CTA's mbarrier counts;
// a warp sends as soon as its rows are done and waits only for the bytes it
// needs.  No CTA barrier, no cluster barrier (whose release fence the warps
// would wait for) and no second pass over the partials.  Measured (B200,
// sets/s) with a cluster barrier per exchange and A_S in shared memory, then
// with st.async, then with A_S in tensor memory, then with no use of P's registers
// outside the passes: k = 384 (1,000 sets) 2.55e4, 3.39e4, 3.51e4, 3.74e4; k = 512
// (600 sets) 8.7e3, 1.19e4, 1.36e4, 1.45e4; with one CTA per set k = 192 (3,000
// sets) 3.06e5, 3.55e5, 4.47e5, 4.56e5.
//
// Thread mapping inside a CTA: NTC threads; a thread holds RPT of the CTA's
// R rows (rows ls, ls + R/RPT, ...), TPR = NTC * RPT / R threads share a row;
// thread g of a row owns the float4 column chunks g, g + TPR, g + 2 TPR, ...
// (CPT = KB / TPR columns of each of its rows).  The lanes of one g are
// adjacent in the warp: a 128-bit load of a broadcast vector in which
// neighbouring lanes share an address takes 2.1 cycles of the shared-memory
// pipe, one in which they do not takes 4.0 whatever else is shared (measured),
// and these loads are a third of the pipe's work.  Row partial sums are combined with
// xor-shuffles over the TPR lanes (TPR divides 32): the first log2(RPT) levels
// halve the rows each lane goes on with (a lane sends the half it drops), so
// TPR / RPT lanes end with each row's sum, one per peer to send it to.  With
// RPT = 2 a thread holds as much of P as with one row of twice the columns,
// but reads half of each broadcast vector per step.
#pragma once
#include <cooperative_groups.h>

#include "pl_engine.cuh"
#include "pl_sturm.cuh"
#include "pl_sync.cuh"
#include "pl_tmem.cuh"

namespace pl {

namespace cg = cooperative_groups;

__host__ __device__ constexpr int pow2_up(int n) {
  int p = 1;
  while (p < n) p *= 2;
  return p;
}

template <int KB, int CS, int NTC, int RPT = 1>
struct CfgC {
  static constexpr int R = KB / CS;       // rows per CTA
  static constexpr int RS = R / RPT;      // row slots: a thread holds rows ls, ls + RS, ...
  static constexpr int TPR = NTC / RS;    // threads per row
  static constexpr int CPT = KB / TPR;    // columns per thread (of each of its rows)
  static constexpr int NCH = CPT / 4;     // float4 chunks per thread and row
  static constexpr int NWC = NTC / 32;    // warps per CTA
  static_assert(R <= NTC, "a thread per own row");
  static_assert(KB % CS == 0 && R % RPT == 0 && NTC % RS == 0 && KB % TPR == 0, "bad shape");
  static constexpr int CPR = TPR / RPT;  // lanes that end with a row's sum
  static constexpr int NP = (CS + CPR - 1) / CPR;  // peers such a lane sends it to
  static_assert(32 % TPR == 0 && CPT % 4 == 0, "bad shape");
  static_assert(TPR % RPT == 0 && (RPT & (RPT - 1)) == 0 && CS <= 32, "bad shape");
};

template <int KB, int CS, int NTC>
struct __align__(16) ClusterSmem {
  static constexpr int NPART = CS * (NTC / 32);  // one partial per warp of the set
  // before the steps, where one CTA mirrors its triangle of A_S: [float4 of a
  // thread][thread]; from then on the own rows of every step's vector: [step][row]
  float4 own[(KB / CS) * KB / 4];
  float vb[3][KB];               // unnormalised Lanczos vectors, rotating: current, previous, next
  float yb[KB];                  // broadcast of y = A v
  float wb[KB];                  // w~, formed locally from yb
  int idx[KB];
  float sc[KB];                  // every step's scale (v = sc * vb)
  float diag[KB / CS];           // own diagonal elements of P, up to step `seen`
  double2 ab[KB];                // T (rank 0 reads it for the bisection)
  double part[4][NPART];         // alpha, ||w||^2, misc, index check
  double ext[2];                 // lambda_min, lambda_max
  double red[NTC / 32];          // warp partials inside the CTA (breakdown argmax)
  unsigned long long key[CS];    // breakdown argmax exchange
  unsigned long long bar[2];     // mbarriers of the y and the w exchange
  int seen;
  int abort;                     // a bounded wait gave up, here or in a peer
  long long lost;                // the item it was on
};

// What one exchange delivers into every CTA: KB rows and the warps' partials.
template <int KB, int CS, int NTC>
__device__ __forceinline__ constexpr uint32_t exchange_bytes() {
  return KB * sizeof(float) + CS * (NTC / 32) * sizeof(double);
}

// Address of this CTA's shared-memory address `a` in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_async(uint32_t a, float x, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a),
               "r"(__float_as_uint(x)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async(uint32_t a, double x, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
               "l"(__double_as_longlong(x)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Barrier over the set's CTAs.  A one-CTA cluster needs only the CTA barrier
// (same ordering of its shared-memory writes, without the cluster-scope
// release/acquire).
template <int CS>
__device__ __forceinline__ void set_sync(cg::cluster_group& cl) {
  if constexpr (CS == 1)
    __syncthreads();
  else
    cl.sync();
}

// Sum of the N partials of an exchange by one warp (the same order in every
// warp of every CTA).
template <int N>
__device__ __forceinline__ double part_sum(const double* p) {
  const int lane = threadIdx.x & 31;
  double s = lane < N ? p[lane] : 0.0;
#pragma unroll
  for (int i = 32; i < N; i += 32)
    if (i + lane < N) s += p[i + lane];
  return warp_sum(s);
}

// Sum over the set's CTAs outside the step loop (cluster barrier).
template <int KB, int CS, int NTC>
__device__ __forceinline__ double cluster_sum(double x, ClusterSmem<KB, CS, NTC>& sm, int slot,
                                              cg::cluster_group& cl, int rank) {
  const double s = warp_sum(x);
  const int lane = threadIdx.x & 31;
  if (lane < CS) {
    ClusterSmem<KB, CS, NTC>* peer = CS == 1 ? &sm : cl.map_shared_rank(&sm, (unsigned)lane);
    peer->part[slot][rank * (NTC / 32) + (threadIdx.x >> 5)] = s;
  }
  set_sync<CS>(cl);
  return part_sum<ClusterSmem<KB, CS, NTC>::NPART>(sm.part[slot]);
}

// Row sums of a thread's RPT rows over the row's TPR lanes: the xor tree
// TPR/2, ..., 1, each level down to one row dropping half of the rows.  Lane
// g0 ends with the sum of row g0 / (TPR / RPT).
template <int RPT, int TPR>
__device__ __forceinline__ float row_reduce(float (&y)[RPT], int g0) {
  constexpr int RPW = 32 / TPR;  // lanes of one g (adjacent)
  int n = RPT;
#pragma unroll
  for (int o = TPR / 2; o > 0; o >>= 1) {
    if (n > 1) {
      n /= 2;
      const bool hi = g0 & o;
#pragma unroll
      for (int e = 0; e < RPT / 2; ++e)
        if (e < n) {
          const float keep = hi ? y[e + n] : y[e], send = hi ? y[e] : y[e + n];
          y[e] = keep + __shfl_xor_sync(0xffffffffu, send, o * RPW);
        }
    } else {
      y[0] += __shfl_xor_sync(0xffffffffu, y[0], o * RPW);
    }
  }
  return y[0];
}

enum ClusterResult { CLUSTER_DONE, CLUSTER_ABORT };

// Solves one set on the cluster.
//   DONE   its outputs are written
//   ABORT  a bounded wait gave up somewhere in the cluster: nothing is written,
//          and every CTA of the cluster must end
// A wait that gives up is a warp's answer first, then the CTA's (a vote in
// every step, and at the end of the steps), then the cluster's: no CTA passes
// the barrier at the end of its steps before every other one is there, and
// behind it all know whether one of them gave up, so they leave together and no
// CTA writes into one that has left.  hold (tests): 1, the last CTA stays out of
// the steps until its peers' waits have run out; 2, it gives up behind the last
// one, when its peers have all they need.
// ph: phase parity of the exchanges, kept across sets.  ta: the thread's tensor
// memory, read NB float4 at a time.
//
// A breakdown restarts from a row of P.  Any use of P's registers outside the two
// passes costs the loop 80 to 400 bytes of spills at 168 and 255 registers (k = 384
// 0.86 -> 1.32 ms a set), and solving a set again with them is twice the work, so
// the restart forms the diagonal and the row anew, by the same operations in the
// same order, from the vectors of the steps so far (in shared memory that the
// steps leave idle; one float a thread and step).  660 sets of k = 384, none, each
// second and all of them with some 39 restarts: 17.4, 19.1 and 20.7 ms (with sets that
// break down solved twice 18.3, 35.9 and 30.7; with P at hand in every loop 23.2,
// 24.4 and 25.5).  The loop of one CTA per set has room for P at hand (k = 192,
// 3,000 sets: 6.6 ms, from the vectors 6.8).
template <int KB, int CS, int NTC, int RPT, int NB>
__device__ __forceinline__ ClusterResult cluster_solve_set(const MatrixF32& M, const int* __restrict__ S,
                                                  int k, long long set, const SetOutputs& out,
                                                  ClusterSmem<KB, CS, NTC>& sm,
                                                  cg::cluster_group& cl, int rank, uint32_t& ph,
                                                  uint32_t ta, int hold) {
  using C = CfgC<KB, CS, NTC, RPT>;
  constexpr int R = C::R, RS = C::RS, TPR = C::TPR, CPT = C::CPT, NCH = C::NCH;
  constexpr int NPART = ClusterSmem<KB, CS, NTC>::NPART;
  constexpr int RPW = 32 / TPR;        // row slots per warp
  const int t = threadIdx.x;
  const int ls = (t >> 5) * RPW + t % RPW;  // row slot: local rows ls + q * RS
  int r[RPT];                          // global rows
#pragma unroll
  for (int q = 0; q < RPT; ++q) r[q] = rank * R + ls + q * RS;
  const int g0 = (t & 31) / RPW;       // owned chunks g0 + TPR * ch
  const int w_id = t >> 5, lane = t & 31;
  // the row whose sums this lane ends with, and the peers it sends them to
  const int ro = rank * R + ls + g0 / C::CPR * RS;
  const bool lead = g0 % C::CPR == 0;  // one lane per row contributes to the scalars
  const uint32_t ybar = smem_u32(&sm.bar[0]), wbar = smem_u32(&sm.bar[1]);
  // One exchange: the lane's row sum x into row ro of dst in every CTA, then
  // the warp's partial into part[slot].  (Peer addresses are formed here: held
  // across the step they would not fit the registers.)
  auto publish_row = [&](float* dst, float x, uint32_t bar) {
    if constexpr (CS == 1) {
      if (lead) dst[ro] = x;
    } else {
      const uint32_t a = smem_u32(dst + ro);
#pragma unroll
      for (int i = 0; i < C::NP; ++i) {
        const int p = g0 % C::CPR + i * C::CPR;
        if (CS % C::CPR == 0 || p < CS) st_async(peer_addr(a, p), x, peer_addr(bar, p));
      }
    }
  };
  auto publish_partial = [&](int slot, double x, uint32_t bar) {
    double* pd = &sm.part[slot][rank * C::NWC + w_id];
    if constexpr (CS == 1) {
      if (lane == 0) *pd = x;
    } else {
      if (lane < CS) st_async(peer_addr(smem_u32(pd), lane), x, peer_addr(bar, lane));
    }
  };
  // Waits for an exchange; false: the thread gave up.  The warp's lanes are
  // together again afterwards, for the matrix products that follow.
  auto arrived = [&](uint32_t bar) -> bool {
    if constexpr (CS == 1) {
      __syncthreads();
      return true;
    } else {
      const bool got = mbar_wait(bar, ph, (volatile int*)&sm.abort, nullptr);
      __syncwarp();
      return got;
    }
  };

  // ---- indices (every CTA keeps the full set), validation -------------------
  const SetMatrix SM = set_matrix(M, set);
  bool bad = false;
  for (int c = t; c < KB; c += NTC) {
    int v = 0;
    if (c < k) {
      v = SM.index(S, c);
      bad |= (v < 0) | (v >= SM.n);
    }
    sm.idx[c] = (c < k && v >= 0 && v < SM.n) ? v : 0;
  }
  const double badsum = cluster_sum<KB, CS, NTC>(__any_sync(0xffffffffu, bad) ? 1.0 : 0.0, sm, 3, cl, rank);
  if (badsum != 0.0) {
    if (rank == 0 && t == 0) write_failed(out, set, 0, 0, SET_BAD_INDEX);
    set_sync<CS>(cl);
    return CLUSTER_DONE;
  }

  // ---- gather own rows of A_S into tensor memory -----------------------------
  constexpr int NF = NCH * RPT;  // float4 of a thread, (q, ch) as number ch * RPT + q
  static_assert(NF % NB == 0 && NF % 4 == 0, "whole buffers");
  // float offset in sm.own of the CTA's element (row, col): chunk cc = col / 4 of
  // row q * RS + ls belongs to the thread of slot ls and g = cc % TPR as its
  // (q, cc / TPR)
  auto at = [](int row, int col) {
    const int cc = col >> 2, sl = row % RS;
    const int th = (sl / RPW) * 32 + (cc % TPR) * RPW + sl % RPW;
    return (((cc / TPR * RPT + row / RS) * NTC + th) << 2) + (col & 3);
  };
  float* __restrict__ own = reinterpret_cast<float*>(sm.own);
  [[maybe_unused]] float4* __restrict__ my = sm.own + t;  // number i at my[i * NTC]
  double fro = 0.0;
  if constexpr (CS == 1) {
    // One CTA holds all of A_S, which is symmetric: load only its upper
    // triangle (k(k+1)/2 random elements, each its own L1 request) and store
    // each off-diagonal element twice.  Rows p and KB-1-p form a pair of KB+1
    // upper elements, shared by TPP threads.
    constexpr int NP = KB / 2, TPP = NTC / NP, PER = (KB + TPP) / TPP;
    static_assert(NP * TPP == NTC, "row pairs per CTA");
    const int p = t % NP, i0 = (t / NP) * PER;
    const int r0 = p, r1 = KB - 1 - p;
    const float* __restrict__ row0 = SM.A + (size_t)sm.idx[r0] * (size_t)SM.lda;
    const float* __restrict__ row1 = SM.A + (size_t)sm.idx[r1] * (size_t)SM.lda;
#pragma unroll 16
    for (int ii = 0; ii < PER; ++ii) {
      const int i = i0 + ii;
      if (i > KB) break;
      const bool first = i < KB - p;
      const int rr = first ? r0 : r1;
      const int c = first ? p + i : i - 1;  // c >= rr
      const float e = (rr < k && c < k) ? __ldg((first ? row0 : row1) + sm.idx[c]) : 0.f;
      const double e2 = (double)e * (double)e;
      fro += (c == rr) ? e2 : 2.0 * e2;
      own[at(rr, c)] = e;
      if (c != rr) own[at(c, rr)] = e;
    }
    __syncthreads();
#pragma unroll 4
    for (int i = 0; i < NF; ++i) tmem_st4(ta, 4 * i, my[i * NTC]);
  } else {
    // (a rolled loop: 4 U loads in flight)
    constexpr int U = NF % 8 ? 4 : 8;
#pragma unroll 1
    for (int i0 = 0; i0 < NF; i0 += U) {
      float e[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int q = (i0 + u) % RPT, ch = (i0 + u) / RPT;
        const int row = rank * R + ls + q * RS;
        const bool rv = row < k;
        const float* __restrict__ arow = SM.A + (size_t)sm.idx[row] * (size_t)SM.lda;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int c = 4 * (g0 + TPR * ch) + v;
          e[u][v] = (rv && c < k) ? __ldg(arow + sm.idx[c]) : 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int v = 0; v < 4; ++v) fro += (double)e[u][v] * (double)e[u][v];
        tmem_st4(ta, 4 * (i0 + u), make_float4(e[u][0], e[u][1], e[u][2], e[u][3]));
      }
    }
  }
  tmem_st_wait();
  const double fro2 = cluster_sum<KB, CS, NTC>(fro, sm, 2, cl, rank);
  const double tau2 = (32.0 * (double)kEps32) * (32.0 * (double)kEps32) * fro2;

  // vb[cur] holds the unnormalised v_j (v_j = sc * vb[cur]), vb[prv] v_{j-1}
  // (scaled by scp); w is published into vb[nxt].  No buffer is written while
  // it may still be read: a CTA sends y of step j + 1 only after every warp of
  // the set has sent w of step j, hence after its reads of yb and part[0]; it
  // sends w of step j only after every warp has sent y of step j, hence after
  // step j - 1's reads of what is now vb[nxt] and of part[1].
  const float v0 = (float)(1.0 / sqrt((double)k));
  float v[RPT];
#pragma unroll
  for (int q = 0; q < RPT; ++q) v[q] = r[q] < k ? v0 : 0.f;
  float vo = ro < k ? v0 : 0.f;  // v of row ro
  for (int c = t; c < KB; c += NTC) {
    sm.vb[0][c] = c < k ? v0 : 0.f;
    sm.vb[1][c] = 0.f;
  }
  if (t == 0) {
    sm.ab[0].y = 0.0;
    sm.seen = 0;
  }
  float sc = 1.f, scp = 0.f, bprev = 0.f;
  int status = 0;
  int cur = 0, prv = 1, nxt = 2;
  __syncthreads();
  TmemBuf<NB> buf[2];
  float2 Pr[RPT][CPT / 2];
#pragma unroll
  for (int q = 0; q < RPT; ++q)
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {  // I
      const int c = 4 * (g0 + TPR * ch);
      const bool rv = r[q] < k;
      Pr[q][2 * ch] = make_float2(rv && c == r[q], rv && c + 1 == r[q]);
      Pr[q][2 * ch + 1] = make_float2(rv && c + 2 == r[q], rv && c + 3 == r[q]);
    }
  [[maybe_unused]] float pd = ro < k ? 1.f : 0.f;  // (one CTA) P's diagonal element of row ro
  if (CS > 1 && hold == 1 && rank == CS - 1) {
    for (const unsigned long long t0 = globaltimer(); globaltimer() - t0 < kWaitNs + kWaitNs / 4;) __nanosleep(10000);
    goto lost;
  }
  buf[0].load(ta, 0);
  for (int j = 0;; ++j) {
    if constexpr (CS > 1) {
      if (t == 0) {
        mbar_expect(ybar, exchange_bytes<KB, CS, NTC>());
        mbar_expect(wbar, exchange_bytes<KB, CS, NTC>());
      }
    }
    // P -= v v^T and y = A v over the owned row slices
    if constexpr (CS == 1) pd = fmaf(-vo * sc, sm.vb[cur][ro], pd);
    float2 ya[RPT], yb[RPT], nc[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const float cq = -v[q] * sc;
      nc[q] = make_float2(cq, cq);
      ya[q] = make_float2(0.f, 0.f);
      yb[q] = make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      const float4 b4 = *reinterpret_cast<const float4*>(&sm.vb[cur][4 * (g0 + TPR * ch)]);
      const float2 b01 = make_float2(b4.x, b4.y), b23 = make_float2(b4.z, b4.w);
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const int i = ch * RPT + q, bi = i / NB;
        if (i % NB == 0) {
          buf[bi & 1].ready();
          if ((bi + 1) * NB < NF) buf[(bi + 1) & 1].load(ta, 4 * NB * (bi + 1));
        }
        const float4 a4 = buf[bi & 1].f4(i % NB);
        Pr[q][2 * ch] = __ffma2_rn(nc[q], b01, Pr[q][2 * ch]);
        Pr[q][2 * ch + 1] = __ffma2_rn(nc[q], b23, Pr[q][2 * ch + 1]);
        ya[q] = __ffma2_rn(make_float2(a4.x, a4.y), b01, ya[q]);
        yb[q] = __ffma2_rn(make_float2(a4.z, a4.w), b23, yb[q]);
      }
    }
    float y[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) y[q] = ((ya[q].x + ya[q].y) + (yb[q].x + yb[q].y)) * sc;
    const float yo = row_reduce<RPT, TPR>(y, g0);
    publish_row(sm.yb, yo, ybar);
    publish_partial(0, warp_sum(lead ? (double)vo * (double)yo : 0.0), ybar);
    // w~ = y - alpha v_j - beta_j v_{j-1}, every element formed locally (what
    // does not wait for alpha first)
    constexpr int NE = (KB + NTC - 1) / NTC;
    float ve[NE], we[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) {
      const int c = t + e * NTC;
      ve[e] = c < KB ? sc * sm.vb[cur][c] : 0.f;
      we[e] = c < KB ? scp * sm.vb[prv][c] : 0.f;
    }
    const bool got_y = arrived(ybar);
#pragma unroll
    for (int e = 0; e < NE; ++e) we[e] = fmaf(-bprev, we[e], t + e * NTC < KB ? sm.yb[t + e * NTC] : 0.f);
    const double alpha = part_sum<NPART>(sm.part[0]);
    const float af = (float)alpha;
#pragma unroll
    for (int e = 0; e < NE; ++e)
      if (t + e * NTC < KB) sm.wb[t + e * NTC] = fmaf(-af, ve[e], we[e]);
    if constexpr (CS == 1) {
      __syncthreads();
    } else {
      if (__syncthreads_or(!got_y)) goto failed;
    }

    // w = P w~ over the owned row slices
    float2 wa[RPT], wc[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      wa[q] = make_float2(0.f, 0.f);
      wc[q] = make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      const float4 x4 = *reinterpret_cast<const float4*>(&sm.wb[4 * (g0 + TPR * ch)]);
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        wa[q] = __ffma2_rn(Pr[q][2 * ch], make_float2(x4.x, x4.y), wa[q]);
        wc[q] = __ffma2_rn(Pr[q][2 * ch + 1], make_float2(x4.z, x4.w), wc[q]);
      }
    }
    float w[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) w[q] = (wa[q].x + wa[q].y) + (wc[q].x + wc[q].y);
    const float wo = row_reduce<RPT, TPR>(w, g0);
    publish_row(sm.vb[nxt], wo, wbar);
    publish_partial(1, warp_sum(lead ? (double)wo * (double)wo : 0.0), wbar);
    buf[0].load(ta, 0);  // the next pass's first buffer
    if constexpr (CS > 1) {  // (here, while w travels)
      if (t < R) own[j * R + t] = sm.vb[cur][rank * R + t];
      if (t == 0) sm.sc[j] = sc;
    }
    const bool got_w = arrived(wbar);
#pragma unroll
    for (int q = 0; q < RPT; ++q) v[q] = sm.vb[nxt][r[q]];
    const double b2v = part_sum<NPART>(sm.part[1]);
    // (such a warp votes at once, the CTA's others at their next vote; asked here,
    // behind the sum, it is free: before it, 1.02 times the step at k = 512)
    if (CS > 1 && __any_sync(0xffffffffu, !got_w)) goto lost;
    ph ^= 1u;
    if (t == 0 && rank == 0) {
      sm.ab[j].x = alpha;
      if (j + 1 < k) sm.ab[j + 1].y = b2v;
    }
    if (!isfinite(alpha) || !isfinite(b2v)) {
      status |= SET_NONFINITE;
      goto steps_done;
    }
    if (j + 1 == k) goto steps_done;
    if (b2v > tau2) {
      const float bf = sqrtf((float)b2v);
      scp = sc;
      sc = 1.0f / bf;
      bprev = bf;
      vo = wo * sc;
#pragma unroll
      for (int q = 0; q < RPT; ++q) v[q] *= sc;
    } else {
      // Breakdown: restart from the row of P with the largest diagonal
      // (cluster-wide argmax, ties to the smaller row), published into vb[nxt].
      status |= SET_BREAKDOWN;
      if constexpr (CS > 1) {
        if (__syncthreads_or(0)) goto failed;
        set_sync<CS>(cl);
        if (sm.abort) goto leave;
      }
      unsigned long long kk = 0ull;
      if constexpr (CS == 1) {
        if (ro < k) kk = ((unsigned long long)__float_as_uint(fmaxf(pd, 0.f)) << 32) | (unsigned)(0x7fffffff - ro);
      } else if (t < R && rank * R + t < k) {
        const int row = rank * R + t;
        float d = sm.seen ? sm.diag[t] : 1.f;
#pragma unroll 8
        for (int i = sm.seen; i <= j; ++i) {
          const float b = own[i * R + t], c = sm.sc[i];
          d = fmaf(-(b * c) * c, b, d);
        }
        sm.diag[t] = d;
        kk = ((unsigned long long)__float_as_uint(fmaxf(d, 0.f)) << 32) | (unsigned)(0x7fffffff - row);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long y2 = __shfl_xor_sync(0xffffffffu, kk, o);
        kk = y2 > kk ? y2 : kk;
      }
      if ((t & 31) == 0) sm.red[t >> 5] = __longlong_as_double((long long)kk);
      __syncthreads();
      if (t == 0) sm.seen = j + 1;
      if (t < CS) {
        unsigned long long m = 0;
        for (int i = 0; i < NTC / 32; ++i) {
          const unsigned long long y2 = (unsigned long long)__double_as_longlong(sm.red[i]);
          m = y2 > m ? y2 : m;
        }
        cl.map_shared_rank(&sm, (unsigned)t)->key[rank] = m;
      }
      set_sync<CS>(cl);
      unsigned long long best = 0;
      for (int q = 0; q < CS; ++q) best = sm.key[q] > best ? sm.key[q] : best;
      const int mrow = 0x7fffffff - (int)(best & 0xffffffffu);
      if constexpr (CS == 1) {
#pragma unroll
        for (int q = 0; q < RPT; ++q)
          if (r[q] == mrow) {
#pragma unroll
            for (int ch = 0; ch < NCH; ++ch)
              *reinterpret_cast<float4*>(&sm.vb[nxt][4 * (g0 + TPR * ch)]) =
                  make_float4(Pr[q][2 * ch].x, Pr[q][2 * ch].y, Pr[q][2 * ch + 1].x, Pr[q][2 * ch + 1].y);
          }
      } else {
        // row mrow of P: its owner sends the coefficients of the steps, every CTA forms
        // its own columns' elements (one thread each) and sends them
        if (mrow / R == rank) {
          for (int e = t; e < CS * (j + 1); e += NTC) {
            const int p = e / (j + 1), i = e - p * (j + 1);
            const float b = own[i * R + mrow - rank * R], c = sm.sc[i];
            ClusterSmem<KB, CS, NTC>* peer = cl.map_shared_rank(&sm, (unsigned)p);
            peer->wb[i] = -(b * c) * c;
          }
        }
        set_sync<CS>(cl);
        if (t < R) {
          float z = rank * R + t == mrow ? 1.f : 0.f;
#pragma unroll 8
          for (int i = 0; i <= j; ++i) z = fmaf(sm.wb[i], own[i * R + t], z);
#pragma unroll 1
          for (int p = 0; p < CS; ++p) {
            ClusterSmem<KB, CS, NTC>* peer = cl.map_shared_rank(&sm, (unsigned)p);
            peer->vb[nxt][rank * R + t] = z;
          }
        }
      }
      set_sync<CS>(cl);
      const float zo = sm.vb[nxt][ro];
      const double zz = cluster_sum<KB, CS, NTC>(lead ? (double)zo * (double)zo : 0.0, sm, 2, cl, rank);
      if (t == 0 && rank == 0) sm.ab[j + 1].y = 0x1p-600;  // decoupled block (see sturm_count)
      scp = sc;
      sc = 1.0f / sqrtf((float)zz);
      bprev = 0.f;
      vo = zo * sc;
#pragma unroll
      for (int q = 0; q < RPT; ++q) v[q] = sm.vb[nxt][r[q]] * sc;
    }
    const int old_prv = prv;
    prv = cur;
    cur = nxt;
    nxt = old_prv;
  }
steps_done:
  buf[0].ready();  // no load outlives the set
  if constexpr (CS > 1) {
    if (__syncthreads_or(hold == 2 && rank == CS - 1)) goto failed;
  }
  set_sync<CS>(cl);  // every rank done with the step loop before T is read
  if constexpr (CS > 1) {
    if (sm.abort) goto leave;
  }

  // ---- extremes on rank 0: warp 0 lambda_min, warp 1 lambda_max, 33-way -----
  if (rank == 0) {
    if (status & SET_NONFINITE) {
      if (t == 0) write_failed(out, set, 0, 0, status);
    } else {
      double glo = 1e300, ghi = -1e300;
      if (t < 64) {
        for (int i = t & 31; i < k; i += 32) {
          const double rad = (i > 0 ? sqrt(sm.ab[i].y) : 0.0) + (i + 1 < k ? sqrt(sm.ab[i + 1].y) : 0.0);
          glo = fmin(glo, sm.ab[i].x - rad);
          ghi = fmax(ghi, sm.ab[i].x + rad);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          glo = fmin(glo, __shfl_xor_sync(0xffffffffu, glo, o));
          ghi = fmax(ghi, __shfl_xor_sync(0xffffffffu, ghi, o));
        }
        const double pad = 0x1p-51 * fmax(fabs(glo), fabs(ghi)) + 1e-300;
        const double e = multisect_warp(sm.ab, k, glo - pad, ghi + pad, t < 32 ? 1 : k);
        if ((t & 31) == 0) sm.ext[t >> 5] = e;
      }
      __syncthreads();
      if (t == 0) {
        const double lmin = sm.ext[0], lmax = sm.ext[1];
        if (out.lmin) out.lmin[set] = lmin;
        if (out.lmax) out.lmax[set] = lmax;
        if (out.delta) out.delta[set] = fmax(1.0 - lmin, lmax - 1.0);
        if (out.err) out.err[set] = status;
      }
    }
  }
  set_sync<CS>(cl);  // rank 0's reads of T precede the next set's writes
  return CLUSTER_DONE;

lost:  // this warp: its vote
  __syncthreads_or(1);
failed:  // this CTA
  if (t < CS) *(volatile int*)&cl.map_shared_rank(&sm, (unsigned)t)->abort = 1;
  set_sync<CS>(cl);
leave:  // every CTA of the cluster
  // (what a peer sent and no wait here counted has long arrived after 1 ms)
  for (const unsigned long long t0 = globaltimer(); globaltimer() - t0 < 1000000ull;) __nanosleep(1000);
  set_sync<CS>(cl);
  return CLUSTER_ABORT;
}

}  // namespace pl
