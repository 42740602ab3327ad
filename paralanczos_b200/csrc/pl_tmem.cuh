// pl_tmem.cuh -- A[S,S] held in tensor memory (TMEM) as plain storage.
//
// A step of every engine reads all of a set's A_S once and, from the same
// shared-memory pipe, the broadcast Lanczos vectors.  That pipe (128 bytes a
// cycle per SM) is what bounds the steps, while TMEM, 256 KB per SM, has a
// read path of its own: tcgen05.ld.32x32b, double-buffered, delivered 300 to
// 330 bytes a cycle per SM to 8 warps, and as much next to a saturated
// shared-memory pipe (measured, B200).  A_S does not change during a set, so a
// thread writes its row parts once per set and streams them every step.
//
// A thread's part of A_S is a sequence of NF float4 (row q of chunk ch at
// ch * RPT + q: the order in which a pass uses them), in 4 NF consecutive
// columns of its TMEM lane.  Warp w of a CTA can reach lanes 32 (w % 4) ..
// + 31 only, so warps w, w + 4, ... take column ranges of their own.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pl_sync.cuh"

namespace pl {

// Columns to allocate for `n` used ones: a power of two, at least 32.
__host__ __device__ constexpr int tmem_cols(int n) {
  int c = 32;
  while (c < n) c *= 2;
  return c;
}

// One warp of the CTA calls alloc at the start and free at the end (every
// reader done); `slot` in shared memory receives the base address.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, int cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base, int cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}

// Four columns from column `c` on.
__device__ __forceinline__ void tmem_st4(uint32_t a, int c, float4 v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a + (uint32_t)c),
               "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)),
               "r"(__float_as_uint(v.w))
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// A buffer of NB float4 being loaded; its values may be used after ready().
template <int NB>
struct TmemBuf {
  static_assert(NB == 4, "the tcgen05.ld width used");
  uint32_t r[4 * NB];
  // starts the load of columns c .. c + 4 NB - 1
  __device__ __forceinline__ void load(uint32_t a, int c) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(a + (uint32_t)c));
  }
  // waits for every load issued so far; the operands tie the uses of r to it
  __device__ __forceinline__ void ready() {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])
                 :
                 : "memory");
  }
  __device__ __forceinline__ float4 f4(int i) const {
    return make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                       __uint_as_float(r[4 * i + 3]));
  }
};

// The tensor memory of a CTA of CTA threads, COLS columns for every thread
// (NB = 0: none).  A kernel that allocates tensor memory runs one CTA per SM
// (what the occupancy query answers for it), so its CTA holds every set that
// the SM is to work on.
template <int COLS, int CTA, int NB>
struct TmemA {
  static constexpr int kAlloc = tmem_cols(COLS * ((CTA / 32 + 3) / 4));
  static_assert(NB == 0 || kAlloc <= 512, "tensor memory of an SM");
  uint32_t ta = 0;  // this thread's columns (lane bits included)
  uint32_t base = 0;
  // every thread of the CTA, before and after the sets
  __device__ __forceinline__ void begin() {
    if constexpr (NB > 0) {
      __shared__ uint32_t slot;
      const int w = threadIdx.x >> 5;
      if (w == 0) tmem_alloc(&slot, kAlloc);
      __syncthreads();
      base = slot;
      ta = base + ((uint32_t)(32 * (w & 3)) << 16) + (uint32_t)(COLS * (w >> 2));
    }
  }
  __device__ __forceinline__ void end() {
    if constexpr (NB > 0) {
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");  // (a set given up leaves a load behind)
      __syncthreads();
      if (threadIdx.x < 32) tmem_free(base, kAlloc);
    }
  }
};

}  // namespace pl
