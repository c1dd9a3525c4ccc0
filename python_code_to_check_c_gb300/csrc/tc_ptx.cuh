// Inline-PTX wrappers of the tensor-core kernels (gemm_tc.cu, gemm_deep.cu):
// mbarrier, TMA, tcgen05 and TMEM access, and their bounded waits.
#pragma once

#include <cuda.h>

#include <cstdint>

#include "gemm_tc.h"

namespace tdcc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t c) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(c));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t a, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t a) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: false after `limit` polls (each poll may suspend briefly)
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity, int limit) {
  for (int i = 0; i < limit; ++i)
    if (mbar_try(a, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma3d(uint32_t dst, const CUtensorMap* tm, int x, int y, int z, uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          dst),
      "l"((uint64_t)tm), "r"(x), "r"(y), "r"(z), "r"(mbar)
      : "memory");
}
// UMMA shared-memory descriptor: K-major, SWIZZLE_128B, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// instruction descriptor: kind::f16, A = B = BF16, D = F32, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// A slice product issued by the whole warp, executed where `lane_on` is set (one
// lane): the warp stays converged, so descriptors and addresses live in
// uniform registers.  From a single-lane branch every MMA first moves its six
// operand words there, which costs more than the MMA.
__device__ __forceinline__ void umma_warp(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t acc, uint32_t lane_on) {
  asm volatile(
      "{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 e, %5, 0;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(id), "r"(acc), "r"(lane_on));
}
// 8-bit floating-point operands (E5M2, 32 K a step), the same descriptor bits as idesc_bf16
__device__ __forceinline__ void umma_f8_warp(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t acc, uint32_t lane_on) {
  asm volatile(
      "{\n .reg .pred p, e;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 e, %5, 0;\n"
      " @e tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(d),
      "l"(a), "l"(b), "r"(id), "r"(acc), "r"(lane_on));
}
__device__ __forceinline__ void umma_commit_warp(uint32_t mbar, uint32_t lane_on) {
  asm volatile(
      "{\n .reg .pred e;\n setp.ne.b32 e, %1, 0;\n"
      " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(mbar),
      "r"(lane_on)
      : "memory");
}
// one result for the warp
__device__ __forceinline__ bool mbar_wait_warp(uint32_t a, uint32_t parity, int limit) {
  return __all_sync(0xffffffffu, mbar_wait(a, parity, limit)) != 0;
}
// issue only: the caller waits (tcgen05.wait::ld) before reading r
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st16u(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
constexpr int kWaitLimit = kTcWaitLimit;

// The MMA warp's side of a ring of slice pairs (A_j, B_j): the products of one
// K block with s + t <= S + 1 into the accumulators of their levels, BN columns
// each.  Step j runs the products that pair j completes; a pair is released
// after its last product.  Slots and descriptor words are computed once per
// slice (per product they cost more than the products: the FP64 form's ladder
// at o=10, v=38 took 90 us so, 75 with them hoisted).
template <int STAGES, int A_BYTES, int B_BYTES>
struct PairRing {
  uint64_t hi64;
  uint32_t a0, b0, full0, empty0;
  int wait = kWaitLimit;     // polls of a wait
  uint32_t st0 = 0, ph = 0;  // ring slot and phase of the block's first pair
  __device__ __forceinline__ PairRing(const uint8_t* stA, const uint8_t* stB, const uint64_t* full, const uint64_t* empty)
      : hi64(sdesc(0)),
        a0((smem_u32(stA) & 0x3FFFF) >> 4),
        b0((smem_u32(stB) & 0x3FFFF) >> 4),
        full0(smem_u32(full)),
        empty0(smem_u32(empty)) {}
  // `first`: the block starts the sums.  False when a wait expired.
  template <int S, int BN>
  __device__ __forceinline__ bool issue(uint32_t tmem, uint32_t id, bool first, uint32_t on) {
    static_assert(S <= STAGES, "the ring holds one K block's slices");
    uint32_t la[S], lb[S], slot[S];
#pragma unroll
    for (int j = 0; j < S; ++j) {
      slot[j] = st0 + j < STAGES ? st0 + j : st0 + j - STAGES;
      la[j] = a0 + slot[j] * (A_BYTES >> 4);
      lb[j] = b0 + slot[j] * (B_BYTES >> 4);
    }
    bool ok = true;
#pragma unroll
    for (int j = 1; j <= S; ++j) {
      if (ok) ok = mbar_wait_warp(full0 + 8 * slot[j - 1], st0 + j - 1 < STAGES ? ph : ph ^ 1u, wait);
      asm volatile("tcgen05.fence::after_thread_sync;");
      if (ok) {
        auto product = [&](int s, int t) {
          const bool lead = s == t || s == t + 1;  // the first product of its level in a block
#pragma unroll
          for (int k = 0; k < TC_BK / 16; ++k)
            umma_warp(tmem + (uint32_t)((s + t - 2) * BN), hi64 | (uint64_t)(la[s - 1] + 2 * k),
                      hi64 | (uint64_t)(lb[t - 1] + 2 * k), id, (lead && k == 0 && first) ? 0u : 1u, on);
        };
        const int last = S + 1 - j;  // largest partner of slice j
#pragma unroll
        for (int t = 1; t <= S; ++t)
          if (t <= j && t <= last) product(j, t);
#pragma unroll
        for (int q = 1; q <= S; ++q)
          if (q < j && q <= last) product(q, j);
        if (j >= last) {  // pairs j and S + 1 - j have had their last use
          umma_commit_warp(empty0 + 8 * slot[j - 1], on);
          if (j > last) umma_commit_warp(empty0 + 8 * slot[last - 1], on);
        }
      }
    }
    st0 += S;
    if (st0 >= STAGES) {
      st0 -= STAGES;
      ph ^= 1u;
    }
    return ok;
  }
  // The range guard's plane of 128 K (64 where `half`) into columns [0, BN).
  template <int BN>
  __device__ __forceinline__ bool guard(uint32_t tmem, uint32_t id, bool first, bool half, uint32_t on) {
    const bool ok = mbar_wait_warp(full0 + 8 * st0, ph, wait);
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (ok) {
      const uint32_t la = a0 + st0 * (A_BYTES >> 4), lb = b0 + st0 * (B_BYTES >> 4);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < 2 || !half)
          umma_f8_warp(tmem, hi64 | (uint64_t)(la + 2 * k), hi64 | (uint64_t)(lb + 2 * k), id, (k == 0 && first) ? 0u : 1u,
                       on);
      umma_commit_warp(empty0 + 8 * st0, on);
    }
    if (++st0 == STAGES) {
      st0 = 0;
      ph ^= 1u;
    }
    return ok;
  }
};

// records an expired wait: every role of the CTA stops
template <class SH>
__device__ __forceinline__ void fail(SH* sh, int* err, int code) {
  sh->abort = 1;
  atomicCAS(err, 0, code);
}

}  // namespace tdcc
