// Contractions of the FP64 form on the tensor cores: exact BF16 slice products
// (as gemm_tc.cu) with 8 slices of 7 bits a side, 56 bits under each row's
// maximum, the last one rounded.
//
// The 36 products A_s B_t with s + t <= 9 go to the accumulators of their
// levels L = s + t, FP32 sums of integers that stay exact over a K chunk of 6
// K blocks.  The 8 levels of a 128 x 64 tile fill TMEM, so the drain warps
// keep the sums over all chunks in registers: two int64 per output, levels
// 2..5 and 6..9, rounded to FP64 once at the end.  What is dropped (levels
// above 9, the operands' rounding) is about 2^-58 of the product of the two
// row maxima per term and of either sign.  Against extended precision the
// four residuals at o=8, v=26 (amplitudes near an MP2 guess or normal) are off
// by 0.61 to 1.02 times what FP64 multiply-add chains gave.
//
// Order of a K block: the slices arrive in pairs (A_j, B_j), j = 1..8, and
// step j runs the products that pair j completes, (j, t <= min(j, 9 - j)) and
// (s < j, j) with s <= 9 - j, so the tensor pipe starts with the first pair;
// pairs j and 9 - j have their last use in step j >= 5.  Bound: shared memory.
// A K block's 144 MMAs read their operands in 48 clocks each (6.9 k), its 192
// KB arrive by TMA at 32 bytes a clock (6.1 k), and the two add up: 13.3 k
// clocks (6.4 us) measured, of which the MMA queue is busy 10.2 k; then 13 us
// of drain.  The 64-column tile is what 8 levels leave room for in TMEM.
//
// A row whose maximum is not finite (or that holds subnormals only) is marked
// by the packing; its outputs are done by FP64 dot products over the operands.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>
#include <stdexcept>

#include "engine.h"
#include "fx_tile.cuh"
#include "gemm_tc.h"
#include "slice_math.cuh"
#include "tc_ptx.cuh"

namespace tdcc {

CUtensorMap slice_map(const void* base, int S, int rows_pad, int K_pad, int box_rows);

namespace {

struct DeepShared {
  uint64_t full[TcDeep::STAGES], empty[TcDeep::STAGES];
  uint64_t accfull, accempty, done;
  uint32_t tmem;
  volatile int abort;
  long long col_off[TcDeep::BN];  // output offset of each logical column (-1: outside)
  int col_exp[TcDeep::BN];        // stored exponent of each packed column of B
};

// sum over k in [k0, k1) of A[m, k] B[k, n] of batch z, operands as they are
__device__ __noinline__ double2 direct_dot(const TcArgs& g, int m, int n, int z, int k0, int k1) {
  long long ao, bo, dummy;
  decode2(g.gmA, m, ao, dummy);
  decode2(g.gnB, n, bo, dummy);
  ao += z * g.bsA;
  bo += z * g.bsB;
  const double *A = static_cast<const double*>(g.srcA), *B = static_cast<const double*>(g.srcB);
  double2 s = make_double2(0.0, 0.0);
  for (int k = k0; k < k1; ++k) {
    long long ka, kb;
    decode2(g.gkAB, k, ka, kb);
    const double2 x = g.ac ? load1<true>(A, ao + ka) : load1<false>(A, ao + ka);
    const double2 y = g.bc ? load1<true>(B, bo + kb) : load1<false>(B, bo + kb);
    if (g.ac && g.bc) {
      fmac(s, x, y);
    } else if (g.ac) {
      s = make_double2(fma(x.x, y.x, s.x), fma(x.y, y.x, s.y));
    } else {
      s = make_double2(fma(x.x, y.x, s.x), fma(x.x, y.y, s.y));
    }
  }
  return s;
}

template <bool AC, bool BC>
__global__ void __launch_bounds__(TcDeep::THREADS, 1)
    ozaki_deep_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ TcArgs g) {
  using C = TcDeep;
  constexpr int S = TC_DEEP_SLICES;
  extern __shared__ uint8_t smraw[];
  uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  uint8_t* stA = sm;                                // STAGES x 16 KB
  uint8_t* stB = sm + C::STAGES * C::A_BYTES;       // STAGES x 8 KB
  DeepShared* sh = (DeepShared*)(stB + C::STAGES * C::B_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::STAGES; ++i) {
      mbar_init(smem_u32(&sh->full[i]), 1);
      mbar_init(smem_u32(&sh->empty[i]), 1);
    }
    mbar_init(smem_u32(&sh->accfull), 1);
    mbar_init(smem_u32(&sh->accempty), 32 * C::EPI);
    mbar_init(smem_u32(&sh->done), 1);
    sh->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
    asm volatile("fence.proxy.async.shared::cta;");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = sh->tmem;

  const int mt = g.m_fast ? blockIdx.x : blockIdx.y, nt = g.m_fast ? blockIdx.y : blockIdx.x;
  const int zb = blockIdx.z / g.nsplit;
  const int kb0 = (blockIdx.z - zb * g.nsplit) * g.kb_per_split;
  const int kb1 = min(g.kblocks, kb0 + g.kb_per_split);
  const int rowA0 = g.bat_a ? zb * g.rowsA_pad : 0, rowB0 = g.bat_b ? zb * g.rowsB_pad : 0;
  const int nchunks = (kb1 - kb0 + C::CHUNK_KB - 1) / C::CHUNK_KB;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int it = 0;
      for (int kb = kb0; kb < kb1 && !sh->abort; ++kb)
        for (int s = 0; s < S && !sh->abort; ++s, ++it) {
          const int st = it % C::STAGES;
          if (!mbar_wait(smem_u32(&sh->empty[st]), (uint32_t)((it / C::STAGES) & 1) ^ 1u, kWaitLimit)) {
            fail(sh, g.err, 1);
            break;
          }
          const uint32_t fb = smem_u32(&sh->full[st]);
          mbar_expect_tx(fb, C::A_BYTES + C::B_BYTES);
          tma3d(smem_u32(stA + st * C::A_BYTES), &tmA, kb * TC_BK, rowA0 + mt * TC_BM, s, fb);
          tma3d(smem_u32(stB + st * C::B_BYTES), &tmB, kb * TC_BK, rowB0 + nt * C::BN, s, fb);
        }
      // every issued load lands before the CTA exits
      for (int j = (it > C::STAGES ? it - C::STAGES : 0); j < it; ++j)
        mbar_wait(smem_u32(&sh->full[j % C::STAGES]), (uint32_t)((j / C::STAGES) & 1), kWaitLimit);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the whole warp, one lane executing) ----------------
    constexpr uint32_t id = idesc_bf16(TC_BM, C::BN);
    const uint64_t hi64 = sdesc(0);
    const uint32_t a0 = (smem_u32(stA) & 0x3FFFF) >> 4, b0 = (smem_u32(stB) & 0x3FFFF) >> 4;
    const uint32_t full0 = smem_u32(&sh->full[0]), empty0 = smem_u32(&sh->empty[0]);
    const uint32_t on = lane == 0 ? 1u : 0u;
    uint32_t st0 = 0, ph = 0;  // ring slot and phase of the block's first pair
    bool ok = true;
    for (int c = 0; c < nchunks && ok; ++c) {
      if (c > 0 && !mbar_wait_warp(smem_u32(&sh->accempty), (uint32_t)((c - 1) & 1), kWaitLimit)) {
        fail(sh, g.err, 2);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const int kbs = kb0 + c * C::CHUNK_KB, kbe = min(kb1, kbs + C::CHUNK_KB);
#pragma unroll 1
      for (int kb = kbs; kb < kbe && ok; ++kb) {
        const bool first = kb == kbs;
        // what an MMA needs beside constants of the unrolled loops, once per slice
        uint32_t la[S], lb[S], slot[S];  // descriptor low words and ring slots of the block's slices
#pragma unroll
        for (int j = 0; j < S; ++j) {
          slot[j] = st0 + j < C::STAGES ? st0 + j : st0 + j - C::STAGES;
          la[j] = a0 + slot[j] * (C::A_BYTES >> 4);
          lb[j] = b0 + slot[j] * (C::B_BYTES >> 4);
        }
#pragma unroll
        for (int j = 1; j <= S; ++j) {
          if (ok) ok = mbar_wait_warp(full0 + 8 * slot[j - 1], st0 + j - 1 < C::STAGES ? ph : ph ^ 1u, kWaitLimit);
          asm volatile("tcgen05.fence::after_thread_sync;");
          if (ok) {
            auto product = [&](int s, int t) {
              // the first product of each level in a chunk starts its sum
              const bool lead = (s == t || s == t + 1) && s <= 5;
#pragma unroll
              for (int k = 0; k < TC_BK / 16; ++k)
                umma_warp(tmem + (uint32_t)((s + t - 2) * C::BN), hi64 | (uint64_t)(la[s - 1] + 2 * k),
                          hi64 | (uint64_t)(lb[t - 1] + 2 * k), id, (lead && k == 0 && first) ? 0u : 1u, on);
            };
            const int last = S + 1 - j;  // largest partner of slice j
#pragma unroll
            for (int t = 1; t <= S; ++t)
              if (t <= j && t <= last) product(j, t);
#pragma unroll
            for (int q = 1; q <= S; ++q)
              if (q < j && q <= last) product(q, j);
            if (j > S / 2) {  // pairs j and S + 1 - j have had their last use
              umma_commit_warp(empty0 + 8 * slot[j - 1], on);
              umma_commit_warp(empty0 + 8 * slot[last - 1], on);
            }
          }
        }
        if (!ok) fail(sh, g.err, 3);
        st0 += S;
        if (st0 >= C::STAGES) {
          st0 -= C::STAGES;
          ph ^= 1u;
        }
      }
      if (ok) umma_commit_warp(smem_u32(&sh->accfull), on);
      ok = __all_sync(0xffffffffu, ok && sh->abort == 0) != 0;
    }
    // all issued MMAs complete before TMEM is released
    umma_commit_warp(smem_u32(&sh->done), on);
    mbar_wait(smem_u32(&sh->done), 0, kWaitLimit);
  } else {
    // ---------------- drain warps (2 .. 17): 16 packed columns each ----------------
    const int q = warp & 3, j0 = ((warp - 2) >> 2) * 16;
    const int row = q * 32 + lane;
    {
      const int t = threadIdx.x - 64;
      constexpr int ncl = BC ? C::BN / 2 : C::BN;
      if (t < ncl) {
        const int n = nt * ncl + t;
        long long o = -1;
        if (n < g.N) decomp_tc(g.gnC, n, o);
        sh->col_off[t] = o;
      }
      if (t < C::BN) sh->col_exp[t] = g.expB[rowB0 + nt * C::BN + t];
      asm volatile("bar.sync 1, %0;" ::"n"(32 * C::EPI) : "memory");
    }
    const uint32_t tl = (uint32_t)(q * 32) << 16;
    long long hi[16], lo[16];  // levels 2..5 in units of 2^-35, 6..9 in units of 2^-63
#pragma unroll
    for (int j = 0; j < 16; ++j) hi[j] = lo[j] = 0;
    bool ok = true;
    for (int c = 0; c < nchunks; ++c) {
      if (__any_sync(0xffffffffu, sh->abort != 0)) {
        ok = false;
        break;
      }
      const bool got = mbar_wait(smem_u32(&sh->accfull), (uint32_t)(c & 1), kWaitLimit);
      if (!__all_sync(0xffffffffu, got)) {
        fail(sh, g.err, 4);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          uint32_t v0[16], v1[16];  // levels 2 + 4 h + 2 p and the next
          tmem_ld16_nowait(tmem + tl + (uint32_t)((4 * h + 2 * p) * C::BN + j0), v0);
          tmem_ld16_nowait(tmem + tl + (uint32_t)((4 * h + 2 * p + 1) * C::BN + j0), v1);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            // |v| <= 2^24: exact in 32 bits; two levels join in 64
            const long long x = ((long long)__float2int_rn(__uint_as_float(v0[j])) << 7) +
                                (long long)__float2int_rn(__uint_as_float(v1[j]));
            (h ? lo : hi)[j] += p ? x : x << 14;
          }
        }
      asm volatile("tcgen05.fence::before_thread_sync;");
      mbar_arrive(smem_u32(&sh->accempty));
    }
    if (ok && __any_sync(0xffffffffu, sh->abort != 0)) ok = false;
    if (ok) {
      const bool odd = AC && (lane & 1);
      constexpr int NJ = BC ? 8 : 16;          // logical columns of this warp
      constexpr int rows_out = AC ? 16 : 32;    // logical rows
      constexpr int RS = NJ + 1;
      double2* stage = reinterpret_cast<double2*>(sm) + (size_t)(warp - 2) * (32 * RS);  // the ring is idle
      const int lr = AC ? (lane >> 1) : lane;
      const int prow = mt * TC_BM + row;
      const int m = AC ? (prow >> 1) : prow;
      const int ea = prow < g.rowsA_pad ? g.expA[rowA0 + prow] : 0;
      const bool neg = g.alpha_pow2 && g.alpha_neg;
      const int ebase = row_exp(ea) - 63 + (g.alpha_pow2 ? g.alpha_e : 0);
      long long coffm = 0;
      if (m < g.M) decomp_tc(g.gmC, m, coffm);
      double2* Cc = static_cast<double2*>(g.C) + (g.cc ? zb * g.bsC : 0);
      double* Cr = static_cast<double*>(g.C) + (g.cc ? 0 : zb * g.bsC);
      const int m0w = AC ? ((mt * TC_BM + q * 32) >> 1) : (mt * TC_BM + q * 32);
      const int nrows = min(rows_out, g.M - m0w);
      const bool red = g.acc || g.atomic;
#pragma unroll
      for (int k = 0; k < NJ; ++k) {
        const int jj = (BC ? j0 / 2 : j0) + k;
        long long rh, rl, ih = 0, il = 0;  // real and imaginary part, high and low sum
        if constexpr (BC) {
          const long long h0 = hi[2 * k], h1 = hi[2 * k + 1], l0 = lo[2 * k], l1 = lo[2 * k + 1];
          if constexpr (AC) {
            const long long p0 = __shfl_xor_sync(0xffffffffu, h0, 1), p1 = __shfl_xor_sync(0xffffffffu, h1, 1);
            const long long s0 = __shfl_xor_sync(0xffffffffu, l0, 1), s1 = __shfl_xor_sync(0xffffffffu, l1, 1);
            // even lane: (re re, re im) own, (im re, im im) the partner's
            rh = odd ? p0 - h1 : h0 - p1;
            ih = odd ? p1 + h0 : h1 + p0;
            rl = odd ? s0 - l1 : l0 - s1;
            il = odd ? s1 + l0 : l1 + s0;
          } else {
            rh = h0;
            ih = h1;
            rl = l0;
            il = l1;
          }
        } else if constexpr (AC) {
          const long long p = __shfl_xor_sync(0xffffffffu, hi[k], 1), s = __shfl_xor_sync(0xffffffffu, lo[k], 1);
          rh = odd ? p : hi[k];
          ih = odd ? hi[k] : p;
          rl = odd ? s : lo[k];
          il = odd ? lo[k] : s;
        } else {
          rh = hi[k];
          rl = lo[k];
        }
        // with complex A the two lanes of a pair hold the same output: split columns
        if (AC && ((k & 1) != (lane & 1))) continue;
        const int eb = sh->col_exp[BC ? 2 * jj : jj];
        double2 v;
        if (ea == kExpMarked || eb == kExpMarked) {
          const int n = nt * (BC ? C::BN / 2 : C::BN) + jj;
          v = make_double2(0.0, 0.0);
          if (m < g.M && n < g.N)
            v = direct_dot(g, m, n, zb, kb0 * TC_BK, min(g.K, kb1 * TC_BK));
          if (g.alpha_pow2) {
            v.x *= g.ar;
            v.y *= g.ar;
          }
        } else {
          const int E = ebase + row_exp(eb);
          v.x = joined(neg ? -rh : rh, neg ? -rl : rl, E);
          v.y = (AC || BC) ? joined(neg ? -ih : ih, neg ? -il : il, E) : 0.0;
        }
        if (!g.alpha_pow2) v = make_double2(g.ar * v.x - g.ai * v.y, g.ar * v.y + g.ai * v.x);
        stage[lr * RS + k] = v;
      }
      __syncwarp();
      constexpr int RPP = 32 / NJ, NPASS = rows_out / RPP;
      const int lc = lane % NJ, lrw = lane / NJ;
      const long long cn = sh->col_off[(BC ? j0 / 2 : j0) + lc];
#pragma unroll 4
      for (int p = 0; p < NPASS; ++p) {
        const int r = p * RPP + lrw;
        const long long cm = __shfl_sync(0xffffffffu, coffm, (AC ? 2 * r : r) & 31);
        if (r >= nrows || cn < 0) continue;
        const long long off = cm + cn;
        const double2 v = stage[r * RS + lc];
        if (g.cc) {
          if (red) {
            atomicAdd(&Cc[off].x, v.x);
            atomicAdd(&Cc[off].y, v.y);
          } else {
            Cc[off] = v;
          }
        } else {
          if (red)
            atomicAdd(&Cr[off], v.x);
          else
            Cr[off] = v.x;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

}  // namespace

cudaError_t launch_deep(const TcArgs& a0, const void* packA, const void* packB, cudaStream_t st) {
  using C = TcDeep;
  static_assert(sizeof(DeepShared) <= 2560, "shared-memory tail");
  constexpr int kMaxDev = 64;
  static std::once_flag once[kMaxDev];
  static cudaError_t attr_err[kMaxDev] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [dev] {
    cudaError_t e = cudaSuccess;
    for (auto fn : {ozaki_deep_kernel<true, true>, ozaki_deep_kernel<true, false>, ozaki_deep_kernel<false, true>,
                    ozaki_deep_kernel<false, false>}) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    attr_err[dev] = e;
  });
  if (attr_err[dev] != cudaSuccess) return attr_err[dev];
  TcArgs a = a0;
  if (a.S != TC_DEEP_SLICES || a.rowsB_pad % C::BN != 0 || a.rowsA_pad % TC_BM != 0) return cudaErrorInvalidValue;
  a.tmem_cols = 512;
  const CUtensorMap ma = slice_map(packA, a.S, (a.bat_a ? a.nb : 1) * a.rowsA_pad, a.kblocks * TC_BK, TC_BM);
  const CUtensorMap mb = slice_map(packB, a.S, (a.bat_b ? a.nb : 1) * a.rowsB_pad, a.kblocks * TC_BK, C::BN);
  // the tiles of the smaller operand side vary fastest: that side stays in L2
  const unsigned mtiles = (unsigned)(a.rowsA_pad / TC_BM), ntiles = (unsigned)(a.rowsB_pad / C::BN);
  a.m_fast = (a.rowsA_pad < a.rowsB_pad && ntiles <= 65535u) ? 1 : 0;
  if ((a.m_fast ? ntiles : mtiles) > 65535u || (long long)a.nb * a.nsplit > 65535LL) return cudaErrorInvalidConfiguration;
  dim3 grid(a.m_fast ? mtiles : ntiles, a.m_fast ? ntiles : mtiles, (unsigned)((long long)a.nb * a.nsplit));
  if (a.ac && a.bc)
    ozaki_deep_kernel<true, true><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  else if (a.ac)
    ozaki_deep_kernel<true, false><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  else if (a.bc)
    ozaki_deep_kernel<false, true><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  else
    ozaki_deep_kernel<false, false><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  count_launch();
  return cudaGetLastError();
}

}  // namespace tdcc
