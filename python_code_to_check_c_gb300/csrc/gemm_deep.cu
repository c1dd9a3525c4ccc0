// Exact BF16 slice products on tcgen05 with the sums over all of K in the drain
// warps' registers: the FP64 form's contractions (8 slices of 8 bits a side, the
// first of 7: 63 bits under each real row's maximum, the last digit rounded) and the
// mixed form's with up to 5 slices of 7 bits and K beyond two blocks.
//
// The products A_s B_t with s + t <= S + 1 go to the accumulators of their
// levels L = s + t, FP32 sums of integers that stay exact over a K chunk
// (TcDeep::CHUNK_KB).  The S levels of a 128 x BN tile fill TMEM (BN = 128, 96,
// 64 for S <= 4, 5, 8); after every chunk the drain warps add them to int64
// sums (two per output for S = 8, levels 2..5 and 6..9), which are rounded to
// FP64 once at the end.  With 8 slices the real and the imaginary part of a complex
// row have scales of their own (a small imaginary part keeps its bits), so their
// sums become doubles before they meet; and rows that even 63 bits hold worse than
// FP64 does are found by the range guard below.
//
// Order of a K block: the slices arrive in pairs (A_j, B_j), j = 1..S, and
// step j runs the products that pair j completes, (j, t <= min(j, S + 1 - j))
// and (s < j, j) with s <= S + 1 - j, so the tensor pipe starts with the first
// pair; a pair is released after its last product.  Bound: shared memory.  A K
// block's MMAs read their operands at 128 bytes a clock (S = 8: 144 of 48
// clocks, 6.9 k), its slices arrive by TMA at 32 (192 KB, 6.1 k), and the two
// add up: 13.3 k clocks measured (with a drain every 6 blocks; 8-bit digits drain
// every 2, and the guard takes 0.4 k a block: the ladder at o=10, v=38, 1444 x 200 x
// 1444 real, 70 us with 7-bit digits, 78 so).  So the wider the tile the better (per
// output column and K block 52, 82 and 204 clocks for S = 4, 5, 8).  Measured:
// the 24-trajectory ladder at o=10, v=38 (S = 4, 1444 x 4800 x 1444 real) 210
// us, 335 as single-chunk 128-column tiles over split K; the ladder
// at o=18, v=82 (S = 5, 6724 x 648 x 6724 real) 829 us, 1842 as 64-column tiles
// with int64 partial sums in TMEM (TcWide).  With complex rows the two lanes of a
// row finish a column each (the ring terms of the former, K = 380: 174 -> 139 us).
//
// A row whose maximum is not finite (or that holds subnormals only) is marked
// by the packing with 8 slices; its outputs, and those that the range guard sends
// on, are done by FP64 multiply-adds over the operands: where few of a warp's outputs are
// marked, its lanes over k for four rows of a column; where many are, a lane a row for
// four columns.  Many are where a molecule's symmetry forbids elements and leaves noise
// in them (10^-16 of the others, three quarters of the outputs): the FP64 pipe is then
// the bound, T2 residual at o=10, v=38 7.5 ms by the former alone, 5.2 so, 0.9 without
// noise, and 5.1 with or without it on the FP64 pipe throughout.
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

// The range guard.  Digits under the maximum of a row hold its small elements worse
// than FP64 does: with the factors in units of their rows' powers of two, K products
// are off by about 2^-63.6 sqrt(K) in all (the levels left out 2^-64.2 a product, the
// rounding of each factor 2^-64.8).  A plane of each packed operand holds the magnitudes
// x, y in 8 bits; after the slices one more product on the tensor cores gives S = sum
// x y, against which FP64 chains are off by 0.46 x 2^-53 (normal rows) to 0.9 (the
// residuals' own, K = 81 .. 1444).  An output with S < 2^-10 sqrt(K), that is with
// an error above 0.65 x 2^-53 S (rms), is done by FP64 multiply-adds; S = 0 has no product
// that is not zero.  A part of a K split takes its S for its share of the whole.  The
// planes hold 2^15 x, from 2^-31 of a row's maximum up, and what lies below it as that:
// K such products reach the limit for no K below 2^42 (2^-16, without the factor, did
// from K = 4096 on).
constexpr float kGuardDeep = 0x1p20f;  // 2^-10 in the planes' units

template <class C>
struct DeepShared {
  uint64_t full[C::STAGES], empty[C::STAGES];
  uint64_t accfull, accempty, done;
  uint32_t tmem;
  volatile int abort;
  long long col_off[C::BN];  // output offset of each logical column (-1: outside)
  int col_exp[C::BN];        // stored exponent of each packed column of B
  long long col_offT[C::S > 5 ? C::BN : 1];  // offset of each column as a row (symmetric products)
};

// Rows m[0 .. 3] of A times column n of B over k in [k0, k1), batch z, the operands
// as they are: FP64 multiply-adds, the lanes of the warp over k (every lane returns
// the sums).
constexpr int kDirect = 4;
template <bool AC, bool BC>
__device__ __noinline__ void direct_dots(const TcArgs& g, const int (&m)[kDirect], int n, int z, int k0, int k1,
                                         double2 (&s)[kDirect]) {
  const int lane = threadIdx.x & 31;
  long long ao[kDirect], bo, dummy;
  double2 c[kDirect];
#pragma unroll
  for (int i = 0; i < kDirect; ++i) {
    decode2(g.gmA, m[i], ao[i], dummy);
    ao[i] += z * g.bsA;
    c[i] = make_double2(0.0, 0.0);
  }
  decode2(g.gnB, n, bo, dummy);
  bo += z * g.bsB;
  const double *A = static_cast<const double*>(g.srcA), *B = static_cast<const double*>(g.srcB);
#pragma unroll 2
  for (int k = k0 + lane; k < k1; k += 32) {
    long long ka, kb;
    decode2(g.gkAB, k, ka, kb);
    const double2 y = load1<BC>(B, bo + kb);
#pragma unroll
    for (int i = 0; i < kDirect; ++i) {
      const double2 x = load1<AC>(A, ao[i] + ka);
      if constexpr (AC && BC) {
        fmac(c[i], x, y);
      } else if constexpr (AC) {
        c[i] = make_double2(fma(x.x, y.x, c[i].x), fma(x.y, y.x, c[i].y));
      } else {
        c[i].x = fma(x.x, y.x, c[i].x);
        if constexpr (BC) c[i].y = fma(x.x, y.y, c[i].y);
      }
    }
  }
  // the 4 or 8 sums meet across the warp, halving what a lane holds while it can (9
  // additions instead of 40)
  constexpr int NV = AC || BC ? 2 * kDirect : kDirect;
  double v[NV];
#pragma unroll
  for (int i = 0; i < kDirect; ++i) {
    if constexpr (AC || BC) {
      v[2 * i] = c[i].x;
      v[2 * i + 1] = c[i].y;
    } else {
      v[i] = c[i].x;
    }
  }
  int d = 16;
#pragma unroll
  for (int n = NV / 2; n >= 1; n >>= 1, d >>= 1)
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const double send = lane & d ? v[i] : v[i + n], keep = lane & d ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
    }
  for (; d > 0; d >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], d);
  constexpr int LV = 32 / NV;  // lanes that hold the same sum
#pragma unroll
  for (int i = 0; i < kDirect; ++i) {
    s[i].x = __shfl_sync(0xffffffffu, v[0], LV * (AC || BC ? 2 * i : i));
    s[i].y = AC || BC ? __shfl_sync(0xffffffffu, v[0], LV * (2 * i + 1)) : 0.0;
  }
}

// The same for row m of each lane and columns n .. n + 3, one lane over all of k (the
// two lanes of a complex row share it): nothing to meet but those two, and the four
// columns read a row's elements once.  m, n may lie outside (their sums are not used).
template <bool AC, bool BC>
__device__ __noinline__ void direct_rows(const TcArgs& g, int m, int n, int z, int k0, int k1, double2 (&s)[kDirect]) {
  const int lane = threadIdx.x & 31;
  long long ao, bo[kDirect], dummy;
  decode2(g.gmA, min(m, g.M - 1), ao, dummy);
  ao += z * g.bsA;
#pragma unroll
  for (int i = 0; i < kDirect; ++i) {
    decode2(g.gnB, min(n + i, g.N - 1), bo[i], dummy);
    bo[i] += z * g.bsB;
    s[i] = make_double2(0.0, 0.0);
  }
  const double *A = static_cast<const double*>(g.srcA), *B = static_cast<const double*>(g.srcB);
  for (int kk = k0; kk < k1; kk += 32) {  // a K offset a lane, handed round
    const int kn = min(32, k1 - kk);
    long long ka = 0, kb = 0;
    if (lane < kn) decode2(g.gkAB, kk + lane, ka, kb);
    double2 c[kDirect];
#pragma unroll
    for (int i = 0; i < kDirect; ++i) c[i] = make_double2(0.0, 0.0);
#pragma unroll 2
    for (int j = 0; j < kn; j += AC ? 2 : 1) {
      const int k = AC ? j + (lane & 1) : j;
      const long long xa = __shfl_sync(0xffffffffu, ka, k), yb = __shfl_sync(0xffffffffu, kb, k);
      if (k >= kn) continue;
      const double2 x = load1<AC>(A, ao + xa);
#pragma unroll
      for (int i = 0; i < kDirect; ++i) {
        const double2 y = load1<BC>(B, bo[i] + yb);
        if constexpr (AC && BC) {
          fmac(c[i], x, y);
        } else if constexpr (AC) {
          c[i] = make_double2(fma(x.x, y.x, c[i].x), fma(x.y, y.x, c[i].y));
        } else {
          c[i].x = fma(x.x, y.x, c[i].x);
          if constexpr (BC) c[i].y = fma(x.x, y.y, c[i].y);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kDirect; ++i) {
      s[i].x += c[i].x;
      if constexpr (AC || BC) s[i].y += c[i].y;
    }
  }
  if constexpr (AC)
#pragma unroll
    for (int i = 0; i < kDirect; ++i) {
      s[i].x += __shfl_xor_sync(0xffffffffu, s[i].x, 1);
      s[i].y += __shfl_xor_sync(0xffffffffu, s[i].y, 1);
    }
}

template <class C, bool AC, bool BC>
__global__ void __launch_bounds__(C::THREADS, 1)
    ozaki_deep_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ TcArgs g) {
  constexpr int S = C::S;
  extern __shared__ uint8_t smraw[];
  uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  uint8_t* stA = sm;                                // STAGES x 16 KB
  uint8_t* stB = sm + C::STAGES * C::A_BYTES;       // STAGES x BN x 128 B
  DeepShared<C>* sh = (DeepShared<C>*)(stB + C::STAGES * C::B_BYTES);
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
  constexpr bool SYM = !AC && !BC && S > 5;
  // a symmetric product's tile below the diagonal comes from its mirror image
  const bool skip = SYM && g.sym && (nt + 1) * C::BN <= mt * TC_BM;
  const int zb = blockIdx.z / g.nsplit;
  const int kb0 = (blockIdx.z - zb * g.nsplit) * g.kb_per_split;
  const int kb1 = skip ? kb0 : min(g.kblocks, kb0 + g.kb_per_split);
  const int rowA0 = g.bat_a ? zb * g.rowsA_pad : 0, rowB0 = g.bat_b ? zb * g.rowsB_pad : 0;
  const int nchunks = (kb1 - kb0 + C::CHUNK_KB - 1) / C::CHUNK_KB;
  const int wait = g.wait == 0 ? kWaitLimit : g.wait;
  // 8 slices: digits of 8 bits, a scale for each real row; after the chunks, the range
  // guard over the same K
  constexpr bool GUARD = S == TC_DEEP_SLICES;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int it = 0;
      auto load = [&](int kb, int s) {
        const int st = it % C::STAGES;
        if (!mbar_wait(smem_u32(&sh->empty[st]), (uint32_t)((it / C::STAGES) & 1) ^ 1u, wait)) {
          fail(sh, g.err, 1);
          return;
        }
        const uint32_t fb = smem_u32(&sh->full[st]);
        mbar_expect_tx(fb, C::A_BYTES + C::B_BYTES);
        const int x = GUARD && s == S ? kb * (TC_BK / 2) : kb * TC_BK;  // (a byte a number)
        tma3d(smem_u32(stA + st * C::A_BYTES), &tmA, x, rowA0 + mt * TC_BM, s, fb);
        tma3d(smem_u32(stB + st * C::B_BYTES), &tmB, x, rowB0 + nt * C::BN, s, fb);
        ++it;
      };
      for (int kb = kb0; kb < kb1 && !sh->abort; ++kb)
        for (int s = 0; s < S && !sh->abort; ++s) load(kb, s);
      if (GUARD)
        for (int kb = kb0; kb < kb1 && !sh->abort; kb += 2) load(kb, S);
      // every issued load lands before the CTA exits
      for (int j = (it > C::STAGES ? it - C::STAGES : 0); j < it; ++j)
        mbar_wait(smem_u32(&sh->full[j % C::STAGES]), (uint32_t)((j / C::STAGES) & 1), kWaitLimit);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the whole warp, one lane executing) ----------------
    constexpr uint32_t id = idesc_bf16(TC_BM, C::BN);
    const uint32_t on = lane == 0 ? 1u : 0u;
    PairRing<C::STAGES, C::A_BYTES, C::B_BYTES> ring(stA, stB, &sh->full[0], &sh->empty[0]);
    ring.wait = wait;
    bool ok = true;
    for (int c = 0; c < nchunks && ok; ++c) {
      if (c > 0 && !mbar_wait_warp(smem_u32(&sh->accempty), (uint32_t)((c - 1) & 1), wait)) {
        fail(sh, g.err, 2);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const int kbs = kb0 + c * C::CHUNK_KB, kbe = min(kb1, kbs + C::CHUNK_KB);
#pragma unroll 1
      for (int kb = kbs; kb < kbe && ok; ++kb) ok = ring.template issue<S, C::BN>(tmem, id, kb == kbs, on);
      if (!ok) fail(sh, g.err, 3);
      if (ok) umma_commit_warp(smem_u32(&sh->accfull), on);
      ok = __all_sync(0xffffffffu, ok && sh->abort == 0) != 0;
    }
    if (GUARD && ok && nchunks > 0) {
      ok = mbar_wait_warp(smem_u32(&sh->accempty), (uint32_t)((nchunks - 1) & 1), wait);
      if (!ok) fail(sh, g.err, 2);
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
      for (int kb = kb0; kb < kb1 && ok; kb += 2) {
        ok = ring.template guard<C::BN>(tmem, id, kb == kb0, kb + 1 == kb1, on);
        if (!ok) fail(sh, g.err, 3);
      }
      if (ok) umma_commit_warp(smem_u32(&sh->accfull), on);
    }
    // all issued MMAs complete before TMEM is released
    umma_commit_warp(smem_u32(&sh->done), on);
    mbar_wait(smem_u32(&sh->done), 0, kWaitLimit);
  } else {
    // ---------------- drain warps (2 .. 17): NC packed columns each ----------------
    constexpr int NC = C::BN / (C::EPI / 4), HL = S > 5 ? 2 : 1;
    const int q = warp & 3, j0 = ((warp - 2) >> 2) * NC;
    const int row = q * 32 + lane;
    {
      const int t = threadIdx.x - 64;
      constexpr int ncl = BC ? C::BN / 2 : C::BN;
      if (t < ncl) {
        const int n = nt * ncl + t;
        long long o = -1;
        if (n < g.N) decomp_tc(g.gnC, n, o);
        sh->col_off[t] = o;
        if constexpr (SYM) {
          if (g.sym && n < g.N) decomp_tc(g.gmC, n, o);
          sh->col_offT[t] = o;
        }
      }
      // the last tile may reach beyond the packed rows (its loads read zeros
      // or the next batch there; those columns are not stored)
      if (t < C::BN) sh->col_exp[t] = nt * C::BN + t < g.rowsB_pad ? g.expB[rowB0 + nt * C::BN + t] : 0;
      asm volatile("bar.sync 1, %0;" ::"n"(32 * C::EPI) : "memory");
    }
    const int prow = mt * TC_BM + row;
    const int ea = prow < g.rowsA_pad ? g.expA[rowA0 + prow] : 0;
    const uint32_t tl = (uint32_t)(q * 32) << 16;
    // exact sums in units of 2^-u: all levels (u = 7 (S + 1)), or with S = 8
    // levels 2..5 (u = 38) and 6..9 (u = 70)
    long long acc[HL][NC];
#pragma unroll
    for (int h = 0; h < HL; ++h)
#pragma unroll
      for (int j = 0; j < NC; ++j) acc[h][j] = 0;
    bool ok = true;
    unsigned direct = 0u;  // this row's columns that the guard sends to FP64 multiply-adds
    for (int c = 0; c < nchunks; ++c) {
      if (__any_sync(0xffffffffu, sh->abort != 0)) {
        ok = false;
        break;
      }
      const bool got = mbar_wait(smem_u32(&sh->accfull), (uint32_t)(c & 1), wait);
      if (!__all_sync(0xffffffffu, got)) {
        fail(sh, g.err, 4);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      constexpr int SL = S / HL, BITS = HL == 2 ? 8 : 7;  // levels per sum, bits between them
#pragma unroll
      for (int h = 0; h < HL; ++h)
#pragma unroll
        for (int w = 0; w < NC; w += 8) {
          uint32_t v[SL][8];
#pragma unroll
          for (int p = 0; p < SL; ++p) tmem_ld8_nowait(tmem + tl + (uint32_t)((SL * h + p) * C::BN + j0 + w), v[p]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            // |v| <= 2^24: exact in 32 bits, Horner in 64
            long long x = (long long)__float2int_rn(__uint_as_float(v[0][j]));
#pragma unroll
            for (int p = 1; p < SL; ++p) x = (x << BITS) + (long long)__float2int_rn(__uint_as_float(v[p][j]));
            acc[h][w + j] += x;
          }
        }
      asm volatile("tcgen05.fence::before_thread_sync;");
      mbar_arrive(smem_u32(&sh->accempty));
    }
    const int k0 = kb0 * TC_BK, k1 = min(g.K, kb1 * TC_BK);  // (with 8 slices)
    if (GUARD && ok && nchunks > 0) {
      const bool got = mbar_wait(smem_u32(&sh->accfull), (uint32_t)(nchunks & 1), wait);
      if (!__all_sync(0xffffffffu, got)) {
        fail(sh, g.err, 4);
        ok = false;
      } else {
        asm volatile("tcgen05.fence::after_thread_sync;");
        const float share = (float)(k1 - k0) / (float)g.K, limit = kGuardDeep * sqrtf((float)g.K) * share;
#pragma unroll
        for (int w = 0; w < NC; w += 8) {
          uint32_t a8[8];
          tmem_ld8_nowait(tmem + tl + (uint32_t)(j0 + w), a8);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float sxy = __uint_as_float(a8[j]);
            if ((sxy != 0.f && !(sxy >= limit)) || sh->col_exp[j0 + w + j] == kExpMarked)
              direct |= 1u << (w + j);
          }
        }
        if (ea == kExpMarked) direct = ~0u;
        if (AC) direct |= __shfl_xor_sync(0xffffffffu, direct, 1);  // the row's other part
      }
    }
    if (__any_sync(0xffffffffu, sh->abort != 0)) ok = false;
    // a wait that ran out leaves no numbers behind: NaN, straight from the registers
    // (loads may still be on their way to the ring)
    const bool lost = !ok;
    if (!skip) {
      const bool odd = AC && (lane & 1);
      constexpr int GC = NC > 24 ? NC / 2 : NC;  // packed columns staged at a time
      constexpr int NL = BC ? GC / 2 : GC;       // logical columns of them
      constexpr int rows_out = AC ? 16 : 32;     // logical rows
      constexpr int RS = NL + 1;
      static_assert(C::EPI * 32 * RS * 16 <= C::STAGES * (C::A_BYTES + C::B_BYTES), "staging fits the ring");
      double2* stage = reinterpret_cast<double2*>(sm) + (size_t)(warp - 2) * (32 * RS);  // the ring is idle
      const int lr = AC ? (lane >> 1) : lane;
      const int m = AC ? (prow >> 1) : prow;
      const bool neg = g.alpha_pow2 && g.alpha_neg;
      const int ebase = row_exp(ea) - (HL == 2 ? 70 : 7 * (S + 1)) + (g.alpha_pow2 ? g.alpha_e : 0);
      long long coffm = 0;
      if (m < g.M) decomp_tc(g.gmC, m, coffm);
      long long coffT = 0;  // this row as a column
      if (SYM && g.sym && m < g.M) decomp_tc(g.gnC, m, coffT);
      double2* Cc = static_cast<double2*>(g.C) + (g.cc ? zb * g.bsC : 0);
      double* Cr = static_cast<double*>(g.C) + (g.cc ? 0 : zb * g.bsC);
      const int m0w = AC ? ((mt * TC_BM + q * 32) >> 1) : (mt * TC_BM + q * 32);
      const int nrows = min(rows_out, g.M - m0w);
      const bool red = g.acc || g.atomic;
      const double nan = __longlong_as_double(0x7FF8000000000000ll);
#pragma unroll
      for (int g0 = 0; g0 < NC; g0 += GC) {
        if (g0) __syncwarp();  // the previous group's stores have read the staging area
        auto put = [&](int k, double2 v) {
          if (lost) return;
          if (!g.alpha_pow2) v = make_double2(g.ar * v.x - g.ai * v.y, g.ar * v.y + g.ai * v.x);
          stage[lr * RS + k] = v;
        };
        if constexpr (HL == 2) {
          // every real row and column has a scale of its own: the sums become
          // doubles first.  A complex row's two parts lie in neighbouring lanes:
          // the even one finishes column k, the odd one k + 1, each with what the
          // other holds of it
          auto value = [&](int j) {
            const int E = ebase + row_exp(sh->col_exp[j0 + g0 + j]);
            const long long h = acc[0][g0 + j], l = acc[HL - 1][g0 + j];
            return joined<32>(neg ? -h : h, neg ? -l : l, E);
          };
          if constexpr (AC) {
            static_assert(NL % 2 == 0, "columns in pairs");
#pragma unroll
            for (int k = 0; k < NL; k += 2) {
              if constexpr (BC) {
                const double x0 = value(2 * k), x1 = value(2 * k + 1), y0 = value(2 * k + 2), y1 = value(2 * k + 3);
                const double p0 = __shfl_xor_sync(0xffffffffu, odd ? x0 : y0, 1);
                const double p1 = __shfl_xor_sync(0xffffffffu, odd ? x1 : y1, 1);
                // even: (re re, re im) own, (im re, im im) the partner's
                put(k + (odd ? 1 : 0), odd ? make_double2(p0 - y1, p1 + y0) : make_double2(x0 - p1, x1 + p0));
              } else {
                const double x = value(k), y = value(k + 1);
                const double p = __shfl_xor_sync(0xffffffffu, odd ? x : y, 1);
                put(k + (odd ? 1 : 0), odd ? make_double2(p, y) : make_double2(x, p));
              }
            }
          } else {
#pragma unroll
            for (int k = 0; k < NL; ++k)
              put(k, BC ? make_double2(value(2 * k), value(2 * k + 1)) : make_double2(value(k), 0.0));
          }
          // what the guard found, four columns at a time: where few of their outputs
          // are marked, the warp's lanes over k for four rows of one column
#pragma unroll 1
          for (int kq = 0; !lost && __any_sync(0xffffffffu, direct != 0u) && kq < NL; kq += kDirect) {
            static_assert(NL % kDirect == 0, "columns in fours");
            const int n = nt * (BC ? C::BN / 2 : C::BN) + (BC ? (j0 + g0) / 2 : j0 + g0) + kq;
            unsigned mine = 0u;  // bit i: this row's column n + i
#pragma unroll
            for (int i = 0; i < kDirect; ++i)
              if (m < g.M && n + i < g.N && !(AC && odd) && ((direct >> (BC ? g0 + 2 * (kq + i) : g0 + kq + i)) & (BC ? 3u : 1u)))
                mine |= 1u << i;
            __syncwarp();  // the staged values are written
            const int marked = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(mine));
            // (the lanes over k: a quarter of K and some 64 multiply-adds' time to meet for
            // four outputs; a lane a row: 8 K for 128)
            if (marked * (k1 - k0 + 256) > (AC ? 64 : 128) * (k1 - k0)) {
              double2 s[kDirect];
              direct_rows<AC, BC>(g, m, n, zb, k0, k1, s);
#pragma unroll
              for (int i = 0; i < kDirect; ++i)
                if (mine >> i & 1u) {
                  if (g.alpha_pow2) s[i] = make_double2(g.ar * s[i].x, g.ar * s[i].y);
                  put(kq + i, s[i]);
                }
              continue;
            }
#pragma unroll 1
            for (int k = 0; k < kDirect; ++k) {
              unsigned rows = __ballot_sync(0xffffffffu, (mine >> k) & 1u);
              while (rows) {
                int src[kDirect], mm[kDirect];
#pragma unroll
                for (int i = 0; i < kDirect; ++i) {
                  src[i] = rows ? __ffs(rows) - 1 : -1;
                  rows &= rows - 1u;
                  mm[i] = __shfl_sync(0xffffffffu, m, max(src[i], src[0]));
                }
                double2 s[kDirect];
                direct_dots<AC, BC>(g, mm, n + k, zb, k0, k1, s);
#pragma unroll
                for (int i = 0; i < kDirect; ++i)
                  if (lane == src[i]) {
                    if (g.alpha_pow2) s[i] = make_double2(g.ar * s[i].x, g.ar * s[i].y);
                    put(kq + k, s[i]);
                  }
              }
            }
          }
        } else {
          // value of the staged column k from its exact sums
          auto finish = [&](int k, long long re, long long im) {
            const int E = ebase + row_exp(sh->col_exp[(BC ? 2 * ((j0 + g0) / 2 + k) : j0 + g0 + k)]);
            put(k, make_double2(scaled_i64_to_double(neg ? -re : re, E),
                                (AC || BC) ? scaled_i64_to_double(neg ? -im : im, E) : 0.0));
          };
          if constexpr (AC) {
            // (lanes as above; the two parts share a scale, so the sums meet exactly)
            static_assert(NL % 2 == 0, "columns in pairs");
#pragma unroll
            for (int k = 0; k < NL; k += 2) {
              if constexpr (BC) {
                const long long* c = &acc[0][g0 + 2 * k];
                const long long p0 = __shfl_xor_sync(0xffffffffu, odd ? c[0] : c[2], 1);
                const long long p1 = __shfl_xor_sync(0xffffffffu, odd ? c[1] : c[3], 1);
                const long long x0 = odd ? c[2] : c[0], x1 = odd ? c[3] : c[1];
                finish(k + (odd ? 1 : 0), odd ? p0 - x1 : x0 - p1, odd ? p1 + x0 : x1 + p0);
              } else {
                const long long* c = &acc[0][g0 + k];
                const long long p = __shfl_xor_sync(0xffffffffu, odd ? c[0] : c[1], 1);
                const long long x = odd ? c[1] : c[0];
                finish(k + (odd ? 1 : 0), odd ? p : x, odd ? x : p);
              }
            }
          } else {
#pragma unroll
            for (int k = 0; k < NL; ++k) finish(k, BC ? acc[0][g0 + 2 * k] : acc[0][g0 + k], BC ? acc[0][g0 + 2 * k + 1] : 0);
          }
        }
        __syncwarp();
        if constexpr (SYM) {  // the mirror image: lanes along the rows, which are its columns
          if (g.sym && lane < nrows)
#pragma unroll 4
            for (int k = 0; k < NL; ++k) {
              const long long cT = sh->col_offT[j0 + g0 + k];
              if (cT >= 0 && m <= nt * C::BN + j0 + g0 + k) Cr[cT + coffT] = lost ? nan : stage[lane * RS + k].x;
            }
        }
        // every lane owns a (row, column) pair per pass
#pragma unroll 4
        for (int i = lane; i < rows_out * NL; i += 32) {
          const int r = i / NL, lc = i - r * NL;
          const long long cm = __shfl_sync(0xffffffffu, coffm, (AC ? 2 * r : r) & 31);
          const long long cn = sh->col_off[(BC ? (j0 + g0) / 2 : j0 + g0) + lc];
          if (r >= nrows || cn < 0) continue;
          if (SYM && g.sym && m0w + r > nt * C::BN + j0 + g0 + lc) continue;  // stored by the mirror image's tile
          const long long off = cm + cn;
          const double2 v = lost ? make_double2(nan, nan) : stage[r * RS + lc];
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
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

template <class C>
cudaError_t launch_deep_form(const TcArgs& a0, const void* packA, const void* packB, cudaStream_t st) {
  static_assert(sizeof(DeepShared<C>) <= C::TAIL && C::SMEM <= 232448, "shared memory");
  constexpr int kMaxDev = 64;
  static std::once_flag once[kMaxDev];
  static cudaError_t attr_err[kMaxDev] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [dev] {
    cudaError_t e = cudaSuccess;
    for (auto fn : {ozaki_deep_kernel<C, true, true>, ozaki_deep_kernel<C, true, false>,
                    ozaki_deep_kernel<C, false, true>, ozaki_deep_kernel<C, false, false>}) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    attr_err[dev] = e;
  });
  if (attr_err[dev] != cudaSuccess) return attr_err[dev];
  TcArgs a = a0;
  if (a.sym && (C::S <= 5 || a.ac || a.bc || a.cc || a.acc || a.atomic || a.nb != 1 || a.M != a.N || packA != packB))
    return cudaErrorInvalidValue;
  if (a.S != C::S || a.rowsB_pad < 1 || a.rowsA_pad % TC_BM != 0) return cudaErrorInvalidValue;
  a.tmem_cols = 512;
  const CUtensorMap ma = slice_map(packA, tc_planes(a.S), (a.bat_a ? a.nb : 1) * a.rowsA_pad, a.kblocks * TC_BK, TC_BM);
  const CUtensorMap mb = slice_map(packB, tc_planes(a.S), (a.bat_b ? a.nb : 1) * a.rowsB_pad, a.kblocks * TC_BK, C::BN);
  // the tiles of the smaller operand side vary fastest: that side stays in L2
  const unsigned mtiles = (unsigned)(a.rowsA_pad / TC_BM);
  const unsigned ntiles = (unsigned)(((long long)a.N * (a.bc ? 2 : 1) + C::BN - 1) / C::BN);
  // (a side of more than 65535 tiles, v^3 rows at v > 203, has to)
  a.m_fast = mtiles > 65535u || (a.rowsA_pad < a.rowsB_pad && ntiles <= 65535u) ? 1 : 0;
  if ((a.m_fast ? ntiles : mtiles) > 65535u || (long long)a.nb * a.nsplit > 65535LL) return cudaErrorInvalidConfiguration;
  dim3 grid(a.m_fast ? mtiles : ntiles, a.m_fast ? ntiles : mtiles, (unsigned)((long long)a.nb * a.nsplit));
  if (a.ac && a.bc)
    ozaki_deep_kernel<C, true, true><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  else if (a.ac)
    ozaki_deep_kernel<C, true, false><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  else if (a.bc)
    ozaki_deep_kernel<C, false, true><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  else
    ozaki_deep_kernel<C, false, false><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_deep(const TcArgs& a, const void* packA, const void* packB, cudaStream_t st) {
  switch (a.S) {
    case 2: return launch_deep_form<TcDeep<2, 128, 6>>(a, packA, packB, st);
    case 3: return launch_deep_form<TcDeep<3, 128, 6>>(a, packA, packB, st);
    case 4: return launch_deep_form<TcDeep<4, 128, 6>>(a, packA, packB, st);
    case 5: return launch_deep_form<TcDeep<5, 96, 8>>(a, packA, packB, st);
    case 8: return launch_deep_form<TcDeep<8, 64, 9>>(a, packA, packB, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace tdcc
