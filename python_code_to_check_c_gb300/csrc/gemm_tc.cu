// Tensor-core backend of the mixed-precision mode: FP64 contractions
// computed as exact integer products of BF16 slices on tcgen05.
//
// Operand packing (pack_kernel): each row of A (an M x K view) and each
// column of B (a K x N view) is scaled by 2^-e with e the binary exponent of
// its largest magnitude, then cut into S slices of 7 bits,
//     x * 2^-e = sum_s q_s 2^(-7s),  q_s integers, |q_1| <= 128, |q_s| <= 64
// (balanced digits: each lower digit in [-64, 63], carries into the next),
// each exactly representable in BF16.  Complex operands contribute two packed
// rows (real, imaginary) per logical row.  Packed layout: [S][rows][K] BF16,
// K contiguous (K-major for UMMA), rows and K zero-padded to the tile sizes.
//
// Products (ozaki_kernel): for every pair (s, t) with s + t <= S + 1 the
// slice product A_s B_t^T is accumulated by tcgen05.mma (kind::f16, BF16
// inputs, FP32 accumulate in TMEM) into the accumulator of its level
// L = s + t.  With |q_1| <= 128 and |q_s| <= 64 the products of one level
// at one K index add up to at most 2^14 + 2^13 + 2^13 = 2^15 in magnitude
// (level 7 of S = 6; 2^14 + 2^13 + 2^12 for level 6), so the FP32 level sums
// over a 512-wide K chunk stay within 2^24 and are exact integers; after
// every chunk the drain warps join the levels exactly, as integers (sums over
// several chunks as int64 in spare TMEM columns).  The final sum becomes a
// double once, scaled back by 2^(e_row + e_col); real/imaginary rows of complex
// operands are combined with a lane-pair shuffle and written through a
// strided output decoder.
//
// Pipeline (two variants, TcCfg in gemm_tc.h): warp 0 issues TMA loads
// (SWIZZLE_128B) into a shared-memory ring, one (A_s, B_s) slice pair per
// stage; warp 1 owns TMEM and issues the MMAs from one thread; the other
// warps drain TMEM, EPI / 4 per TMEM lane quarter, each taking a slice of
// the tile's columns.  The wide variant (64 columns, 8 stages, 16 drain
// warps) runs one CTA per SM; the narrow one (32 columns, 5 stages, 8 drain
// warps) two, so that one CTA's drain overlaps the other's MMAs -- for
// contractions with short K, whose time is per-CTA latency.
// Every wait has an iteration limit: on expiry the kernel records an error
// code, stops issuing work, waits (bounded) for its own operations and frees
// TMEM before returning.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstdint>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <tuple>

#include "engine.h"
#include "gemm_tc.h"
#include "slice_math.cuh"
#include "tc_ptx.cuh"

namespace tdcc {

// ---------------------------------------------------------------------------
// packing
// ---------------------------------------------------------------------------
// Stored exponent of a row whose largest |x| has bits mx (biased exponent E).
// The deep form marks rows that digits cannot hold (infinities, NaNs, nothing
// but subnormals): its drain does their outputs by FP64 dot products.
template <int SMAX>
__device__ __forceinline__ int packed_exponent(unsigned long long mx, int E) {
  if (mx == 0) return 0;
  if (SMAX > TC_MAX_SLICES && (E == 0 || E == 2047)) return kExpMarked;
  return (E > 0 ? E - 1022 : -1022) + kExpBias;
}

// |x| 2^-e in FP32, x < 2^e; below the normal range zero
__device__ __forceinline__ float scaled_magnitude(double x, int e) {
  const uint32_t h = (uint32_t)__double2hiint(x) & 0x7FFFFFFFu;
  const int E = (int)(h >> 20) - 1023 + 127 - e;
  return (h >> 20) == 0u || E < 1 ? 0.f : __uint_as_float(((uint32_t)min(E, 126) << 23) | ((h & 0xFFFFFu) << 3) | ((uint32_t)__double2loint(x) >> 29));
}

// Digits of two neighbouring elements of a packed row (same exponent e), one
// BF16 pair per slice: out is the packed buffer as BF16 pairs, plane2 the
// pairs per slice, idx2 the pair's index within a slice, k its place in the row.
template <int SMAX>
__device__ __forceinline__ void store_digit_pair(uint32_t* out, size_t plane2, size_t idx2, int k, double x0, double x1,
                                                  int e, int S) {
  uint32_t h0, l0, h1, l1;
  cut_digits<SMAX>(x0, e, S, h0, l0);
  cut_digits<SMAX>(x1, e, S, h1, l1);
  const uint32_t sgn = (((uint32_t)__double2hiint(x0) >> 16) & 0x8000u) | ((uint32_t)__double2hiint(x1) & 0x80000000u);
  out += idx2;
  if constexpr (SMAX == 8) {
    out[0] = digit_pair<24, true>(h0, h1, sgn);
    out[plane2] = digit_pair<16, false, 8>(h0, h1, sgn);
    out[2 * plane2] = digit_pair<8, false, 8>(h0, h1, sgn);
    out[3 * plane2] = digit_pair<0, false, 8>(h0, h1, sgn);
    out[4 * plane2] = digit_pair<24, false, 8>(l0, l1, sgn);
    out[5 * plane2] = digit_pair<16, false, 8>(l0, l1, sgn);
    out[6 * plane2] = digit_pair<8, false, 8>(l0, l1, sgn);
    out[7 * plane2] = digit_pair<0, false, 8>(l0, l1, sgn);
    // the range guard's plane (gemm_deep.cu): 2^15 |x| 2^-e in 8 bits, which reach down to
    // 2^-31 of the maximum; only zeros as zero; a row fills half of a slice's
    const float f0 = scaled_magnitude(x0, e) * 0x1p15f, f1 = scaled_magnitude(x1, e) * 0x1p15f;
    const float2 f = make_float2(x0 != 0.0 ? fmaxf(f0, 0x1p-16f) : 0.f, x1 != 0.0 ? fmaxf(f1, 0x1p-16f) : 0.f);
    const size_t row = 2 * (idx2 - k / 2);  // the row's first BF16
    reinterpret_cast<uint16_t*>(out - idx2)[16 * plane2 + row + k / 2] = __nv_cvt_float2_to_fp8x2(f, __NV_SATFINITE, __NV_E5M2);
    return;
  }
  out[0] = digit_pair<21, true>(h0, h1, sgn);
  if (S > 1) out[plane2] = digit_pair<14, false>(h0, h1, sgn);
  if (S > 2) out[2 * plane2] = digit_pair<7, false>(h0, h1, sgn);
  if (S > 3) out[3 * plane2] = digit_pair<0, false>(h0, h1, sgn);
  if constexpr (SMAX == 6) {
    if (S > 4) out[4 * plane2] = digit_pair<7, false>(l0, l1, sgn);
    if (S > 5) out[5 * plane2] = digit_pair<0, false>(l0, l1, sgn);
  }
}

// One block per logical row (per batch; the real and imaginary rows of a
// complex row together): pass 1 takes the binary exponent e of the row's
// max |x| (max = f 2^e, f in [0.5, 1); integer ops on the bit patterns, the
// order of |x| for finite doubles), pass 2 cuts |x| 2^-e truncated to 7S
// bits into S balanced digits (|q_1| <= 128, |q_s| <= 64, exact in BF16) and
// gives them the sign of x:
//   x 2^-e ~= sum_s q_s 2^(-7s).
// The real and imaginary rows share e, so that the slice-product epilogue
// combines re*re - im*im and re*im + im*re exactly in integers; with 8 slices
// each has its own (a small imaginary part keeps all of its bits).  K padding
// is written as zero; padding rows (up to the tile multiple of each batch)
// are not written at all: they only feed accumulator rows (A) or columns (B)
// that the product kernel never stores, and their exponent entries only
// scale those values, so whatever the buffer holds there is harmless.
// With tab set, the K offsets (the same for every row) are decoded once per
// block into shared memory as 32-bit integers (K of them) and both passes
// read them there.
//
// CL = 8: a cluster of eight blocks per row, a segment of K each; the segments'
// maxima meet through distributed shared memory.  For few long rows (K = o v^2
// with 36 rows at o=18, v=82: 190 us as a block per row, 41 so).
template <int SMAX, int CL>
__global__ void __launch_bounds__(1024) pack_kernel(const PackArgs p, int tab) {
  extern __shared__ int kofs[];
  const int per = p.cplx ? 2 : 1;
  const int br = blockIdx.x / CL, part_k = CL > 1 ? blockIdx.x % CL : 0;
  const int z = br / p.rows, m = br - z * p.rows;  // one block or cluster per live row
  // this block's K indices: [kb, ke) of the row, [kb, kpe) with its padding
  const int seg = (p.K_pad / 2 + CL - 1) / CL * 2;
  const int kb = min(part_k * seg, p.K_pad), kpe = min(kb + seg, p.K_pad), ke = min(p.K, kpe);
  long long ro = 0;
  decomp_tc(p.gr, m, ro);
  ro += z * p.bs;
  if (tab) {
    for (int k = kb + threadIdx.x; k < ke; k += blockDim.x) {
      long long ko;
      decomp_tc(p.gk, k, ko);
      kofs[k - kb] = (int)ko;
    }
    __syncthreads();
  }
  auto koff = [&](int k) -> long long {
    if (tab) return kofs[k - kb];
    long long ko;
    decomp_tc(p.gk, k, ko);
    return ko;
  };
  const unsigned long long* bits = static_cast<const unsigned long long*>(p.src);
  const double* src = static_cast<const double*>(p.src);
  constexpr unsigned long long kAbs = 0x7FFFFFFFFFFFFFFFull;
  constexpr int PX = SMAX == TC_DEEP_SLICES ? 2 : 1;  // exponents per logical row
  unsigned long long mx[PX] = {};
  // four independent loads in flight per thread (complex elements as one 16-byte load)
  constexpr int U = 4;
  for (int k0 = kb + threadIdx.x; k0 < ke; k0 += U * blockDim.x) {
    unsigned long long v[U][2];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int k = k0 + j * blockDim.x;
      v[j][0] = v[j][1] = 0ull;
      if (k < ke) {
        const long long e = ro + koff(k);
        if (p.cplx) {
          const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(bits + 2 * e);
          v[j][0] = w.x;
          v[j][1] = w.y;
        } else {
          v[j][0] = bits[e];
        }
      }
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
      mx[0] = max(mx[0], v[j][0] & kAbs);
      mx[PX - 1] = max(mx[PX - 1], v[j][1] & kAbs);
    }
  }
  __shared__ unsigned long long wmax[32][PX];
#pragma unroll
  for (int x = 0; x < PX; ++x) {
    for (int d = 16; d > 0; d >>= 1) mx[x] = max(mx[x], __shfl_xor_sync(0xffffffffu, mx[x], d));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5][x] = mx[x];
  }
  __syncthreads();
#pragma unroll
  for (int x = 0; x < PX; ++x) {
    mx[x] = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) mx[x] = max(mx[x], wmax[w][x]);
  }
  if constexpr (CL > 1) {
    namespace cg = cooperative_groups;
    __shared__ unsigned long long cmax[PX];
    cg::cluster_group cl = cg::this_cluster();
    if (threadIdx.x == 0)
      for (int x = 0; x < PX; ++x) cmax[x] = mx[x];
    cl.sync();
#pragma unroll
    for (int x = 0; x < PX; ++x)
      for (int r = 0; r < CL; ++r) mx[x] = max(mx[x], cl.map_shared_rank(cmax, r)[x]);
    cl.sync();  // every block has read the others'
  }
  int eb[2], e[2];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    eb[x] = packed_exponent<SMAX>(mx[x < PX ? x : 0], (int)(mx[x < PX ? x : 0] >> 52));
    e[x] = row_exp(eb[x]);
  }
  const size_t prow = (size_t)z * p.rows_pad + (size_t)m * per;  // first packed row
  if (threadIdx.x == 0 && part_k == 0) {
    p.exps[prow] = eb[0];
    if (p.cplx) p.exps[prow + 1] = eb[1];
  }
  uint32_t* out = static_cast<uint32_t*>(p.out);  // BF16 pairs (K_pad is even)
  const size_t plane2 = (size_t)p.nb * p.rows_pad * (p.K_pad / 2);
  // pass 2 over pairs of neighbouring K indices (one 4-byte store per slice
  // and part), two pairs per thread: four loads in flight
  constexpr int U2 = 2;
  for (int k0 = kb + 2 * threadIdx.x; k0 < kpe; k0 += 2 * U2 * blockDim.x) {
    double x[U2][2][2];  // [pair][element][part]
#pragma unroll
    for (int j = 0; j < U2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = k0 + 2 * j * blockDim.x + h;
        x[j][h][0] = x[j][h][1] = 0.0;
        if (k < ke) {
          const long long el = ro + koff(k);
          if (p.cplx) {
            const double2 w = *reinterpret_cast<const double2*>(src + 2 * el);
            x[j][h][0] = w.x;
            x[j][h][1] = w.y;
          } else {
            x[j][h][0] = src[el];
          }
        }
      }
#pragma unroll
    for (int j = 0; j < U2; ++j) {
      const int k = k0 + 2 * j * blockDim.x;
      if (k >= kpe) break;
      for (int part = 0; part < per; ++part)
        store_digit_pair<SMAX>(out, plane2, ((prow + part) * p.K_pad + k) / 2, k, x[j][0][part], x[j][1][part],
                               part ? e[1] : e[0], p.S);
    }
  }
}

// Rows of up to 64 W KP elements: W warps per logical row, 8 / W rows per
// 256-thread block.  Each lane keeps KP pairs of neighbours in registers
// (pair index 32 w + lane + 32 W j for warp w of the row), so the row is read
// once: the exponent comes from shuffles (and shared memory across the W
// warps), the digits from the registers (same exponent, digits and layout as
// pack_kernel).
template <int KP, int W, int SMAX>
__global__ void __launch_bounds__(256) pack_rows_regs_kernel(const PackArgs p) {
  static_assert(W == 1 || W == 2 || W == 4 || W == 8, "warps per row divide the block");
  constexpr int RPB = 8 / W;
  const int per = p.cplx ? 2 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wr = warp % W;  // warp within the row
  const long long lr = (long long)blockIdx.x * RPB + warp / W;  // logical row over all batches
  const bool live = lr < (long long)p.nb * p.rows;              // uniform over the row's warps
  const int z = live ? (int)(lr / p.rows) : 0, m = live ? (int)(lr - (long long)z * p.rows) : 0;
  long long ro = 0;
  decomp_tc(p.gr, m, ro);
  ro += z * p.bs;
  const double* src = static_cast<const double*>(p.src);
  constexpr unsigned long long kAbs = 0x7FFFFFFFFFFFFFFFull;
  double x[KP][2][2];  // [pair][element][part]
  constexpr int PX = SMAX == TC_DEEP_SLICES ? 2 : 1;  // exponents per logical row
  unsigned long long mx[PX] = {};
#pragma unroll
  for (int j = 0; j < KP; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = 2 * (32 * wr + lane + 32 * W * j) + h;
      x[j][h][0] = x[j][h][1] = 0.0;
      if (live && k < p.K) {
        long long ko;
        decomp_tc(p.gk, k, ko);
        const long long el = ro + ko;
        if (p.cplx) {
          const double2 v = *reinterpret_cast<const double2*>(src + 2 * el);
          x[j][h][0] = v.x;
          x[j][h][1] = v.y;
        } else {
          x[j][h][0] = src[el];
        }
      }
      mx[0] = max(mx[0], (unsigned long long)__double_as_longlong(x[j][h][0]) & kAbs);
      mx[PX - 1] = max(mx[PX - 1], (unsigned long long)__double_as_longlong(x[j][h][1]) & kAbs);
    }
#pragma unroll
  for (int q = 0; q < PX; ++q)
    for (int d = 16; d > 0; d >>= 1) mx[q] = max(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], d));
  if (W > 1) {
    __shared__ unsigned long long wmax[8][PX];
    if (lane == 0)
      for (int q = 0; q < PX; ++q) wmax[warp][q] = mx[q];
    __syncthreads();  // every thread of the block arrives (no return above)
    const int w0 = warp - wr;
#pragma unroll
    for (int w = 0; w < W; ++w)
#pragma unroll
      for (int q = 0; q < PX; ++q) mx[q] = max(mx[q], wmax[w0 + w][q]);
  }
  if (!live) return;
  int eb[2], e[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    eb[q] = packed_exponent<SMAX>(mx[q < PX ? q : 0], (int)(mx[q < PX ? q : 0] >> 52));
    e[q] = row_exp(eb[q]);
  }
  const size_t prow = (size_t)z * p.rows_pad + (size_t)m * per;
  if (wr == 0 && lane == 0) {
    p.exps[prow] = eb[0];
    if (p.cplx) p.exps[prow + 1] = eb[1];
  }
  uint32_t* out = static_cast<uint32_t*>(p.out);  // BF16 pairs (K_pad is even)
  const size_t plane2 = (size_t)p.nb * p.rows_pad * (p.K_pad / 2);
#pragma unroll
  for (int j = 0; j < KP; ++j) {
    const int k = 2 * (32 * wr + lane + 32 * W * j);
    if (k >= p.K_pad) break;
    for (int part = 0; part < per; ++part)
      store_digit_pair<SMAX>(out, plane2, ((prow + part) * p.K_pad + k) / 2, k, x[j][0][part], x[j][1][part],
                               part ? e[1] : e[0], p.S);
  }
}

// ---------------------------------------------------------------------------
// slice-product kernel
// ---------------------------------------------------------------------------
template <class C>
struct TcShared {
  uint64_t full[C::STAGES];
  uint64_t empty[C::STAGES];
  uint64_t accfull, accempty, done;
  uint32_t tmem;
  volatile int abort;  // set by any role on an expired wait; polled by all
  long long col_off[C::BN];  // output offset of each logical column of the tile (-1: outside)
  int col_exp[C::BN];        // exponent of each packed column of B
};

template <bool AC, bool BC, class C>
__global__ void __launch_bounds__(C::THREADS, C::MINB)
    ozaki_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const TcArgs g) {
  extern __shared__ uint8_t smraw[];
  uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  uint8_t* stA = sm;                                   // STAGES x 16 KB
  uint8_t* stB = sm + C::STAGES * TC_A_BYTES;          // STAGES x BN x 128 B
  TcShared<C>* sh = (TcShared<C>*)(stB + C::STAGES * C::B_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = g.S;
  const int ncols = g.tmem_cols;

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
                 "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = sh->tmem;

  const int mt = g.m_fast ? blockIdx.x : blockIdx.y, nt = g.m_fast ? blockIdx.y : blockIdx.x;
  const int zb = blockIdx.z / g.nsplit;                 // batch
  const int kb0 = (blockIdx.z - zb * g.nsplit) * g.kb_per_split;
  const int rowA0 = (g.bat_a ? zb * g.rowsA_pad : 0);  // packed-row origin of this batch
  const int rowB0 = (g.bat_b ? zb * g.rowsB_pad : 0);
  const int kb1 = min(g.kblocks, kb0 + g.kb_per_split);
  const int nkb = kb1 - kb0;
  const int nchunks = (nkb + TC_CHUNK_KB - 1) / TC_CHUNK_KB;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int it = 0;
      for (int kb = kb0; kb < kb1 && !sh->abort; ++kb)
        for (int s = 0; s < S && !sh->abort; ++s, ++it) {
          const int st = it % C::STAGES;
          const uint32_t ph = (uint32_t)((it / C::STAGES) & 1);
          if (!mbar_wait(smem_u32(&sh->empty[st]), ph ^ 1u, kWaitLimit)) {
            fail(sh, g.err, 1);
            break;
          }
          const uint32_t fb = smem_u32(&sh->full[st]);
          mbar_expect_tx(fb, TC_A_BYTES + C::B_BYTES);
          tma3d(smem_u32(stA + st * TC_A_BYTES), &tmA, kb * TC_BK, rowA0 + mt * TC_BM, s, fb);
          tma3d(smem_u32(stB + st * C::B_BYTES), &tmB, kb * TC_BK, rowB0 + nt * C::BN, s, fb);
        }
      // drain: every issued load must land before the CTA exits
      const int issued = it;
      for (int j = (issued > C::STAGES ? issued - C::STAGES : 0); j < issued; ++j)
        mbar_wait(smem_u32(&sh->full[j % C::STAGES]), (uint32_t)((j / C::STAGES) & 1), kWaitLimit);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the whole warp, one lane executing) ----------------
    constexpr uint32_t id = idesc_bf16(TC_BM, C::BN);
    const uint32_t on = lane == 0 ? 1u : 0u;
    PairRing<C::STAGES, TC_A_BYTES, C::B_BYTES> ring(stA, stB, &sh->full[0], &sh->empty[0]);
    bool ok = true;
    for (int c = 0; c < nchunks && ok; ++c) {
      if (c > 0 && !mbar_wait_warp(smem_u32(&sh->accempty), (uint32_t)((c - 1) & 1), kWaitLimit)) {
        fail(sh, g.err, 2);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const int kbs = kb0 + c * TC_CHUNK_KB, kbe = min(kb1, kbs + TC_CHUNK_KB);
#pragma unroll 1
      for (int kb = kbs; kb < kbe && ok; ++kb)
        switch (S) {
          case 2: ok = ring.template issue<2, C::BN>(tmem, id, kb == kbs, on); break;
          case 3: ok = ring.template issue<3, C::BN>(tmem, id, kb == kbs, on); break;
          case 4: ok = ring.template issue<4, C::BN>(tmem, id, kb == kbs, on); break;
          case 5: ok = ring.template issue<5, C::BN>(tmem, id, kb == kbs, on); break;
          default:
            if constexpr (C::STAGES >= 6) ok = ring.template issue<6, C::BN>(tmem, id, kb == kbs, on);
        }
      if (!ok) fail(sh, g.err, 3);
      if (ok) umma_commit_warp(smem_u32(&sh->accfull), on);
      ok = __all_sync(0xffffffffu, ok && sh->abort == 0) != 0;
    }
    // all issued MMAs complete before TMEM is released
    umma_commit_warp(smem_u32(&sh->done), on);
    mbar_wait(smem_u32(&sh->done), 0, kWaitLimit);
  } else {
    // ---------------- epilogue (warps 2 .. 2 + C::EPI - 1) ----------------
    // C::EPI / 4 warps per TMEM lane quarter, each owning a slice of the
    // tile's columns: the drain is latency-bound per warp, so the work is
    // spread over warps.
    constexpr int kWq = C::EPI / 4;   // warps per lane quarter
    constexpr int kCw = C::BN / kWq;        // packed columns per warp (multiple of 16)
    const int q = warp & 3;             // TMEM lane quarter this warp may access
    const int hcol = (warp - 2) >> 2;   // column slice of this warp
    const int row = q * 32 + lane;      // tile row == TMEM lane
    // Exact sums in integer units of 2^-u, u = 7 (min(S,5) + 1).  The level
    // sums are integers (products of integer slices, FP32-exact per chunk),
    // so sum_L v_L 2^(u - 7L) is exact for S <= 5 (the seventh-slice level of
    // S = 6 is truncated by 7 bits, below its own resolution) and stays
    // below 2^52 per chunk: int64 holds up to 2^11 chunks.  No FP64
    // arithmetic until the final conversion -- the FP64 pipe is narrow.
    const int u = 7 * ((S < 5 ? S : 5) + 1);
    {
      // per-tile column data, shared by all rows: output offsets and B exponents
      const int t = threadIdx.x - 64;  // 0 .. 32 * C::EPI - 1
      constexpr int ncl = BC ? C::BN / 2 : C::BN;
      if (t < ncl) {
        const int n = nt * ncl + t;
        long long o = -1;
        if (n < g.N) decomp_tc(g.gnC, n, o);
        sh->col_off[t] = o;
      }
      if (t < C::BN) sh->col_exp[t] = row_exp(g.expB[rowB0 + nt * C::BN + t]);
      asm volatile("bar.sync 1, %0;" ::"n"(32 * C::EPI) : "memory");  // the epilogue warps
    }
    // Row data and the staging tile of this warp (final chunk): the operand
    // ring is idle once the last accumulators are complete.
    const int prow = mt * TC_BM + row;          // packed row of A (within the batch)
    const int m = AC ? (prow >> 1) : prow;
    const bool odd = AC && (lane & 1);
    constexpr int ncol_log = BC ? C::BN / 2 : C::BN;  // logical output columns in this tile
    constexpr int rows_out = AC ? 16 : 32;             // logical output rows of this warp
    constexpr int RS = ncol_log + 1;                    // staging row stride (double2), padded
    double2* stage = reinterpret_cast<double2*>(sm) + (size_t)q * (32 * RS);
    const int lr = AC ? (lane >> 1) : lane;            // this lane's staging row
    const uint32_t tl = (uint32_t)(q * 32) << 16;      // TMEM lane base of this warp
    const uint32_t t64 = (uint32_t)(S * C::BN);        // int64 partial sums: 2 words per column
    bool ok = true;
    for (int c = 0; c < nchunks; ++c) {
      // warp-uniform decisions: tcgen05.ld/st and the shuffles below are collective
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
      const bool last = c == nchunks - 1;
      int ebase = 0;
      if (last) {
        const int ea = prow < g.rowsA_pad ? row_exp(g.expA[rowA0 + prow]) : 0;
        ebase = ea - u + (g.alpha_pow2 ? g.alpha_e : 0);
      }
      // 16 columns at a time (a runtime loop keeps the code small)
#pragma unroll 1
      for (int j0 = hcol * kCw; j0 < (hcol + 1) * kCw; j0 += 16) {
        // all loads of the group in flight before one wait (TMEM latency)
        constexpr int kMaxLv = 6;  // levels 2..7 (S <= 6)
        long long a16[16];
        if (c > 0) {
          uint32_t lo[16], hi[16];
          tmem_ld16_nowait(tmem + tl + t64 + 2 * j0, lo);
          tmem_ld16_nowait(tmem + tl + t64 + 2 * j0 + 16, hi);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j) a16[j] = (long long)(((unsigned long long)hi[j] << 32) | lo[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) a16[j] = 0;
        }
        // levels in batches of three loads before one wait
#pragma unroll
        for (int L0 = 2; L0 <= kMaxLv + 1; L0 += 3) {
          if (L0 > S + 1) break;
          uint32_t lv[3][16];
#pragma unroll
          for (int i = 0; i < 3; ++i)
            if (L0 + i <= S + 1) tmem_ld16_nowait(tmem + tl + (uint32_t)((L0 + i - 2) * C::BN + j0), lv[i]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const int L = L0 + i;
            if (L > S + 1) break;
            const int sh = u - 7 * L;
            // |v| <= 2^24: a 32-bit conversion is exact and stays off the FP64 pipe
            if (sh >= 0) {
#pragma unroll
              for (int j = 0; j < 16; ++j) a16[j] += (long long)__float2int_rn(__uint_as_float(lv[i][j])) << sh;
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) a16[j] += (long long)__float2int_rn(__uint_as_float(lv[i][j])) >> (-sh);
            }
          }
        }
        if (!last) {
          uint32_t lo[16], hi[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            lo[j] = (uint32_t)(unsigned long long)a16[j];
            hi[j] = (uint32_t)((unsigned long long)a16[j] >> 32);
          }
          tmem_st16u(tmem + tl + t64 + 2 * j0, lo);
          tmem_st16u(tmem + tl + t64 + 2 * j0 + 16, hi);
          continue;
        }
        // final chunk: combine, scale back, stage (lanes own rows here)
        const bool neg = g.alpha_pow2 && g.alpha_neg;
        constexpr int NJ = BC ? 8 : 16;  // logical columns in this group
        auto put = [&](int k, long long re, long long im) {
          const int jj = (BC ? j0 / 2 : j0) + k;
          const int E = ebase + sh->col_exp[BC ? 2 * jj : jj];
          double vr, vi;
          if (g.alpha_pow2) {
            vr = scaled_i64_to_double(neg ? -re : re, E);
            vi = scaled_i64_to_double(neg ? -im : im, E);
          } else {
            const double dr = scaled_i64_to_double(re, E), di = scaled_i64_to_double(im, E);
            vr = g.ar * dr - g.ai * di;
            vi = g.ar * di + g.ai * dr;
          }
          stage[lr * RS + jj] = make_double2(vr, vi);
        };
        // integer combine: the pair exponents are shared, so these are exact
        if constexpr (AC) {
          // a row's real and imaginary parts lie in neighbouring lanes: the even
          // one finishes column k, the odd one k + 1, each with what the other
          // holds of it
#pragma unroll
          for (int k = 0; k < NJ; k += 2) {
            if constexpr (BC) {
              const long long p0 = __shfl_xor_sync(0xffffffffu, odd ? a16[2 * k] : a16[2 * k + 2], 1);
              const long long p1 = __shfl_xor_sync(0xffffffffu, odd ? a16[2 * k + 1] : a16[2 * k + 3], 1);
              const long long x0 = odd ? a16[2 * k + 2] : a16[2 * k], x1 = odd ? a16[2 * k + 3] : a16[2 * k + 1];
              // even: (re re, re im) own, (im re, im im) the partner's
              put(k + (odd ? 1 : 0), odd ? p0 - x1 : x0 - p1, odd ? p1 + x0 : x1 + p0);
            } else {
              const long long p = __shfl_xor_sync(0xffffffffu, odd ? a16[k] : a16[k + 1], 1);
              const long long x = odd ? a16[k + 1] : a16[k];
              put(k + (odd ? 1 : 0), odd ? p : x, odd ? x : p);
            }
          }
        } else {
#pragma unroll
          for (int k = 0; k < NJ; ++k) put(k, BC ? a16[2 * k] : a16[k], BC ? a16[2 * k + 1] : 0);
        }
      }
      if (!last) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;");
      mbar_arrive(smem_u32(&sh->accempty));
    }
    if (ok && !__any_sync(0xffffffffu, sh->abort != 0)) {
      // write the staged tile: rows of contiguous columns per pass
      __syncwarp();
      long long coffm = 0;
      if (m < g.M) decomp_tc(g.gmC, m, coffm);
      double2* Cc = static_cast<double2*>(g.C) + (g.cc ? zb * g.bsC : 0);
      double* Cr = static_cast<double*>(g.C) + (g.cc ? 0 : zb * g.bsC);
      const int m0w = AC ? ((mt * TC_BM + q * 32) >> 1) : (mt * TC_BM + q * 32);
      constexpr int NCW = ncol_log / kWq;  // logical columns of this warp (<= 32)
      // every lane owns a (row, column) pair: NCW columns by 32 / NCW rows per
      // pass.  Accumulated outputs are added in L2 (reductions without a
      // return value), so the pass issues no load: one writer per element
      // and launch (split K aside), so the single addition c + v is the same
      // as a read-modify-write.
      static_assert(32 % NCW == 0, "columns per warp divide the warp");
      constexpr int RPP = 32 / NCW;
      constexpr int NPASS = (rows_out + RPP - 1) / RPP;
      const int lc = lane % NCW, lrw = lane / NCW;
      const int cc = hcol * NCW + lc;  // this lane's column while storing
      const long long cn = sh->col_off[cc];
      const int nrows = min(rows_out, g.M - m0w);
      const bool red = g.acc || g.atomic;
#pragma unroll 4
      for (int p = 0; p < NPASS; ++p) {
        const int r = p * RPP + lrw;
        // row offsets live in the lanes of the rows' TMEM rows
        const long long cm = __shfl_sync(0xffffffffu, coffm, (AC ? 2 * r : r) & 31);
        if (r >= nrows || cn < 0) continue;
        const long long off = cm + cn;
        const double2 v = stage[r * RS + cc];
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
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}

// ---------------------------------------------------------------------------
// Persistent 64-column form for S <= 4 slices (TcPersist).  One CTA per SM
// walks the output tiles t = blockIdx.x, blockIdx.x + gridDim.x, ... (each
// at most one exact K chunk).  Two TMEM buffers of
// S level accumulators: the MMA issuer fills buffer j & 1 for its j-th tile
// once the drain warps have released it (accempty), the drain warps empty it
// once its MMAs are complete (accfull) and release it as soon as the levels
// are in registers, before they convert and store -- so a tile's drain runs
// under the next tile's loads and MMAs.  A and B slices have rings of their
// own (A1 .. AS and B1 .. BS per K block, products row by row, each slice
// released after its last product).  Bound: the drain; as one group of 16 warps,
// all in the same phase of it, it took 11 k to 20 k clocks a tile against 5 k a
// K block for loads and products.  Two groups of eight, a buffer each: the o=10,
// v=38 contractions of 24 trajectories with mnij 160 -> 119 us, with the 38 x 38
// intermediates 158 -> 98.  Accumulated outputs are reductions in L2: as loads
// and stores the former took 180 us.
// ---------------------------------------------------------------------------
struct PersistShared {
  uint64_t fullA[TcPersist::RA], emptyA[TcPersist::RA];
  uint64_t fullB[TcPersist::RB], emptyB[TcPersist::RB];
  uint64_t accfull[2], accempty[2], done;
  uint32_t tmem;
  volatile int abort;
  int stop[2];                              // each drain group's common decision for a tile
  long long col_off[2][TcPersist::BN];      // output offset of each logical column (-1: outside)
  int col_exp[2][TcPersist::BN];
};

static_assert(sizeof(PersistShared) <= 2048, "fits behind the staging areas");

struct TileCoord {
  int mt, nt, zb, kb0, kb1, rowA0, rowB0;
};

__device__ __forceinline__ TileCoord persist_tile(const TcArgs& g, int t, int mtiles, int ntiles) {
  TileCoord c;
  const int per = mtiles * ntiles;
  const int zs = t / per, rem = t - zs * per;
  if (g.m_fast) {
    c.mt = rem % mtiles;
    c.nt = rem / mtiles;
  } else {
    c.nt = rem % ntiles;
    c.mt = rem / ntiles;
  }
  c.zb = zs / g.nsplit;
  c.kb0 = (zs - c.zb * g.nsplit) * g.kb_per_split;
  c.kb1 = min(g.kblocks, c.kb0 + g.kb_per_split);
  c.rowA0 = g.bat_a ? c.zb * g.rowsA_pad : 0;
  c.rowB0 = g.bat_b ? c.zb * g.rowsB_pad : 0;
  return c;
}

// The MMA warp of the persistent form.  The ring slots and descriptor words of
// a K block's slices are computed once per slice; with them worked out for
// every product (a ring index, a modulo, a descriptor) the issue of 10
// products took longer than the products.
template <int S>
__device__ __forceinline__ void persist_issue(const TcArgs& g, PersistShared* sh, const uint8_t* ringA,
                                              const uint8_t* ringB, uint32_t tmem, int ntiles_total, int mtiles,
                                              int ntiles, int lane) {
  using C = TcPersist;
  constexpr uint32_t id = idesc_bf16(TC_BM, C::BN);
  const uint64_t hi64 = sdesc(0);
  const uint32_t a0 = (smem_u32(ringA) & 0x3FFFF) >> 4, b0 = (smem_u32(ringB) & 0x3FFFF) >> 4;
  const uint32_t fullA = smem_u32(&sh->fullA[0]), emptyA = smem_u32(&sh->emptyA[0]);
  const uint32_t fullB = smem_u32(&sh->fullB[0]), emptyB = smem_u32(&sh->emptyB[0]);
  const uint32_t on = lane == 0 ? 1u : 0u;
  uint32_t sa0 = 0, pa = 0, sb0 = 0, pb = 0;  // ring slot and phase of the block's first slices
  int jt = 0;
  bool ok = true;
  for (int t = blockIdx.x; t < ntiles_total && ok; t += gridDim.x, ++jt) {
    const TileCoord c = persist_tile(g, t, mtiles, ntiles);
    const int b = jt & 1, use = jt >> 1;
    if (use > 0 && !mbar_wait_warp(smem_u32(&sh->accempty[b]), (uint32_t)((use - 1) & 1), kWaitLimit)) {
      fail(sh, g.err, 2);
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t dbuf = tmem + (uint32_t)(b * S * C::BN);
#pragma unroll 1
    for (int kb = c.kb0; kb < c.kb1 && ok; ++kb) {
      const bool first = kb == c.kb0;
      uint32_t la[S], lb[S], qa[S], qb[S];
#pragma unroll
      for (int j = 0; j < S; ++j) {
        qa[j] = sa0 + j < C::RA ? sa0 + j : sa0 + j - C::RA;
        qb[j] = sb0 + j < C::RB ? sb0 + j : sb0 + j - C::RB;
        la[j] = a0 + qa[j] * (C::A_SLOT >> 4);
        lb[j] = b0 + qb[j] * (C::B_SLOT >> 4);
      }
#pragma unroll
      for (int s = 1; s <= S; ++s) {
        if (ok) ok = mbar_wait_warp(fullA + 8 * qa[s - 1], sa0 + s - 1 < C::RA ? pa : pa ^ 1u, kWaitLimit);
#pragma unroll
        for (int tt = 1; tt <= S; ++tt) {
          if (tt > S + 1 - s) continue;
          if (s == 1 && ok) ok = mbar_wait_warp(fullB + 8 * qb[tt - 1], sb0 + tt - 1 < C::RB ? pb : pb ^ 1u, kWaitLimit);
          asm volatile("tcgen05.fence::after_thread_sync;");
          if (ok) {
#pragma unroll
            for (int k = 0; k < TC_BK / 16; ++k)
              umma_warp(dbuf + (uint32_t)((s + tt - 2) * C::BN), hi64 | (uint64_t)(la[s - 1] + 2 * k),
                        hi64 | (uint64_t)(lb[tt - 1] + 2 * k), id, (first && s == 1 && k == 0) ? 0u : 1u, on);
          }
        }
        if (ok) {  // A_s and B_(S+1-s) have had their last use in this K block
          umma_commit_warp(emptyA + 8 * qa[s - 1], on);
          umma_commit_warp(emptyB + 8 * qb[S - s], on);
        }
      }
      sa0 += S;
      if (sa0 >= C::RA) {
        sa0 -= C::RA;
        pa ^= 1u;
      }
      sb0 += S;
      if (sb0 >= C::RB) {
        sb0 -= C::RB;
        pb ^= 1u;
      }
    }
    if (!ok) {
      fail(sh, g.err, 3);
      break;
    }
    umma_commit_warp(smem_u32(&sh->accfull[b]), on);
    ok = __all_sync(0xffffffffu, sh->abort == 0) != 0;
  }
  // all issued MMAs complete before TMEM is released
  umma_commit_warp(smem_u32(&sh->done), on);
  mbar_wait(smem_u32(&sh->done), 0, kWaitLimit);
}

template <bool AC, bool BC>
__global__ void __launch_bounds__(TcPersist::THREADS, 1)
    ozaki_persist_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                         const TcArgs g, int ntiles_total) {
  using C = TcPersist;
  extern __shared__ uint8_t smraw[];
  uint8_t* sm = (uint8_t*)(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
  uint8_t* ringA = sm;                                   // RA x 16 KB
  uint8_t* ringB = ringA + C::RA * C::A_SLOT;            // RB x 8 KB
  uint8_t* stg = ringB + C::RB * C::B_SLOT;              // EPI x STAGE_WARP
  PersistShared* sh = (PersistShared*)(stg + C::EPI * C::STAGE_WARP);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = g.S;
  const int ncols = g.tmem_cols;
  const int mtiles = g.rowsA_pad / TC_BM, ntiles = g.rowsB_pad / C::BN;
  const uint32_t buf_cols = (uint32_t)(S * C::BN);  // one buffer of S levels

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::RA; ++i) {
      mbar_init(smem_u32(&sh->fullA[i]), 1);
      mbar_init(smem_u32(&sh->emptyA[i]), 1);
    }
    for (int i = 0; i < C::RB; ++i) {
      mbar_init(smem_u32(&sh->fullB[i]), 1);
      mbar_init(smem_u32(&sh->emptyB[i]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sh->accfull[b]), 1);
      mbar_init(smem_u32(&sh->accempty[b]), 32 * C::EPI / 2);
    }
    mbar_init(smem_u32(&sh->done), 1);
    sh->abort = 0;
    sh->stop[0] = sh->stop[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
    asm volatile("fence.proxy.async.shared::cta;");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem)),
                 "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = sh->tmem;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int ja = 0, jb = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < ntiles_total && ok && !sh->abort; t += gridDim.x) {
        const TileCoord c = persist_tile(g, t, mtiles, ntiles);
        for (int kb = c.kb0; kb < c.kb1 && ok && !sh->abort; ++kb)
          for (int i = 0; i < 2 * S; ++i) {
            const bool isA = i == 0 || i > S;  // A1, B1 .. BS, A2 .. AS
            const int j = isA ? ja : jb, R = isA ? C::RA : C::RB;
            const int st = j % R;
            const uint32_t ph = (uint32_t)((j / R) & 1);
            const uint32_t eb = smem_u32(isA ? &sh->emptyA[st] : &sh->emptyB[st]);
            if (!mbar_wait(eb, ph ^ 1u, kWaitLimit)) {
              fail(sh, g.err, 1);
              ok = false;
              break;
            }
            const uint32_t fb = smem_u32(isA ? &sh->fullA[st] : &sh->fullB[st]);
            if (isA) {
              mbar_expect_tx(fb, C::A_SLOT);
              tma3d(smem_u32(ringA + st * C::A_SLOT), &tmA, kb * TC_BK, c.rowA0 + c.mt * TC_BM, i == 0 ? 0 : i - S,
                    fb);
              ++ja;
            } else {
              mbar_expect_tx(fb, C::B_SLOT);
              tma3d(smem_u32(ringB + st * C::B_SLOT), &tmB, kb * TC_BK, c.rowB0 + c.nt * C::BN, i - 1, fb);
              ++jb;
            }
          }
      }
      // every issued load lands before the CTA exits
      for (int q = (ja > C::RA ? ja - C::RA : 0); q < ja; ++q)
        mbar_wait(smem_u32(&sh->fullA[q % C::RA]), (uint32_t)((q / C::RA) & 1), kWaitLimit);
      for (int q = (jb > C::RB ? jb - C::RB : 0); q < jb; ++q)
        mbar_wait(smem_u32(&sh->fullB[q % C::RB]), (uint32_t)((q / C::RB) & 1), kWaitLimit);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the whole warp, one lane executing) ----------------
    switch (S) {
      case 2: persist_issue<2>(g, sh, ringA, ringB, tmem, ntiles_total, mtiles, ntiles, lane); break;
      case 3: persist_issue<3>(g, sh, ringA, ringB, tmem, ntiles_total, mtiles, ntiles, lane); break;
      default: persist_issue<4>(g, sh, ringA, ringB, tmem, ntiles_total, mtiles, ntiles, lane); break;
    }
  } else {
    // ---------------- drain warps (2 .. 17): two groups of eight ----------------
    // Group b empties buffer b, so one group's chain of loads, conversions and
    // stores runs under the other's; a warp owns 32 columns, 16 at a time.
    const int grp = (warp - 2) >> 3, q = warp & 3;
    const int j00 = (((warp - 2) >> 2) & 1) * 32;  // this warp's packed columns
    const int row = q * 32 + lane;
    const bool odd = AC && (lane & 1);
    constexpr int NJ = BC ? 8 : 16;        // logical columns of 16 packed ones
    constexpr int rows_out = AC ? 16 : 32;  // logical rows of this warp
    constexpr int RS = NJ + 1;              // staging row stride, padded
    constexpr bool REAL_ONLY = !AC && !BC;  // real operands: stage the real part only
    double2* stage2 = reinterpret_cast<double2*>(stg + (size_t)(warp - 2) * C::STAGE_WARP);
    double* stage1 = reinterpret_cast<double*>(stg + (size_t)(warp - 2) * C::STAGE_WARP);
    const int lr = AC ? (lane >> 1) : lane;
    const uint32_t tl = (uint32_t)(q * 32) << 16;
    const int u = 7 * (S + 1);
    const bool neg = g.alpha_pow2 && g.alpha_neg;
    const bool red = g.acc || g.atomic;
    constexpr int RPP = 32 / NJ;
    constexpr int NPASS = rows_out / RPP;
    const int lc = lane % NJ, lrw = lane / NJ;
    const int td = threadIdx.x - 64 - 32 * (C::EPI / 2) * grp;
    auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(32 * (C::EPI / 2)) : "memory"); };
    int use = 0;
    for (int t = blockIdx.x + grp * gridDim.x; t < ntiles_total; t += 2 * gridDim.x, ++use) {
      const TileCoord c = persist_tile(g, t, mtiles, ntiles);
      // one decision for the group, and the tile's column data
      group_sync();
      if (td == 0) sh->stop[grp] = sh->abort;
      {
        constexpr int ncl = BC ? C::BN / 2 : C::BN;
        if (td < ncl) {
          const int n = c.nt * ncl + td;
          long long o = -1;
          if (n < g.N) decomp_tc(g.gnC, n, o);
          sh->col_off[grp][td] = o;
        }
        if (td < C::BN) sh->col_exp[grp][td] = row_exp(g.expB[c.rowB0 + c.nt * C::BN + td]);
      }
      const int prow = c.mt * TC_BM + row;
      const int m = AC ? (prow >> 1) : prow;
      const int ea = prow < g.rowsA_pad ? row_exp(g.expA[c.rowA0 + prow]) : 0;
      const int ebase = ea - u + (g.alpha_pow2 ? g.alpha_e : 0);
      long long coffm = 0;
      if (m < g.M) decomp_tc(g.gmC, m, coffm);
      double2* Cc = static_cast<double2*>(g.C) + (g.cc ? c.zb * g.bsC : 0);
      double* Cr = static_cast<double*>(g.C) + (g.cc ? 0 : c.zb * g.bsC);
      const int m0w = AC ? ((c.mt * TC_BM + q * 32) >> 1) : (c.mt * TC_BM + q * 32);
      const int nrows = min(rows_out, g.M - m0w);
      group_sync();
      if (sh->stop[grp]) break;  // the same value for every warp of the group
      const bool got = mbar_wait(smem_u32(&sh->accfull[grp]), (uint32_t)(use & 1), kWaitLimit);
      if (!__all_sync(0xffffffffu, got)) {
        fail(sh, g.err, 4);
        continue;  // the next tile's decision stops the group
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      if (nrows <= 0) {  // rows of padding only
        mbar_arrive(smem_u32(&sh->accempty[grp]));
        continue;
      }
#pragma unroll 1
      for (int j0 = j00; j0 < j00 + 32; j0 += 16) {
        // Level sums of at most two K blocks stay below 2^22 (24576 x 128), so
        // adding 1.5 x 2^23 leaves the integer in the low bits of the float,
        // and two levels (2^7 apart) meet in 32 bits.
        static_assert(24576LL * C::MAX_KB * TC_BK <= (1 << 22), "level sums of a persistent tile");
        int p01[16], p23[16];
#pragma unroll
        for (int L0 = 2; L0 <= 5; L0 += 2) {
          int* p = L0 == 2 ? p01 : p23;
#pragma unroll
          for (int j = 0; j < 16; ++j) p[j] = 0;
          if (L0 > S + 1) continue;
          uint32_t lv[2][16];
          const uint32_t ta = tmem + tl + (uint32_t)grp * buf_cols + (uint32_t)((L0 - 2) * C::BN + j0);
          tmem_ld16_nowait(ta, lv[0]);
          if (L0 < S + 1) tmem_ld16_nowait(ta + C::BN, lv[1]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            p[j] = (int)(__float_as_uint(__fadd_rn(__uint_as_float(lv[0][j]), 12582912.f)) - 0x4B400000u);
            if (L0 < S + 1)
              p[j] = (p[j] << 7) + (int)(__float_as_uint(__fadd_rn(__uint_as_float(lv[1][j]), 12582912.f)) - 0x4B400000u);
          }
        }
        if (j0 != j00) {  // all levels read: the MMAs of a later tile may refill this buffer
          asm volatile("tcgen05.fence::before_thread_sync;");
          mbar_arrive(smem_u32(&sh->accempty[grp]));
        }
        // units of 2^-u: level L weighs 2^(u - 7 L), u = 7 (S + 1)
        long long a16[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) a16[j] = S <= 2 ? p01[j] : ((long long)p01[j] << (7 * (S - 2))) + p23[j];
        __syncwarp();  // the previous stores have read the staging area
        auto put = [&](int k, long long re, long long im) {
          const int jj = (BC ? j0 / 2 : j0) + k;
          const int E = ebase + sh->col_exp[grp][BC ? 2 * jj : jj];
          double vr, vi;
          if (g.alpha_pow2) {
            vr = scaled_i64_to_double(neg ? -re : re, E);
            vi = scaled_i64_to_double(neg ? -im : im, E);
          } else {
            const double dr = scaled_i64_to_double(re, E), di = scaled_i64_to_double(im, E);
            vr = g.ar * dr - g.ai * di;
            vi = g.ar * di + g.ai * dr;
          }
          if constexpr (REAL_ONLY)
            stage1[lr * RS + k] = vr;
          else
            stage2[lr * RS + k] = make_double2(vr, vi);
        };
        if constexpr (AC) {
          // a row's real and imaginary parts lie in neighbouring lanes: the even
          // one finishes column k, the odd one k + 1, each with what the other
          // holds of it
#pragma unroll
          for (int k = 0; k < NJ; k += 2) {
            if constexpr (BC) {
              const long long p0 = __shfl_xor_sync(0xffffffffu, odd ? a16[2 * k] : a16[2 * k + 2], 1);
              const long long p1 = __shfl_xor_sync(0xffffffffu, odd ? a16[2 * k + 1] : a16[2 * k + 3], 1);
              const long long x0 = odd ? a16[2 * k + 2] : a16[2 * k], x1 = odd ? a16[2 * k + 3] : a16[2 * k + 1];
              // even: (re re, re im) own, (im re, im im) the partner's
              put(k + (odd ? 1 : 0), odd ? p0 - x1 : x0 - p1, odd ? p1 + x0 : x1 + p0);
            } else {
              const long long p = __shfl_xor_sync(0xffffffffu, odd ? a16[k] : a16[k + 1], 1);
              const long long x = odd ? a16[k + 1] : a16[k];
              put(k + (odd ? 1 : 0), odd ? p : x, odd ? x : p);
            }
          }
        } else {
#pragma unroll
          for (int k = 0; k < NJ; ++k) put(k, BC ? a16[2 * k] : a16[k], BC ? a16[2 * k + 1] : 0);
        }
        __syncwarp();
        const long long cn = sh->col_off[grp][(BC ? j0 / 2 : j0) + lc];
#pragma unroll 4
        for (int p = 0; p < NPASS; ++p) {
          const int r = p * RPP + lrw;
          const long long cm = __shfl_sync(0xffffffffu, coffm, (AC ? 2 * r : r) & 31);
          if (r >= nrows || cn < 0) continue;
          const long long off = cm + cn;
          const double2 v = REAL_ONLY ? make_double2(stage1[r * RS + lc], 0.0) : stage2[r * RS + lc];
          if (g.cc) {
            if (red) {
              atomicAdd(&Cc[off].x, v.x);
              if (!REAL_ONLY) atomicAdd(&Cc[off].y, v.y);
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
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}

// ---------------------------------------------------------------------------
// Short contractions (K <= 64) of the mixed mode on the FP32 pipe: the same
// exact slice products as the tensor-core path, without packing.  One output
// tile per block: the block takes the binary exponents of its rows of A and
// columns of B over all of K (real and imaginary parts share one), cuts K
// chunks of both into S signed 7-bit digits in shared memory, and every
// thread accumulates the levels L = s + t of its 4 outputs with FP32 FMAs.  A complex level sum grows by at most
// 2 (2^14 + 2^13 + 2^13) = 2^16 per K index, so up to K = 64 every partial
// sum is an integer below 2^22, exact in FP32.  The epilogue recombines the
// levels in int64 and converts with the exponents, as the tensor-core drain
// does.  GB300's FP64 pipe runs about 2 FMA per clock per SM, its FP32 pipe
// 128: 60 FP32 FMAs per complex multiply-add still finish 4x sooner than 4
// FP64 ones, and the FP64 pipe stays free for the elementwise ops.
// ---------------------------------------------------------------------------
constexpr int kSimtMaxK = 64;

// d += a * b on two FP32 pairs: one instruction, each half rounded as fmaf does
__device__ __forceinline__ void fma_f32x2(float2& d, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}

// Tile BM x BN (32 x 32, 16 x 64 or 64 x 16), 256 threads on a 16 x 16 grid,
// 4 outputs each: rows ty + 16 i, columns tx + 16 j.  Digits in shared memory
// per K index and row: S x (2 if complex) floats, contiguous, read as float2.
// Three blocks per SM: a block's exponents, digits and stores are chains of
// loads that the others' multiply-adds cover (the K = 10 contractions at o=10,
// v=38 with 24 trajectories: 198 us with two, 181 with three, 166 with a chunk's
// loads all in flight and kept for its digits; K = 18 at o=18, v=82: 258, 228,
// 207).
template <bool AC, bool BC, bool CC, int S, int BM, int BN>
__global__ void __launch_bounds__(256, 3) simt_slices_kernel(const GemmArgs g, int alpha_pow2, int alpha_e,
                                                             int alpha_neg) {
  constexpr int PA = AC ? 2 : 1, PB = BC ? 2 : 1;
  constexpr int SPA = (S * PA + 1) / 2 * 2, SPB = (S * PB + 1) / 2 * 2;  // floats per row, even
  // shared row strides: B's columns are read by the 16 tx values of a half
  // warp at once, so their stride is twice an odd number of floats (the 16
  // float2 reads fall in distinct bank pairs); A's rows by two ty values only
  constexpr int STA = SPA, STB = (SPB / 2) % 2 == 1 ? SPB : SPB + 2;
  constexpr int MI = BM / 16, NJ = BN / 16;
  static_assert(MI * NJ == 4, "four outputs per thread");
  constexpr int KC = (BM > 32 || BN > 32) ? 8 : 16;  // K chunk (static shared memory <= 48 KB)
  __shared__ __align__(8) float sa[KC][BM][STA];
  __shared__ __align__(8) float sb[KC][BN][STB];
  __shared__ long long aoff[BM], boff[BN], coffm[BM], coffn[BN];
  __shared__ long long kofa[kSimtMaxK], kofb[kSimtMaxK];
  __shared__ int ea[BM], eb[BN];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, zb = blockIdx.z;
  const double* A = static_cast<const double*>(g.A) + (size_t)zb * g.bsA * PA;
  const double* B = static_cast<const double*>(g.B) + (size_t)zb * g.bsB * PB;
  auto dec = [](const ModeGroup& gr, int l, long long& o0, long long& o1) {
    o0 = 0;
    o1 = 0;
    for (int q = kMaxModes - 1; q >= 0; --q)
      if (q < gr.n) {
        const int r = l % gr.dim[q];
        l /= gr.dim[q];
        o0 += (long long)r * gr.s0[q];
        o1 += (long long)r * gr.s1[q];
      }
  };
  if (tid < BM) {
    long long o0 = -1, o1 = -1;
    if (m0 + tid < g.M) dec(g.gm, m0 + tid, o0, o1);
    aoff[tid] = o0;
    coffm[tid] = o1;
  } else if (tid < BM + BN) {
    const int c = tid - BM;
    long long o0 = -1, o1 = -1;
    if (n0 + c < g.N) dec(g.gn, n0 + c, o0, o1);
    boff[c] = o0;
    coffn[c] = o1;
  } else if (tid < BM + BN + g.K) {
    const int k = tid - BM - BN;
    dec(g.gk, k, kofa[k], kofb[k]);
  }
  __syncthreads();
  // a chunk's elements of A (BM x KC) and B (KC x BN), E to a thread, all loads
  // in flight
  constexpr int E = ((BM + BN) * KC + 255) / 256;
  double x[E][2];
  auto place = [&](int i, bool& isA, int& r, int& kk) {
    const int idx = tid + 256 * i;
    isA = idx < BM * KC;
    const int id2 = isA ? idx : idx - BM * KC, nr = isA ? BM : BN;
    r = id2 % nr;
    kk = id2 / nr;
    return idx < (BM + BN) * KC;
  };
  auto load_chunk = [&](int kc) {
#pragma unroll
    for (int i = 0; i < E; ++i) {
      bool isA;
      int r, kk;
      const bool in = place(i, isA, r, kk);
      const int k = kc + kk;
      x[i][0] = x[i][1] = 0.0;
      const long long base = !in ? -1 : isA ? aoff[r] : boff[r];
      if (base >= 0 && k < g.K) {
        const double* src = isA ? A : B;
        const long long el = base + (isA ? kofa[k] : kofb[k]);
        if ((isA ? PA : PB) == 2) {
          const double2 v = *reinterpret_cast<const double2*>(src + 2 * el);
          x[i][0] = v.x;
          x[i][1] = v.y;
        } else {
          x[i][0] = src[el];
        }
      }
    }
  };
  // exponents of the tile's rows of A and columns of B over all of K, as twice
  // the biased exponent of the largest |x| plus one where there is a nonzero
  __shared__ unsigned rmax[BM + BN];
  if (tid < BM + BN) rmax[tid] = 0u;
  __syncthreads();
  for (int kc = 0; kc < g.K; kc += KC) {
    load_chunk(kc);
#pragma unroll
    for (int i = 0; i < E; ++i) {
      bool isA;
      int r, kk;
      if (!place(i, isA, r, kk)) continue;
      unsigned v = 0u;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        const unsigned h = (unsigned)__double2hiint(x[i][part]) & 0x7FFFFFFFu;
        if (h | (unsigned)__double2loint(x[i][part])) v = max(v, 2u * (h >> 20) + 1u);
      }
      if (v) atomicMax(&rmax[isA ? r : BM + r], v);
    }
  }
  __syncthreads();
  if (tid < BM + BN) {
    const int E2 = (int)(rmax[tid] >> 1);
    const int e = rmax[tid] != 0u ? (E2 > 0 ? E2 - 1022 : -1022) : 0;
    if (tid < BM)
      ea[tid] = e;
    else
      eb[tid - BM] = e;
  }
  __syncthreads();
  const int tx = tid % 16, ty = tid / 16;
  float2 acc[MI][NJ][S];  // levels, (re, im)
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int L = 0; L < S; ++L) acc[i][j][L] = make_float2(0.f, 0.f);
  for (int kc = 0; kc < g.K; kc += KC) {
    if (g.K > KC) load_chunk(kc);  // one chunk: as loaded for the exponents
#pragma unroll
    for (int i = 0; i < E; ++i) {
      bool isA;
      int r, kk;
      if (!place(i, isA, r, kk)) continue;
      const int per = isA ? PA : PB, e = isA ? ea[r] : eb[r];
      float* dst = isA ? &sa[kk][r][0] : &sb[kk][r][0];
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        if (part >= per) continue;
        uint32_t hi, lo;
        cut_digits<(S <= 4 ? 4 : 6)>(x[i][part], e, S, hi, lo);
        const uint32_t sgn = (uint32_t)__double2hiint(x[i][part]) & 0x80000000u;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          // 2^23 + u is the float 0x4B000000 + u; digits after the first are biased by 64
          const uint32_t w = s < 4 ? hi : lo, bit = s < 4 ? 21 - 7 * s : 7 * (5 - s);
          const uint32_t uf = ((w >> bit) & (s == 0 ? 0xFFu : 0x7Fu)) | 0x4B000000u;
          const float d = __uint_as_float(uf) - (s == 0 ? 8388608.f : 8388672.f);
          dst[s * per + part] = __uint_as_float(__float_as_uint(d) ^ sgn);
        }
      }
    }
    __syncthreads();
    const int kn = min(KC, g.K - kc);
    for (int kk = 0; kk < kn; ++kk) {
      // real times complex: re and im share a packed FP32 multiply-add (97 -> 73 us
      // on a K = 10 contraction; complex times complex, which needs B's digits
      // swapped as well: 176 us so, 166 with single ones)
      float2 b[NJ][S];  // B's digits (re, im), or the real one twice
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int t = 0; t < S; ++t) {
          const float* p = &sb[kk][tx + 16 * j][t * PB];
          if constexpr (BC) {
            b[j][t] = *reinterpret_cast<const float2*>(p);
          } else {
            b[j][t] = make_float2(p[0], p[0]);
          }
        }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const float* p = &sa[kk][ty + 16 * i][s * PA];
          const float2 a = AC ? *reinterpret_cast<const float2*>(p) : make_float2(p[0], p[0]);
#pragma unroll
          for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int t = 0; t < S - s; ++t) {  // level s + t (0-based), s + t <= S - 1
              float2& c = acc[i][j][s + t];
              if constexpr (AC && BC) {
                c.x = fmaf(a.x, b[j][t].x, c.x);
                c.x = fmaf(-a.y, b[j][t].y, c.x);
                c.y = fmaf(a.x, b[j][t].y, c.y);
                c.y = fmaf(a.y, b[j][t].x, c.y);
              } else if constexpr (AC || BC) {
                fma_f32x2(c, a, b[j][t]);
              } else {
                c.x = fmaf(a.x, b[j][t].x, c.x);
              }
            }
        }
    }
    __syncthreads();
  }
  // recombine the levels in int64 (0-based level l weighs 2^(-7(l + 2))) and store
  const int u = 7 * ((S < 5 ? S : 5) + 1);
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int r = ty + 16 * i, c = tx + 16 * j;
      if (m0 + r >= g.M || n0 + c >= g.N) continue;
      long long X[2] = {0, 0};
#pragma unroll
      for (int L = 0; L < S; ++L) {
        const int sh = u - 7 * (L + 2);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const long long v = (long long)__float2int_rn(p ? acc[i][j][L].y : acc[i][j][L].x);
          X[p] += sh >= 0 ? (v << sh) : (v >> (-sh));
        }
      }
      const int E = ea[r] + eb[c] - u + (alpha_pow2 ? alpha_e : 0);
      double vr, vi;
      if (alpha_pow2) {
        vr = scaled_i64_to_double(alpha_neg ? -X[0] : X[0], E);
        vi = scaled_i64_to_double(alpha_neg ? -X[1] : X[1], E);
      } else {
        const double dr = scaled_i64_to_double(X[0], E), di = scaled_i64_to_double(X[1], E);
        vr = g.ar * dr - g.ai * di;
        vi = g.ar * di + g.ai * dr;
      }
      const long long off = coffm[r] + coffn[c];
      // accumulation as an L2 reduction (one writer per element)
      if constexpr (CC) {
        double2* C = static_cast<double2*>(g.C) + (size_t)zb * g.bsC;
        if (g.acc) {
          atomicAdd(&C[off].x, vr);
          atomicAdd(&C[off].y, vi);
        } else {
          C[off] = make_double2(vr, vi);
        }
      } else {
        double* C = static_cast<double*>(g.C) + (size_t)zb * g.bsC;
        if (g.acc)
          atomicAdd(&C[off], vr);
        else
          C[off] = vr;
      }
    }
}

template <bool AC, bool BC, bool CC, int S>
static void launch_simt_tile(int tile, const GemmArgs& g, int nb, int p2, int e2, int n2, cudaStream_t st) {
  const int bm = tile == 1 ? 16 : tile == 2 ? 64 : 32, bn = tile == 1 ? 64 : tile == 2 ? 16 : 32;
  dim3 grid((unsigned)((g.N + bn - 1) / bn), (unsigned)((g.M + bm - 1) / bm), (unsigned)nb);
  if (tile == 1)
    simt_slices_kernel<AC, BC, CC, S, 16, 64><<<grid, 256, 0, st>>>(g, p2, e2, n2);
  else if (tile == 2)
    simt_slices_kernel<AC, BC, CC, S, 64, 16><<<grid, 256, 0, st>>>(g, p2, e2, n2);
  else
    simt_slices_kernel<AC, BC, CC, S, 32, 32><<<grid, 256, 0, st>>>(g, p2, e2, n2);
}

template <bool AC, bool BC, bool CC>
static void launch_simt_typed(int tile, const GemmArgs& g, int nb, int S, int p2, int e2, int n2, cudaStream_t st) {
  if (S == 6)
    launch_simt_tile<AC, BC, CC, 6>(tile, g, nb, p2, e2, n2, st);
  else if (S == 5)
    launch_simt_tile<AC, BC, CC, 5>(tile, g, nb, p2, e2, n2, st);
  else
    launch_simt_tile<AC, BC, CC, 4>(tile, g, nb, p2, e2, n2, st);
}

bool simt_slices_supported(int K, int S) { return K >= 1 && K <= kSimtMaxK && S >= 4 && S <= 6; }

cudaError_t launch_simt_slices(const Op& op, const void* A, const void* B, void* C, cudaStream_t st) {
  GemmArgs g = op.g;
  g.A = A;
  g.B = B;
  g.C = C;
  const TcArgs& t = op.tc;
  if (!simt_slices_supported(g.K, t.S) || g.atomic) return cudaErrorInvalidValue;
  const int nb = g.nb < 1 ? 1 : g.nb;
  // the tile with the least padding: 32 x 32, 16 x 64, 64 x 16
  const long long M = g.M, N = g.N;
  const long long pad[3] = {((M + 31) / 32 * 32) * ((N + 31) / 32 * 32), ((M + 15) / 16 * 16) * ((N + 63) / 64 * 64),
                            ((M + 63) / 64 * 64) * ((N + 15) / 16 * 16)};
  int tile = 0;
  for (int q = 1; q < 3; ++q)
    if (pad[q] < pad[tile]) tile = q;
  const int bm = tile == 1 ? 16 : tile == 2 ? 64 : 32;
  if ((M + bm - 1) / bm > 65535 || nb > 65535) return cudaErrorInvalidConfiguration;
  const bool ac = op.dta == C64, bc = op.dtb == C64, cc = op.dtc == C64;
  if (!cc && (ac || bc)) return cudaErrorInvalidValue;
  if (ac && bc)
    launch_simt_typed<true, true, true>(tile, g, nb, t.S, t.alpha_pow2, t.alpha_e, t.alpha_neg, st);
  else if (ac)
    launch_simt_typed<true, false, true>(tile, g, nb, t.S, t.alpha_pow2, t.alpha_e, t.alpha_neg, st);
  else if (bc)
    launch_simt_typed<false, true, true>(tile, g, nb, t.S, t.alpha_pow2, t.alpha_e, t.alpha_neg, st);
  else if (cc)
    launch_simt_typed<false, false, true>(tile, g, nb, t.S, t.alpha_pow2, t.alpha_e, t.alpha_neg, st);
  else
    launch_simt_typed<false, false, false>(tile, g, nb, t.S, t.alpha_pow2, t.alpha_e, t.alpha_neg, st);
  count_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
bool tc_available() { return true; }

// the driver's tensor-map encoder, looked up once (thread-safe static init)
static PFN_cuTensorMapEncodeTiled_v12000 encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        !p)
      return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
    return (PFN_cuTensorMapEncodeTiled_v12000)p;
  }();
  if (!fn) throw std::runtime_error("cuTensorMapEncodeTiled unavailable");
  return fn;
}

// [S][rows_pad][K_pad] BF16, box = (64 K, box_rows rows, 1 slice).
// Encoded maps are cached by (address, layout), which determine them: a packed
// buffer keeps its address for the life of its program.  The cache is emptied when
// it has grown to kMapsMax (scratch addresses come and go).
constexpr size_t kMapsMax = 4096;
CUtensorMap slice_map(const void* base, int S, int rows_pad, int K_pad, int box_rows) {
  static std::mutex mu;
  static std::map<std::tuple<const void*, int, int, int, int>, CUtensorMap> cache;
  const auto key = std::make_tuple(base, S, rows_pad, K_pad, box_rows);
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
  }
  CUtensorMap m;
  cuuint64_t dims[3] = {(cuuint64_t)K_pad, (cuuint64_t)rows_pad, (cuuint64_t)S};
  cuuint64_t strides[2] = {(cuuint64_t)K_pad * 2, (cuuint64_t)K_pad * 2 * rows_pad};
  cuuint32_t box[3] = {TC_BK, (cuuint32_t)box_rows, 1};
  cuuint32_t es[3] = {1, 1, 1};
  const CUresult r = encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box,
                               es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  std::lock_guard<std::mutex> lk(mu);
  if (cache.size() >= kMapsMax) cache.clear();
  cache[key] = m;
  return m;
}

template <int SMAX>
static cudaError_t launch_pack_slices(const PackArgs& p, long long blocks, cudaStream_t st) {
  if (p.K_pad <= 2048) {
    // rows held in registers, read once: up to 256 elements per warp (8 per
    // lane), up to eight warps per row.  Three pairs a lane where they suffice:
    // fewer idle lanes and registers (K = 1444, 6.9 M numbers: 37 -> 32 us; K =
    // 380: 43 -> 37)
    auto go = [&](auto kern, int rows_per_block) {
      kern<<<(unsigned)((blocks + rows_per_block - 1) / rows_per_block), 256, 0, st>>>(p);
    };
    if (p.K_pad <= 64)
      go(pack_rows_regs_kernel<1, 1, SMAX>, 8);
    else if (p.K_pad <= 128)
      go(pack_rows_regs_kernel<2, 1, SMAX>, 8);
    else if (p.K_pad <= 192)
      go(pack_rows_regs_kernel<3, 1, SMAX>, 8);
    else if (p.K_pad <= 384)
      go(pack_rows_regs_kernel<3, 2, SMAX>, 4);
    else if (p.K_pad <= 768)
      go(pack_rows_regs_kernel<3, 4, SMAX>, 2);
    else if (p.K_pad <= 1024)
      go(pack_rows_regs_kernel<4, 4, SMAX>, 2);
    else if (p.K_pad <= 1536)
      go(pack_rows_regs_kernel<3, 8, SMAX>, 1);
    else
      go(pack_rows_regs_kernel<4, 8, SMAX>, 1);
  } else {
    // long rows: a block per row, of more threads where there are few; fewer than
    // the SMs, a cluster of eight blocks per row
    constexpr int CL = 8;
    const bool cluster = blocks <= 152 && p.K_pad >= 8192;
    const int threads = cluster ? 512 : (p.K_pad >= 4096 && blocks < 4 * 152) ? 1024 : 256;
    // the K offsets as a shared-memory table when they fit (64 KB, 32 bits)
    constexpr int kTabMax = 16384;
    constexpr int kMaxDev = 64;
    static std::once_flag once[kMaxDev];
    static cudaError_t attr_err[kMaxDev] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
    std::call_once(once[dev], [dev] {
      attr_err[dev] = cudaFuncSetAttribute(pack_kernel<SMAX, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           kTabMax * (int)sizeof(int));
      if (attr_err[dev] == cudaSuccess)
        attr_err[dev] = cudaFuncSetAttribute(pack_kernel<SMAX, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             kTabMax * (int)sizeof(int));
    });
    long long span = 0;  // largest K offset
    for (int q = 0; q < p.gk.n && q < kMaxModes; ++q) span += (long long)(p.gk.dim[q] - 1) * std::llabs(p.gk.s0[q]);
    const int seg = cluster ? (p.K_pad / 2 + CL - 1) / CL * 2 : p.K;
    const int tab = (attr_err[dev] == cudaSuccess && seg <= kTabMax && span < (1LL << 31)) ? 1 : 0;
    const size_t smem = tab ? (size_t)seg * sizeof(int) : 0;
    if (cluster) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(blocks * CL));
      cfg.blockDim = dim3(threads);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = st;
      cudaLaunchAttribute at[1] = {};
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = CL;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      const cudaError_t e = cudaLaunchKernelEx(&cfg, pack_kernel<SMAX, CL>, p, tab);
      if (e != cudaSuccess) return e;
    } else {
      pack_kernel<SMAX, 1><<<(unsigned)blocks, threads, smem, st>>>(p, tab);
    }
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_pack(const PackArgs& p, cudaStream_t st) {
  if (p.nb < 1 || p.rows < 1 || p.rows_pad % (p.cplx ? 2 : 1) != 0 || p.rows * (p.cplx ? 2 : 1) > p.rows_pad ||
      p.K_pad % 2 != 0 || p.K > p.K_pad)
    return cudaErrorInvalidValue;
  const long long blocks = (long long)p.nb * p.rows;
  if (blocks > 0x7FFFFFFFLL) return cudaErrorInvalidConfiguration;
  if (p.S < 1 || (p.S > TC_MAX_SLICES && p.S != TC_DEEP_SLICES)) return cudaErrorInvalidValue;
  return p.S > TC_MAX_SLICES ? launch_pack_slices<TC_DEEP_SLICES>(p, blocks, st)
         : p.S > 4           ? launch_pack_slices<TC_MAX_SLICES>(p, blocks, st)
                             : launch_pack_slices<4>(p, blocks, st);
}

template <class C>
static cudaError_t launch_variant(const TcArgs& a0, const void* packA, const void* packB, cudaStream_t st) {
  // kernel attributes act on the current device's context: set them once
  // per device (engines on several host threads may launch their first
  // slice products together)
  constexpr int kMaxDev = 64;
  static std::once_flag once[kMaxDev];
  static cudaError_t attr_err[kMaxDev] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [dev] {
    cudaError_t e = cudaFuncSetAttribute(ozaki_kernel<true, true, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ozaki_kernel<true, false, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ozaki_kernel<false, true, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ozaki_kernel<false, false, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    // all of L1 as shared memory, so that MINB CTAs fit on an SM
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ozaki_kernel<true, true, C>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ozaki_kernel<true, false, C>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ozaki_kernel<false, true, C>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ozaki_kernel<false, false, C>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    attr_err[dev] = e;
  });
  if (attr_err[dev] != cudaSuccess) return attr_err[dev];
  TcArgs a = a0;
  if (a.S < 2 || a.S > C::STAGES) return cudaErrorInvalidValue;  // the ring holds one K block's slices
  int cols = 32;
  while (cols < (a.S + 2) * C::BN) cols *= 2;  // level accumulators + int64 partial sums
  if (cols > 512 / C::MINB) return cudaErrorInvalidValue;
  a.tmem_cols = cols;
  if (a.rowsB_pad % C::BN != 0) return cudaErrorInvalidValue;
  const CUtensorMap ma = slice_map(packA, a.S, (a.bat_a ? a.nb : 1) * a.rowsA_pad, a.kblocks * TC_BK, TC_BM);
  const CUtensorMap mb = slice_map(packB, a.S, (a.bat_b ? a.nb : 1) * a.rowsB_pad, a.kblocks * TC_BK, C::BN);
  // CTA order: the tiles of the smaller operand side vary fastest, so that
  // side stays in L2 while each tile of the larger side is read from DRAM
  // once (the N-fastest order re-read the 69 MB of packed amplitudes of the
  // 24-trajectory ladder for each of its 12 M strips: 430 MB per launch)
  const unsigned mtiles = (unsigned)(a.rowsA_pad / TC_BM), ntiles = (unsigned)(a.rowsB_pad / C::BN);
  a.m_fast = (a.rowsA_pad < a.rowsB_pad && ntiles <= 65535u) ? 1 : 0;
  dim3 grid(a.m_fast ? mtiles : ntiles, a.m_fast ? ntiles : mtiles, (unsigned)((long long)a.nb * a.nsplit));
  if (a.ac && a.bc)
    ozaki_kernel<true, true, C><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  else if (a.ac)
    ozaki_kernel<true, false, C><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  else if (a.bc)
    ozaki_kernel<false, true, C><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  else
    ozaki_kernel<false, false, C><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a);
  count_launch();
  return cudaGetLastError();
}

static cudaError_t launch_persist(const TcArgs& a0, const void* packA, const void* packB, cudaStream_t st) {
  using C = TcPersist;
  constexpr int kMaxDev = 64;
  static std::once_flag once[kMaxDev];
  static cudaError_t attr_err[kMaxDev] = {};
  static int sm_count[kMaxDev] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [dev] {
    cudaError_t e = cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
    for (auto fn : {ozaki_persist_kernel<true, true>, ozaki_persist_kernel<true, false>,
                    ozaki_persist_kernel<false, true>, ozaki_persist_kernel<false, false>}) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    attr_err[dev] = e;
  });
  if (attr_err[dev] != cudaSuccess) return attr_err[dev];
  TcArgs a = a0;
  // two TMEM buffers of S levels, short K per tile
  if (a.S < 2 || a.S > TC_PERSIST_MAX_S || a.kb_per_split > C::MAX_KB) return cudaErrorInvalidValue;
  int cols = 32;
  while (cols < 2 * a.S * C::BN) cols *= 2;
  a.tmem_cols = cols;
  if (a.rowsB_pad % C::BN != 0 || a.rowsA_pad % TC_BM != 0) return cudaErrorInvalidValue;
  const CUtensorMap ma = slice_map(packA, a.S, (a.bat_a ? a.nb : 1) * a.rowsA_pad, a.kblocks * TC_BK, TC_BM);
  const CUtensorMap mb = slice_map(packB, a.S, (a.bat_b ? a.nb : 1) * a.rowsB_pad, a.kblocks * TC_BK, C::BN);
  const long long mtiles = a.rowsA_pad / TC_BM, ntiles = a.rowsB_pad / C::BN;
  a.m_fast = a.rowsA_pad < a.rowsB_pad ? 1 : 0;
  const long long total = mtiles * ntiles * a.nb * a.nsplit;
  if (total > 0x7FFFFFFFLL) return cudaErrorInvalidConfiguration;
  const unsigned grid = (unsigned)std::min<long long>(total, std::max(sm_count[dev], 1));
  if (a.ac && a.bc)
    ozaki_persist_kernel<true, true><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a, (int)total);
  else if (a.ac)
    ozaki_persist_kernel<true, false><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a, (int)total);
  else if (a.bc)
    ozaki_persist_kernel<false, true><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a, (int)total);
  else
    ozaki_persist_kernel<false, false><<<grid, C::THREADS, C::SMEM, st>>>(ma, mb, a, (int)total);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_ozaki(const TcArgs& a, const void* packA, const void* packB, cudaStream_t st) {
  if (a.nb < 1 || a.nsplit < 1 || (long long)a.nsplit * a.kb_per_split < a.kblocks) return cudaErrorInvalidValue;
  if (a.variant == 3) return launch_deep(a, packA, packB, st);
  if (a.variant == 2) return launch_persist(a, packA, packB, st);
  return a.variant == 1 ? launch_variant<TcNarrow>(a, packA, packB, st) : launch_variant<TcWide>(a, packA, packB, st);
}

}  // namespace tdcc
