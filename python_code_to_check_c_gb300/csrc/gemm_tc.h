// Tensor-core (tcgen05) slice-product backend: tile constants.  The argument
// blocks PackArgs / TcArgs live in engine.h; see gemm_tc.cu for the method.
#pragma once

#include <cuda_runtime.h>

#include "engine.h"

namespace tdcc {

constexpr int TC_BM = 128;                   // UMMA M (rows of A per CTA)
constexpr int TC_BN = 64;                    // packed B rows are padded to this (both variants)
constexpr int TC_BK = 64;                    // K per TMA box (128 B of BF16)
constexpr int TC_CHUNK_KB = 8;               // 512-wide K chunks (exact FP32 level sums)
constexpr int TC_A_BYTES = TC_BM * TC_BK * 2;
constexpr int kTcWaitLimit = 1 << 22;        // polls after which a tensor-core kernel gives up a wait
constexpr int TC_MAX_SLICES = 6;
constexpr int TC_DEEP_SLICES = 8;            // the FP64 form's tensor-core contractions
// planes of a packed operand: its slices, and with 8 the range guard's (gemm_deep.cu)
constexpr int tc_planes(int S) { return S + (S == TC_DEEP_SLICES ? 1 : 0); }

// Kernel variants: tile width BN (UMMA N), ring depth, TMEM-drain warps and
// CTAs per SM.  The ring must hold the S slices of one K block (STAGES >= S).
template <int BN_, int STAGES_, int EPI_, int MINB_>
struct TcCfg {
  static constexpr int BN = BN_, STAGES = STAGES_, EPI = EPI_, MINB = MINB_;
  static constexpr int B_BYTES = BN * TC_BK * 2;
  static constexpr int THREADS = 64 + 32 * EPI;  // + TMA producer warp + MMA warp
  static constexpr int SMEM = 1024 + STAGES * (TC_A_BYTES + B_BYTES) + 2048;
};
// one CTA per SM: 64-wide tile, 8 stages, 16 drain warps (four per lane quarter)
using TcWide = TcCfg<64, 8, 16, 1>;
// two CTAs per SM (one's drain overlaps the other's MMAs): 32-wide tile, 5
// stages, 8 drain warps; TMEM (S + 2) x 32 <= 256 columns, so S <= 5
using TcNarrow = TcCfg<32, 5, 8, 2>;
constexpr int TC_PERSIST_MAX_S = 4;

// Persistent 64-column form for S <= 4 slices: one CTA per SM walks a list
// of output tiles; S level accumulators of 64 columns make one TMEM buffer
// (S x 64 <= 256 columns), two buffers fill TMEM, so that the drain warps
// empty tile i's buffer while the MMAs of tile i + 1 fill the other.  Slices
// of A (128 x 64, 16 KB) and of B (64 x 64, 8 KB) have rings of their own;
// the drain stages 16 columns per warp in an area of its own (the rings keep
// loading the next tile meanwhile).
struct TcPersist {
  static constexpr int BN = 64, EPI = 16, MINB = 1;
  static constexpr int MAX_KB = 2;                   // K blocks per tile
  static constexpr int RA = 5, RB = 6;               // ring slots of A and B slices
  static constexpr int A_SLOT = TC_BM * TC_BK * 2;   // 16 KB
  static constexpr int B_SLOT = BN * TC_BK * 2;      // 8 KB
  static constexpr int STAGE_WARP = 4608;            // staging bytes per drain warp
  static constexpr int THREADS = 64 + 32 * EPI;
  static constexpr int SMEM = 1024 + RA * A_SLOT + RB * B_SLOT + EPI * STAGE_WARP + 2048;
};

// Deep form (gemm_deep.cu): a 128 x BN tile whose S level accumulators fill
// TMEM, a ring of (A, B) slice pairs, sums over K in the drain warps'
// registers across exact chunks of CHUNK_KB K blocks: a level of p pairs grows
// by at most 2 x 128 x 64 + (p - 2) x 64 x 64 per K index (7-bit digits; the 8-bit
// ones of S = 8: p x 128 x 128) and must stay within 2^24.
template <int S_, int BN_, int STAGES_>
struct TcDeep {
  static constexpr int S = S_, BN = BN_, STAGES = STAGES_, EPI = 16;
  static constexpr int A_BYTES = TC_BM * TC_BK * 2, B_BYTES = BN * TC_BK * 2;
  static constexpr int THREADS = 64 + 32 * EPI;
  static constexpr int TAIL = 2048;
  static constexpr int SMEM = 1024 + STAGES * (A_BYTES + B_BYTES) + TAIL;
  static constexpr int CHUNK_KB =
      (1 << 24) / ((S == TC_DEEP_SLICES ? S * 16384 : 16384 + (S > 2 ? S - 2 : 0) * 4096) * TC_BK);
  static_assert(S * BN <= 512 && STAGES >= S, "TMEM columns, ring");
};

cudaError_t launch_deep(const TcArgs& a, const void* packA, const void* packB, cudaStream_t st);

}  // namespace tdcc
