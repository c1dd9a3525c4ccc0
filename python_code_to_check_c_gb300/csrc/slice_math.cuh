// Device helpers of the slice-product kernels (gemm_tc.cu): strided index
// decoding, the per-row binary exponents, the
// cut of a scaled double into balanced BF16-exact digits, and the exact
// conversion of an int64 sum back to a scaled double.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

#include "engine.h"

namespace tdcc {

// Offset of index l < prod(dim) of a mode group (last mode fastest).
__device__ __forceinline__ void decomp_tc(const ModeGroup& g, int l, long long& o0) {
  if (g.n == 1) {  // l < dim[0]: no division
    o0 = (long long)l * g.s0[0];
    return;
  }
  o0 = 0;
#pragma unroll
  for (int q = kMaxModes - 1; q >= 1; --q) {
    if (q < g.n) {
      const int d = g.dim[q];
      const int r = l % d;
      l /= d;
      o0 += (long long)r * g.s0[q];
    }
  }
  o0 += (long long)l * g.s0[0];  // l < dim[0]: the outermost mode needs no division
}

// Row exponents are stored biased (e + kExpBias; 0 = all-zero row) so that
// zero-initialised memory and atomicMax give the maximum directly.
constexpr int kExpBias = 4096;
constexpr int kExpMarked = 1 << 30;  // a row that digits cannot hold (deep form)
__device__ __forceinline__ int row_exp(int biased) { return biased > 0 ? biased - kExpBias : 0; }

// |x| 2^(nbits - e) rounded to the nearest integer (ties away) from the bits of x
// (no FP64 arithmetic).  Requires |x| < 2^e and nbits <= 63: at most 2^nbits.
__device__ __forceinline__ unsigned long long fixed_point_rounded(double x, int e, int nbits) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
  const int E = (int)(u >> 52);
  if (E == 0) return 0ull;
  const unsigned long long M = (u & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
  const int sh = E - 1075 - e + nbits;
  if (sh >= 0) return M << sh;
  if (sh < -54) return 0ull;
  return ((M >> (-sh - 1)) + 1ull) >> 1;
}

// |x| 2^-e cut into SMAX balanced digits of 7 bits (the packing keeps the first S),
// in two words: hi holds digits 1 .. 4, the first in [0, 128] at bit 21, lo the
// others.  The digits after the first are biased by 64: f plus 64 at each of their
// places has them in its 7-bit fields, carries included.  SMAX = 4 and 6 cut after
// 7 S bits; SMAX = 8 has digits of 8 bits (the first in [0, 128] at bit 24, the
// others biased by 128) and rounds to 63.  |x| < 2^e; integer operations only, of 32 bits for
// SMAX = 4.  (Packing 6.9 M numbers, o=10, v=38 with 24 trajectories: 51 us with
// digits cut one by one in 64 bits, 38 so, 16 for their bytes.)
template <int SMAX>
__device__ __forceinline__ void cut_digits(double x, int e, int S, uint32_t& hi, uint32_t& lo) {
  constexpr uint32_t kB3 = 64u * (1u + (1u << 7) + (1u << 14)), kB2 = 64u * (1u + (1u << 7));
  lo = 0u;
  if constexpr (SMAX == 8) {
    const unsigned long long f = fixed_point_rounded(x, e, 63) + 0x0080808080808080ull;
    lo = (uint32_t)f;
    hi = (uint32_t)(f >> 32);
  } else {
    const uint32_t xh = (uint32_t)__double2hiint(x) & 0x7FFFFFFFu, xl = (uint32_t)__double2loint(x);
    const int E = (int)(xh >> 20);
    const uint32_t mh = (xh & 0xFFFFFu) | 0x100000u;
    const int drop = 1022 + e - E;  // bits of the row's scale above x; >= 0
    if constexpr (SMAX == 4) {
      uint32_t t = (mh << 7) | (xl >> 25);  // the top 28 bits of the significand
      t >>= min(drop, 31);
      t &= ~((1u << (7 * (4 - S))) - 1u);
      hi = (E == 0 ? 0u : t) + kB3;  // zero or subnormal: below every slice
    } else {
      static_assert(SMAX == 6, "4, 6 or 8");
      unsigned long long t = (((unsigned long long)mh << 32) | xl) >> 11;  // the top 42
      t >>= min(drop, 63);
      t &= ~((1ull << (7 * (6 - S))) - 1ull);
      if (E == 0) t = 0ull;
      lo = (uint32_t)(t & 0x3FFFull) + kB2;
      hi = (uint32_t)(t >> 14) + (lo >> 14) + kB3;
    }
  }
}

// A digit of two neighbouring elements as a BF16 pair, w0's in the low half (the
// lower address): 0x4300 + u is the BF16 number 128 + u (u <= 128), so the
// subtraction of the bias is exact.  sgn: the elements' signs in bits 15 and 31.
// BITS = 8: u + 128 with u's upper bit in the bias, 256 or 128.
template <int BIT, bool TOP, int BITS = 7>
__device__ __forceinline__ uint32_t digit_pair(uint32_t w0, uint32_t w1, uint32_t sgn) {
  constexpr uint32_t m = TOP || BITS == 8 ? 0xFFu : 0x7Fu;
  const uint32_t a = w0 >> BIT, b = BIT <= 16 ? w1 << (16 - BIT) : w1 >> (BIT - 16);
  uint32_t p = (a & m) | (b & (m << 16));
  uint32_t bias = TOP ? 0x43004300u : 0x43404340u;  // 128, 192
  if (!TOP && BITS == 8) {
    bias = (p & 0x00800080u) ^ 0x43804380u;
    p &= 0x007F007Fu;
  }
  p |= 0x43004300u;
  const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&p), *reinterpret_cast<const __nv_bfloat162*>(&bias));
  return *reinterpret_cast<const uint32_t*>(&r) ^ sgn;
}

// Subnormal or overflowing results (not met by the contractions here) take
// the FP64 path, out of line so that nothing of it is evaluated on the
// normal path.
static __device__ __noinline__ double scaled_i64_to_double_rare(long long x, int E) { return ldexp((double)x, E); }

// x * 2^E rounded to nearest (ties to even) from the integer's bits, without
// branches on the normal-range path and no FP64 arithmetic (GB300's FP64
// pipe is narrow): the magnitude is normalised to bit 63, its top 53 bits
// are the significand, the 11 bits below round it, and a carry out of the
// significand rounds up into the exponent field by the integer addition.
__device__ __forceinline__ double scaled_i64_to_double(long long x, int E) {
  const unsigned long long sgn = (unsigned long long)(x >> 63);  // all ones when negative
  const unsigned long long u = ((unsigned long long)x ^ sgn) - sgn;
  if (u == 0ull) return 0.0;
  const int lz = __clzll((long long)u);
  const unsigned long long m = u << lz;  // leading one at bit 63
  const unsigned long long mant = m >> 11;  // 53 bits, leading one at bit 52
  const unsigned rem = (unsigned)(m & 0x7FFull);
  const unsigned long long up = (rem > 0x400u || (rem == 0x400u && (mant & 1ull))) ? 1ull : 0ull;
  const int be = 63 - lz + E + 1023;  // biased exponent before rounding
  if (be <= 0 || be >= 2047) return scaled_i64_to_double_rare(x, E);
  // the leading one of mant adds 1 to the exponent field (be - 1 + 1)
  const unsigned long long bits = ((unsigned long long)(be - 1) << 52) + mant + up;
  return __longlong_as_double((long long)(bits | (sgn << 63)));
}

}  // namespace tdcc
