// FP64 contractions on the integer pipe: block fixed point with exact sums.
//
// GB300's FP64 pipe does 1.9 multiply-adds per clock and SM (0.58 T/s for the
// chip), its integer pipe 26 of 32 x 32 + 64 bits (both measured, operands
// from shared memory).  So a
// contraction C[m,n] (+)= alpha sum_k A[m,k] B[k,n] is cut into K chunks of
// at most 60; in a chunk each real row of A and column of B (the real and
// imaginary parts of a complex one are two) is scaled by the power of two
// above its largest magnitude and written as v = h 2^28 + l + r, |v| < 2^56,
// |h| <= 2^28, -2^27 <= l < 2^27, |r| <= 1/2: 56 bits as integers, the rest
// of a small element as an FP32 number.  A product is h h' 2^56 + (h l' + l h')
// 2^28, three multiply-adds into two 64-bit sums that cannot overflow (60
// terms of 2^56, 2 x 60 of 2^55), and l l' + v r' + r v', three FP32
// multiply-adds of at most 2^-57 of the row maxima: about 78 bits under the
// maxima altogether.  The integer sums are exact; each chunk is rounded to FP64
// once, where an FP64 chain rounds every term.  Rows that span more still are
// found by the range guard below and done by FP64 multiply-adds.  So an output's
// error against the sum of its products' magnitudes is below an FP64 chain's,
// not only the error against the largest output.
//
// Bound: issue, the integer multiply-adds (4.9 clocks a warp and scheduler each) and
// the FP32 ones beside them; then index work and cutting (16 warps, 512 threads and
// 64 registers, gain 8 % on one tile and lose 5 % on many).  With the integer sums
// alone, 56 bits and one scale for both parts of a complex row, a launch took 35 us
// where this takes 49 (100 x 100 x 196 complex, o=10, v=14) and 24 where this takes 37
// (380 x 38 x 38 complex by 100, o=10, v=38); the FP64 kernel before (64 x 64 tile, at
// 96 % of the FP64 pipe) 1450 us for 1444 x 100 x 1444 complex by real, where the
// integers alone took 320.
//
// A chunk whose maxima are not finite, or so large or small that scaling by
// them would leave the normal range, is done by FP64 multiply-adds from
// global memory instead (the same operands, infinities and NaNs as they are).
#pragma once

#include <cstdint>

#include "elementwise.cuh"
#include "engine.h"
#include "slice_math.cuh"

namespace tdcc {

constexpr int kFxThreads = 256;
constexpr int kChunk = 60;                 // K per chunk: keeps the 64-bit sums below 2^63
constexpr int kExpLo = 101, kExpHi = 1946;  // biased exponents of a chunk maximum that scaling handles

// a real number of a chunk: its limbs, the remainder r and x = v 2^-56, both FP32
struct __align__(16) FxNum {
  int h, l;
  float r, x;
};

__device__ __forceinline__ void decode2(const ModeGroup& g, int l, long long& o0, long long& o1) {
  o0 = 0;
  o1 = 0;
  unsigned u = (unsigned)l;
#pragma unroll
  for (int q = kMaxModes - 1; q >= 0; --q) {
    if (q < g.n) {
      const unsigned d = (unsigned)g.dim[q];
      const unsigned w = q == 0 ? 0u : u / d;
      const unsigned r = q == 0 ? u : u - w * d;
      u = w;
      o0 += (long long)r * g.s0[q];
      o1 += (long long)r * g.s1[q];
    }
  }
}

// Upper word of |x|: its order is that of |x| down to the low word.
__device__ __forceinline__ unsigned upper_abs(double x) {
  return (unsigned)__double2hiint(x) & 0x7FFFFFFFu;
}

// x 2^(56 - e), e = Emax - 1022, as limbs and remainder: the significand
// left-justified in 64 bits, shifted down by Emax - E; h = bits 36.. rounded to
// nearest, l = the signed 28 bits below it, r = what rounding at bit 8 left.  A
// nonzero element too small for FP32 (2^-125 of the maximum) is marked by a NaN.
__device__ __forceinline__ FxNum cut_number(double x, int Emax) {
  const unsigned bh = (unsigned)__double2hiint(x), bl = (unsigned)__double2loint(x);
  const int E = (int)(bh >> 20) & 0x7FF;
  const unsigned d = (unsigned)(Emax - E);  // 0 .. 2046
  unsigned w2 = 0x80000000u | (bh << 11) | (bl >> 21), w1 = bl << 11, w0 = 0u;
  if (d >= 32u) {
    w0 = w1;
    w1 = w2;
    w2 = 0u;
  }
  const unsigned out = __funnelshift_r(w0, w1, d & 31u), ul = __funnelshift_r(w1, w2, d & 31u);
  unsigned uh = w2 >> (d & 31u);
  const unsigned rl = ul + 128u;  // round at bit 8
  uh += rl < ul ? 1u : 0u;
  int h = (int)((uh >> 4) + ((uh >> 3) & 1u));  // up to 2^28
  int l = (int)(__funnelshift_r(rl, uh, 8) << 4) >> 4;
  float r = (float)(int)((ul << 24) | (out >> 8)) * 0x1p-32f;
  float f = __uint_as_float(((126u - d) << 23) | ((bh & 0xFFFFFu) << 3) | (bl >> 29));
  if (E == 0 || d > 125u) f = ((bh << 1) | bl) == 0u ? 0.f : __uint_as_float(0x7FC00000u);
  if (E == 0 || d >= 64u) {
    h = l = 0;
    r = f * 0x1p56f;
  }
  const int s = (int)bh >> 31;
  FxNum q;
  q.h = (h ^ s) - s;
  q.l = (l ^ s) - s;
  q.r = s ? -r : r;
  q.x = s ? -f : f;
  return q;
}

__device__ __forceinline__ void imad(long long& c, int a, int b) { c += (long long)a * (long long)b; }

// The FP32 companions of a number: l 2^-28, and |x| 2^60 for the range guard.
struct FxAux {
  float l, g;
};
__device__ __forceinline__ FxAux fx_aux(const FxNum& a) {
  // (the integer l / 64 in the low bits of a number between 2 and 4)
  return {__int_as_float((a.l >> 6) + 0x40400000) - 3.f, fabsf(a.x) * 0x1p60f};
}

// One product into its sums: hh, mm the integers, f = sum l l' 2^-56 + x r' + r x',
// s = 2^120 sum |x x'|.
__device__ __forceinline__ void fx_mac(long long& hh, long long& mm, float& f, float& s, const FxNum& a, const FxAux& ax,
                                       const FxNum& b, const FxAux& bx) {
  imad(hh, a.h, b.h);
  imad(mm, a.h, b.l);
  imad(mm, a.l, b.h);
  f = fmaf(ax.l, bx.l, f);
  f = fmaf(a.x, b.r, f);
  f = fmaf(a.r, b.x, f);
  s = fmaf(ax.g, bx.g, s);
}

// The range guard.  FP32 leaves the small part f of a product off by some 2^-78 of
// the row maxima, so an output whose products' magnitudes add up to less than 2^-22
// a product (rows that fall along K by 10^6 against columns that rise by it) is
// done by FP64 multiply-adds instead.  s = 0 has no product that is not zero.
__device__ __forceinline__ bool out_of_range(float s, int K) { return !(s == 0.f || s >= 0x1p98f * (float)K); }

// (h 2^SH + m) 2^E as a double: the two sums joined in 64 bits at the top of
// their common magnitude, then rounded to nearest.
template <int SH = 28>
__device__ __forceinline__ double joined(long long h, long long m, int E) {
  const long long t = h + (m >> SH);                 // top part
  const unsigned long long lo = (unsigned long long)m & ((1ull << SH) - 1ull);  // SH bits below it
  const int lz = __clzll(t ^ (t >> 63)) - 1;         // redundant sign bits (63 for 0 and -1)
  const int s = lz < SH ? lz : SH;
  const long long X = (long long)(((unsigned long long)t << s) | (lo >> (SH - s)));
  return scaled_i64_to_double(X, E + SH - s);
}

__device__ __forceinline__ void fmac(double2& c, double2 a, double2 b) {
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(-a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(a.y, b.x, c.y);
}

template <bool CX>
__device__ __forceinline__ double2 load1(const double* p, long long off) {
  if constexpr (CX)
    return *reinterpret_cast<const double2*>(p + 2 * off);
  else
    return make_double2(p[off], 0.0);
}

// shared memory of a K index of a tile, rounded so that each operand's planes are
// whole; K indices per chunk: two blocks on an SM
__host__ __device__ __forceinline__ constexpr int fx_k_bytes(int bm, int bn, bool ac, bool bc) {
  return (int)sizeof(FxNum) * ((bm + 1) * (ac ? 2 : 1) + (bn + 1) * (bc ? 2 : 1));
}
__host__ __device__ __forceinline__ constexpr int fx_chunk(int bm, int bn, bool ac, bool bc) {
  const int k = 104 * 1024 / fx_k_bytes(bm, bn, ac, bc);
  return k < kChunk ? k : kChunk;
}

// This thread's elements of an R x kn piece of an operand (kn <= kChunk), all
// loads in flight at once and kept in registers between the exponent pass and
// the cutting; neighbouring threads take neighbouring k (kfast: k < 2^lw, no
// index division) or rows.
template <bool CX, int R>
struct Piece {
  static constexpr int U = R * 64 / kFxThreads;
  double x[U][CX ? 2 : 1];
  int at[U];  // row | k << 8, or -1
  __device__ __forceinline__ void load(const double* p, const long long* roff, const long long* koff, int kn, int lw,
                                       int kfast) {
    const unsigned total = kfast ? (unsigned)R << lw : (unsigned)(R * kn);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned i = threadIdx.x + (unsigned)kFxThreads * u;
      at[u] = -1;
      if (i < total) {
        const unsigned r = kfast ? i >> lw : i % R, k = kfast ? i & ((1u << lw) - 1u) : i / R;
        const long long o = roff[r];
        if (o >= 0 && k < (unsigned)kn) {
          at[u] = (int)(r | (k << 8));
          if constexpr (CX) {
            const double2 v = *reinterpret_cast<const double2*>(p + 2 * (o + koff[k]));
            x[u][0] = v.x;
            x[u][1] = v.y;
          } else {
            x[u][0] = p[o + koff[k]];
          }
        }
      }
    }
  }
  // the largest upper word of each row, met in shared memory; real and imaginary
  // parts are rows of their own (e[0][r], e[1][r])
  __device__ __forceinline__ void maxima(unsigned (*e)[64]) const {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0)
#pragma unroll
        for (int p = 0; p < (CX ? 2 : 1); ++p) {
          const unsigned w = upper_abs(x[u][p]);
          unsigned* q = &e[p][at[u] & 255];
          if (w > *(volatile unsigned*)q) atomicMax(q, w);
        }
  }
  // into planes [part][k][pitch]
  __device__ __forceinline__ void cut(FxNum* s, int pitch, int kc, const unsigned (*e)[64]) const {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0) {
        const int r = at[u] & 255, k = at[u] >> 8;
#pragma unroll
        for (int p = 0; p < (CX ? 2 : 1); ++p) s[(p * kc + k) * pitch + r] = cut_number(x[u][p], (int)(e[p][r] >> 20));
      }
  }
};

// Shared index tables of a tile.
struct FxScratch {
  long long aoff[64], boff[64], coffm[64], coffn[64];
  long long kofa[kChunk], kofb[kChunk];
  unsigned eA[2][64], eB[2][64];
};

// One tile (number `tile` of the output, batch and K split z) by a block of
// 256 threads on a 16 x 16 grid, TM x TN outputs each (rows ty + 16 i, columns
// tx + 16 j).  flags: bit 0 / 1: the K modes of A / B are the contiguous ones,
// so neighbouring threads load neighbouring k (else neighbouring rows).
// alpha = +-2^e2 when p2.  The scratch may be reused after a __syncthreads.
template <bool AC, bool BC, bool CC, int BM, int BN>
__device__ __forceinline__ void fx_tile(const GemmArgs& g, const FxPlan& f, unsigned tile, unsigned z,
                                        unsigned char* smraw, FxScratch& sh) {
  constexpr int TM = BM / 16, TN = BN / 16;
  constexpr bool CX = AC || BC;
  constexpr int NP = CX ? 2 : 1;
  constexpr int PA = BM + 1, PB = BN + 1;  // limb row pitches (a k-fast store strides by them)
  const int kc = f.kc, flags = f.flags, alpha_pow2 = f.p2, alpha_e = f.e2, alpha_neg = f.neg;
  FxNum* sA = reinterpret_cast<FxNum*>(smraw);       // [part][kc][PA]
  FxNum* sB = sA + (size_t)kc * PA * (AC ? 2 : 1);  // [part][kc][PB]
  long long *aoff = sh.aoff, *boff = sh.boff, *coffm = sh.coffm, *coffn = sh.coffn, *kofa = sh.kofa, *kofb = sh.kofb;
  unsigned (*eA)[64] = sh.eA, (*eB)[64] = sh.eB;  // upper word of each row's / column's chunk maximum
  const int tid = threadIdx.x;
  const int mt = (int)(tile % (unsigned)f.mtiles), nt = (int)(tile / (unsigned)f.mtiles);
  const int m0 = mt * BM, n0 = nt * BN;
  const int zb = (int)z / g.nsplit, ks = (int)z - zb * g.nsplit;
  const int kbeg = ks * g.kchunk, kend = min(g.K, kbeg + g.kchunk);
  const double* A = static_cast<const double*>(g.A) + (size_t)zb * g.bsA * (AC ? 2 : 1);
  const double* B = static_cast<const double*>(g.B) + (size_t)zb * g.bsB * (BC ? 2 : 1);
  const int tx = tid & 15, ty = tid >> 4;
  double sum[TM][TN][NP];
  for (int k0 = kbeg; k0 < kend; k0 += kc) {
    const int kn = min(kc, kend - k0);
    if (k0 != kbeg) __syncthreads();  // the previous chunk's limbs and offsets have been read
    // one thread per row, column and k (BM + BN + kc <= 156)
    if (tid < BM + BN) {
      if (tid < BM)
        eA[0][tid] = eA[1][tid] = 0;
      else
        eB[0][tid - BM] = eB[1][tid - BM] = 0;
      if (k0 == kbeg) {
        long long o0 = -1, o1 = -1;
        if (tid < BM) {
          if (m0 + tid < g.M) decode2(g.gm, m0 + tid, o0, o1);
          aoff[tid] = o0;
          coffm[tid] = o1;
        } else {
          if (n0 + tid - BM < g.N) decode2(g.gn, n0 + tid - BM, o0, o1);
          boff[tid - BM] = o0;
          coffn[tid - BM] = o1;
        }
      }
    } else if (tid < BM + BN + kn) {
      const int k = tid - BM - BN;
      decode2(g.gk, k0 + k, kofa[k], kofb[k]);
    }
    __syncthreads();
    Piece<AC, BM> pa;
    Piece<BC, BN> pb;
    const int lw = 32 - __clz(kn - 1 > 0 ? kn - 1 : 1);
    pa.load(A, aoff, kofa, kn, lw, flags & 1);
    pb.load(B, boff, kofb, kn, lw, flags & 2);
    pa.maxima(eA);
    pb.maxima(eB);
    __syncthreads();
    int bad = 0;
    if (tid < BM + BN)
      for (int p = 0; p < 2; ++p) {
        const unsigned w = tid < BM ? eA[p][tid] : eB[p][tid - BM];
        if (w != 0u && ((w >> 20) < (unsigned)kExpLo || (w >> 20) > (unsigned)kExpHi)) bad = 1;
      }
    bad = __syncthreads_or(bad);
    if (!bad) {
      pa.cut(sA, PA, kc, eA);
      pb.cut(sB, PB, kc, eB);
      __syncthreads();
    }
    // complex by complex: the real parts of A by B, then the imaginary parts (a
    // row's two parts have scales of their own)
#pragma unroll
    for (int pass = 0; pass < (AC && BC ? 2 : 1); ++pass) {
      // outputs to do in FP64, bit (i TN + j) NP + q: the whole chunk, or what the guard finds
      unsigned direct = 0u;
      double val[TM][TN][NP];
      if (!bad) {
        long long hh[TM][TN][NP], mm[TM][TN][NP];
        float fs[TM][TN][NP], gs[TM][TN][NP];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j)
#pragma unroll
            for (int p = 0; p < NP; ++p) {
              hh[i][j][p] = mm[i][j][p] = 0;
              fs[i][j][p] = gs[i][j][p] = 0.f;
            }
        // the parts of a complex operand by the real numbers of the other
        constexpr int QA = AC && !BC ? 2 : 1, QB = BC ? 2 : 1;
        const FxNum* ra = sA + (AC && BC ? (size_t)pass * kc * PA : 0) + ty;
        const FxNum* rb = sB + tx;
#pragma unroll 2
        for (int k = 0; k < kn; ++k) {
          FxNum a[TM][QA];
          FxAux ax[TM][QA];
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int p = 0; p < QA; ++p) {
              a[i][p] = ra[(p * kc + k) * PA + 16 * i];
              ax[i][p] = fx_aux(a[i][p]);
            }
#pragma unroll
          for (int j = 0; j < TN; ++j)
#pragma unroll
            for (int p = 0; p < QB; ++p) {
              const FxNum b = rb[(p * kc + k) * PB + 16 * j];
              const FxAux bx = fx_aux(b);
#pragma unroll
              for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int pp = 0; pp < QA; ++pp) {
                  const int q = QA == 2 ? pp : p;
                  fx_mac(hh[i][j][q], mm[i][j][q], fs[i][j][q], gs[i][j][q], a[i][pp], ax[i][pp], b, bx);
                }
            }
        }
        // each chunk is rounded to FP64 once
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j)
#pragma unroll
            for (int q = 0; q < NP; ++q) {
              // h carries 2^56 / 2^112: value = (h 2^28 + m) 2^(28 - 112 + ea + eb)
              const int E = (int)(eA[AC && !BC ? q : pass][ty + 16 * i] >> 20) + (int)(eB[BC ? q : 0][tx + 16 * j] >> 20) -
                            2 * 1022 - 84 + alpha_e;
              const long long h = hh[i][j][q], m = mm[i][j][q] + __float2ll_rn(fs[i][j][q] * 0x1p28f);
              val[i][j][q] = joined(alpha_neg ? -h : h, alpha_neg ? -m : m, E);
              if (out_of_range(gs[i][j][q], kn)) direct |= 1u << ((i * TN + j) * NP + q);
            }
      } else {
        direct = (1u << (TM * TN * NP)) - 1u;
      }
      // FP64 multiply-adds on the operands as they are
      while (direct) {
        const int bit = __ffs(direct) - 1, q = bit % NP, j = bit / NP % TN, i = bit / (NP * TN);
        direct &= direct - 1u;
        const long long ao = aoff[ty + 16 * i], bo = boff[tx + 16 * j];
        double s = 0.0;
        if (ao >= 0 && bo >= 0) {
          const double* x = A + (AC ? 2 * ao + (BC ? pass : q) : ao);
          const double* y = B + (BC ? 2 * bo + q : bo);
#pragma unroll 4
          for (int k = 0; k < kn; ++k) s = fma(x[(AC ? 2 : 1) * kofa[k]], y[(BC ? 2 : 1) * kofb[k]], s);
        }
        if (alpha_pow2) s *= g.ar;  // the sums below carry alpha
#pragma unroll
        for (int ii = 0; ii < TM; ++ii)
#pragma unroll
          for (int jj = 0; jj < TN; ++jj)
#pragma unroll
            for (int qq = 0; qq < NP; ++qq)
              if ((ii * TN + jj) * NP + qq == bit) val[ii][jj][qq] = s;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          double v[NP];
#pragma unroll
          for (int q = 0; q < NP; ++q) v[q] = val[i][j][q];
          if constexpr (AC && BC)
            if (pass == 1) {  // i (re + i im)
              v[0] = -val[i][j][1];
              v[1] = val[i][j][0];
            }
#pragma unroll
          for (int q = 0; q < NP; ++q) sum[i][j][q] = k0 == kbeg && pass == 0 ? v[q] : sum[i][j][q] + v[q];
        }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = ty + 16 * i;
    if (m0 + m >= g.M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = tx + 16 * j;
      if (n0 + n >= g.N) continue;
      const double2 s = make_double2(sum[i][j][0], CX ? sum[i][j][NP - 1] : 0.0);
      const long long off = coffm[m] + coffn[n];
      if constexpr (CC) {
        double2* C = static_cast<double2*>(g.C) + (size_t)zb * g.bsC;
        const double2 v = alpha_pow2 ? s : make_double2(g.ar * s.x - g.ai * s.y, g.ar * s.y + g.ai * s.x);
        if (g.atomic || g.acc) {  // L2 reductions (one writer per element unless split)
          atomicAdd(&C[off].x, v.x);
          atomicAdd(&C[off].y, v.y);
        } else {
          C[off] = v;
        }
      } else {
        double* C = static_cast<double*>(g.C) + (size_t)zb * g.bsC;
        const double v = alpha_pow2 ? s.x : g.ar * s.x;
        if (g.atomic || g.acc)
          atomicAdd(&C[off], v);
        else
          C[off] = v;
      }
    }
  }
}

// Small contractions, straight in FP64: 2^lw lanes per output share out its
// k and meet by shuffles; the K offsets of up to kDotK indices at a time are
// decoded once per block into shared memory.  A warp's FP64 instruction holds
// its scheduler's pipe for 64 clocks, so the lanes per output are as few as
// still give every scheduler of the chip a warp (fx_plan): the time is then
// (K / lanes x 2 or 4 + 2 lw) x 64 clocks plus a load's latency, 1-5 k clocks
// up to about a million multiply-adds, where a fixed-point tile takes 7-15 k
// whatever part of it is padding.
constexpr int kDotK = 1024;

template <bool AC, bool BC, bool CC>
__device__ __forceinline__ void dot_tile(const GemmArgs& g, const FxPlan& f, unsigned tile, unsigned z,
                                         unsigned char* smraw) {
  const int lw = f.flags, L = 1 << lw;  // lanes per output
  const int kcap = min(g.K, kDotK);
  long long* kofa = reinterpret_cast<long long*>(smraw);
  long long* kofb = kofa + kcap;
  const int tid = threadIdx.x, lane = tid & (L - 1);
  const long long out = (long long)tile * (kFxThreads >> lw) + (tid >> lw);
  const bool live = out < (long long)g.M * g.N;
  const double* A = static_cast<const double*>(g.A) + (size_t)z * g.bsA * (AC ? 2 : 1);
  const double* B = static_cast<const double*>(g.B) + (size_t)z * g.bsB * (BC ? 2 : 1);
  long long ao = 0, bo = 0, cm = 0, cn = 0;
  if (live) {
    const int m = (int)(out / g.N), n = (int)(out - (long long)m * g.N);
    decode2(g.gm, m, ao, cm);
    decode2(g.gn, n, bo, cn);
  }
  double2 s = make_double2(0.0, 0.0);
  for (int k0 = 0; k0 < g.K; k0 += kDotK) {
    const int kn = min(kDotK, g.K - k0);
    if (k0) __syncthreads();
    for (int k = tid; k < kn; k += kFxThreads) decode2(g.gk, k0 + k, kofa[k], kofb[k]);
    __syncthreads();
    if (live) {
      constexpr int U = 4;
      for (int k = lane; k < kn; k += U * L) {
        double2 x[U], y[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u * L < kn) {
            x[u] = load1<AC>(A, ao + kofa[k + u * L]);
            y[u] = load1<BC>(B, bo + kofb[k + u * L]);
          }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u * L < kn) {
            if constexpr (AC && BC) {
              fmac(s, x[u], y[u]);
            } else if constexpr (AC) {
              s.x = fma(x[u].x, y[u].x, s.x);
              s.y = fma(x[u].y, y[u].x, s.y);
            } else {
              s.x = fma(x[u].x, y[u].x, s.x);
              if constexpr (BC) s.y = fma(x[u].x, y[u].y, s.y);
            }
          }
      }
    }
  }
  for (int d = L >> 1; d > 0; d >>= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, d);
    if constexpr (AC || BC) s.y += __shfl_xor_sync(0xffffffffu, s.y, d);
  }
  if (!live || lane != 0) return;
  if (f.p2) {
    const unsigned long long sgn = f.neg ? 0x8000000000000000ull : 0ull;
    if (f.e2 != 0 || f.neg) {
      s.x = scale_pow2(s.x, g.ar, sgn, f.e2);
      s.y = scale_pow2(s.y, g.ar, sgn, f.e2);
    }
  } else {
    s = make_double2(g.ar * s.x - g.ai * s.y, g.ar * s.y + g.ai * s.x);
  }
  const long long off = cm + cn;
  if constexpr (CC) {
    double2* C = static_cast<double2*>(g.C) + (size_t)z * g.bsC;
    if (g.acc) {
      atomicAdd(&C[off].x, s.x);
      atomicAdd(&C[off].y, s.y);
    } else {
      C[off] = s;
    }
  } else {
    double* C = static_cast<double*>(g.C) + (size_t)z * g.bsC;
    if (g.acc)
      atomicAdd(&C[off], s.x);
    else
      C[off] = s.x;
  }
}

}  // namespace tdcc
