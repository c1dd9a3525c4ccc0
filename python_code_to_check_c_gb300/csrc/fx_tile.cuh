// FP64 contractions on the integer pipe: block fixed point with exact sums.
//
// GB300's FP64 pipe does 1.9 multiply-adds per clock and SM (0.58 T/s for the
// chip), its integer pipe 26 of 32 x 32 + 64 bits (both measured, operands
// from shared memory).  So a
// contraction C[m,n] (+)= alpha sum_k A[m,k] B[k,n] is cut into K chunks of
// at most 60; in a chunk each row of A and column of B is scaled by the power
// of two above its largest magnitude (real and imaginary parts share it) and
// written as v = h 2^28 + l, |v| < 2^56, |h| <= 2^28, -2^27 <= l < 2^27: 56
// bits, three more than an FP64 significand at the row's maximum.  A product
// is h h' 2^56 + (h l' + l h') 2^28, three multiply-adds into two 64-bit sums
// that cannot overflow (2 x 60 terms of 2^56, 4 x 60 of 2^55); l l', at most
// 2^-58 of the product of the two maxima and of either sign, is left out.
// The sums are exact; each chunk is rounded to FP64 once, where an FP64 chain
// rounds every term, so the error against 64 bits is no larger than the
// FP64 kernel's (measured over both on the residuals' own operands and on
// random ones, K = 2..2000).
//
// Bound: the integer multiply-adds, at 85-90 % of that rate while they run
// (a complex 16 x 16 x 60 tile: 8.5 of 16.4 k clocks), then index
// work and cutting; 16 warps (512 threads, 64 registers) gain 8 % on one tile
// and lose 5 % on many.  Against the FP64 kernel it replaced (64 x 64 tile, at 96
// % of the FP64 pipe), one launch: real 2304 x 2304 x 144 1324 -> 484 us;
// complex by real 1444 x 100 x 1444 1450 -> 320 us; the T2 residual at o=10,
// v=38 5.13 -> 1.66 ms.
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

template <bool AC>
struct Limbs;  // one element: h, l (and the imaginary part's h, l)
template <>
struct Limbs<true> {
  using T = int4;
};
template <>
struct Limbs<false> {
  using T = int2;
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

// x 2^(56 - e) rounded to an integer, e = Emax - 1022, as limbs h, l: the
// significand left-justified in 64 bits, shifted down by Emax - E; h = bits
// 36.. rounded to nearest, l = the signed 28 bits below it.
__device__ __forceinline__ int2 limbs(double x, int Emax) {
  const unsigned bh = (unsigned)__double2hiint(x), bl = (unsigned)__double2loint(x);
  const int E = (int)(bh >> 20) & 0x7FF;
  const unsigned d = (unsigned)(Emax - E);  // 0 .. 2046
  unsigned uh = 0x80000000u | (bh << 11) | (bl >> 21), ul = bl << 11;
  if (d >= 32u) {
    ul = uh;
    uh = 0u;
  }
  ul = __funnelshift_r(ul, uh, d & 31u);
  uh >>= (d & 31u);
  if (d >= 64u || E == 0) uh = ul = 0u;
  const unsigned rl = ul + 128u;  // round at bit 8
  uh += rl < ul ? 1u : 0u;
  int h = (int)((uh >> 4) + ((uh >> 3) & 1u));  // up to 2^28
  int l = (int)(__funnelshift_r(rl, uh, 8) << 4) >> 4;
  const int s = (int)bh >> 31;
  return make_int2((h ^ s) - s, (l ^ s) - s);
}

__device__ __forceinline__ void imad(long long& c, int a, int b) { c += (long long)a * (long long)b; }

// one product into its sums: hh and mm hold the real (and imaginary) part
template <bool AC, bool BC, int NP>
__device__ __forceinline__ void fx_mac(long long (&hh)[NP], long long (&mm)[NP], const typename Limbs<AC>::T& a,
                                       const typename Limbs<BC>::T& b) {
  imad(hh[0], a.x, b.x);
  imad(mm[0], a.x, b.y);
  imad(mm[0], a.y, b.x);
  if constexpr (AC && BC) {
    const int nh = -a.z, nl = -a.w;
    imad(hh[1], a.x, b.z);
    imad(mm[1], a.x, b.w);
    imad(mm[1], a.y, b.z);
    imad(hh[0], nh, b.z);
    imad(mm[0], nh, b.w);
    imad(mm[0], nl, b.z);
    imad(hh[1], a.z, b.x);
    imad(mm[1], a.z, b.y);
    imad(mm[1], a.w, b.x);
  } else if constexpr (AC) {
    imad(hh[1], a.z, b.x);
    imad(mm[1], a.z, b.y);
    imad(mm[1], a.w, b.x);
  } else if constexpr (BC) {
    imad(hh[1], a.x, b.z);
    imad(mm[1], a.x, b.w);
    imad(mm[1], a.y, b.z);
  }
}

// (h 2^28 + m) 2^E as a double: the two sums joined in 64 bits at the top of
// their common magnitude, then rounded to nearest.
__device__ __forceinline__ double joined(long long h, long long m, int E) {
  const long long t = h + (m >> 28);                 // top part
  const unsigned long long lo = (unsigned long long)m & 0xFFFFFFFull;  // 28 bits below it
  const int lz = __clzll(t ^ (t >> 63)) - 1;         // redundant sign bits (63 for 0 and -1)
  const int s = lz < 28 ? lz : 28;
  const long long X = (long long)(((unsigned long long)t << s) | (lo >> (28 - s)));
  return scaled_i64_to_double(X, E + 28 - s);
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

// bytes of kc rows of limbs, rounded so that what follows is 16-byte aligned
__host__ __device__ __forceinline__ size_t limb_bytes(int kc, int pitch, size_t esz) {
  return ((size_t)kc * pitch * esz + 15) & ~(size_t)15;
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
  // the largest upper word of each row, met in shared memory
  __device__ __forceinline__ void maxima(unsigned* e) const {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0) {
        unsigned w = upper_abs(x[u][0]);
        if constexpr (CX) w = max(w, upper_abs(x[u][1]));
        unsigned* q = &e[at[u] & 255];
        if (w > *(volatile unsigned*)q) atomicMax(q, w);
      }
  }
  template <class L>
  __device__ __forceinline__ void cut(L* s, int pitch, const unsigned* e) const {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0) {
        const int r = at[u] & 255, k = at[u] >> 8;
        const int Em = (int)(e[r] >> 20);
        const int2 h = limbs(x[u][0], Em);
        if constexpr (CX) {
          const int2 q = limbs(x[u][1], Em);
          s[k * pitch + r] = make_int4(h.x, h.y, q.x, q.y);
        } else {
          s[k * pitch + r] = h;
        }
      }
  }
};

// Shared index tables of a tile.
struct FxScratch {
  long long aoff[64], boff[64], coffm[64], coffn[64];
  long long kofa[kChunk], kofb[kChunk];
  unsigned eA[64], eB[64];
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
  using LA = typename Limbs<AC>::T;
  using LB = typename Limbs<BC>::T;
  constexpr int PA = BM + 1, PB = BN + 1;  // limb row pitches (a k-fast store strides by them)
  const int kc = f.kc, flags = f.flags, alpha_pow2 = f.p2, alpha_e = f.e2, alpha_neg = f.neg;
  LA* sA = reinterpret_cast<LA*>(smraw);                                      // [kc][PA]
  LB* sB = reinterpret_cast<LB*>(smraw + limb_bytes(kc, PA, sizeof(LA)));       // [kc][PB]
  long long *aoff = sh.aoff, *boff = sh.boff, *coffm = sh.coffm, *coffn = sh.coffn, *kofa = sh.kofa, *kofb = sh.kofb;
  unsigned *eA = sh.eA, *eB = sh.eB;  // upper word of each row's / column's chunk maximum
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
        eA[tid] = 0;
      else
        eB[tid - BM] = 0;
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
    if (tid < BM + BN) {
      const unsigned w = tid < BM ? eA[tid] : eB[tid - BM];
      if (w != 0u && ((w >> 20) < (unsigned)kExpLo || (w >> 20) > (unsigned)kExpHi)) bad = 1;
    }
    if (__syncthreads_or(bad)) {
      // FP64 multiply-adds on the operands as they are
      for (int i = 0; i < TM; ++i)
        for (int j = 0; j < TN; ++j) {
          const long long ao = aoff[ty + 16 * i], bo = boff[tx + 16 * j];
          double2 s = make_double2(0.0, 0.0);
          if (ao >= 0 && bo >= 0)
            for (int k = 0; k < kn; ++k) {
              const double2 x = load1<AC>(A, ao + kofa[k]), y = load1<BC>(B, bo + kofb[k]);
              if constexpr (AC && BC)
                fmac(s, x, y);
              else if constexpr (AC)
                s = make_double2(fma(x.x, y.x, s.x), fma(x.y, y.x, s.y));
              else
                s = make_double2(fma(x.x, y.x, s.x), fma(x.x, y.y, s.y));
            }
          if (alpha_pow2) {  // the sums below carry alpha
            s.x *= g.ar;
            s.y *= g.ar;
          }
#pragma unroll
          for (int ii = 0; ii < TM; ++ii)
#pragma unroll
            for (int jj = 0; jj < TN; ++jj)
              if (ii == i && jj == j) {
                sum[ii][jj][0] = k0 == kbeg ? s.x : sum[ii][jj][0] + s.x;
                if constexpr (CX) sum[ii][jj][1] = k0 == kbeg ? s.y : sum[ii][jj][1] + s.y;
              }
        }
      continue;
    }
    pa.cut(sA, PA, eA);
    pb.cut(sB, PB, eB);
    __syncthreads();
    long long hh[TM][TN][NP], mm[TM][TN][NP];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int p = 0; p < NP; ++p) hh[i][j][p] = mm[i][j][p] = 0;
#pragma unroll 2
    for (int k = 0; k < kn; ++k) {
      LA a[TM];
      LB b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = sA[k * PA + ty + 16 * i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = sB[k * PB + tx + 16 * j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) fx_mac<AC, BC>(hh[i][j], mm[i][j], a[i], b[j]);
    }
    // each chunk is rounded to FP64 once
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        // h carries 2^56 / 2^112: value = (h 2^28 + m) 2^(28 - 112 + ea + eb)
        const int E = (int)(eA[ty + 16 * i] >> 20) + (int)(eB[tx + 16 * j] >> 20) - 2 * 1022 - 84 + alpha_e;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const long long h = alpha_neg ? -hh[i][j][p] : hh[i][j][p], m = alpha_neg ? -mm[i][j][p] : mm[i][j][p];
          const double x = joined(h, m, E);
          sum[i][j][p] = k0 == kbeg ? x : sum[i][j][p] + x;
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
