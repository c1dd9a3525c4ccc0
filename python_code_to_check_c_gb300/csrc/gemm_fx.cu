// FP64 contractions on the integer pipe: block fixed point with exact sums.
//
// GB300's FP64 pipe does 1.9 FMA per clock and SM (measured; 0.58 T FMA/s for
// the chip), its integer pipe 55 multiply-adds of 32 x 32 + 64 bits.  So a
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
// Bound: issue slots (cutting the limbs, index work) beside the integer
// multiply-adds, 27 % of the instructions of a 32 x 64 real tile at K = 48 a
// chunk (ncu: issue 45 %, 2 blocks of 8 warps per SM).  Against the FP64
// kernel it replaced (64 x 64 tile, at 96 % of the FP64 pipe), one launch:
// real 2304 x 2304 x 144 1324 -> 484 us; complex by real 1444 x 100 x 1444
// 1450 -> 320 us; whole calls: the T2 residual at o=10, v=38 5.13 -> 1.66 ms,
// eight steps at o=10, v=14 14.1 -> 7.4 ms.
//
// A chunk whose maxima are not finite, or so large or small that scaling by
// them would leave the normal range, is done by FP64 multiply-adds from
// global memory instead (the same operands, infinities and NaNs as they are).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <utility>

#include "engine.h"
#include "slice_math.cuh"

namespace tdcc {

namespace {

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
  static constexpr int U = R * 64 / 256;
  double x[U][CX ? 2 : 1];
  int at[U];  // row | k << 8, or -1
  __device__ __forceinline__ void load(const double* p, const long long* roff, const long long* koff, int kn, int lw,
                                       int kfast) {
    const unsigned total = kfast ? (unsigned)R << lw : (unsigned)(R * kn);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned i = threadIdx.x + 256u * u;
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

}  // namespace

// BM x BN outputs per block of 256 threads on a 16 x 16 grid, TM x TN each
// (rows ty + 16 i, columns tx + 16 j).  flags: bit 0 / 1: the K modes of A / B
// are the contiguous ones, so neighbouring threads load neighbouring k (else
// neighbouring rows).  alpha = +-2^alpha_e when alpha_pow2.
template <bool AC, bool BC, bool CC, int BM, int BN>
__global__ void __launch_bounds__(256, 2) gemm_fx_kernel(const GemmArgs g, int mtiles, int kc, int flags, int alpha_pow2,
                                                      int alpha_e, int alpha_neg) {
  constexpr int TM = BM / 16, TN = BN / 16;
  constexpr bool CX = AC || BC;
  constexpr int NP = CX ? 2 : 1;
  using LA = typename Limbs<AC>::T;
  using LB = typename Limbs<BC>::T;
  constexpr int PA = BM + 1, PB = BN + 1;  // limb row pitches (a k-fast store strides by them)
  extern __shared__ __align__(16) unsigned char smraw[];
  LA* sA = reinterpret_cast<LA*>(smraw);                                      // [kc][PA]
  LB* sB = reinterpret_cast<LB*>(smraw + limb_bytes(kc, PA, sizeof(LA)));       // [kc][PB]
  __shared__ long long aoff[BM], boff[BN], coffm[BM], coffn[BN];
  __shared__ long long kofa[kChunk], kofb[kChunk];
  __shared__ unsigned eA[BM], eB[BN];  // upper word of each row's / column's chunk maximum
  const int tid = threadIdx.x;
  const int mt = (int)(blockIdx.x % (unsigned)mtiles), nt = (int)(blockIdx.x / (unsigned)mtiles);
  const int m0 = mt * BM, n0 = nt * BN;
  const int zb = blockIdx.z / g.nsplit, ks = blockIdx.z - zb * g.nsplit;
  const int kbeg = ks * g.kchunk, kend = min(g.K, kbeg + g.kchunk);
  const double* A = static_cast<const double*>(g.A) + (size_t)zb * g.bsA * (AC ? 2 : 1);
  const double* B = static_cast<const double*>(g.B) + (size_t)zb * g.bsB * (BC ? 2 : 1);
  for (int i = tid; i < BM + BN; i += 256) {
    long long o0 = -1, o1 = -1;
    if (i < BM) {
      if (m0 + i < g.M) decode2(g.gm, m0 + i, o0, o1);
      aoff[i] = o0;
      coffm[i] = o1;
    } else {
      if (n0 + i - BM < g.N) decode2(g.gn, n0 + i - BM, o0, o1);
      boff[i - BM] = o0;
      coffn[i - BM] = o1;
    }
  }
  const int tx = tid & 15, ty = tid >> 4;
  double sum[TM][TN][NP];
  for (int k0 = kbeg; k0 < kend; k0 += kc) {
    const int kn = min(kc, kend - k0);
    if (k0 != kbeg) __syncthreads();  // the previous chunk's limbs and offsets have been read
    for (int i = tid; i < kn; i += 256) decode2(g.gk, k0 + i, kofa[i], kofb[i]);
    for (int i = tid; i < BM + BN; i += 256) {
      if (i < BM)
        eA[i] = 0;
      else
        eB[i - BM] = 0;
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
    for (int i = tid; i < BM + BN; i += 256) {
      const unsigned w = i < BM ? eA[i] : eB[i - BM];
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
        for (int j = 0; j < TN; ++j) {
          imad(hh[i][j][0], a[i].x, b[j].x);
          imad(mm[i][j][0], a[i].x, b[j].y);
          imad(mm[i][j][0], a[i].y, b[j].x);
          if constexpr (AC && BC) {
            const int nh = -a[i].z, nl = -a[i].w;
            imad(hh[i][j][0], nh, b[j].z);
            imad(mm[i][j][0], nh, b[j].w);
            imad(mm[i][j][0], nl, b[j].z);
            imad(hh[i][j][1], a[i].x, b[j].z);
            imad(mm[i][j][1], a[i].x, b[j].w);
            imad(mm[i][j][1], a[i].y, b[j].z);
            imad(hh[i][j][1], a[i].z, b[j].x);
            imad(mm[i][j][1], a[i].z, b[j].y);
            imad(mm[i][j][1], a[i].w, b[j].x);
          } else if constexpr (AC) {
            imad(hh[i][j][1], a[i].z, b[j].x);
            imad(mm[i][j][1], a[i].z, b[j].y);
            imad(mm[i][j][1], a[i].w, b[j].x);
          } else if constexpr (BC) {
            imad(hh[i][j][1], a[i].x, b[j].z);
            imad(mm[i][j][1], a[i].x, b[j].w);
            imad(mm[i][j][1], a[i].y, b[j].z);
          }
        }
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

// Output tiles {BM, BN}: a block's cutting work grows with BM + BN and its
// multiply-adds with BM BN; the narrow ones serve outputs with a side of o.
// The last one for real operands only (complex sums of 2 x 4 outputs a thread
// would not fit the registers).
const int kTiles[kNumTiles][2] = {{32, 32}, {16, 64}, {64, 16}, {16, 16}, {32, 64}};

bool tile_fits(int t, bool real) { return t >= 0 && t < kNumTiles && (t != 4 || real); }

// Tile and K splits of a contraction.  A block's time is a fixed part (index
// decoding, the loads, the stores), the cutting of its operands and its
// multiply-adds; blocks beyond one per SM share the SM's pipes.  All in SM
// clocks, from the rates above; splits cost a second pass of the outputs
// through L2 and, when not accumulating, a zeroing launch before.
void choose_fx(long long M, long long N, long long K, long long nb, bool ac, bool bc, bool allow_split, int tile,
               int* best_tile, int* best_splits) {
  const double im = (ac && bc) ? 12.0 : (ac || bc) ? 6.0 : 3.0;
  double best = 1e300;
  *best_tile = 0;
  *best_splits = 1;
  for (int t = 0; t < kNumTiles; ++t) {
    if (tile >= 0 && t != tile) continue;
    if (!tile_fits(t, !ac && !bc)) continue;
    const long long bm = kTiles[t][0], bn = kTiles[t][1];
    const long long tiles = ((M + bm - 1) / bm) * ((N + bn - 1) / bn) * nb;
    for (long long sp = 1; sp <= (allow_split ? std::max<long long>(1, K / 16) : 1); sp += sp < 8 ? 1 : sp / 4) {
      const long long kper = (K + sp - 1) / sp, chunks = (kper + kChunk - 1) / kChunk;
      const double fixed = 3000.0 + 1500.0 * (double)(chunks - 1) + (sp > 1 ? 2500.0 : 0.0);
      const double cut = (double)kper * (double)(bm * (ac ? 2 : 1) + bn * (bc ? 2 : 1)) * 30.0 / 128.0;
      const double mul = (double)(bm * bn) * (double)kper * im / 55.0;
      const double out = (double)(bm * bn) * (double)chunks * 1.2 + (sp > 1 ? (double)(bm * bn) * 0.5 : 0.0);
      const double per_sm = std::ceil((double)(tiles * sp) / 152.0);
      const double cost = fixed + per_sm * (cut + mul + out + 400.0);
      if (cost < best * 0.999) {
        best = cost;
        *best_tile = t;
        *best_splits = (int)sp;
      }
    }
  }
}

namespace {

template <bool AC, bool BC, bool CC, int BM, int BN>
cudaError_t launch_fx_tile(const GemmArgs& g, int kc, int flags, int p2, int e2, int neg, cudaStream_t st) {
  constexpr size_t ea = sizeof(typename Limbs<AC>::T), eb = sizeof(typename Limbs<BC>::T);
  constexpr int kMaxDev = 64;
  static std::once_flag once[kMaxDev];
  static cudaError_t attr_err[kMaxDev] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [dev] {
    attr_err[dev] =
        cudaFuncSetAttribute(gemm_fx_kernel<AC, BC, CC, BM, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(limb_bytes(kChunk, BM + 1, ea) + limb_bytes(kChunk, BN + 1, eb)));
  });
  if (attr_err[dev] != cudaSuccess) return attr_err[dev];
  const long long mt = (g.M + BM - 1) / BM, nt = (g.N + BN - 1) / BN, z = (long long)g.nb * g.nsplit;
  if (mt * nt > 0x7FFFFFFFLL || z > 65535) return cudaErrorInvalidConfiguration;
  const size_t smem = limb_bytes(kc, BM + 1, ea) + limb_bytes(kc, BN + 1, eb);
  gemm_fx_kernel<AC, BC, CC, BM, BN><<<dim3((unsigned)(mt * nt), 1, (unsigned)z), 256, smem, st>>>(g, (int)mt, kc, flags,
                                                                                                 p2, e2, neg);
  return cudaGetLastError();
}

template <bool AC, bool BC, bool CC>
cudaError_t launch_fx_typed(int tile, const GemmArgs& g, int kc, int flags, int p2, int e2, int neg, cudaStream_t st) {
  if constexpr (!AC && !BC)
    if (tile == 4) return launch_fx_tile<AC, BC, CC, 32, 64>(g, kc, flags, p2, e2, neg, st);
  switch (tile) {
    case 0: return launch_fx_tile<AC, BC, CC, 32, 32>(g, kc, flags, p2, e2, neg, st);
    case 1: return launch_fx_tile<AC, BC, CC, 16, 64>(g, kc, flags, p2, e2, neg, st);
    case 2: return launch_fx_tile<AC, BC, CC, 64, 16>(g, kc, flags, p2, e2, neg, st);
    case 3: return launch_fx_tile<AC, BC, CC, 16, 16>(g, kc, flags, p2, e2, neg, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_gemm(const Op& op, const void* A, const void* B, void* C, cudaStream_t st) {
  GemmArgs g = op.g;
  g.A = A;
  g.B = B;
  g.C = C;
  bool ac = op.dta == C64, bc = op.dtb == C64;
  const bool cc = op.dtc == C64;
  int tile = op.tile;
  if (!cc && (ac || bc)) return cudaErrorInvalidValue;
  if (g.nb < 1) g.nb = 1;
  if (g.nsplit < 1) g.nsplit = 1;
  if ((long long)g.nsplit * g.kchunk < g.K) return cudaErrorInvalidValue;
  // neighbouring threads store neighbouring columns: the operand that carries
  // the output's contiguous mode becomes B (C^T = B^T A^T)
  auto unit = [](const ModeGroup& q) { return q.n > 0 && q.s1[q.n - 1] == 1 && q.dim[q.n - 1] > 1; };
  if (!unit(g.gn) && unit(g.gm)) {
    std::swap(g.gm, g.gn);
    std::swap(g.M, g.N);
    std::swap(g.A, g.B);
    std::swap(g.bsA, g.bsB);
    std::swap(ac, bc);
    for (int i = 0; i < kMaxModes; ++i) std::swap(g.gk.s0[i], g.gk.s1[i]);
    tile = tile == 1 ? 2 : tile == 2 ? 1 : tile;  // {32, 64} serves both orders
  }
  const int chunks = (g.kchunk + kChunk - 1) / kChunk;
  const int kc = std::min(kChunk, (std::min(g.kchunk, std::max(g.K, 1)) + chunks - 1) / chunks);
  auto kfast = [&](const long long* ks, const ModeGroup& rows) {
    const int q = g.gk.n - 1;
    if (q < 0 || ks[q] != 1 || g.gk.dim[q] < 4) return 0;
    return (rows.n > 0 && rows.s0[rows.n - 1] == 1 && rows.dim[rows.n - 1] > 1) ? 0 : 1;
  };
  const int flags = kfast(g.gk.s0, g.gm) | (kfast(g.gk.s1, g.gn) << 1);
  int e2 = 0;
  const double fr = std::frexp(std::fabs(g.ar), &e2);
  const int p2 = (g.ai == 0.0 && fr == 0.5) ? 1 : 0;
  e2 = p2 ? e2 - 1 : 0;
  const int neg = (p2 && g.ar < 0.0) ? 1 : 0;
  cudaError_t e;
  if (ac && bc)
    e = launch_fx_typed<true, true, true>(tile, g, kc, flags, p2, e2, neg, st);
  else if (ac)
    e = launch_fx_typed<true, false, true>(tile, g, kc, flags, p2, e2, neg, st);
  else if (bc)
    e = launch_fx_typed<false, true, true>(tile, g, kc, flags, p2, e2, neg, st);
  else if (cc)
    e = launch_fx_typed<false, false, true>(tile, g, kc, flags, p2, e2, neg, st);
  else
    e = launch_fx_typed<false, false, false>(tile, g, kc, flags, p2, e2, neg, st);
  count_launch();
  return e;
}

}  // namespace tdcc
