// Launches of the fixed-point contraction (fx_tile.cuh): tile shapes, the
// choice of a shape and K splits, and the kernel entry points.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <utility>

#include "engine.h"
#include "fx_tile.cuh"

namespace tdcc {

// Output tiles {BM, BN}: a block's cutting work grows with BM + BN and its
// multiply-adds with BM BN; the narrow ones serve outputs with a side of o,
// the fifth real operands only (complex sums of 2 x 2 outputs a thread would
// not fit the registers).  The last is no tile: FP64 dot products.
const int kTiles[kNumTiles][2] = {{32, 32}, {16, 64}, {64, 16}, {16, 16}, {32, 64}, {1, 1}};

bool tile_fits(int t, bool real) { return t >= 0 && t < kNumTiles && (t != 4 || real); }

// log2 of the lanes per output of a dot product: as few as give the chip's
// 608 schedulers a warp each, at most one lane per two k
int dot_lanes(long long outputs, long long K) {
  int lw = 0;
  while (lw < 5 && (outputs << lw) < 608LL * 32 && (K >> (lw + 1)) >= 2) ++lw;
  return lw;
}

// clocks of the dot products (dot_tile) with 2^lw lanes per output
double dot_cost(long long outputs, long long K, int lw, bool ac, bool bc) {
  const double warps = std::ceil((double)outputs * (double)(1 << lw) / 32.0);
  const double per = std::ceil((double)K / (double)(1 << lw)) * ((ac && bc) ? 4.0 : (ac || bc) ? 2.0 : 1.0) + 2.0 * lw;
  return 2200.0 + std::ceil(warps / 608.0) * per * 66.0;
}

// Form and K splits of a contraction, by a model in SM clocks.  Fixed-point
// tiles: a fixed part (index decoding, the loads' latency, the stores), the
// cutting of its operands and its multiply-adds; blocks beyond one per SM
// share the SM's pipes; splits cost a second pass of the outputs through L2
// and, when not accumulating, a zeroing launch before.  Dot products: see
// dot_tile.  The rates are fitted to whole calls, whose ops run several at a
// time.  Integer multiply-adds a clock and cutting clocks a number (26, 0.7) against
// (40, 0.3) and (31, 0.45): a gradient of 8 steps at o=6, v=12 17.7 ms, 22.7 and 26.4;
// the propagation at o=10, v=14 10.06 ms for 8 steps, 9.81 and 9.96; 60 residuals of
// o=5..14, v=14..50 32.7 ms in all, 32.9 and 32.8.
double choose_fx(long long M, long long N, long long K, long long nb, bool ac, bool bc, bool allow_split, int tile,
                 int* best_tile, int* best_splits) {
  const double im = (ac && bc) ? 12.0 : (ac || bc) ? 6.0 : 3.0;
  double best = 1e300;
  *best_tile = 0;
  *best_splits = 1;
  for (int t = 0; t < kNumTiles; ++t) {
    if (tile >= 0 && t != tile) continue;
    if (tile == -2 && t != 3) continue;  // the shape of the phase kernel
    if (t == 5 && tile != -3) continue;
    if (!tile_fits(t, !ac && !bc)) continue;
    if (t == 5) {
      const double cost = dot_cost(M * N * nb, K, dot_lanes(M * N * nb, K), ac, bc);
      if (cost < best * 0.999) {
        best = cost;
        *best_tile = t;
        *best_splits = 1;
      }
      continue;
    }
    const long long bm = kTiles[t][0], bn = kTiles[t][1];
    const long long tiles = ((M + bm - 1) / bm) * ((N + bn - 1) / bn) * nb;
    for (long long sp = 1; sp <= (allow_split ? std::max<long long>(1, K / 16) : 1); sp += sp < 8 ? 1 : sp / 4) {
      const long long kper = (K + sp - 1) / sp, most = fx_chunk((int)bm, (int)bn, ac, bc), chunks = (kper + most - 1) / most;
      const double fixed = 3400.0 + 1500.0 * (double)(chunks - 1) + (sp > 1 ? 2500.0 : 0.0);
      const double cut = (double)kper * (double)(bm * (ac ? 2 : 1) + bn * (bc ? 2 : 1)) * 0.7;
      const double mul = (double)(bm * bn) * (double)kper * im / 26.0;
      const double out = (double)(bm * bn) * (double)chunks * 1.2 + (sp > 1 ? (double)(bm * bn) * 0.5 : 0.0);
      const double per_sm = std::ceil((double)(tiles * sp) / 152.0);
      const double cost = fixed + cut / (double)chunks + per_sm * (cut + mul + out + 400.0);
      if (cost < best * 0.999) {
        best = cost;
        *best_tile = t;
        *best_splits = (int)sp;
      }
    }
  }
  return best;
}

namespace {

template <bool AC, bool BC, bool CC, int BM, int BN>
__global__ void __launch_bounds__(kFxThreads, 2) gemm_fx_kernel(const GemmArgs g, const FxPlan f) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ FxScratch sh;
  fx_tile<AC, BC, CC, BM, BN>(g, f, blockIdx.x, blockIdx.z, smraw, sh);
}

template <bool AC, bool BC, bool CC, int BM, int BN>
cudaError_t launch_fx_tile(const GemmArgs& g, const FxPlan& f, cudaStream_t st) {
  constexpr int kbytes = fx_k_bytes(BM, BN, AC, BC);
  constexpr int kMaxDev = 64;
  static std::once_flag once[kMaxDev];
  static cudaError_t attr_err[kMaxDev] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [dev] {
    attr_err[dev] =
        cudaFuncSetAttribute(gemm_fx_kernel<AC, BC, CC, BM, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kbytes * fx_chunk(BM, BN, AC, BC));
  });
  if (attr_err[dev] != cudaSuccess) return attr_err[dev];
  const long long z = (long long)g.nb * g.nsplit;
  if (f.tiles > 0x7FFFFFFFLL || z > 65535) return cudaErrorInvalidConfiguration;
  const size_t smem = (size_t)kbytes * f.kc;
  gemm_fx_kernel<AC, BC, CC, BM, BN><<<dim3((unsigned)f.tiles, 1, (unsigned)z), kFxThreads, smem, st>>>(g, f);
  return cudaGetLastError();
}

template <bool AC, bool BC, bool CC>
__global__ void __launch_bounds__(kFxThreads, 2) gemm_dot_kernel(const GemmArgs g, const FxPlan f) {
  extern __shared__ __align__(16) unsigned char smraw[];
  dot_tile<AC, BC, CC>(g, f, blockIdx.x, blockIdx.z, smraw);
}

template <bool AC, bool BC, bool CC>
cudaError_t launch_fx_typed(const GemmArgs& g, const FxPlan& f, cudaStream_t st) {
  if (f.tile == 5) {
    if (f.tiles > 0x7FFFFFFFLL || g.nb > 65535) return cudaErrorInvalidConfiguration;
    gemm_dot_kernel<AC, BC, CC><<<dim3((unsigned)f.tiles, 1, (unsigned)g.nb), kFxThreads, f.kc, st>>>(g, f);
    return cudaGetLastError();
  }
  if constexpr (!AC && !BC)
    if (f.tile == 4) return launch_fx_tile<AC, BC, CC, 32, 64>(g, f, st);
  switch (f.tile) {
    case 0: return launch_fx_tile<AC, BC, CC, 32, 32>(g, f, st);
    case 1: return launch_fx_tile<AC, BC, CC, 16, 64>(g, f, st);
    case 2: return launch_fx_tile<AC, BC, CC, 64, 16>(g, f, st);
    case 3: return launch_fx_tile<AC, BC, CC, 16, 16>(g, f, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t fx_plan(const Op& op, GemmArgs& g, FxPlan& f) {
  g = op.g;
  f = FxPlan{};
  f.ac = op.dta == C64;
  f.bc = op.dtb == C64;
  f.cc = op.dtc == C64;
  f.tile = op.tile;
  if (!f.cc && (f.ac || f.bc)) return cudaErrorInvalidValue;
  if (g.nb < 1) g.nb = 1;
  if (g.nsplit < 1) g.nsplit = 1;
  if ((long long)g.nsplit * g.kchunk < g.K) return cudaErrorInvalidValue;
  // neighbouring threads store neighbouring columns: the operand that carries
  // the output's contiguous mode becomes B (C^T = B^T A^T)
  auto unit = [](const ModeGroup& q) { return q.n > 0 && q.s1[q.n - 1] == 1 && q.dim[q.n - 1] > 1; };
  if (!unit(g.gn) && unit(g.gm)) {
    f.swapped = 1;
    std::swap(g.gm, g.gn);
    std::swap(g.M, g.N);
    std::swap(g.bsA, g.bsB);
    std::swap(f.ac, f.bc);
    for (int i = 0; i < kMaxModes; ++i) std::swap(g.gk.s0[i], g.gk.s1[i]);
    f.tile = f.tile == 1 ? 2 : f.tile == 2 ? 1 : f.tile;  // {32, 64} serves both orders
  }
  if (!tile_fits(f.tile, !f.ac && !f.bc)) return cudaErrorInvalidValue;
  int e2 = 0;
  const double fr = std::frexp(std::fabs(g.ar), &e2);
  f.p2 = (g.ai == 0.0 && fr == 0.5) ? 1 : 0;
  f.e2 = f.p2 ? e2 - 1 : 0;
  f.neg = (f.p2 && g.ar < 0.0) ? 1 : 0;
  if (f.tile == 5) {  // flags: log2 of the lanes per output; kc: bytes of the offset tables
    if (g.nsplit != 1 || g.atomic) return cudaErrorInvalidValue;
    if (op.dot < 0 || op.dot > 5) return cudaErrorInvalidValue;
    f.flags = op.dot;
    f.kc = 16 * std::min(g.K, kDotK);
    f.mtiles = 1;
    f.tiles = ((long long)g.M * g.N + (kFxThreads >> f.flags) - 1) / (kFxThreads >> f.flags);
    return cudaSuccess;
  }
  const int bm = kTiles[f.tile][0], bn = kTiles[f.tile][1];
  f.mtiles = (g.M + bm - 1) / bm;
  f.tiles = (long long)f.mtiles * ((g.N + bn - 1) / bn);
  const int most = fx_chunk(bm, bn, f.ac, f.bc), chunks = (g.kchunk + most - 1) / most;
  f.kc = std::min(most, (std::min(g.kchunk, std::max(g.K, 1)) + chunks - 1) / chunks);
  auto kfast = [&](const long long* ks, const ModeGroup& rows) {
    const int q = g.gk.n - 1;
    if (q < 0 || ks[q] != 1 || g.gk.dim[q] < 4) return 0;
    return (rows.n > 0 && rows.s0[rows.n - 1] == 1 && rows.dim[rows.n - 1] > 1) ? 0 : 1;
  };
  f.flags = kfast(g.gk.s0, g.gm) | (kfast(g.gk.s1, g.gn) << 1);
  return cudaSuccess;
}

cudaError_t launch_gemm(const Op& op, const void* A, const void* B, void* C, cudaStream_t st) {
  GemmArgs g;
  FxPlan f;
  cudaError_t e = fx_plan(op, g, f);
  if (e != cudaSuccess) return e;
  g.A = f.swapped ? B : A;
  g.B = f.swapped ? A : B;
  g.C = C;
  if (f.ac && f.bc)
    e = launch_fx_typed<true, true, true>(g, f, st);
  else if (f.ac)
    e = launch_fx_typed<true, false, true>(g, f, st);
  else if (f.bc)
    e = launch_fx_typed<false, true, true>(g, f, st);
  else if (f.cc)
    e = launch_fx_typed<false, false, true>(g, f, st);
  else
    e = launch_fx_typed<false, false, false>(g, f, st);
  count_launch();
  return e;
}

}  // namespace tdcc
