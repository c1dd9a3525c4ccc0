// Elementwise accumulate with antisymmetrisers, reductions and the dipole
// trace, in FP64.  All complex data is interleaved (double2).
#include <atomic>
#include <cstdio>
#include <type_traits>

#include "elementwise.cuh"
#include "engine.h"

namespace tdcc {

static std::atomic<long long> g_launches{0};
void count_launch(long long k) { g_launches.fetch_add(k, std::memory_order_relaxed); }
long long launch_count() { return g_launches.load(); }

// ---------------------------------------------------------------------------
// elementwise: C[idx] (+)= sum_t coef_t * A_t[idx] (* B_t[idx])
// ---------------------------------------------------------------------------
template <typename IDX>
__global__ void __launch_bounds__(256) add_kernel(const AddArgs a) {
  const IDX stride = (IDX)gridDim.x * blockDim.x;
  const AddStart st(a);
  for (IDX idx = (IDX)blockIdx.x * blockDim.x + threadIdx.x; idx < (IDX)a.total; idx += stride)
    add_element<IDX>(a, st, idx);
}

// The sums that make up a step (one to four tensors with real coefficients, fewer
// than 2^31 elements, offsets of 32 bits): divisions by the extents as
// multiplications (Granlund and Montgomery, PLDI 1994: n < 2^31, sh = ceil log2 d,
// mul = floor(2^32 (2^sh - d) / d) + 1, n / d = (mulhi(n, mul) + n) >> sh), all
// loads of an element's terms in flight, nothing 64 bits wide but the data.
// Bound: the memory system, the L2 reductions and the FP64 pipe (two operations an
// element and term after the first).  3.5 M elements: three terms 98 us through
// add_kernel, 72 here (two elements a thread); two terms accumulated 56, 46 (one
// element a thread: with two, 58; as loads and stores instead of reductions, whose
// additions the FP64 pipe would do, 70).
constexpr int kFastTerms = 4;
struct AddFast {
  void* C;
  unsigned total;
  int nd, cc, acc;
  unsigned d[kAddDims], mul[kAddDims], sh[kAddDims];
  int sC[kAddDims];
  const void* A[kFastTerms];
  double cr[kFastTerms];
  int ac[kFastTerms];
  int sA[kFastTerms][kAddDims];
};

template <int NT, int U>
__global__ void __launch_bounds__(256) add_fast_kernel(const __grid_constant__ AddFast a) {
  const unsigned long long cb = (unsigned long long)__double_as_longlong(a.cr[0]);
  const int ce = (int)((cb >> 52) & 0x7FF);
  const bool p2 = (cb & 0x000FFFFFFFFFFFFFull) == 0ull && ce > 0 && ce < 2047;
  double2 x[U][NT];
  int oc[U];
  bool in[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const unsigned idx = (blockIdx.x * U + u) * 256u + threadIdx.x;
    in[u] = idx < a.total;
    unsigned l = in[u] ? idx : 0u;
    int oa[NT];
    oc[u] = 0;
#pragma unroll
    for (int t = 0; t < NT; ++t) oa[t] = 0;
#pragma unroll
    for (int q = kAddDims - 1; q >= 0; --q)
      if (q < a.nd) {
        const unsigned quo = q > 0 ? (__umulhi(l, a.mul[q]) + l) >> a.sh[q] : 0u;
        const int r = (int)(l - quo * a.d[q]);
        l = quo;
        oc[u] += r * a.sC[q];
#pragma unroll
        for (int t = 0; t < NT; ++t) oa[t] += r * a.sA[t][q];
      }
#pragma unroll
    for (int t = 0; t < NT; ++t) x[u][t] = ld(a.A[t], oa[t], a.ac[t]);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    if (!in[u]) continue;
    double2 s = cz();
    if (p2)
      s = make_double2(scale_pow2(x[u][0].x, a.cr[0], cb & 0x8000000000000000ull, ce - 1023),
                       scale_pow2(x[u][0].y, a.cr[0], cb & 0x8000000000000000ull, ce - 1023));
#pragma unroll
    for (int t = 0; t < NT; ++t)
      if (t > 0 || !p2) {
        s.x = fma(a.cr[t], x[u][t].x, s.x);
        s.y = fma(a.cr[t], x[u][t].y, s.y);
      }
    if (a.cc) {
      double2* C = static_cast<double2*>(a.C) + oc[u];
      if (a.acc) {
        atomicAdd(&C->x, s.x);
        atomicAdd(&C->y, s.y);
      } else {
        *C = s;
      }
    } else {
      double* C = static_cast<double*>(a.C) + oc[u];
      if (a.acc)
        atomicAdd(C, s.x);
      else
        *C = s.x;
    }
  }
}

// false where the general kernel has to run
static bool fast_add(const AddArgs& a, AddFast& f) {
  constexpr long long kMax = 0x7FFFFFFFLL;
  if (a.nt < 1 || a.nt > kFastTerms || a.total >= kMax - 512) return false;
  auto spans = [&](const long long* s) {  // every offset fits 32 bits
    long long lo = 0, hi = 0;
    for (int q = 0; q < a.nd; ++q) (s[q] < 0 ? lo : hi) += (long long)(a.d[q] - 1) * s[q];
    return lo >= -kMax && hi <= kMax;
  };
  if (!spans(a.sC)) return false;
  for (int t = 0; t < a.nt; ++t)
    if (a.t[t].B || a.t[t].ci != 0.0 || !spans(a.t[t].sA)) return false;
  f.C = a.C;
  f.total = (unsigned)a.total;
  f.nd = a.nd;
  f.cc = a.cc;
  f.acc = a.acc;
  for (int q = 0; q < a.nd; ++q) {
    const unsigned long long d = (unsigned long long)a.d[q];
    if (d < 1) return false;
    unsigned sh = 0;
    while ((1ull << sh) < d) ++sh;
    f.d[q] = (unsigned)d;
    f.sh[q] = sh;
    f.mul[q] = (unsigned)(((1ull << 32) * ((1ull << sh) - d)) / d + 1);
    f.sC[q] = a.d[q] > 1 ? (int)a.sC[q] : 0;
    for (int t = 0; t < a.nt; ++t) f.sA[t][q] = a.d[q] > 1 ? (int)a.t[t].sA[q] : 0;
  }
  for (int t = 0; t < a.nt; ++t) {
    f.A[t] = a.t[t].A;
    f.cr[t] = a.t[t].cr;
    f.ac[t] = a.t[t].ac;
  }
  return true;
}

cudaError_t launch_add(const AddArgs& a, cudaStream_t st) {
  if (a.total <= 0) return cudaSuccess;
  if (a.nd < 1 || a.nd > kAddDims) return cudaErrorInvalidValue;
  AddFast f{};
  if (fast_add(a, f)) {
    auto go = [&](auto one, auto two) {
      if (a.acc)
        one<<<(unsigned)((a.total + 255) / 256), 256, 0, st>>>(f);
      else
        two<<<(unsigned)((a.total + 511) / 512), 256, 0, st>>>(f);
    };
    switch (a.nt) {
      case 1: go(add_fast_kernel<1, 1>, add_fast_kernel<1, 2>); break;
      case 2: go(add_fast_kernel<2, 1>, add_fast_kernel<2, 2>); break;
      case 3: go(add_fast_kernel<3, 1>, add_fast_kernel<3, 2>); break;
      default: go(add_fast_kernel<4, 1>, add_fast_kernel<4, 2>); break;
    }
    count_launch();
    return cudaGetLastError();
  }
  long long blocks = (a.total + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  // 32-bit index arithmetic unless the index space needs 64 bits
  if (a.total + (long long)blocks * 256 < (1LL << 32))
    add_kernel<unsigned><<<(unsigned)blocks, 256, 0, st>>>(a);
  else
    add_kernel<unsigned long long><<<(unsigned)blocks, 256, 0, st>>>(a);
  count_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// reduction: out[o] (+)= c * sum_r X[o, r] (* Y[o, r]).  One warp per output
// element, lanes over the reduction index, fixed-order shuffle sum.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) reduce_kernel(const ReduceArgs r) {
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < r.nout; w += nw)
    reduce_element(r, w, lane);
}

cudaError_t launch_reduce(const ReduceArgs& r, cudaStream_t st) {
  if (r.nout <= 0) return cudaSuccess;
  if (r.no < 0 || r.no > kRedDims || r.nr < 0 || r.nr > kRedDims) return cudaErrorInvalidValue;
  long long blocks = (r.nout + 7) / 8;
  if (blocks > 152 * 16) blocks = 152 * 16;
  reduce_kernel<<<(unsigned)blocks, 256, 0, st>>>(r);
  count_launch();
  return cudaGetLastError();
}

struct TraceBatch {
  long long bs[4];  // batch strides of Dij, l1, Dai, Dab (elements)
  long long bsres;
};

// dipole trace: res[k] = sum_ij mu_k[i,j] rho[i,j], rho = [[Dij, l1],[Dai, Dab]]
// One CTA per dipole component; warp-shuffle + shared-memory reduction, so
// the sum order is fixed (deterministic).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) trace_kernel(int n, int o, const double* mu,
                                                     const double2* dij, const double2* l1,
                                                     const double2* dai, const double2* dab,
                                                     double2* res, TraceBatch tb) {
  const int k = blockIdx.x;
  const int z = blockIdx.y;  // trajectory
  dij += z * tb.bs[0];
  l1 += z * tb.bs[1];
  dai += z * tb.bs[2];
  dab += z * tb.bs[3];
  res += z * tb.bsres;
  const int v = n - o;
  const double* M = mu + (long long)k * n * n;
  double sr = 0.0, si = 0.0;
  const long long nn = (long long)n * n;
  for (long long e = threadIdx.x; e < nn; e += blockDim.x) {
    const int p = (int)(e / n), q = (int)(e % n);
    double2 r;
    if (p < o && q < o)
      r = dij[p * o + q];
    else if (p < o)
      r = l1[p * v + (q - o)];
    else if (q < o)
      r = dai[(p - o) * o + q];
    else
      r = dab[(long long)(p - o) * v + (q - o)];
    const double m = M[e];
    sr = fma(m, r.x, sr);
    si = fma(m, r.y, si);
  }
  for (int d = 16; d > 0; d >>= 1) {
    sr += __shfl_down_sync(0xffffffffu, sr, d);
    si += __shfl_down_sync(0xffffffffu, si, d);
  }
  __shared__ double wr[32], wi[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    wr[w] = sr;
    wi[w] = si;
  }
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    sr = lane < nw ? wr[lane] : 0.0;
    si = lane < nw ? wi[lane] : 0.0;
    for (int d = 16; d > 0; d >>= 1) {
      sr += __shfl_down_sync(0xffffffffu, sr, d);
      si += __shfl_down_sync(0xffffffffu, si, d);
    }
    if (lane == 0) res[k] = make_double2(sr, si);
  }
}

cudaError_t launch_trace(int n, int o, int n_mu, const double* mu, const void* dij, const void* l1,
                         const void* dai, const void* dab, void* res, int nb, const long long* bs,
                         long long bsres, cudaStream_t st) {
  TraceBatch tb;
  for (int k = 0; k < 4; ++k) tb.bs[k] = nb > 1 ? bs[k] : 0;
  tb.bsres = nb > 1 ? bsres : 0;
  trace_kernel<<<dim3(n_mu, nb > 1 ? nb : 1), 1024, 0, st>>>(n, o, mu, static_cast<const double2*>(dij),
                                                             static_cast<const double2*>(l1),
                                                             static_cast<const double2*>(dai),
                                                             static_cast<const double2*>(dab),
                                                             static_cast<double2*>(res), tb);
  count_launch();
  return cudaGetLastError();
}

}  // namespace tdcc
