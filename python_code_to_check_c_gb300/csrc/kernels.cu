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

cudaError_t launch_add(const AddArgs& a, cudaStream_t st) {
  if (a.total <= 0) return cudaSuccess;
  if (a.nd < 1 || a.nd > kAddDims) return cudaErrorInvalidValue;
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
