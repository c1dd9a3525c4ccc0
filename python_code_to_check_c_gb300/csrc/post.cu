// Integral build from density-fitting factors and the dipole spectrum.
//
// tei_antisym_kernel: <pq||rs> = (pr|qs) - (ps|qr) in place over the
//   Coulomb-ordered product X[p,q,r,s] = (pr|qs) (the GEMM sum_Q B_Q,pr B_Q,qs
//   is written in that order by the strided GEMM).
// spectrum_kernel: the shifted discrete Fourier transforms of Re mu(t) and
//   Im mu(t), as the reference's post-processing computes them
//   (Plots.py:20-25: np.fft.fft of the real and imaginary parts, fftshift).
#include <cuda_runtime.h>

#include "engine.h"
#include "post.h"

namespace tdcc {

// A block owns one (p, q) slice's tile pairs (rt, st), (st, rt) in turn: both
// tiles are read along their rows, exchanged through shared memory and written
// along their rows, so every access is a 128-byte run.  (One thread per element
// with the partner read down a column took 52 us at n = 48, 85 MB.)
__global__ void __launch_bounds__(256) tei_antisym_kernel(double* __restrict__ X, int n, long long pairs, int tiles,
                                                          const int* __restrict__ err) {
  constexpr int T = 16;
  __shared__ double ta[T][T + 1], tb[T][T + 1];
  const int i = threadIdx.x / T, j = threadIdx.x % T;
  // a contraction that gave up on a wait leaves no numbers behind
  const bool bad = err && *err;
  const double nan = __longlong_as_double(0x7FF8000000000000ll);
  const int per = tiles * (tiles + 1) / 2;
  for (long long w = blockIdx.x; w < pairs; w += gridDim.x) {
    double* base = X + (w / per) * (long long)n * n;
    int st = 0, rem = (int)(w % per);
    while (rem > st) rem -= ++st;  // rt <= st, row-wise over the triangle
    const int rt = rem;
    const int r = rt * T + i, s = st * T + j;    // the tile above the diagonal, this thread's element
    const int r2 = st * T + i, s2 = rt * T + j;  // and the one below
    const bool in1 = r < n && s < n, in2 = r2 < n && s2 < n;
    const double a = in1 ? base[(long long)r * n + s] : 0.0;
    const double b = in2 ? base[(long long)r2 * n + s2] : 0.0;
    ta[i][j] = a;
    tb[i][j] = b;
    __syncthreads();
    // out[r][s] = x[r][s] - x[s][r]
    if (in1) base[(long long)r * n + s] = bad ? nan : r == s ? 0.0 : a - tb[j][i];
    if (in2 && rt != st) base[(long long)r2 * n + s2] = bad ? nan : b - ta[j][i];
    __syncthreads();
  }
}

cudaError_t launch_tei_antisym(double* X, int n, const int* err, cudaStream_t st) {
  const int tiles = (n + 15) / 16;
  const long long pairs = (long long)n * n * (tiles * (tiles + 1) / 2);
  const long long blocks = pairs < 152LL * 8 ? pairs : 152LL * 8;
  tei_antisym_kernel<<<(unsigned)blocks, 256, 0, st>>>(X, n, pairs, tiles, err);
  count_launch();
  return cudaGetLastError();
}

// tw[r] = exp(-2 pi i r / N)
__global__ void twiddle_kernel(double2* __restrict__ tw, long long N) {
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < N; r += (long long)gridDim.x * blockDim.x) {
    double s, c;
    sincospi(2.0 * (double)r / (double)N, &s, &c);
    tw[r] = make_double2(c, -s);
  }
}

// One block per output position j of the shifted spectra: frequency index
// k = (j + N - N/2) mod N; Yr[j] = sum_n Re mu[n] tw[k n mod N], Yi likewise
// with Im mu.
__global__ void __launch_bounds__(256) spectrum_kernel(const double2* __restrict__ mu, long long N, long long stride,
                                                       const double2* __restrict__ tw, double2* __restrict__ Yr,
                                                       double2* __restrict__ Yi) {
  const long long j = blockIdx.x;
  const long long k = (j + N - N / 2) % N;
  const long long step = (k * (long long)blockDim.x) % N;
  long long r = (k * (long long)threadIdx.x) % N;
  double rr = 0.0, ri = 0.0, ir = 0.0, ii = 0.0;
  for (long long nn = threadIdx.x; nn < N; nn += blockDim.x) {
    const double2 m = mu[nn * stride];
    const double2 w = tw[r];
    rr = fma(m.x, w.x, rr);
    ri = fma(m.x, w.y, ri);
    ir = fma(m.y, w.x, ir);
    ii = fma(m.y, w.y, ii);
    r += step;
    if (r >= N) r -= N;
  }
  for (int d = 16; d > 0; d >>= 1) {
    rr += __shfl_down_sync(0xffffffffu, rr, d);
    ri += __shfl_down_sync(0xffffffffu, ri, d);
    ir += __shfl_down_sync(0xffffffffu, ir, d);
    ii += __shfl_down_sync(0xffffffffu, ii, d);
  }
  __shared__ double red[4][8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    red[0][w] = rr;
    red[1][w] = ri;
    red[2][w] = ir;
    red[3][w] = ii;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
      a += red[0][q];
      b += red[1][q];
      c += red[2][q];
      d += red[3][q];
    }
    Yr[j] = make_double2(a, b);
    Yi[j] = make_double2(c, d);
  }
}

cudaError_t launch_spectrum(const double2* mu, long long N, long long stride, double2* tw, double2* Yr, double2* Yi,
                            cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  long long tb = (N + 255) / 256;
  if (tb > 152LL * 8) tb = 152LL * 8;
  twiddle_kernel<<<(unsigned)tb, 256, 0, st>>>(tw, N);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (N > 0x7fffffffLL) return cudaErrorInvalidValue;
  spectrum_kernel<<<(unsigned)N, 256, 0, st>>>(mu, N, stride, tw, Yr, Yi);
  count_launch();
  return cudaGetLastError();
}

}  // namespace tdcc
