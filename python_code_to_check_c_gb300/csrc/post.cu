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

// Frequencies k = 0 .. N/2 of the transforms of the two real sequences Re mu and
// Im mu; those of N - k are their conjugates.  64 threads per frequency, each
// with four partial sums of every 256th term.  Bound: the FP64 pipe (8 N^2/2
// operations, 14 us at N = 2000) and the table's reads.  A block of 256 threads
// per frequency, all N of them, spent 160 of its 416 FP64 instructions per
// warp-column on shuffle sums: 58 us; this form adds in the same depth with a
// sixth of them and does half the frequencies (a call of 7934 samples 835 ->
// 333 us, one of 2000, with its scratch no longer mapped anew, 376 -> 108).
constexpr int kSpecLanes = 64;
__global__ void __launch_bounds__(256) spectrum_kernel(const double2* __restrict__ mu, long long N, long long stride,
                                                       const double2* __restrict__ tw, double2* __restrict__ Yr,
                                                       double2* __restrict__ Yi) {
  constexpr int L = kSpecLanes, Q = 256 / L;
  const int t = threadIdx.x % L, q = threadIdx.x / L;
  const long long k = (long long)blockIdx.x * Q + q;
  double rr[4] = {}, ri[4] = {}, ir[4] = {}, ii[4] = {};
  if (k <= N / 2) {
    const long long step = (k * L) % N;
    long long r = (k * t) % N;
    for (long long n0 = t; n0 < N; n0 += 4 * L)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const long long n = n0 + u * L;
        if (n < N) {
          const double2 m = mu[n * stride];
          const double2 w = tw[r];
          rr[u] = fma(m.x, w.x, rr[u]);
          ri[u] = fma(m.x, w.y, ri[u]);
          ir[u] = fma(m.y, w.x, ir[u]);
          ii[u] = fma(m.y, w.y, ii[u]);
          r += step;
          if (r >= N) r -= N;
        }
      }
  }
  double v[4] = {(rr[0] + rr[1]) + (rr[2] + rr[3]), (ri[0] + ri[1]) + (ri[2] + ri[3]),
                 (ir[0] + ir[1]) + (ir[2] + ir[3]), (ii[0] + ii[1]) + (ii[2] + ii[3])};
  __shared__ double red[256 / 32][4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    for (int d = 16; d > 0; d >>= 1) v[p] += __shfl_down_sync(0xffffffffu, v[p], d);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][p] = v[p];
  }
  __syncthreads();
  if (t == 0 && k <= N / 2) {
    const int w = threadIdx.x >> 5;
    const double2 a = make_double2(red[w][0] + red[w + 1][0], red[w][1] + red[w + 1][1]);
    const double2 b = make_double2(red[w][2] + red[w + 1][2], red[w][3] + red[w + 1][3]);
    const long long j = (k + N / 2) % N, j2 = (N - k + N / 2) % N;  // shifted positions of k and N - k
    Yr[j] = a;
    Yi[j] = b;
    if (j2 != j) {
      Yr[j2] = make_double2(a.x, -a.y);
      Yi[j2] = make_double2(b.x, -b.y);
    }
  }
}

cudaError_t launch_spectrum(const double2* mu, long long N, long long stride, double2* tw, double2* Yr, double2* Yi,
                            cudaStream_t st) {
  if (N <= 0) return cudaSuccess;
  if (N > 0x7fffffffLL) return cudaErrorInvalidValue;
  long long tb = (N + 63) / 64;
  if (tb > 152LL * 16) tb = 152LL * 16;
  twiddle_kernel<<<(unsigned)tb, 64, 0, st>>>(tw, N);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  constexpr int Q = 256 / kSpecLanes;
  spectrum_kernel<<<(unsigned)((N / 2 + 1 + Q - 1) / Q), 256, 0, st>>>(mu, N, stride, tw, Yr, Yi);
  count_launch();
  return cudaGetLastError();
}

}  // namespace tdcc
