// Device bodies of the elementwise and reduction ops, shared by their own
// kernels (kernels.cu) and by the kernel that runs a whole program phase
// (phase.cu).
#pragma once

#include "engine.h"

namespace tdcc {

__device__ __forceinline__ double2 cz() { return make_double2(0.0, 0.0); }

// elementwise: C[idx] (+)= sum_t coef_t * A_t[idx] (* B_t[idx])
__device__ __forceinline__ double2 ld(const void* p, long long off, int cplx) {
  if (cplx) return static_cast<const double2*>(p)[off];
  return make_double2(static_cast<const double*>(p)[off], 0.0);
}

// c x for c = +-2^k from the bits of x, with no FP64 operation, where x and
// the product are normal; otherwise (and for infinities and NaNs) fma(c, x,
// +0), whose value the bit path also gives: a zero x gives +0, and a normal
// product is exact.  sgn = c's sign bit, k its unbiased exponent.
__device__ __forceinline__ double scale_pow2(double x, double c, unsigned long long sgn, int k) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const unsigned long long mag = u & 0x7FFFFFFFFFFFFFFFull;
  if (mag == 0ull) return 0.0;
  const int E = (int)(mag >> 52), Er = E + k;
  if (E == 0 || E == 2047 || Er <= 0 || Er >= 2047) return fma(c, x, 0.0);
  return __longlong_as_double((long long)((u ^ sgn) + ((unsigned long long)(long long)k << 52)));
}

// What an elementwise op's first term needs once per thread: when it is A
// alone with a real coefficient +-2^k (the antisymmetrisers' +-1, the 1/2 and
// 1/4 of tau) it starts the sum with no FP64 operation (the FP64 pipe is the
// one these sums wait on).
struct AddStart {
  bool p2;
  unsigned long long sgn;
  int k;
  __device__ __forceinline__ explicit AddStart(const AddArgs& a) {
    const unsigned long long cb = (unsigned long long)__double_as_longlong(a.t[0].cr);
    const int ce = (int)((cb >> 52) & 0x7FF);
    p2 = a.nt > 0 && a.t[0].B == nullptr && __double_as_longlong(a.t[0].ci) == 0 &&
         (cb & 0x000FFFFFFFFFFFFFull) == 0ull && ce > 0 && ce < 2047;
    sgn = cb & 0x8000000000000000ull;
    k = ce - 1023;
  }
};

template <typename IDX>
__device__ __forceinline__ void add_element(const AddArgs& a, const AddStart& st, IDX idx) {
  // decode the (coalesced) index, last dimension fastest
  IDX l = idx;
  int ii[kAddDims];
#pragma unroll
  for (int q = kAddDims - 1; q >= 0; --q) {
    ii[q] = 0;
    if (q < a.nd) {
      const IDX d = (IDX)a.d[q];
      ii[q] = (int)(l % d);
      l /= d;
    }
  }
  double2 s = cz();
  int t0 = 0;
  if (st.p2) {
    long long oa = 0;
#pragma unroll
    for (int q = 0; q < kAddDims; ++q)
      if (q < a.nd) oa += (long long)ii[q] * a.t[0].sA[q];
    const double2 x = ld(a.t[0].A, oa, a.t[0].ac);
    s = make_double2(scale_pow2(x.x, a.t[0].cr, st.sgn, st.k), scale_pow2(x.y, a.t[0].cr, st.sgn, st.k));
    t0 = 1;
  }
  for (int t = t0; t < a.nt; ++t) {
    const AddTerm& T = a.t[t];
    long long oa = 0, ob = 0;
#pragma unroll
    for (int q = 0; q < kAddDims; ++q) {
      if (q < a.nd) {
        oa += (long long)ii[q] * T.sA[q];
        ob += (long long)ii[q] * T.sB[q];
      }
    }
    double2 x = ld(T.A, oa, T.ac);
    if (T.B) {
      const double2 y = ld(T.B, ob, T.bc);
      x = make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x);
    }
    if (T.ci == 0.0) {  // real coefficients (almost all): half the FP64 operations
      s.x = fma(T.cr, x.x, s.x);
      s.y = fma(T.cr, x.y, s.y);
    } else {
      s.x += T.cr * x.x - T.ci * x.y;
      s.y += T.cr * x.y + T.ci * x.x;
    }
  }
  long long oc = 0;
#pragma unroll
  for (int q = 0; q < kAddDims; ++q)
    if (q < a.nd) oc += (long long)ii[q] * a.sC[q];
  // accumulation as an L2 reduction (no return value): one writer per
  // element, so the single addition c + s equals a read-modify-write, and
  // neither the load nor the add occupies the SM (its FP64 pipe is narrow)
  if (a.cc) {
    double2* C = static_cast<double2*>(a.C);
    if (a.acc) {
      atomicAdd(&C[oc].x, s.x);
      atomicAdd(&C[oc].y, s.y);
    } else {
      C[oc] = s;
    }
  } else {
    double* C = static_cast<double*>(a.C);
    if (a.acc)
      atomicAdd(&C[oc], s.x);
    else
      C[oc] = s.x;
  }
}

__device__ __forceinline__ long long red_off(const int* d, const long long* s, int nd, long long l) {
  long long off = 0;
#pragma unroll
  for (int q = kRedDims - 1; q >= 0; --q) {
    if (q < nd) {
      off += (l % d[q]) * s[q];
      l /= d[q];
    }
  }
  return off;
}

// output element w of a reduction, by one warp: lanes over the reduction
// index, fixed-order shuffle sum
__device__ __forceinline__ void reduce_element(const ReduceArgs& r, long long w, int lane) {
  const long long oo = red_off(r.dout, r.so_out, r.no, w);
  const long long ox = red_off(r.dout, r.so_x, r.no, w);
  const long long oy = red_off(r.dout, r.so_y, r.no, w);
  double sr = 0.0, si = 0.0;
  for (long long k = lane; k < r.nred; k += 32) {
    const double2 x = static_cast<const double2*>(r.X)[ox + red_off(r.dred, r.sr_x, r.nr, k)];
    double2 v = x;
    if (r.Y) {
      const long long yo = oy + red_off(r.dred, r.sr_y, r.nr, k);
      const double2 y = ld(r.Y, yo, r.ycplx);
      v = make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x);
    }
    sr += v.x;
    si += v.y;
  }
  for (int dd = 16; dd > 0; dd >>= 1) {
    sr += __shfl_down_sync(0xffffffffu, sr, dd);
    si += __shfl_down_sync(0xffffffffu, si, dd);
  }
  if (lane == 0) {
    double2* out = static_cast<double2*>(r.out);
    const double vr = r.cr * sr - r.ci * si, vi = r.cr * si + r.ci * sr;
    if (r.acc) {
      atomicAdd(&out[oo].x, vr);
      atomicAdd(&out[oo].y, vi);
    } else {
      out[oo] = make_double2(vr, vi);
    }
  }
}

}  // namespace tdcc
