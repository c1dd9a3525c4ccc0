// A whole phase of a small FP64 program in one cooperative launch.
//
// A residual of a few orbitals is 20 to 70 ops of a few microseconds in 5 to
// 15 dependency levels; as launches of their own they cost the host 3-4 us
// each (events included) and the device 4-5 us per dependent pair.  Here the
// op records lie in device memory, grouped in levels; the blocks share out
// the tiles of a level, meet at a grid barrier and go on to the next.  Bound:
// per level the barrier (about 2 k clocks) and the latency of one tile, so
// everything that does not depend on the level before is done ahead of the
// barrier: index tables are made by the host, a block's next record and its
// threads' first table entries are read before it waits.  FP64 instructions
// hold a scheduler's pipe for 64 clocks per warp, so small ops are spread a
// warp per scheduler over all blocks rather than packed into a few.
//
// The launch is cooperative, so all blocks are resident; every wait on the
// barrier has an iteration limit, after which the kernel records an error
// code, stops, leaves NaN in all that it writes and returns.
#include <algorithm>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <stdexcept>
#include <utility>

#include "elementwise.cuh"
#include "fx_tile.cuh"
#include "phase.h"

namespace tdcc {

namespace {

constexpr int kPhaseSlots = 128;   // pointers passed by value
constexpr int kPhaseOps = 160;
constexpr int kBarrierLimit = 1 << 21;
constexpr unsigned kLost = 1u << 16;  // in the count of blocks that are out: one gave up a wait
// Phases with more work keep a launch per op: there the blocks of several ops
// fill the chip without waiting for one another.  Measured (one launch per phase
// against one per op; Mflop of the phase, us): T2 residuals of o=4..6, v=8..13 2.5 111
// 248, 4.7 130 220, 8.2 155 225, 16 200 226, 27 262 242.  But a phase of few large
// contractions, as T1's and L1's of larger systems are, loses far below that: with the
// line at 9 instead of 3 8 steps at o=10, v=14 took 15.2 ms for 10.1, a step at o=8, v=12
// 1.63 for 1.28, the ground state at o=10, v=14 16.6 for 9.9.
constexpr double kPhaseFlops = 3e6;
constexpr size_t kPhaseTempMax = 64u << 20;
constexpr size_t kPhaseTableMax = 1u << 20;   // index table entries (8 bytes each)
constexpr int kPtrs = 2 * kMaxAddTerms + 1;

struct TraceRec {
  const double* mu;
  const double2 *dij, *l1, *dai, *dab;
  double2* res;
  int n, o, n_mu, pad;
  long long bs[4], bsres;
};

struct GemmRec {  // fixed-point tiles
  GemmArgs g;
  FxPlan f;
};

// Dot products: 2^lw lanes per output, `threads` of a block at work; offsets
// (elements) of the rows (A, C), the columns (B, C) and the k (A, B) in tables.
struct DotRec {
  const double *A, *B;
  double2* C;
  const int2 *mt, *nt, *kt;
  int M, N, K, ntiles, lw, threads;
  int acc, p2, e2, neg;
  double ar, ai;
  long long bsA, bsB, bsC;
};

struct AddRecTerm {
  const void *A, *B;
  int sA[kAddDims], sB[kAddDims];
  int ac, bc;
  double cr, ci;
};
struct AddRec {
  void* C;
  int nd, nt, cc, acc, per, pad;  // acc 1: one atomic addition; 2: read, add term by term, write
  unsigned total, d[kAddDims];
  int sC[kAddDims];
  AddRecTerm t[kMaxAddTerms];
};

// One op; pointers are filled in from (slot, byte offset) at run time.
struct alignas(16) PhaseOp {
  int kind;          // OP_GEMM, OP_ADD, OP_REDUCE, OP_TRACE
  int form;          // GEMM: operand types and tile (3..5: dot products)
  int nptr, pad;
  int pslot[kPtrs], poff[kPtrs];  // slot (-1: none, -2: pbyte is the address); where in this record the pointer goes
  long long pbyte[kPtrs];
  union {
    GemmRec gemm;
    DotRec dot;
    AddRec add;
    ReduceArgs red;
    TraceRec tr;
  };
};

struct PhaseOut {  // a buffer that the phase writes
  int slot, pad;
  long long doubles;
};

struct PhaseArgs {
  const PhaseOp* ops;
  const PhaseOut* outs;
  int nouts, wait;
  const int* tab;      // [nlevels + 1] first op of each level, [nops] first tile within its level, [nops] end tile
  int nops, nlevels;
  unsigned* bar;
  int* err;
  void* base[kPhaseSlots];
};

// The grid barrier in two halves.  arrive: every thread's writes are ordered
// before the block's arrival.  wait: polls (thread 0, then the block); false
// when the wait expired.
__device__ __forceinline__ void grid_arrive(unsigned* bar) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}
__device__ __forceinline__ bool grid_wait(unsigned* bar, unsigned target, int limit, int* err, int* shared_ok) {
  if (threadIdx.x == 0) {
    int good = 0;
    for (int i = 0; i < limit; ++i) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if (v >= target) {
        good = 1;
        break;
      }
    }
    if (!good) {
      atomicCAS(err, 0, 9);
      atomicAdd(bar + 1, kLost);  // this launch's results are lost
    }
    *shared_ok = good;
  }
  __syncthreads();
  return *shared_ok != 0;
}

constexpr int kDotU = 4;  // k entries in flight per lane
struct DotAhead {         // a thread's offsets of a tile, read ahead of the barrier
  int m, n;               // element offsets of its row of A and column of B, -1: no output
  int c;
  int2 k[kDotU];
};

__device__ __forceinline__ void dot_ahead(const DotRec& r, unsigned tile, DotAhead& a) {
  const unsigned z = tile / (unsigned)r.ntiles, q = tile - z * (unsigned)r.ntiles;
  const unsigned out = q * ((unsigned)r.threads >> r.lw) + (threadIdx.x >> r.lw);
  a.m = -1;
  if ((int)threadIdx.x < r.threads && out < (unsigned)r.M * (unsigned)r.N) {
    const unsigned m = out / (unsigned)r.N, n = out - m * (unsigned)r.N;
    const int2 u = __ldg(r.mt + m), v = __ldg(r.nt + n);
    a.m = u.x;
    a.n = v.x;
    a.c = u.y + v.y;
    const int L = 1 << r.lw, lane = threadIdx.x & (L - 1);
#pragma unroll
    for (int i = 0; i < kDotU; ++i)
      if (lane + i * L < r.K) a.k[i] = __ldg(r.kt + lane + i * L);
  }
}

template <bool AC, bool BC>
__device__ __forceinline__ void dot_run(const DotRec& r, unsigned tile, const DotAhead& a) {
  if ((int)(threadIdx.x & ~31u) >= r.threads) return;  // whole warps
  const unsigned z = tile / (unsigned)r.ntiles;
  const int L = 1 << r.lw, lane = threadIdx.x & (L - 1);
  const double* A = r.A + z * r.bsA * (AC ? 2 : 1);
  const double* B = r.B + z * r.bsB * (BC ? 2 : 1);
  double2 s = make_double2(0.0, 0.0);
  if (a.m >= 0) {
    for (int k = lane; k < r.K; k += kDotU * L) {
      double2 x[kDotU], y[kDotU];
#pragma unroll
      for (int i = 0; i < kDotU; ++i)
        if (k + i * L < r.K) {
          const int2 o = k == lane ? a.k[i] : __ldg(r.kt + k + i * L);
          x[i] = load1<AC>(A, a.m + o.x);
          y[i] = load1<BC>(B, a.n + o.y);
        }
#pragma unroll
      for (int i = 0; i < kDotU; ++i)
        if (k + i * L < r.K) {
          if constexpr (AC && BC) {
            fmac(s, x[i], y[i]);
          } else if constexpr (AC) {
            s.x = fma(x[i].x, y[i].x, s.x);
            s.y = fma(x[i].y, y[i].x, s.y);
          } else {
            s.x = fma(x[i].x, y[i].x, s.x);
            s.y = fma(x[i].x, y[i].y, s.y);
          }
        }
    }
  }
  for (int d = L >> 1; d > 0; d >>= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, d);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, d);
  }
  if (a.m < 0 || lane != 0) return;
  if (!r.p2) {
    s = make_double2(r.ar * s.x - r.ai * s.y, r.ar * s.y + r.ai * s.x);
  } else if (r.e2 != 0 || r.neg) {
    const unsigned long long sgn = r.neg ? 0x8000000000000000ull : 0ull;
    s = make_double2(scale_pow2(s.x, r.ar, sgn, r.e2), scale_pow2(s.y, r.ar, sgn, r.e2));
  }
  double2* C = r.C + z * r.bsC + a.c;
  if (r.acc) {
    atomicAdd(&C->x, s.x);
    atomicAdd(&C->y, s.y);
  } else {
    *C = s;
  }
}

// elements [per tile, + per) of an elementwise op: the terms' loads first, then
// the sum in term order (as add_element)
__device__ __forceinline__ void add_tile(const AddRec& a, unsigned tile) {
  const unsigned end = min((tile + 1) * (unsigned)a.per, a.total);
  for (unsigned idx = tile * (unsigned)a.per + threadIdx.x; idx < end; idx += kFxThreads) {
    int ii[kAddDims];
    unsigned l = idx;
#pragma unroll
    for (int q = kAddDims - 1; q >= 1; --q) {
      ii[q] = 0;
      if (q < a.nd) {
        const unsigned w = l / a.d[q];
        ii[q] = (int)(l - w * a.d[q]);
        l = w;
      }
    }
    ii[0] = (int)l;
    auto off = [&](const int* st) {
      int o = 0;
#pragma unroll
      for (int q = 0; q < kAddDims; ++q)
        if (q < a.nd) o += ii[q] * st[q];
      return o;
    };
    double2 x[kMaxAddTerms];
#pragma unroll
    for (int t = 0; t < kMaxAddTerms; ++t)
      if (t < a.nt) x[t] = ld(a.t[t].A, off(a.t[t].sA), a.t[t].ac);
    const int oc = off(a.sC);
    double2 s = cz();
    if (a.acc == 2) s = static_cast<const double2*>(a.C)[oc];  // the terms join it one by one
#pragma unroll
    for (int t = 0; t < kMaxAddTerms; ++t) {
      if (t >= a.nt) break;
      double2 v = x[t];
      if (a.t[t].B) {
        const double2 y = ld(a.t[t].B, off(a.t[t].sB), a.t[t].bc);
        v = make_double2(v.x * y.x - v.y * y.y, v.x * y.y + v.y * y.x);
      }
      const double cr = a.t[t].cr, ci = a.t[t].ci;
      if (t == 0 && cr == 1.0 && ci == 0.0 && a.acc != 2) {
        s = v;  // the sum starts with no FP64 operation
      } else if (ci == 0.0) {
        s.x = fma(cr, v.x, s.x);
        s.y = fma(cr, v.y, s.y);
      } else {
        s.x += cr * v.x - ci * v.y;
        s.y += cr * v.y + ci * v.x;
      }
    }
    if (a.cc) {
      double2* C = static_cast<double2*>(a.C) + oc;
      if (a.acc == 1) {
        atomicAdd(&C->x, s.x);
        atomicAdd(&C->y, s.y);
      } else {
        *C = s;
      }
    } else {
      double* C = static_cast<double*>(a.C) + oc;
      if (a.acc)
        atomicAdd(C, s.x);
      else
        *C = s.x;
    }
  }
}

__device__ __forceinline__ void trace_tile(const TraceRec& t, unsigned tile, double* red) {
  const int k = (int)(tile % (unsigned)t.n_mu), z = (int)(tile / (unsigned)t.n_mu);
  const int n = t.n, o = t.o, v = n - o;
  const double2 *dij = t.dij + z * t.bs[0], *l1 = t.l1 + z * t.bs[1], *dai = t.dai + z * t.bs[2],
                *dab = t.dab + z * t.bs[3];
  const double* M = t.mu + (long long)k * n * n;
  double sr = 0.0, si = 0.0;
  for (int e = threadIdx.x; e < n * n; e += kFxThreads) {
    const int p = e / n, q = e - p * n;
    double2 r;
    if (p < o)
      r = q < o ? dij[p * o + q] : l1[p * v + (q - o)];
    else
      r = q < o ? dai[(p - o) * o + q] : dab[(p - o) * v + (q - o)];
    sr = fma(M[e], r.x, sr);
    si = fma(M[e], r.y, si);
  }
  for (int d = 16; d > 0; d >>= 1) {
    sr += __shfl_down_sync(0xffffffffu, sr, d);
    si += __shfl_down_sync(0xffffffffu, si, d);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    red[2 * w] = sr;
    red[2 * w + 1] = si;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < kFxThreads / 32; ++q) {
      sr += red[2 * q];
      si += red[2 * q + 1];
    }
    t.res[z * t.bsres + k] = make_double2(sr, si);
  }
}

__global__ void __launch_bounds__(kFxThreads, 2) phase_kernel(const __grid_constant__ PhaseArgs p) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ FxScratch sh;
  __shared__ PhaseOp rec[2];
  __shared__ int tab[kPhaseOps + 1 + 2 * kPhaseOps];
  __shared__ double red[2 * kFxThreads / 32];
  __shared__ int ok;
  const int tid = threadIdx.x;
  for (int i = tid; i < p.nlevels + 1 + 2 * p.nops; i += kFxThreads) tab[i] = p.tab[i];
  __syncthreads();
  const int* first = tab;
  const int* beg = tab + p.nlevels + 1;
  const int* end = beg + p.nops;
  // copies record o into rec[w] (a __syncthreads must follow before its use)
  auto fetch = [&](int w, int o) {
    const uint4* src = reinterpret_cast<const uint4*>(p.ops + o);
    uint4* dst = reinterpret_cast<uint4*>(&rec[w]);
    for (int i = tid; i < (int)(sizeof(PhaseOp) / 16); i += kFxThreads) dst[i] = __ldg(src + i);
  };
  auto bind = [&](int w) {
    PhaseOp& op = rec[w];
    if (tid < op.nptr)
      *reinterpret_cast<void**>(reinterpret_cast<char*>(&op) + op.poff[tid]) =
          op.pslot[tid] >= 0    ? static_cast<char*>(p.base[op.pslot[tid]]) + op.pbyte[tid]
          : op.pslot[tid] == -2 ? reinterpret_cast<char*>(op.pbyte[tid])
                                : nullptr;
  };
  bool good = true;
  int w = 0, cur = -1;  // record in use and its op
  DotAhead ahead;
  bool have = false;    // `ahead` holds this block's first tile of the level
  for (int l = 0; l < p.nlevels && good; ++l) {
    const int total = end[first[l + 1] - 1];
    int o = first[l];
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
      while (t >= end[o]) ++o;
      if (o != cur) {
        __syncthreads();  // the previous tile is done with its record
        w ^= 1;
        fetch(w, o);
        __syncthreads();
        bind(w);
        cur = o;
        have = false;
      }
      if (!have) __syncthreads();  // record bound; scratch of the previous tile free
      const PhaseOp& op = rec[w];
      const unsigned tile = (unsigned)(t - beg[o]);
      if (op.kind == OP_GEMM && op.form >= 3) {
        if (!have) dot_ahead(op.dot, tile, ahead);
        if (op.form == 3)
          dot_run<true, true>(op.dot, tile, ahead);
        else if (op.form == 4)
          dot_run<true, false>(op.dot, tile, ahead);
        else
          dot_run<false, true>(op.dot, tile, ahead);
      } else if (op.kind == OP_GEMM) {
        const GemmArgs& g = op.gemm.g;
        const FxPlan& f = op.gemm.f;
        const unsigned z = tile / (unsigned)f.tiles, q = tile - z * (unsigned)f.tiles;
        switch (op.form) {
          case 0: fx_tile<true, true, true, 16, 16>(g, f, q, z, smraw, sh); break;
          case 1: fx_tile<true, false, true, 16, 16>(g, f, q, z, smraw, sh); break;
          default: fx_tile<false, true, true, 16, 16>(g, f, q, z, smraw, sh); break;
        }
      } else if (op.kind == OP_ADD) {
        add_tile(op.add, tile);
      } else if (op.kind == OP_REDUCE) {
        const long long x = (long long)tile * 4 + (tid >> 5);
        if (tid < 128 && x < op.red.nout) reduce_element(op.red, x, tid & 31);
      } else {
        trace_tile(op.tr, tile, red);
      }
      have = false;
    }
    if (l + 1 < p.nlevels) {
      grid_arrive(p.bar);
      // ahead of the wait: this block's first record of the next level and
      // its threads' offsets (neither depends on what the levels write)
      const int next = end[first[l + 2] - 1];
      if ((int)blockIdx.x < next) {
        o = first[l + 1];
        while ((int)blockIdx.x >= end[o]) ++o;
        if (o != cur) {
          w ^= 1;
          fetch(w, o);
          __syncthreads();
          bind(w);
          cur = o;
        }
        __syncthreads();
        if (rec[w].kind == OP_GEMM && rec[w].form >= 3) dot_ahead(rec[w].dot, (unsigned)((int)blockIdx.x - beg[o]), ahead);
        have = true;
      }
      good = grid_wait(p.bar, (unsigned)(l + 1) * gridDim.x, p.wait, p.err, &ok);
    }
  }
  // The last block out resets the barrier for the next launch.  Where a wait ran
  // out it then writes NaN over all that the phase writes: no other block has
  // anything left to store.
  int lost = 0;
  __syncthreads();  // this block has stored all it will
  if (tid == 0) {
    __threadfence();
    const unsigned out = atomicAdd(p.bar + 1, 1u);  // blocks out before; what is lost, above
    if ((out & (kLost - 1u)) == gridDim.x - 1) {
      p.bar[0] = 0u;
      p.bar[1] = 0u;
      __threadfence();
      lost = out >= kLost ? 1 : 0;
    }
  }
  if (__syncthreads_or(lost)) {
    const double nan = __longlong_as_double(0x7FF8000000000000ll);
    for (int i = 0; i < p.nouts; ++i) {
      double* x = static_cast<double*>(p.base[p.outs[i].slot]);
      for (long long k = tid; k < p.outs[i].doubles; k += kFxThreads) x[k] = nan;
    }
  }
}

// Does the op's output view cover its whole slot, each element once?
bool covers(const Program& p, const Op& op) {
  const long long numel = p.slots[op.write].numel;
  long long n = 1, last = 0;
  if (op.kind == OP_GEMM) {
    if (op.oc != 0 || op.dtc != C64) return false;
    for (const ModeGroup* g : {&op.g.gm, &op.g.gn})
      for (int i = 0; i < g->n; ++i) {
        n *= g->dim[i];
        last += (g->dim[i] - 1) * g->s1[i];
      }
    if (op.g.nb > 1) {
      n *= op.g.nb;
      last += (op.g.nb - 1) * op.g.bsC;
    }
  } else {
    if (op.add_oc != 0 || !op.a.cc) return false;
    for (int i = 0; i < op.a.nd; ++i) {
      n *= op.a.d[i];
      last += (op.a.d[i] - 1) * op.a.sC[i];
    }
  }
  return n == numel && last == numel - 1;
}

// doubles of the op's output buffer up to the last one that it writes
long long out_doubles(const Op& op) {
  long long last = 0;
  if (op.kind == OP_GEMM) {
    last = op.oc + (op.g.nb > 1 ? (op.g.nb - 1) * op.g.bsC : 0);
    for (const ModeGroup* g : {&op.g.gm, &op.g.gn})
      for (int i = 0; i < g->n; ++i) last += (g->dim[i] - 1) * g->s1[i];
    return (last + 1) * (op.dtc == C64 ? 2 : 1);
  }
  if (op.kind == OP_ADD) {
    last = op.add_oc;
    for (int i = 0; i < op.a.nd; ++i) last += (op.a.d[i] - 1) * op.a.sC[i];
    return (last + 1) * (op.a.cc ? 2 : 1);
  }
  if (op.kind == OP_REDUCE) {
    last = op.rd_oout;
    for (int i = 0; i < op.rd.no; ++i) last += (op.rd.dout[i] - 1) * op.rd.so_out[i];
    return 2 * (last + 1);
  }
  const int nb = std::max(op.tr_nb, 1);
  return 2 * ((nb > 1 ? (nb - 1) * op.tr_bsres : 0) + op.tr_n_mu);
}

// The ops of a phase with their dependency levels, sums into one output taken
// apart into temporaries (slots from p.slots.size() on, complex elements in
// `temps`; 0: unused) and one addition.
struct PhaseOps {
  std::vector<Op> ops;
  std::vector<int> level;
  std::vector<long long> temps;
};

// Several ops that add to one output wait for one another in program order
// (a fixed order of the roundings).  Here they write to temporaries instead,
// in one level, and an elementwise op adds these to it in the same order:
// slots beyond p.slots are the temporaries, their extents in `temps`.
PhaseOps phase_ops(const Program& p, Program::Phase ph) {
  PhaseOps r;
  const int n0 = (int)p.slots.size();
  const bool shared = !p.slot_buf.empty();  // shared buffers: keep the order they were planned for
  std::vector<std::vector<int>> pending(n0);  // per slot: indices into r.ops of ops moved to temporaries
  auto flush = [&](int c) {
    std::vector<int> q;
    q.swap(pending[c]);
    if (q.empty()) return;
    if (q.size() == 1) {  // alone: back to its own output
      Op& o = r.ops[q[0]];
      r.temps[o.write - n0] = 0;
      o.write = c;
      (o.kind == OP_GEMM ? o.sc : o.add_sc) = c;
      (o.kind == OP_GEMM ? o.g.acc : o.a.acc) = 1;
      o.reads.push_back(c);
      return;
    }
    for (size_t k = 0; k < q.size(); k += kMaxAddTerms) {
      Op o;
      o.kind = OP_ADD;
      o.tag = p.name + ":sum";
      memset(&o.a, 0, sizeof(o.a));
      const long long numel = p.slots[c].numel;
      for (int i = 0; i < kAddDims; ++i) o.a.d[i] = 1;
      o.a.nd = 1;
      o.a.d[0] = (int)numel;
      o.a.sC[0] = 1;
      o.a.total = numel;
      o.a.cc = 1;
      o.a.acc = 2;  // C + x1 + x2 ..: the roundings of a launch per op
      o.add_sc = o.write = c;
      o.add_oc = 0;
      o.reads = {c};
      for (size_t t = k; t < q.size() && t < k + kMaxAddTerms; ++t) {
        const int x = r.ops[q[t]].write, j = o.a.nt++;
        o.a.t[j].sA[0] = 1;
        o.a.t[j].ac = 1;
        o.a.t[j].cr = 1.0;
        o.add_slots[j][0] = x;
        o.add_slots[j][1] = -1;
        o.add_off[j][0] = o.add_off[j][1] = 0;
        o.reads.push_back(x);
      }
      r.ops.push_back(o);
    }
  };
  for (const Op& op : p.ops) {
    if (!Program::in_phase(op, ph)) continue;
    const bool acc = (op.kind == OP_GEMM && op.g.acc) || (op.kind == OP_ADD && op.a.acc);
    for (int s : op.reads)
      if (s >= 0 && s < n0 && !(acc && s == op.write)) flush(s);
    if (acc && !shared && op.write >= 0 && p.slots[op.write].numel < (1LL << 30) && covers(p, op)) {
      Op o = op;
      const int t = n0 + (int)r.temps.size();
      r.temps.push_back(p.slots[op.write].numel);
      o.write = t;
      (o.kind == OP_GEMM ? o.sc : o.add_sc) = t;
      (o.kind == OP_GEMM ? o.g.acc : o.a.acc) = 0;
      o.reads.clear();
      for (int s : op.reads)
        if (s != op.write) o.reads.push_back(s);
      pending[op.write].push_back((int)r.ops.size());
      r.ops.push_back(o);
      continue;
    }
    if (op.write >= 0) flush(op.write);
    r.ops.push_back(op);
  }
  for (int c = 0; c < n0; ++c) flush(c);
  // levels: after every op whose output it reads or overwrites, and after
  // every reader of what it overwrites
  const size_t n = n0 + r.temps.size();
  std::vector<int> wr(n, -1), rd(n, -1);
  auto buf = [&](int s) { return shared && s < (int)p.slot_buf.size() ? p.slot_buf[s] : s; };
  for (const Op& op : r.ops) {
    int l = 0;
    for (int s : op.reads)
      if (s >= 0) l = std::max(l, wr[buf(s)] + 1);
    if (op.write >= 0) l = std::max(l, std::max(wr[buf(op.write)], rd[buf(op.write)]) + 1);
    for (int s : op.reads)
      if (s >= 0) rd[buf(s)] = std::max(rd[buf(s)], l);
    if (op.write >= 0) wr[buf(op.write)] = l;
    r.level.push_back(l);
  }
  return r;
}

}  // namespace

void PhaseKernel::build(const Program& p, Program::Phase ph, std::vector<void*>& owned, long long& bytes) {
  ok = false;
  double flops = 0.0;
  int n = 0;
  for (const Op& op : p.ops) {
    if (!Program::in_phase(op, ph)) continue;
    ++n;
    flops += (double)op.flops;
    if (op.kind == OP_GEMM) {
      if (op.backend != GB_FP64 || op.dtc != C64 || (op.dta != C64 && op.dtb != C64)) return;
    } else if (op.kind == OP_ADD) {
      if (op.a.total <= 0 || op.a.total > 0x3FFFFFFFLL) return;
    } else if (op.kind == OP_REDUCE) {
      if (op.rd.nout <= 0 || op.rd.nout > 0x3FFFFFFFLL) return;
    } else if (op.kind != OP_TRACE) {
      return;
    }
  }
  if (n < 2 || n > kPhaseOps || flops > kPhaseFlops) return;
  const PhaseOps q = phase_ops(p, ph);
  n = (int)q.ops.size();
  if (n > kPhaseOps || p.slots.size() > (size_t)kPhaseSlots) return;
  const std::vector<int>& lev = q.level;
  std::vector<int> order(n);
  for (int i = 0; i < n; ++i) order[i] = i;
  // contractions first within a level: they take longest
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return lev[a] != lev[b] ? lev[a] < lev[b] : (q.ops[a].kind == OP_GEMM) > (q.ops[b].kind == OP_GEMM);
  });
  // the temporaries follow the records in one allocation
  const int n0 = (int)p.slots.size();
  std::vector<size_t> toff;
  size_t tbytes = 0;
  for (long long t : q.temps) {
    toff.push_back(tbytes);
    tbytes += ((size_t)t * 16 + 255) / 256 * 256;
  }
  if (tbytes > kPhaseTempMax) return;
  char* tmem = nullptr;
  if (tbytes) {
    if (cudaMalloc(&tmem, tbytes) != cudaSuccess) {
      cudaGetLastError();
      return;  // a launch per op needs none
    }
    owned.push_back(tmem);
    bytes += (long long)tbytes;
    // all-ones bytes are NaN: a read of memory no op wrote cannot pass silently
    if (cudaMemset(tmem, 0xFF, tbytes) != cudaSuccess) throw std::runtime_error("clearing the phase temporaries failed");
  }
  std::vector<PhaseOp> recs(n);
  std::vector<int> first, beg(n), end(n);
  std::vector<int2> tables;
  std::vector<std::pair<int, int>> table_at;  // (record, pointer) of each table, its pbyte the offset in bytes
  smem_ = 0;
  widest_ = 1;
  int at = 0, cur = -1;
  for (int k = 0; k < n; ++k) {
    const Op& op = q.ops[order[k]];
    PhaseOp& r = recs[k];
    memset(&r, 0, sizeof(r));
    auto ptr = [&](size_t where, int slot, long long byte) {
      const bool temp = slot >= n0;
      r.pslot[r.nptr] = temp ? -2 : slot;
      r.poff[r.nptr] = (int)where;
      r.pbyte[r.nptr] = temp ? (long long)(uintptr_t)(tmem + toff[slot - n0]) + byte : byte;
      ++r.nptr;
    };
    r.kind = op.kind;
    long long tiles = 0;
    if (op.kind == OP_GEMM) {
      Op u = op;
      Program::plan_gemm(u, false, -2);  // no K splits: a fixed order of the roundings
      GemmArgs g;
      FxPlan f;
      if (fx_plan(u, g, f) != cudaSuccess) return;
      r.form = (f.tile == 5 ? 3 : 0) + (f.ac && f.bc ? 0 : f.ac ? 1 : 2);
      size_t pa, pb, pc;
      if (f.tile == 5) {
        DotRec& d = r.dot;
        d.M = g.M;
        d.N = g.N;
        d.K = g.K;
        d.lw = f.flags;
        // a warp per scheduler where that still fits one round of blocks
        const long long threads = ((long long)g.M * g.N << d.lw) * g.nb;
        d.threads = kFxThreads;
        while (d.threads > 128 && threads <= (long long)(d.threads / 2) * 152) d.threads /= 2;
        d.ntiles = (int)(((long long)g.M * g.N + (d.threads >> d.lw) - 1) / (d.threads >> d.lw));
        d.acc = g.acc;
        d.p2 = f.p2;
        d.e2 = f.e2;
        d.neg = f.neg;
        d.ar = g.ar;
        d.ai = g.ai;
        d.bsA = g.bsA;
        d.bsB = g.bsB;
        d.bsC = g.bsC;
        tiles = (long long)d.ntiles * g.nb;
        const size_t w = offsetof(PhaseOp, dot);
        const ModeGroup* grp[3] = {&g.gm, &g.gn, &g.gk};
        const size_t where[3] = {offsetof(DotRec, mt), offsetof(DotRec, nt), offsetof(DotRec, kt)};
        const int len[3] = {g.M, g.N, g.K};
        for (int q3 = 0; q3 < 3; ++q3) {
          table_at.push_back({k, (int)r.nptr});
          ptr(w + where[q3], -1, (long long)(tables.size() * sizeof(int2)));  // made an address once allocated
          for (int i = 0; i < len[q3]; ++i) {
            long long o0 = 0, o1 = 0;
            int l = i;
            for (int m = grp[q3]->n - 1; m >= 0; --m) {
              o0 += (long long)(l % grp[q3]->dim[m]) * grp[q3]->s0[m];
              o1 += (long long)(l % grp[q3]->dim[m]) * grp[q3]->s1[m];
              l /= grp[q3]->dim[m];
            }
            if (o0 > 0x3FFFFFFFLL || o1 > 0x3FFFFFFFLL) return;
            tables.push_back(make_int2((int)o0, (int)o1));
          }
        }
        if (tables.size() > kPhaseTableMax) return;
        pa = w + offsetof(DotRec, A);
        pb = w + offsetof(DotRec, B);
        pc = w + offsetof(DotRec, C);
      } else {
        r.gemm.g = g;
        r.gemm.f = f;
        tiles = f.tiles * g.nb * g.nsplit;
        const int bm = kTiles[f.tile][0], bn = kTiles[f.tile][1];
        smem_ = std::max(smem_, (size_t)fx_k_bytes(bm, bn, f.ac, f.bc) * f.kc);
        const size_t w = offsetof(PhaseOp, gemm) + offsetof(GemmRec, g);
        pa = w + offsetof(GemmArgs, A);
        pb = w + offsetof(GemmArgs, B);
        pc = w + offsetof(GemmArgs, C);
      }
      ptr(f.swapped ? pb : pa, op.sa, op.oa * elem_bytes(op.dta));
      ptr(f.swapped ? pa : pb, op.sb, op.ob * elem_bytes(op.dtb));
      ptr(pc, op.sc, op.oc * elem_bytes(op.dtc));
    } else if (op.kind == OP_ADD) {
      AddRec& d = r.add;
      const AddArgs& x = op.a;
      d.nd = x.nd;
      d.nt = x.nt;
      d.cc = x.cc;
      d.acc = x.acc;
      d.total = (unsigned)x.total;
      // a warp per block before a second one
      d.per = 32 * (int)std::max<long long>(1, (x.total + 32 * 152 - 1) / (32 * 152));
      tiles = (x.total + d.per - 1) / d.per;
      auto narrow = [&](const long long* from, int* to) {
        long long last = 0;
        for (int i = 0; i < kAddDims; ++i) {
          to[i] = (int)from[i];
          if (i < x.nd) last += (x.d[i] - 1) * std::llabs(from[i]);
        }
        return last <= 0x3FFFFFFFLL;
      };
      bool fits = narrow(x.sC, d.sC);
      for (int i = 0; i < kAddDims; ++i) d.d[i] = (unsigned)std::max(x.d[i], 1);
      ptr(offsetof(PhaseOp, add) + offsetof(AddRec, C), op.add_sc, op.add_oc * (x.cc ? 16 : 8));
      for (int t = 0; t < x.nt; ++t) {
        AddRecTerm& dt = d.t[t];
        fits = narrow(x.t[t].sA, dt.sA) && fits;
        fits = narrow(x.t[t].sB, dt.sB) && fits;
        dt.ac = x.t[t].ac;
        dt.bc = x.t[t].bc;
        dt.cr = x.t[t].cr;
        dt.ci = x.t[t].ci;
        const size_t w = offsetof(PhaseOp, add) + offsetof(AddRec, t) + t * sizeof(AddRecTerm);
        ptr(w + offsetof(AddRecTerm, A), op.add_slots[t][0], op.add_off[t][0] * (x.t[t].ac ? 16 : 8));
        ptr(w + offsetof(AddRecTerm, B), op.add_slots[t][1],
            op.add_slots[t][1] >= 0 ? op.add_off[t][1] * (x.t[t].bc ? 16 : 8) : 0);
      }
      if (!fits) return;
    } else if (op.kind == OP_REDUCE) {
      r.red = op.rd;
      tiles = (op.rd.nout + 3) / 4;
      const size_t w = offsetof(PhaseOp, red);
      ptr(w + offsetof(ReduceArgs, out), op.rd_out, op.rd_oout * 16);
      ptr(w + offsetof(ReduceArgs, X), op.rd_x, op.rd_ox * 16);
      ptr(w + offsetof(ReduceArgs, Y), op.rd_y, op.rd_y >= 0 ? op.rd_oy * (op.rd.ycplx ? 16 : 8) : 0);
    } else {
      TraceRec& t = r.tr;
      t.n = p.dims.n;
      t.o = p.dims.o;
      t.n_mu = op.tr_n_mu;
      const int nb = std::max(op.tr_nb, 1);
      for (int q = 0; q < 4; ++q) t.bs[q] = nb > 1 ? op.tr_bs[q] : 0;
      t.bsres = nb > 1 ? op.tr_bsres : 0;
      tiles = (long long)op.tr_n_mu * nb;
      const size_t w = offsetof(PhaseOp, tr);
      ptr(w + offsetof(TraceRec, mu), S_MU, 0);
      ptr(w + offsetof(TraceRec, dij), op.tr_slots[0], 0);
      ptr(w + offsetof(TraceRec, l1), op.tr_slots[1], 0);
      ptr(w + offsetof(TraceRec, dai), op.tr_slots[2], 0);
      ptr(w + offsetof(TraceRec, dab), op.tr_slots[3], 0);
      ptr(w + offsetof(TraceRec, res), S_RES, 0);
    }
    if (lev[order[k]] != cur) {
      cur = lev[order[k]];
      first.push_back(k);
      at = 0;
    }
    if (tiles < 1 || at + tiles > 0x3FFFFFFFLL) return;
    beg[k] = at;
    at += (int)tiles;
    end[k] = at;
    widest_ = std::max(widest_, at);
  }
  nlevels_ = (int)first.size();
  nops_ = n;
  nslots_ = n0;
  std::vector<PhaseOut> outs;
  for (const Op& op : q.ops) {
    if (op.write < 0 || op.write >= n0) continue;
    const long long doubles = out_doubles(op);
    bool known = false;
    for (PhaseOut& x : outs)
      if (x.slot == op.write) {
        known = true;
        x.doubles = std::max(x.doubles, doubles);
      }
    if (!known) outs.push_back(PhaseOut{op.write, 0, doubles});
  }
  nouts_ = (int)outs.size();
  first.push_back(n);
  std::vector<int> tab(first);
  tab.insert(tab.end(), beg.begin(), beg.end());
  tab.insert(tab.end(), end.begin(), end.end());
  const size_t rb = recs.size() * sizeof(PhaseOp), tb = (tab.size() * sizeof(int) + 255) / 256 * 256,
               ob = (tables.size() * sizeof(int2) + 255) / 256 * 256, wb = (outs.size() * sizeof(PhaseOut) + 255) / 256 * 256;
  char* d = nullptr;
  if (cudaMalloc(&d, rb + tb + 256 + ob + wb) != cudaSuccess) {
    cudaGetLastError();
    return;  // a launch per op needs no records
  }
  owned.push_back(d);
  bytes += (long long)(rb + tb + 256 + ob + wb);
  for (const auto& at : table_at) {
    recs[at.first].pslot[at.second] = -2;
    recs[at.first].pbyte[at.second] += (long long)(uintptr_t)(d + rb + tb + 256);
  }
  std::vector<char> host(rb + tb + 256 + ob + wb, 0);  // one copy, the barrier's words zero
  memcpy(host.data(), recs.data(), rb);
  memcpy(host.data() + rb, tab.data(), tab.size() * sizeof(int));
  if (!tables.empty()) memcpy(host.data() + rb + tb + 256, tables.data(), tables.size() * sizeof(int2));
  if (!outs.empty()) memcpy(host.data() + rb + tb + 256 + ob, outs.data(), outs.size() * sizeof(PhaseOut));
  if (cudaMemcpy(d, host.data(), host.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaDeviceSynchronize() != cudaSuccess)
    throw std::runtime_error("uploading the phase records failed");
  ops_ = d;
  tab_ = reinterpret_cast<int*>(d + rb);
  bar_ = reinterpret_cast<unsigned*>(d + rb + tb);
  err_ = reinterpret_cast<int*>(d + rb + tb + 128);
  outs_ = d + rb + tb + 256 + ob;
  ok = true;
}

cudaError_t PhaseKernel::launch(const std::vector<void*>& bases, int blocks, cudaStream_t st) const {
  constexpr int kMaxDev = 64;
  static std::once_flag once[kMaxDev];
  static cudaError_t attr_err[kMaxDev] = {};
  static int resident[kMaxDev] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  std::call_once(once[dev], [dev] {
    const int most = fx_k_bytes(16, 16, true, true) * fx_chunk(16, 16, true, true);
    int sms = 0, per = 0;
    cudaError_t e = cudaFuncSetAttribute(phase_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, phase_kernel, kFxThreads, most);
    resident[dev] = sms * per;
    attr_err[dev] = e;
  });
  if (attr_err[dev] != cudaSuccess) return attr_err[dev];
  PhaseArgs a;
  a.ops = static_cast<const PhaseOp*>(ops_);
  a.tab = tab_;
  a.outs = static_cast<const PhaseOut*>(outs_);
  a.nouts = nouts_;
  a.wait = wait == 0 ? kBarrierLimit : wait;
  a.nops = nops_;
  a.nlevels = nlevels_;
  a.bar = bar_;
  a.err = err_;
  for (int i = 0; i < nslots_; ++i) a.base[i] = bases[i];
  for (int i = nslots_; i < kPhaseSlots; ++i) a.base[i] = nullptr;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)std::max(1, std::min({blocks, widest_, resident[dev]})));
  cfg.blockDim = dim3(kFxThreads);
  cfg.dynamicSmemBytes = smem_;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  count_launch();
  return cudaLaunchKernelEx(&cfg, phase_kernel, a);
}

}  // namespace tdcc
