// gt_pcg_impl.cuh -- Jacobi-PCG as one persistent kernel: kernels and launches.
// gt_pcg.cu, gt_pcg_ir.cu and gt_pcg_fp32.cu instantiate them for one precision
// each (compiled in parallel).
//
// Two kernels: gt_pcg_local.cuh keeps each CTA's vectors, its halo of p and
// what fits of the matrix in shared memory (every system whose local sets fit);
// k_pcg below works on global vectors.  Both run the iteration described here.
//
// The whole iteration runs inside one launch (chunks of iterations per
// launch): CTA c owns a contiguous range of block rows, every
// phase works on the CTA's own rows, and phases are separated by a grid-wide
// barrier.  A reduction is two-level and identical in every CTA: each CTA
// writes its partial sums, and after the barrier every CTA adds all partials
// in the same fixed order, so alpha, beta and the convergence decisions are
// bitwise the same in all CTAs without a further broadcast.  Per iteration:
//
//   P1  q = A p (own rows), p.q            -> barrier, alpha = rz / pq
//   P2  xs += alpha p, r -= alpha q,       -> barrier, beta, convergence
//       z = Dinv r, r.z, r.r
//   [reliable update, when due]
//   P3  x += xs, xs = 0                    -> barrier
//   P4  r = b - A64 x (FP64), z = Dinv r   -> barrier, r.z, ||r||^2
//   P5  p = z + beta p                     -> barrier
//
// The iteration runs in X (FP64 or FP32) on the correction xs since the last
// update, with SpMV values of type V.  With reliable updates (RELIABLE) the
// FP64 solution takes the correction and the FP64 true residual replaces the
// recurrence residual whenever the recurrence residual fell by delta since
// the last update, claims convergence, or maxit is reached; the direction p
// is then rebuilt from the true residual.  Convergence is decided on the
// FP64 true residual.  Without reliable updates (the FP32-only mode) the
// recurrence residual decides and x takes xs at the end.
//
// Every grid barrier waits with a time limit: a barrier that does not
// complete within a second records an error and the kernel returns (the
// cooperative launch makes all CTAs co-resident, so this does not happen in
// a correct run).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>

#include "gt_internal.cuh"
#include "gt_rowdot.cuh"

namespace gt {
namespace pcg {

constexpr int PT = 256;          // threads per CTA
constexpr int NW = PT / 32;      // warps per CTA
constexpr int PSLOT = 4;         // doubles per CTA partial
constexpr uint64_t BAR_TIMEOUT_NS = 1000000000ull;
constexpr int PCG_STALLED = 1;   // internal status: the FP32 iteration stalled
constexpr int PCG_NOFIT = kPcgNoFit;  // internal status: the sliced form's local sets do not fit

struct PState {
  double rz, rzold, rr, rmax2, bb, tol2;
  double beta;      // of the next direction (local kernel)
  double thr;       // ||r||^2 of the next reliable update (local kernel)
  uint32_t epoch;   // sums done so far (local kernel)
  int32_t iters, nupd;
  int32_t started;  // sliced form: a chunk has run
  int32_t done;     // 1 converged or maxit, 2 FP32 iteration stalled or slowed down: continue in FP64
  int32_t stall;    // consecutive reliable updates with less than a halving of the true residual
  int32_t it_upd;   // iteration of the last reliable update
  int32_t max_cyc;  // longest cycle between reliable updates so far
};

// when an iteration ends, updates its residual or goes on in FP64
struct PRule {
  double rtol2, delta2;
  int maxit;
  double stall_ratio;  // hand-over rule (Ctx::ir_stall_ratio / ir_stall_count)
  int stall_count;
};

struct PArgs : PRule {
  const int64_t* rowptr;
  const int32_t* colind;
  const void* val;       // iteration values (V)
  const double* val64;   // FP64 values (true residual), may be null without reliable updates
  int64_t nrows;         // block rows
  int nb;                // CTAs that solve this system (the grouped launch)
  const double* b;
  double* x;
  void *xs, *r, *z, *p, *q;
  const void* dinv;
  double* part;          // 3 slots x gridDim.x x PSLOT; local kernel: its slots and counters, zero at the start
  int lanes;             // local kernel: entry lanes per scalar row (with_lanes)
  double* resid;         // sliced form: FP64 products of the residual
  int init;              // sliced form: how its first chunk starts
  uint16_t* lcol;        // local kernel: local columns of the entries not held in shared memory
  uint32_t* bar;         // barrier counter, zero at launch
  int32_t* err;          // set to 1 when a barrier timed out
  PState* st;
};

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// grid-wide barrier number `target / gridDim.x`; false when it timed out
// (no arrival for timeout_ns: the error word is set and every CTA returns)
__device__ __forceinline__ bool grid_sync(uint32_t* bar, uint32_t target, int32_t* err, int* s_abort,
                                          uint64_t timeout_ns = BAR_TIMEOUT_NS) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    uint64_t t0 = global_ns();
    while (ld_acquire(bar) < target) {
      if (global_ns() - t0 > timeout_ns) {
        atomicExch(err, 1);
        *s_abort = 1;
        break;
      }
      __nanosleep(32);
    }
    __threadfence();
  }
  __syncthreads();
  return *s_abort == 0;
}

// CTA sum of K values -> out[0..K) (written by thread 0)
template <int K>
__device__ __forceinline__ void cta_sum(double (&v)[K], double* s_red, double* out) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; k++) {
    double t = v[k];
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) s_red[k * NW + w] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      double t = 0.0;
#pragma unroll
      for (int i = 0; i < NW; i++) t += s_red[k * NW + i];
      __stcg(out + k, t);
    }
  }
}

// sum of the CTA partials of a slot, in one fixed order that is identical in
// every CTA: each thread loads its (at most a few) partials at once, warp
// butterflies (whose result is the same in all lanes), then the warp totals
// in warp order; result in s_tot[0..K).  s_red is free again at this point.
template <int K>
__device__ __forceinline__ void grid_total(const double* slot, int nb, double* s_red, double* s_tot) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double t[K];
#pragma unroll
  for (int k = 0; k < K; k++) t[k] = 0.0;
  for (int i = threadIdx.x; i < nb; i += PT) {
    const double2 v01 = __ldcg(reinterpret_cast<const double2*>(slot + (size_t)i * PSLOT));
    t[0] += v01.x;
    if (K > 1) t[1] += v01.y;
    if (K > 2) t[2] += __ldcg(slot + (size_t)i * PSLOT + 2);
  }
#pragma unroll
  for (int k = 0; k < K; k++) {
#pragma unroll
    for (int o = 16; o; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
    if (lane == 0) s_red[k * NW + w] = t[k];
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < NW; i++) s += s_red[threadIdx.x * NW + i];
    s_tot[threadIdx.x] = s;
  }
  __syncthreads();
}

// The solve of one system by nb CTAs, this CTA being number blk of them
// (k_pcg: the whole grid).
// The shared arrays are the caller's.
template <int BS, int G, class V, class X, bool RELIABLE>
__device__ __forceinline__ void pcg_body(const PArgs& a, int nb, int blk, int init, int it_end, double* s_red,
                                         double* s_tot, int& s_abort) {
  constexpr int NG = PT / G;  // row groups per CTA
  if (threadIdx.x == 0) s_abort = 0;
  const int tid = threadIdx.x;
  const int gl = tid % G, grp = tid / G;
  const int64_t rows_per = (a.nrows + nb - 1) / nb;
  const int64_t r0 = min(a.nrows, (int64_t)blk * rows_per), r1 = min(a.nrows, r0 + rows_per);
  const int64_t e0 = r0 * BS, e1 = r1 * BS;
  X* xs = (X*)a.xs;
  X* r = (X*)a.r;
  X* z = (X*)a.z;
  X* p = (X*)a.p;
  X* q = (X*)a.q;
  const X* dinv = (const X*)a.dinv;
  const V* val = (const V*)a.val;
  double* slot0 = a.part;
  double* slot1 = a.part + (size_t)nb * PSLOT;
  double* slot2 = a.part + (size_t)2 * nb * PSLOT;
  uint32_t nbar = 0;
  PState S = *a.st;
  __syncthreads();

  if (init == 2) {
    // continuation of a stalled FP32 run in FP64: x holds the FP64
    // solution; r = b - A x, z = Dinv r, p = z (the iteration count and
    // ||b|| carry over)
    double v[2] = {0.0, 0.0};
    for (int64_t base = r0; base < r1; base += NG) {
      int64_t row = base + grp;
      const bool valid = row < r1;
      if (!valid) row = r1 - 1;
      double o[BS];
      row_dot<BS, G, double, double, double, true>(a.rowptr, a.colind, a.val64, a.x, row, gl, o);
      if (gl == 0 && valid) {
#pragma unroll
        for (int c = 0; c < BS; c++) {
          const int64_t i = row * BS + c;
          const double ri = a.b[i] - o[c];
          const X rx = (X)ri, zx = dinv[i] * rx;
          r[i] = rx;
          z[i] = zx;
          xs[i] = (X)0;
          v[0] += (double)rx * (double)zx;
          v[1] += ri * ri;
        }
      }
    }
    cta_sum<2>(v, s_red, slot2 + (size_t)blk * PSLOT);
    if (!grid_sync(a.bar, (++nbar) * nb, a.err, &s_abort)) return;
    grid_total<2>(slot2, nb, s_red, s_tot);
    // the FP64 iteration restarts from the true residual (p = z): the FP32
    // run stalled, so its direction no longer fits the true residual, and
    // continuing it made the FP64 recurrence stagnate or diverge at
    // tolerances near the attainable accuracy (measured)
    for (int64_t i = e0 + tid; i < e1; i += PT) p[i] = z[i];
    S.rz = s_tot[0];
    S.rr = s_tot[1];
    S.rmax2 = S.rr;
    S.it_upd = S.iters;
    S.max_cyc = 0;
    S.stall = 0;
    S.done = S.rr <= S.tol2;
    if (!grid_sync(a.bar, (++nbar) * nb, a.err, &s_abort)) return;
  } else if (init) {
    // r = b - A x0 (FP64 products), z = Dinv r, p = z, xs = 0; r.z, r.r, b.b
    double v[3] = {0.0, 0.0, 0.0};
    for (int64_t base = r0; base < r1; base += NG) {
      int64_t row = base + grp;
      const bool valid = row < r1;
      if (!valid) row = r1 - 1;
      double o[BS];
      if constexpr (RELIABLE) row_dot<BS, G, double, double, double, true>(a.rowptr, a.colind, a.val64, a.x, row, gl, o);
      else row_dot<BS, G, V, double, double, true>(a.rowptr, a.colind, val, a.x, row, gl, o);
      if (gl == 0 && valid) {
#pragma unroll
        for (int c = 0; c < BS; c++) {
          const int64_t i = row * BS + c;
          const double bi = a.b[i], ri = bi - o[c];
          const X rx = (X)ri, zx = dinv[i] * rx;
          r[i] = rx;
          z[i] = zx;
          p[i] = zx;
          xs[i] = (X)0;
          v[0] += (double)rx * (double)zx;
          v[1] += ri * ri;
          v[2] += bi * bi;
        }
      }
    }
    cta_sum<3>(v, s_red, slot2 + (size_t)blk * PSLOT);
    if (!grid_sync(a.bar, (++nbar) * nb, a.err, &s_abort)) return;
    grid_total<3>(slot2, nb, s_red, s_tot);
    S.rz = s_tot[0];
    S.rr = s_tot[1];
    S.bb = s_tot[2];
    S.tol2 = a.rtol2 * S.bb;
    S.rmax2 = S.rr;
    S.rzold = 0.0;
    S.iters = 0;
    S.nupd = 0;
    S.done = S.rr <= S.tol2;
  }

  while (!S.done && S.iters < it_end) {
    // P1: q = A p, p.q
    double pq;
    {
      X acc = (X)0;
      for (int64_t base = r0; base < r1; base += 2 * NG) {
        int64_t ra = base + grp, rb = base + NG + grp;
        const bool va = ra < r1, vb = rb < r1;
        if (!va) ra = r1 - 1;
        if (!vb) rb = r1 - 1;
        X oa[BS], ob[BS];
        row_dot<BS, G, V, X, X, true>(a.rowptr, a.colind, val, p, ra, gl, oa);
        row_dot<BS, G, V, X, X, true>(a.rowptr, a.colind, val, p, rb, gl, ob);
        if (gl == 0) {
#pragma unroll
          for (int c = 0; c < BS; c++) {
            if (va) {
              q[ra * BS + c] = oa[c];
              acc += oa[c] * __ldcg(p + ra * BS + c);
            }
            if (vb) {
              q[rb * BS + c] = ob[c];
              acc += ob[c] * __ldcg(p + rb * BS + c);
            }
          }
        }
      }
      double v[1] = {(double)acc};
      cta_sum<1>(v, s_red, slot0 + (size_t)blk * PSLOT);
      if (!grid_sync(a.bar, (++nbar) * nb, a.err, &s_abort)) return;
      grid_total<1>(slot0, nb, s_red, s_tot);
      pq = s_tot[0];
    }
    const X alpha = (X)(S.rz / pq);
    // P2: xs += alpha p, r -= alpha q, z = Dinv r; r.z, r.r
    double rzn, rr;
    {
      X v0 = (X)0, v1 = (X)0;
#pragma unroll 4
      for (int64_t i = e0 + tid; i < e1; i += PT) {
        const X ri = r[i] - alpha * q[i];
        const X zi = dinv[i] * ri;
        xs[i] += alpha * p[i];
        r[i] = ri;
        z[i] = zi;
        v0 += ri * zi;
        v1 += ri * ri;
      }
      double v[2] = {(double)v0, (double)v1};
      cta_sum<2>(v, s_red, slot1 + (size_t)blk * PSLOT);
      if (!grid_sync(a.bar, (++nbar) * nb, a.err, &s_abort)) return;
      grid_total<2>(slot1, nb, s_red, s_tot);
      rzn = s_tot[0];
      rr = s_tot[1];
    }
    S.iters += 1;
    double beta = rzn / S.rz;
    S.rzold = S.rz;
    S.rz = rzn;
    S.rr = rr;
    const bool stop = rr <= S.tol2 || S.iters >= a.maxit || !(rr == rr);
    if constexpr (RELIABLE) {
      // an FP32 cycle (recurrence residual down by delta) that runs past 2.5x
      // the longest earlier cycle: the FP32 iteration has lost the rate of
      // the exact iteration (eps32 * cond(A) too large); hand over to FP64
      const int cyc = S.iters - S.it_upd;
      const bool slow = sizeof(X) < sizeof(double) && (cyc > kSlowCycle || (S.max_cyc > 0 && cyc > (5 * S.max_cyc) / 2 + 16));
      if (stop || slow || rr <= a.delta2 * S.rmax2) {
        // P3: x += xs
        for (int64_t i = e0 + tid; i < e1; i += PT) {
          a.x[i] += (double)xs[i];
          xs[i] = (X)0;
        }
        if (!grid_sync(a.bar, (++nbar) * nb, a.err, &s_abort)) return;
        // P4: true residual in FP64
        double v[2] = {0.0, 0.0};
        for (int64_t base = r0; base < r1; base += NG) {
          int64_t row = base + grp;
          const bool valid = row < r1;
          if (!valid) row = r1 - 1;
          double o[BS];
          row_dot<BS, G, double, double, double, true>(a.rowptr, a.colind, a.val64, a.x, row, gl, o);
          if (gl == 0 && valid) {
#pragma unroll
            for (int c = 0; c < BS; c++) {
              const int64_t i = row * BS + c;
              const double ri = a.b[i] - o[c];
              const X rx = (X)ri, zx = dinv[i] * rx;
              r[i] = rx;
              z[i] = zx;
              v[0] += (double)rx * (double)zx;
              v[1] += ri * ri;
            }
          }
        }
        cta_sum<2>(v, s_red, slot2 + (size_t)blk * PSLOT);
        if (!grid_sync(a.bar, (++nbar) * nb, a.err, &s_abort)) return;
        grid_total<2>(slot2, nb, s_red, s_tot);
        beta = S.rzold != 0.0 ? s_tot[0] / S.rzold : 0.0;
        // the recurrence lost track of the true residual (an FP64 run past
        // its attainable accuracy, or FP32 drift): the next direction
        // restarts from the true residual instead of scaling the old one by
        // the true/recurrence mismatch
        if (s_tot[0] > (sizeof(X) == sizeof(double) ? kRestartRatio64 : kRestartRatio) * S.rz) beta = 0.0;
        const double prev = S.rmax2;
        S.rz = s_tot[0];
        S.rr = s_tot[1];
        S.rmax2 = s_tot[1];
        S.nupd += 1;
        S.done = s_tot[1] <= S.tol2 || S.iters >= a.maxit || !(s_tot[1] == s_tot[1]);
        if (sizeof(X) == sizeof(double) && !S.done) {
          // FP64: true-residual checks that do not halve ||r||, kStagnation
          // times running -- the tolerance lies below the attainable accuracy
          // (eps64 * cond(A)); the solve ends, not converged
          S.stall = s_tot[1] > 0.25 * prev ? S.stall + 1 : 0;
          if (S.stall >= kStagnation) S.done = 1;
        }
        if (sizeof(X) < sizeof(double) && !S.done) {
          // the recurrence fell by delta but the true residual did not halve:
          // the FP32 operator no longer resolves the error (eps32 * cond ~ 1)
          S.stall = s_tot[1] > a.stall_ratio * prev ? S.stall + 1 : 0;
          if (S.stall >= a.stall_count || slow) S.done = 2;
        }
        if (cyc > S.max_cyc) S.max_cyc = cyc;
        S.it_upd = S.iters;
      }
    } else {
      S.done = stop;
    }
    if (S.done) break;
    // P5: p = z + beta p
    const X bx = (X)beta;
#pragma unroll 4
    for (int64_t i = e0 + tid; i < e1; i += PT) p[i] = z[i] + bx * p[i];
    if (!grid_sync(a.bar, (++nbar) * nb, a.err, &s_abort)) return;
  }
  if (!RELIABLE && S.done) {
    for (int64_t i = e0 + tid; i < e1; i += PT) {
      a.x[i] += (double)xs[i];
      xs[i] = (X)0;
    }
  }
  if (blk == 0 && tid == 0) *a.st = S;
}

// CTAs an SM (0: the compiler's choice): four, three of block rows of 3, where
// the compiler would spill.  Measured, ms: Q2 hexahedra 30^3 FP64 22.5 (25.3
// by its choice), Q2 elasticity on scattered numberings 16^3 FP64 27.3 (32.6),
// 19^3 FP32 15.0 (20.4); the FP32 iteration with updates is faster by its choice
// (P2 tetrahedra 31^3 21.6, 22.9 with four).
constexpr int pcg_per_sm(int bs, bool fp64, bool reliable) {
  return fp64 ? (bs == 3 ? 3 : 4) : (bs == 3 && !reliable ? 3 : 0);
}
template <int BS, int G, class V, class X, bool RELIABLE>
__global__ void __launch_bounds__(PT, pcg_per_sm(BS, sizeof(X) == sizeof(double), RELIABLE)) k_pcg(PArgs a, int init, int it_end) {
  __shared__ double s_red[3 * NW];
  __shared__ double s_tot[4];
  __shared__ int s_abort;
  pcg_body<BS, G, V, X, RELIABLE>(a, gridDim.x, blockIdx.x, init, it_end, s_red, s_tot, s_abort);
}

#include "gt_pcg_local.cuh"

// Several systems in one launch, for `chunk` more iterations than each one's
// count at entry.  In a cooperative grid CTA c is CTA map[c].y of the
// args[map[c].x].nb CTAs that solve system map[c].x, exactly as that system's
// own launch would (map null: one system, the whole grid); in the cluster
// form cluster c solves system c.
template <int BS, class V, class X, bool RELIABLE, bool CL, bool SL = false>
__device__ __forceinline__ void local_group_entry(const PArgs* args, int sys, int nb, int blk, int init, int chunk,
                                                  unsigned char* smem, int smem_bytes, LShared& S, LCluster* C) {
  const PArgs a = args[sys];
  if (a.st->done) return;  // finished in an earlier launch (the same in all its CTAs)
  int it_end = a.st->iters + chunk;
  if (it_end > a.maxit || it_end < 0) it_end = a.maxit;
  pcg_local_body<BS, V, X, RELIABLE, CL, SL>(a, CL ? nb : a.nb, blk, init, it_end, smem, smem_bytes, S, C);
}
template <int BS, class V, class X, bool RELIABLE>
__global__ void __launch_bounds__(LT, 1) k_pcg_local(const PArgs* __restrict__ args, const int2* __restrict__ map,
                                                         int init, int chunk, int smem_bytes) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ LShared S;
  const int2 m = map ? map[blockIdx.x] : make_int2(0, (int)blockIdx.x);
  local_group_entry<BS, V, X, RELIABLE, false>(args, m.x, 0, m.y, init, chunk, s_dyn, smem_bytes, S, nullptr);
}
template <int BS, class V, class X, bool RELIABLE>
__global__ void __launch_bounds__(LT, 1) k_pcg_cluster(const PArgs* __restrict__ args, int init, int chunk,
                                                    int smem_bytes) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ LShared S;
  __shared__ LCluster C;
  local_group_entry<BS, V, X, RELIABLE, true>(args, blockIdx.x / LCLUSTER, LCLUSTER, blockIdx.x % LCLUSTER, init,
                                                 chunk, s_dyn, smem_bytes, S, &C);
}

// one system in its sliced form (SL), the whole grid
template <class V, class X, bool RELIABLE>
__global__ void __launch_bounds__(LT, 1) k_pcg_sliced(const PArgs* __restrict__ args, int chunk, int smem_bytes) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ LShared S;
  local_group_entry<1, V, X, RELIABLE, false, true>(args, 0, 0, blockIdx.x, args->st->started ? 0 : args->init, chunk, s_dyn, smem_bytes, S, nullptr);
}

template <int BS, class V, class X>
__global__ void k_pdinv(const int64_t* rowptr, const int32_t* diag_pos, const V* val, int64_t nbrows, X* dinv) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nbrows * BS) return;
  int64_t r = t / BS;
  int c = (int)(t - r * BS);
  int64_t k = rowptr[r] + diag_pos[r];
  dinv[t] = (X)(1.0 / (double)val[k * BS * BS + c * BS + c]);
}

// result of one persistent run
struct PRun {
  PState st{};
  bool stalled = false;
};

// One system's persistent solve: its CTA count (as many as give two row
// passes per CTA, at most the co-resident CTAs of k_pcg), its buffers and
// its kernel arguments.  What it still holds when it ends goes back to the
// pool, after the work queued on it.
template <int BS, class V, class X, bool REL>
struct PSolve {
  Ctx* ctx = nullptr;       // owns the buffers (a batch may hold matrices of other contexts)
  Matrix* A = nullptr;
  int nb = 0;
  X *xs = nullptr, *r = nullptr, *z = nullptr, *p = nullptr, *q = nullptr, *dinv = nullptr;
  double* part = nullptr;
  uint16_t* lcol = nullptr; // local kernel only
  double* resid = nullptr;  // sliced form only
  uint32_t* bar = nullptr;  // own (stand-alone) or a slot of a grouped launch's array
  int32_t* err = nullptr;
  PState* st = nullptr;
  bool own_sync = true;     // bar, err and st allocated here
  PArgs* dargs = nullptr;   // args on the device (stand-alone local kernel)
  PArgs args{};
  PSolve() = default;
  PSolve(const PSolve&) = delete;
  PSolve& operator=(const PSolve&) = delete;
  ~PSolve() {
    if (!ctx) return;
    cudaStreamSynchronize(ctx->stream);
    release();
  }
  void release() {
    dfree(ctx, xs);
    dfree(ctx, r);
    dfree(ctx, z);
    dfree(ctx, p);
    dfree(ctx, q);
    dfree(ctx, dinv);
    dfree(ctx, part);
    dfree(ctx, lcol);
    dfree(ctx, resid);
    dfree(ctx, dargs);
    if (own_sync) {
      dfree(ctx, bar);
      dfree(ctx, err);
      dfree(ctx, st);
    }
    ctx = nullptr;
  }
};

// k_pcg of a matrix: lanes per row by its mean row length (row_lanes; block rows
// of 2 are short), and the CTAs that solve it
template <int BS, class V, class X, bool REL>
static int pcg_kernel(Ctx* ctx, const Matrix* A, const void** kern, int* nb) {
  int G = 2;
  *kern = (const void*)k_pcg<BS, 2, V, X, REL>;
  if constexpr (BS != 2)
    if (A->nbrows > 0 && row_lanes((double)A->bnnz / (double)A->nbrows) > 2) {
      G = 4;
      *kern = (const void*)k_pcg<BS, 4, V, X, REL>;
    }
  int per_sm = 0;
  GT_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, *kern, PT, 0));
  if (per_sm < 1) return set_error(ctx, GT_ERR_CUDA, "persistent PCG kernel does not fit on an SM");
  const int NG = PT / G;
  int64_t want = (A->nbrows + 2 * NG - 1) / (2 * NG);  // at least two row passes per CTA
  int64_t cap = (int64_t)per_sm * ctx->num_sms;
  *nb = (int)(want < cap ? (want > 0 ? want : 1) : cap);
  return GT_OK;
}

// The local kernel's launch of one system: one cluster or a grid, its CTA
// count (properties of the system and the device, so a result never depends
// on what else runs) and the shared memory a CTA is given -- est: the
// expected need (the halo about seven times the rows; a grid gets no more
// than it can use, so that systems of several contexts run side by side),
// most: the device's limit, for systems whose local sets do not fit est.
// The kernels' attribute is always set to most: it is the process's, and
// another thread may launch the same kernel with another size.
struct LPlan {
  int nb = 1;
  int est = 0, most = 0;
  bool ok = false;  // the fixed part fits
};
enum class Place { Auto, Cluster, Grid };

template <class K>
static int cta_room(Ctx* ctx, K kern, int* most) {
  cudaFuncAttributes fa{};
  GT_CUDA(ctx, cudaFuncGetAttributes(&fa, (const void*)kern));
  int optin = 0;
  GT_CUDA(ctx, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  *most = (optin - (int)fa.sharedSizeBytes) & ~1023;
  return GT_OK;
}
template <class K>
static int local_plan(Ctx* ctx, const Matrix* A, K kern, bool cluster, size_t xsize, size_t vsize, LPlan* L) {
  const int64_t lsize = xsize == sizeof(float) ? sizeof(float) + sizeof(double) : xsize;  // local set, a component
  GT_TRY(cta_room(ctx, kern, &L->most));
  const int64_t n = A->nbrows * A->bs;
  const int64_t want = (n + kLocalRows - 1) / kLocalRows;
  const int64_t cap = std::min<int64_t>(ctx->num_sms, LMAXCTA);
  L->nb = cluster ? LCLUSTER : (int)std::max<int64_t>(1, std::min(want, cap));
  const int64_t rows = (A->nbrows + L->nb - 1) / L->nb;
  const int64_t tail = ((A->nbrows + 31) / 32) * 6 + 16;
  const int64_t fixed = tail + rows * A->bs * 6 * (int64_t)xsize + (rows + 1) * 4 + 64;
  const int64_t local = std::min<int64_t>(A->nbrows, 8 * rows + 512) * (A->bs * lsize + 4);
  const int64_t ents = (A->bnnz / L->nb + 1) * 5 / 4 + 64;
  const int64_t est = fixed + local + ents * (A->bs * A->bs * (int64_t)vsize + 2);
  L->ok = fixed + rows * (A->bs * (int64_t)xsize + 4) <= L->most && A->bnnz / L->nb < (int64_t(1) << 30);
  L->est = cluster ? L->most : (int)std::min<int64_t>(L->most, (est + 1023) & ~int64_t(1023));
  return GT_OK;
}

// One cluster solves a system whose iteration the barriers dominate: up to
// kClusterWork FP64 operations an iteration, 8/5 of it in FP32, whose
// operations are cheap.  Measured, us a solve, cluster / grid: 2-D Q1 FP64
// 24^2 459 / 659, 64^2 1238 / 1630, 96^2 (190,000) 2522 / 2551, 140^2 4696 /
// 3684; 3-D Q1 FP64 10^3 260 / 352, 19^3 (220,000) 626 / 592, 25^3 1408 / 790;
// FP32 with reliable updates 2-D 96^2 2390 / 2772, 140^2 (400,000) 3814 /
// 3733, 3-D 19^3 625 / 634, 25^3 (540,000) 1107 / 889.
constexpr int64_t kClusterWork = 190000;
static bool cluster_place(const Matrix* A, bool fp64, Place place) {
  if (place != Place::Auto) return place == Place::Cluster;
  const int64_t work = A->bnnz * A->bs * A->bs + row_cost(A->bs) * A->nbrows * A->bs;
  return (fp64 ? work : work * 5 / 8) <= kClusterWork;
}

// entry lanes of a scalar row (with_lanes)
inline int entry_lanes(const Matrix* A, bool fp64) {
  const double avg = A->nbrows > 0 ? (double)A->bnnz / (double)A->nbrows : 1.0;
  return fp64 && avg <= 20 ? 1 : (avg <= 40 ? 2 : 4);
}

// buffers, the start state (zero, or a continuation's) and the Jacobi
// diagonal of one system; bar / err / st come from the caller when given
template <int BS, class V, class X, bool REL>
static int pcg_prepare(Ctx* ctx, PSolve<BS, V, X, REL>& P, Matrix* A, const V* val, const double* b, double* x,
                       double rtol, int maxit, double delta, const PRun* from, int nb, bool local, bool sliced = false,
                       uint32_t* bar = nullptr, int32_t* err = nullptr, PState* st = nullptr) {
  cudaStream_t s = ctx->stream;
  const int64_t n = A->nbrows * BS;
  P.ctx = ctx;
  P.A = A;
  P.nb = nb;
  P.own_sync = bar == nullptr;
  GT_TRY(dalloc(ctx, &P.xs, n));
  GT_TRY(dalloc(ctx, &P.r, n));
  GT_TRY(dalloc(ctx, &P.z, n));
  GT_TRY(dalloc(ctx, &P.p, n));
  GT_TRY(dalloc(ctx, &P.dinv, n));
  if (local) {
    GT_TRY(dalloc(ctx, &P.part, (int64_t)LSLOTS * P.nb + LCTRS));
    GT_TRY(dalloc(ctx, &P.lcol, sliced ? A->sell_total : A->bnnz));
    if (sliced) GT_TRY(dalloc(ctx, &P.resid, n));
    GT_CUDA(ctx, cudaMemsetAsync(P.part, 0, sizeof(double) * (LSLOTS * P.nb + LCTRS), s));
  } else {
    GT_TRY(dalloc(ctx, &P.q, n));
    GT_TRY(dalloc(ctx, &P.part, (int64_t)3 * P.nb * PSLOT));
  }
  if (P.own_sync) {
    GT_TRY(dalloc(ctx, &P.bar, 2));
    GT_TRY(dalloc(ctx, &P.err, 2));
    GT_TRY(dalloc(ctx, (unsigned char**)&P.st, sizeof(PState)));
    GT_CUDA(ctx, cudaMemsetAsync(P.err, 0, 2 * sizeof(int32_t), s));
  } else {
    P.bar = bar;
    P.err = err;
    P.st = st;
  }
  if (from) {
    // continuation: scalars of the FP32 run (iteration count, ||b||, rzold)
    PState* h0 = reinterpret_cast<PState*>(ctx->h_dscratch);
    *h0 = from->st;
    h0->done = 0;
    h0->epoch = 0;
    h0->started = 0;
    GT_CUDA(ctx, cudaMemcpyAsync(P.st, h0, sizeof(PState), cudaMemcpyHostToDevice, s));
    GT_CUDA(ctx, cudaStreamSynchronize(s));
  } else {
    GT_CUDA(ctx, cudaMemsetAsync(P.st, 0, sizeof(PState), s));
  }
  GT_TRY(find_diag(A));
  const double* dval = REL ? A->val64 : (const double*)nullptr;
  if (REL || A->val64)
    k_pdinv<BS, double, X><<<GT_KC(ctx, grid_for(n, 256)), 256, 0, s>>>(A->rowptr, A->diag_pos, A->val64, A->nbrows,
                                                                         P.dinv);
  else
    k_pdinv<BS, V, X><<<GT_KC(ctx, grid_for(n, 256)), 256, 0, s>>>(A->rowptr, A->diag_pos, val, A->nbrows, P.dinv);
  GT_LAUNCH(ctx, "k_pdinv");
  PArgs& args = P.args;
  args.rowptr = A->rowptr;
  args.colind = A->colind;
  args.val = val;
  args.val64 = dval;
  if (sliced) {
    args.rowptr = A->sell_ptr;
    args.colind = A->sell_col;
    args.val = sizeof(V) == sizeof(double) ? (const void*)A->sell_v64 : (const void*)A->sell_v32;
    args.val64 = A->sell_v64;
  }
  args.nrows = A->nbrows;
  args.nb = P.nb;
  args.b = b;
  args.x = x;
  args.xs = P.xs;
  args.r = P.r;
  args.z = P.z;
  args.p = P.p;
  args.q = P.q;
  args.dinv = P.dinv;
  args.part = P.part;
  args.lcol = P.lcol;
  args.resid = P.resid;
  args.init = from ? 2 : 1;
  args.lanes = entry_lanes(A, sizeof(X) == sizeof(double));
  args.bar = P.bar;
  args.err = P.err;
  args.st = P.st;
  args.rtol2 = rtol * rtol;
  args.delta2 = delta * delta;
  args.maxit = maxit;
  args.stall_ratio = ctx->ir_stall_ratio;
  args.stall_count = ctx->ir_stall_count;
  return GT_OK;
}

// the outcome of a finished system (h: its final state; err: a barrier timed
// out) and the release of its buffers
template <int BS, class V, class X, bool REL>
static int pcg_finish(PSolve<BS, V, X, REL>& P, const PState& h, bool err, PRun* out) {
  Ctx* ctx = P.ctx;
  int status = GT_OK;
  if (err) status = set_error(ctx, GT_ERR_TIMEOUT, "persistent PCG: a grid barrier timed out");
  out->st = h;
  if (status == GT_OK && h.done == 2) {
    status = PCG_STALLED;
    out->stalled = true;
  } else if (status == GT_OK && !(h.rr <= h.tol2)) {
    status = GT_ERR_NOT_CONVERGED;
  }
  P.release();
  return status;
}

// place in Matrix::local_sets of a form: iteration type and residuals, sliced
// or not
template <class X, bool REL>
constexpr int local_form(bool sliced) {
  return (sizeof(X) == sizeof(double) ? 0 : REL ? 1 : 2) + 3 * sliced;
}

// One system on the whole device.  The local kernel (gt_pcg_local.cuh) takes
// it unless its local sets do not fit in shared memory -- a numbering that
// scatters a CTA's columns over the whole system; then the kernel on global
// vectors does.  Measured, us a solve, local / global vectors: 2-D Q1 64 x 64
// FP64 1630 / 2790, 3-D Q1 25^3 mixed 889 / 1370, Q2 elasticity 11^3 FP64
// 15200 / 42200.
template <int BS, class V, class X, bool REL>
int run_typed(Ctx* ctx, Matrix* A, const V* val, const double* b, double* x, double rtol, int maxit, double delta,
              const PRun* from, PRun* out) {
  cudaStream_t s = ctx->stream;
  auto lkern = k_pcg_local<BS, V, X, REL>;
  LPlan L;
  GT_TRY(local_plan(ctx, A, lkern, false, sizeof(X), sizeof(V), &L));
  uint8_t& known = A->local_sets[local_form<X, REL>(false)];
  int smem = known ? L.most : L.est;
  for (bool local = L.ok && known < 2;;) {
    int nb = L.nb;
    const void* gkern = nullptr;
    if (!local) GT_TRY((pcg_kernel<BS, V, X, REL>(ctx, A, &gkern, &nb)));
    else GT_CUDA(ctx, cudaFuncSetAttribute(lkern, cudaFuncAttributeMaxDynamicSharedMemorySize, L.most));
    PSolve<BS, V, X, REL> P;
    GT_TRY((pcg_prepare<BS, V, X, REL>(ctx, P, A, val, b, x, rtol, maxit, delta, from, nb, local)));
    PArgs& args = P.args;
    PState h{};
    bool err = false;
    int chunk = local ? 512 : 32, done_iters = from ? from->st.iters : 0;
    const int2* dmap = nullptr;
    if (local) {
      GT_TRY(dalloc(ctx, &P.dargs, 1));
      GT_TRY(copy_in(ctx, P.dargs, (const PArgs*)&args, 1));
    }
    for (int launch = 0;; launch++) {
      int init = launch == 0 ? (from ? 2 : 1) : 0;
      int it_end = done_iters + chunk;
      if (it_end > maxit || it_end < 0) it_end = maxit;
      ctx->launches++;
      if (local) {
        void* kargs[] = {&P.dargs, &dmap, &init, &chunk, &smem};
        GT_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)lkern, dim3(P.nb), dim3(LT), kargs, smem, s));
      } else {
        GT_CUDA(ctx, cudaMemsetAsync(P.bar, 0, sizeof(uint32_t), s));
        void* kargs[] = {&args, &init, &it_end};
        GT_CUDA(ctx, cudaLaunchCooperativeKernel(gkern, dim3(P.nb), dim3(PT), kargs, 0, s));
      }
      GT_CUDA(ctx, cudaMemcpyAsync(ctx->h_dscratch, P.st, sizeof(PState), cudaMemcpyDeviceToHost, s));
      GT_CUDA(ctx, cudaMemcpyAsync(ctx->h_scratch, P.err, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
      GT_CUDA(ctx, cudaStreamSynchronize(s));
      memcpy(&h, ctx->h_dscratch, sizeof(PState));
      int32_t e = 0;
      memcpy(&e, ctx->h_scratch, sizeof(int32_t));
      if (e) {
        err = true;
        break;
      }
      done_iters = h.iters;
      if (h.done || h.iters >= maxit) break;
      if (chunk < 2048) chunk *= 2;
    }
    if (local && !err && h.done == LOVERFLOW) {
      // nothing was computed: more shared memory, or the global vectors
      P.release();
      known = smem < L.most ? 1 : 2;
      if (smem < L.most) smem = L.most;
      else local = false;
      continue;
    }
    return pcg_finish<BS, V, X, REL>(P, h, err, out);
  }
}

// A scalar system in its sliced form; PCG_NOFIT, with nothing done, when it has
// no sliced copy, its local sets do not fit in shared memory or there is no
// memory left for what this form holds beside the other's vectors.  smem: a CTA's
// shared memory (0: the expected need)
template <class V, class X, bool REL>
int run_sliced(Ctx* ctx, Matrix* A, const V* val, const double* b, double* x, double rtol, int maxit, double delta,
               const PRun* from, PRun* out, int smem) {
  cudaStream_t s = ctx->stream;
  auto kern = k_pcg_sliced<V, X, REL>;
  LPlan L;
  GT_TRY(local_plan(ctx, A, kern, false, sizeof(X), sizeof(V), &L));
  // r, q, p and the column numbers (and x) of rows and halo: at most a band of
  // the space's DOF spread on both sides; on a three-dimensional mesh in
  // lexicographic order about three planes' shares
  const int64_t rows = (A->nbrows + L.nb - 1) / L.nb, spread = A->space->dof_spread;
  int64_t local = rows * 13 / 4 + 512;
  if (spread >= 0) local = std::min<int64_t>(local, rows + 2 * spread);
  const int64_t need = rows * 5 / 4 * 2 * (int64_t)sizeof(X) + local * (int64_t)(sizeof(X) + 4 + (REL && sizeof(X) == 4 ? 8 : 0)) + 8192;
  uint8_t& known = A->local_sets[local_form<X, REL>(true)];
  if (need > L.most + 8192 || known == 2) return PCG_NOFIT;
  // out of memory: the copies that only this form takes go back too
  auto without = [&](int s) -> int {
    if (s != GT_ERR_OOM) return s;
    if (A->sell_state != 1) sell_release(A);
    else if (sizeof(V) == 4) sell_release_values64(A);
    return PCG_NOFIT;
  };
  bool ready = false;
  const int rs = sell_ready(A, REL, sizeof(V) == 4, &ready);
  if (rs != GT_OK) return without(rs);
  if (!ready) return PCG_NOFIT;
  if (known == 1) smem = L.most;
  if (smem == 0) smem = (int)std::min<int64_t>(L.most, (need + 1023) & ~int64_t(1023));
  GT_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L.most));
  PSolve<1, V, X, REL> P;
  int ps = pcg_prepare<1, V, X, REL>(ctx, P, A, val, b, x, rtol, maxit, delta, from, L.nb, true, true);
  if (ps == GT_OK) ps = dalloc(ctx, &P.dargs, 1);
  if (ps != GT_OK) {
    cudaStreamSynchronize(s);
    P.release();
    return without(ps);
  }
  GT_TRY(copy_in(ctx, P.dargs, (const PArgs*)&P.args, 1));
  PState h{};
  int32_t e = 0;
  int chunk = 512;
  ChunkGraph graph;
  auto body = [&]() -> int {
    ctx->launches++;
    void* kargs[] = {&P.dargs, &chunk, &smem};
    GT_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)kern, dim3(P.nb), dim3(LT), kargs, smem, s));
    GT_CUDA(ctx, cudaMemcpyAsync(ctx->h_dscratch, P.st, sizeof(PState), cudaMemcpyDeviceToHost, s));
    GT_CUDA(ctx, cudaMemcpyAsync(ctx->h_scratch, P.err, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    return GT_OK;
  };
  while (true) {
    GT_TRY(graph.run(ctx, s, body));
    GT_CUDA(ctx, cudaStreamSynchronize(s));
    memcpy(&h, ctx->h_dscratch, sizeof(PState));
    memcpy(&e, ctx->h_scratch, sizeof(int32_t));
    if (e || h.done || h.iters >= maxit) break;
  }
  if (!e && h.done == LOVERFLOW) {
    P.release();
    known = smem < L.most ? 1 : 2;
    if (smem < L.most) return run_sliced<V, X, REL>(ctx, A, val, b, x, rtol, maxit, delta, from, out, L.most);
    return PCG_NOFIT;
  }
  return pcg_finish<1, V, X, REL>(P, h, e != 0, out);
}

// The clusters of the cluster form: the shared memory a CTA is given, and how
// many clusters the device holds at once (0: none)
struct ClusterRoom {
  int smem = 0, at_once = 0;
};
template <int BS, class V, class X, bool REL>
static int cluster_room_typed(Ctx* ctx, ClusterRoom* room, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
  auto kern = k_pcg_cluster<BS, V, X, REL>;
  GT_TRY(cta_room(ctx, kern, &room->smem));
  GT_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  GT_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, room->smem));
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = LCLUSTER;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg->gridDim = dim3(LCLUSTER);
  cfg->blockDim = dim3(LT);
  cfg->dynamicSmemBytes = (size_t)room->smem;
  cfg->stream = ctx->stream;
  cfg->attrs = at;
  cfg->numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&room->at_once, kern, cfg) != cudaSuccess) {
    cudaGetLastError();
    room->at_once = 0;
  }
  return GT_OK;
}
template <class V, class X, bool REL>
int cluster_room(Ctx* ctx, int bs, ClusterRoom* room) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  return bs == 1 ? cluster_room_typed<1, V, X, REL>(ctx, room, &cfg, at) : cluster_room_typed<3, V, X, REL>(ctx, room, &cfg, at);
}

// Systems of one block size, each on the CTAs its stand-alone
// solve would use (so its partition, its sums and its result are bitwise that
// solve's).  Those placed on a cluster share launches of one cluster per
// system, largest first; the others are packed into cooperative launches
// whose CTAs are co-resident, by falling shared memory per CTA, so that one
// launch's systems need about the same, and each waits only on its own
// bounded sums.  All systems of one call start alike (froms all null, or all
// continuations).  A system whose local sets do not fit goes from a cluster to
// a grid, and from a shared grid to one of its own.
template <int BS, class V, class X, bool REL>
static int run_groups_typed(Ctx* ctx, Place place, const std::vector<Matrix*>& As, const std::vector<const V*>& vals,
                            const std::vector<const double*>& bs, const std::vector<double*>& xs, double rtol,
                            int maxit, double delta, const std::vector<const PRun*>& froms, std::vector<PRun>& outs,
                            std::vector<int>& status) {
  cudaStream_t s = ctx->stream;
  const int n = (int)As.size();
  auto gkern = k_pcg_local<BS, V, X, REL>;
  auto ckern = k_pcg_cluster<BS, V, X, REL>;
  std::vector<LPlan> plan(n);
  std::vector<int> cl, grid, alone;
  LPlan cplan;
  for (int i = 0; i < n; i++) {
    if (cluster_place(As[i], sizeof(X) == sizeof(double), place)) {
      GT_TRY(local_plan(ctx, As[i], ckern, true, sizeof(X), sizeof(V), &cplan));
      if (cplan.ok) {
        cl.push_back(i);
        continue;
      }
    }
    grid.push_back(i);
  }
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  if (!cl.empty()) {
    ClusterRoom room;
    GT_TRY((cluster_room_typed<BS, V, X, REL>(ctx, &room, &cfg, at)));
    if (room.at_once < 1) {
      grid.insert(grid.end(), cl.begin(), cl.end());
      cl.clear();
    }
    std::stable_sort(cl.begin(), cl.end(), [&](int a, int c) { return As[a]->bnnz > As[c]->bnnz; });
  }
  // one launch sequence over the systems `ids`, CTAs given by hmap in a grid
  auto run = [&](const std::vector<int>& ids, bool cluster, int smem, int64_t tot, std::vector<int>& overflow) -> int {
    const int m = (int)ids.size();
    uint32_t* bars = nullptr;
    int32_t* errs = nullptr;
    PState* sts = nullptr;
    PArgs* dargs = nullptr;
    int2* dmap = nullptr;
    std::vector<PSolve<BS, V, X, REL>> P(m);
    int prepared = 0;
    std::vector<PState> h(m);
    std::vector<PArgs> hargs(m);
    std::vector<int2> hmap;
    std::vector<int32_t> e(2 * m, 0);
    bool err = false;
    // every exit below goes through the release of its blocks
    auto body = [&]() -> int {
      GT_TRY(dalloc(ctx, &bars, 2 * (int64_t)m));
      GT_TRY(dalloc(ctx, &errs, 2 * (int64_t)m));
      GT_TRY(dalloc(ctx, (unsigned char**)&sts, (int64_t)sizeof(PState) * m));
      GT_TRY(dalloc(ctx, (unsigned char**)&dargs, (int64_t)sizeof(PArgs) * m));
      GT_CUDA(ctx, cudaMemsetAsync(errs, 0, sizeof(int32_t) * 2 * m, s));
      for (int k = 0; k < m; k++) {
        const int i = ids[k];
        prepared++;
        GT_TRY((pcg_prepare<BS, V, X, REL>(ctx, P[k], As[i], vals[i], bs[i], xs[i], rtol, maxit, delta, froms[i],
                                              cluster ? LCLUSTER : plan[i].nb, true, false, bars + 2 * k, errs + 2 * k,
                                              sts + k)));
        hargs[k] = P[k].args;
        for (int j = 0; !cluster && j < P[k].nb; j++) hmap.push_back(make_int2(k, j));
      }
      GT_TRY(copy_in(ctx, (unsigned char*)dargs, (const unsigned char*)hargs.data(), (int64_t)sizeof(PArgs) * m));
      if (!cluster) {
        GT_TRY(dalloc(ctx, (unsigned char**)&dmap, (int64_t)sizeof(int2) * tot));
        GT_TRY(copy_in(ctx, (unsigned char*)dmap, (const unsigned char*)hmap.data(), (int64_t)sizeof(int2) * tot));
      }
      int chunk = 512;
      for (int launch = 0;; launch++) {
        int init = launch == 0 ? (froms[ids[0]] ? 2 : 1) : 0;
        ctx->launches++;
        if (cluster) {
          cfg.gridDim = dim3((unsigned)(LCLUSTER * m));
          GT_CUDA(ctx, cudaLaunchKernelEx(&cfg, ckern, (const PArgs*)dargs, init, chunk, smem));
        } else {
          void* kargs[] = {&dargs, &dmap, &init, &chunk, &smem};
          GT_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)gkern, dim3((unsigned)tot), dim3(LT), kargs, smem, s));
        }
        GT_CUDA(ctx, cudaMemcpyAsync(h.data(), sts, sizeof(PState) * m, cudaMemcpyDeviceToHost, s));
        GT_CUDA(ctx, cudaMemcpyAsync(e.data(), errs, sizeof(int32_t) * 2 * m, cudaMemcpyDeviceToHost, s));
        GT_CUDA(ctx, cudaStreamSynchronize(s));
        bool all = true;
        for (int k = 0; k < m; k++) {
          err |= e[2 * k] != 0;
          all &= h[k].done != 0 || h[k].iters >= maxit;
        }
        if (err || all) break;
        if (chunk < 2048) chunk *= 2;
      }
      return GT_OK;
    };
    const int ws = body();
    if (ws != GT_OK) cudaStreamSynchronize(s);  // nothing of the launches may be reused before the stream drains
    for (int k = 0; k < prepared; k++) {
      const int i = ids[k];
      if (ws == GT_OK && !err && h[k].done == LOVERFLOW) {
        P[k].release();
        overflow.push_back(i);
        continue;
      }
      const int st = pcg_finish<BS, V, X, REL>(P[k], h[k], err, &outs[i]);
      status[i] = ws == GT_OK ? st : ws;
    }
    dfree(ctx, bars);
    dfree(ctx, errs);
    if (sts) pool_free(ctx, sts);
    if (dargs) pool_free(ctx, dargs);
    if (dmap) pool_free(ctx, dmap);
    return ws;
  };
  if (!cl.empty()) GT_TRY(run(cl, true, cplan.most, 0, grid));
  if (grid.size() == 1) {
    alone = grid;
    grid.clear();
  }
  std::vector<int> order;
  for (int i : grid) {
    GT_TRY(local_plan(ctx, As[i], gkern, false, sizeof(X), sizeof(V), &plan[i]));
    (plan[i].ok && !As[i]->local_sets[local_form<X, REL>(false)] ? order : alone).push_back(i);
  }
  std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return plan[a].est > plan[c].est; });
  size_t i0 = 0;
  while (i0 < order.size()) {
    const int smem = plan[order[i0]].est;
    GT_CUDA(ctx, cudaFuncSetAttribute(gkern, cudaFuncAttributeMaxDynamicSharedMemorySize, plan[order[i0]].most));
    int per_sm = 0;
    GT_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gkern, LT, smem));
    const int64_t cap = (int64_t)per_sm * ctx->num_sms;
    std::vector<int> ids;
    int64_t tot = 0;
    while (i0 < order.size() && tot + plan[order[i0]].nb <= cap) {
      tot += plan[order[i0]].nb;
      ids.push_back(order[i0++]);
    }
    if (ids.empty()) alone.push_back(order[i0++]);
    else GT_TRY(run(ids, false, smem, tot, alone));
  }
  for (int i : alone)
    status[i] =
        run_typed<BS, V, X, REL>(ctx, As[i], vals[i], bs[i], xs[i], rtol, maxit, delta, froms[i], &outs[i]);
  return GT_OK;
}

// kernel instances by block size
template <class V, class X, bool REL>
int run_groups_dispatch(Ctx* ctx, Place place, int bs, const std::vector<Matrix*>& As, const std::vector<const V*>& vals,
                        const std::vector<const double*>& b, const std::vector<double*>& x, double rtol, int maxit,
                        double delta, const std::vector<const PRun*>& froms, std::vector<PRun>& outs,
                        std::vector<int>& status) {
  switch (bs) {
    case 1:
      return run_groups_typed<1, V, X, REL>(ctx, place, As, vals, b, x, rtol, maxit, delta, froms, outs, status);
    case 2:
      return run_groups_typed<2, V, X, REL>(ctx, place, As, vals, b, x, rtol, maxit, delta, froms, outs, status);
    case 3:
      return run_groups_typed<3, V, X, REL>(ctx, place, As, vals, b, x, rtol, maxit, delta, froms, outs, status);
  }
  return set_error(ctx, GT_ERR_UNSUPPORTED, "persistent PCG: unsupported block size");
}

extern template int cluster_room<double, double, true>(Ctx*, int, ClusterRoom*);
extern template int cluster_room<float, float, true>(Ctx*, int, ClusterRoom*);
extern template int cluster_room<float, float, false>(Ctx*, int, ClusterRoom*);
extern template int run_groups_dispatch<double, double, true>(
    Ctx*, Place, int, const std::vector<Matrix*>&, const std::vector<const double*>&,
    const std::vector<const double*>&, const std::vector<double*>&, double, int, double, const std::vector<const PRun*>&,
    std::vector<PRun>&, std::vector<int>&);
extern template int run_groups_dispatch<float, float, true>(
    Ctx*, Place, int, const std::vector<Matrix*>&, const std::vector<const float*>&,
    const std::vector<const double*>&, const std::vector<double*>&, double, int, double, const std::vector<const PRun*>&,
    std::vector<PRun>&, std::vector<int>&);
extern template int run_groups_dispatch<float, float, false>(
    Ctx*, Place, int, const std::vector<Matrix*>&, const std::vector<const float*>&,
    const std::vector<const double*>&, const std::vector<double*>&, double, int, double, const std::vector<const PRun*>&,
    std::vector<PRun>&, std::vector<int>&);
extern template int run_sliced<double, double, true>(Ctx*, Matrix*, const double*, const double*, double*, double, int, double,
                                    const PRun*, PRun*, int);
extern template int run_sliced<float, float, true>(Ctx*, Matrix*, const float*, const double*, double*, double, int, double,
                                    const PRun*, PRun*, int);
extern template int run_sliced<float, float, false>(Ctx*, Matrix*, const float*, const double*, double*, double, int, double,
                                    const PRun*, PRun*, int);

}  // namespace pcg
}  // namespace gt
