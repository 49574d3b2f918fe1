// gt_batch.cu -- many independent solves of uneven size in few launches.
//
// A batch holds n assembled matrices of block size 1 (scalar problems) or
// 3 (3-D linear elasticity).  Instances are split by size (scalar rows):
//
//  * small instances (rows <= kSmallRows) up to kOneCtaRows rows are solved
//    by ONE persistent launch: each CTA takes the next instance from a queue
//    (largest first) and runs its whole Jacobi-PCG alone -- SpMV with G lanes
//    per row, CTA reductions through shared memory, no inter-CTA
//    synchronisation -- then takes the next one, so the device stays full
//    however uneven the sizes;
//  * larger small instances with the arithmetic of one thread-block cluster
//    each (gt_pcg_local.cuh): on clusters, in one launch per block size, or --
//    when there are more of them than the clusters get done in the same time --
//    the smaller ones on one CTA each, from a queue (k_bpcg_cluster);
//  * medium instances (up to the persistent solver's 262,144 rows, matrices
//    of the batch's own context, FP64 or mixed mode) share cooperative
//    launches of the persistent solver: each one on the CTAs its own solve
//    would use, with its own bounded barrier, so many run at once;
//  * large instances, which fill the device by themselves, run one after
//    the other through the single-system solver of gt_solve.cu.
//
// Either way an instance's arithmetic and summation order depend only on
// the instance (one CTA in a fixed order, a cluster's, or the grid layout of
// the instance's own solve), so its result is bitwise the same alone and in
// any mix.  The precision modes match gt_solve: FP64 CG, FP32 CG with FP64
// reliable updates (an FP32 run that stalls or loses its rate continues in
// FP64), and FP32 CG.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "gt_internal.cuh"
#include "gt_pcg_impl.cuh"
#include "gt_rowdot.cuh"

namespace gt {

constexpr int BT = 256;                 // threads per CTA of the batched kernel
constexpr int BNW = BT / 32;
constexpr int64_t kSmallRows = 32768;   // largest instance of the small tier
// Small instances up to this size are solved by k_bpcg, one per CTA, the
// others with a cluster's arithmetic.  Measured on 16 uneven Poisson problems
// of 256 to 4,096 cells (225 to 30,000 rows; assembly and mixed solves to
// 1e-10): 9.1 ms, 119 ms with every one on one CTA, whose SM then holds the
// largest alone.
constexpr int64_t kOneCtaRows = 1024;

struct BInst {
  const int64_t* rowptr;
  const int32_t* colind;
  const double* v64;
  const float* v32;
  const int32_t* diag;  // position of the diagonal block in each block row
  int64_t nrows;        // block rows
  int64_t off;          // offset of the instance in the concatenated vectors (scalar entries)
  int32_t bs, pad;
};

// per-instance outcome of the batched kernel
struct BRes {
  double rr, bb;        // final ||r||^2 (true residual with reliable updates) and ||b||^2
  int32_t iters, nupd;
  int32_t status;       // 0 converged, 1 maxit / breakdown, 2 FP32 stalled (continue in FP64)
  int32_t pad;
};

struct BatchImpl {
  Ctx* ctx = nullptr;
  int n = 0;
  int G = 0;  // lanes per row of k_bpcg; 0: each instance's own (row_lanes of its mean row)
  int64_t ntot = 0;
  std::vector<Matrix*> mats;
  std::vector<BInst> h_inst;
  BInst* d_inst = nullptr;
  int64_t small_rows = kSmallRows;  // scalar rows up to which an instance is of the small tier
  std::vector<int> small, large;   // instance ids by class (small: largest first)
};

// the small tier: instances up to B->small_rows scalar rows, largest first
static void classify(BatchImpl* B) {
  B->small.clear();
  B->large.clear();
  for (int i = 0; i < B->n; i++) {
    if (B->h_inst[i].nrows * B->h_inst[i].bs <= B->small_rows) B->small.push_back(i);
    else B->large.push_back(i);
  }
  std::stable_sort(B->small.begin(), B->small.end(), [&](int a, int c) {
    return B->h_inst[a].nrows * B->h_inst[a].bs > B->h_inst[c].nrows * B->h_inst[c].bs;
  });
}

// CTA sum of K values, identical in every thread (fixed order); sr is one of
// two alternating shared buffers of K * BNW doubles
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K], double* sr) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; k++) {
    double t = v[k];
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) sr[k * BNW + w] = t;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; k++) {
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < BNW; i++) t += sr[k * BNW + i];
    v[k] = t;
  }
}

template <class V>
__device__ __forceinline__ const V* inst_vals(const BInst& in) {
  if constexpr (sizeof(V) == 8) return (const V*)in.v64;
  else return (const V*)in.v32;
}

// One CTA per instance (up to kOneCtaRows rows), instances from a queue.  BS: block size of the
// instances of the launch (G lanes per block row); V: values of the
// iteration, X: vector type; REL: FP64 reliable updates (needs v64).
// from_x: start from the given x (else x = 0).  Jacobi on the scalar
// diagonal, as the single-system solver.
template <int BS, int G, class V, class X, bool REL>
__global__ void __launch_bounds__(BT) k_bpcg(const BInst* __restrict__ insts, const int32_t* __restrict__ queue,
                                             int nq, int32_t* head, const double* __restrict__ b, double* x, X* xs,
                                             X* r, X* z, X* p, X* q, X* dinv, BRes* res, double rtol2, double delta2,
                                             int maxit, int from_x, double stall_ratio, int stall_count) {
  __shared__ double s_red[2][3 * BNW];
  __shared__ int s_k;
  constexpr int NG = BT / G;
  const int tid = threadIdx.x, gl = tid % G, grp = tid / G;
  int buf = 0;
  while (true) {
    if (tid == 0) s_k = atomicAdd(head, 1);
    __syncthreads();
    const int k = s_k;
    __syncthreads();
    if (k >= nq) return;
    const int ii = queue[k];
    const BInst in = insts[ii];
    const int64_t nb = in.nrows, n = nb * BS, off = in.off;
    const V* val = inst_vals<V>(in);
    const double* bi = b + off;
    double* xi = x + off;
    X *xsi = xs + off, *ri = r + off, *zi = z + off, *pi = p + off, *qi = q + off, *di = dinv + off;
    for (int64_t i = tid; i < n; i += BT) {
      const int64_t br = i / BS;
      const int c = (int)(i - br * BS);
      const int64_t pos = (in.rowptr[br] + in.diag[br]) * BS * BS + c * BS + c;
      const double d = in.v64 ? in.v64[pos] : (double)in.v32[pos];
      di[i] = (X)(1.0 / d);
      if (!from_x) xi[i] = 0.0;
    }
    __syncthreads();
    // r = b - A x, z = Dinv r, p = z, xs = 0
    double rz, rr, bb;
    {
      double v[3] = {0.0, 0.0, 0.0};
      for (int64_t base = 0; base < nb; base += NG) {
        int64_t row = base + grp;
        const bool valid = row < nb;
        if (!valid) row = nb - 1;
        double o[BS];
        if constexpr (REL) row_dot<BS, G, double, double, double, false>(in.rowptr, in.colind, in.v64, xi, row, gl, o);
        else row_dot<BS, G, V, double, double, false>(in.rowptr, in.colind, val, xi, row, gl, o);
        if (gl == 0 && valid) {
#pragma unroll
          for (int c = 0; c < BS; c++) {
            const int64_t i = row * BS + c;
            const double bv = bi[i], rv = bv - o[c];
            const X rx = (X)rv, zx = di[i] * rx;
            ri[i] = rx;
            zi[i] = zx;
            pi[i] = zx;
            xsi[i] = (X)0;
            v[0] += (double)rx * (double)zx;
            v[1] += rv * rv;
            v[2] += bv * bv;
          }
        }
      }
      block_sum<3>(v, s_red[buf]);
      buf ^= 1;
      rz = v[0];
      rr = v[1];
      bb = v[2];
    }
    const double tol2 = rtol2 * bb;
    double rmax2 = rr, rzold = 0.0;
    int iters = 0, nupd = 0, status = 0, it_upd = 0, max_cyc = 0, stall = 0;
    bool done = rr <= tol2;
    while (!done) {
      // q = A p, p.q
      double pq;
      {
        X acc = (X)0;
        for (int64_t base = 0; base < nb; base += 2 * NG) {
          int64_t ra = base + grp, rb = base + NG + grp;
          const bool va = ra < nb, vb = rb < nb;
          if (!va) ra = nb - 1;
          if (!vb) rb = nb - 1;
          X oa[BS], ob[BS];
          row_dot<BS, G, V, X, X, false>(in.rowptr, in.colind, val, pi, ra, gl, oa);
          row_dot<BS, G, V, X, X, false>(in.rowptr, in.colind, val, pi, rb, gl, ob);
          if (gl == 0) {
            if (va)
#pragma unroll
              for (int c = 0; c < BS; c++) {
                qi[ra * BS + c] = oa[c];
                acc += oa[c] * pi[ra * BS + c];
              }
            if (vb)
#pragma unroll
              for (int c = 0; c < BS; c++) {
                qi[rb * BS + c] = ob[c];
                acc += ob[c] * pi[rb * BS + c];
              }
          }
        }
        double v[1] = {(double)acc};
        block_sum<1>(v, s_red[buf]);
        buf ^= 1;
        pq = v[0];
      }
      const X alpha = (X)(rz / pq);
      double rzn;
      {
        X v0 = (X)0, v1 = (X)0;
        for (int64_t i = tid; i < n; i += BT) {
          const X rv = ri[i] - alpha * qi[i];
          const X zv = di[i] * rv;
          xsi[i] += alpha * pi[i];
          ri[i] = rv;
          zi[i] = zv;
          v0 += rv * zv;
          v1 += rv * rv;
        }
        double v[2] = {(double)v0, (double)v1};
        block_sum<2>(v, s_red[buf]);
        buf ^= 1;
        rzn = v[0];
        rr = v[1];
      }
      iters++;
      double beta = rzn / rz;
      rzold = rz;
      rz = rzn;
      const bool stop = rr <= tol2 || iters >= maxit || !(rr == rr);
      if constexpr (REL) {
        const int cyc = iters - it_upd;
        const bool slow = sizeof(X) < sizeof(double) && (cyc > kSlowCycle || (max_cyc > 0 && cyc > (5 * max_cyc) / 2 + 16));
        if (stop || slow || rr <= delta2 * rmax2) {
          for (int64_t i = tid; i < n; i += BT) {
            xi[i] += (double)xsi[i];
            xsi[i] = (X)0;
          }
          __syncthreads();
          double v[2] = {0.0, 0.0};
          for (int64_t base = 0; base < nb; base += NG) {
            int64_t row = base + grp;
            const bool valid = row < nb;
            if (!valid) row = nb - 1;
            double o[BS];
            row_dot<BS, G, double, double, double, false>(in.rowptr, in.colind, in.v64, xi, row, gl, o);
            if (gl == 0 && valid) {
#pragma unroll
              for (int c = 0; c < BS; c++) {
                const int64_t i = row * BS + c;
                const double rv = bi[i] - o[c];
                const X rx = (X)rv, zx = di[i] * rx;
                ri[i] = rx;
                zi[i] = zx;
                v[0] += (double)rx * (double)zx;
                v[1] += rv * rv;
              }
            }
          }
          block_sum<2>(v, s_red[buf]);
          buf ^= 1;
          beta = rzold != 0.0 ? v[0] / rzold : 0.0;
          // the recurrence lost track of the true residual: restart the directions
          if (v[0] > (sizeof(X) == sizeof(double) ? kRestartRatio64 : kRestartRatio) * rz) beta = 0.0;
          const double prev = rmax2;
          rz = v[0];
          rr = v[1];
          rmax2 = v[1];
          nupd++;
          done = rr <= tol2 || iters >= maxit || !(rr == rr);
          if (sizeof(X) == sizeof(double) && !done) {
            // FP64: checks that do not halve ||r||, kStagnation times running:
            // the tolerance lies below the attainable accuracy
            stall = rr > 0.25 * prev ? stall + 1 : 0;
            if (stall >= kStagnation) done = true;
          }
          if (sizeof(X) < sizeof(double) && !done) {
            stall = rr > stall_ratio * prev ? stall + 1 : 0;
            if (stall >= stall_count || slow) {
              done = true;
              status = 2;
            }
          }
          if (cyc > max_cyc) max_cyc = cyc;
          it_upd = iters;
        }
      } else {
        done = stop;
      }
      if (done) break;
      const X bx = (X)beta;
      for (int64_t i = tid; i < n; i += BT) pi[i] = zi[i] + bx * pi[i];
      __syncthreads();
    }
    if (!REL) {
      for (int64_t i = tid; i < n; i += BT) {
        xi[i] += (double)xsi[i];
        xsi[i] = (X)0;
      }
    }
    if (tid == 0) {
      BRes o{};
      o.rr = rr;
      o.bb = bb;
      o.iters = iters;
      o.nupd = nupd;
      o.status = status == 2 ? 2 : (rr <= tol2 ? 0 : 1);
      res[ii] = o;
    }
    __syncthreads();
  }
}

// A cluster's arithmetic on one CTA (gt_pcg_local.cuh, CL), bitwise: the rows
// are split among LCLUSTER shares as among a cluster's CTAs, every sum is taken
// by (share, warp of its CTA) -- a warp here takes one after the other -- and
// the vector updates and the scalars are the cluster's own functions.  One
// instance per CTA from a queue (its entry lanes beside it); row pointers and
// vectors in shared memory as far as they fit, else in global memory.
// cont: continuations of FP32 runs in FP64, from x and st.
constexpr int VW = pcg::LCLUSTER * pcg::LNW;  // warps of a cluster
struct VShared {
  pcg::Fx part[3][VW];
  pcg::PState st;
  double alpha;
  int first[pcg::LCLUSTER + 1];
  int act, next;
  int nw;  // warps of a share that hold values in some sum
};
// threads per CTA (scalar rows: two CTAs on an SM; block rows, whose products
// load more per lane: one of twice the warps -- 64 elasticity instances of 1,944
// rows FP64 11.3 ms, 12.5 with 512 threads)
constexpr int vthreads(int bs) { return bs == 1 ? 512 : 1024; }
template <int BS, class V, class X, bool REL>
__global__ void __launch_bounds__(vthreads(BS), BS == 1 ? 2 : 1) k_bpcg_cluster(
    const BInst* __restrict__ insts, const int2* __restrict__ queue, int nq, int32_t* head,
    const double* __restrict__ b, double* x, X* xs, X* r, X* p, X* q, X* dinv, pcg::PState* st, pcg::PRule rule,
    int cont, int smem_bytes) {
  using namespace pcg;
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ VShared S;
  constexpr int VT = vthreads(BS), VNW = VT / 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  while (true) {
    __syncthreads();
    if (tid == 0) S.next = atomicAdd(head, 1);
    __syncthreads();
    if (S.next >= nq) return;
    const int2 job = queue[S.next];
    const BInst in = insts[job.x];
    const int nb = (int)in.nrows, n = nb * BS;
    const V* val = inst_vals<V>(in);
    const double* bi = b + in.off;
    double* xi = x + in.off;
    X *xsi = xs + in.off, *ri = r + in.off, *pi = p + in.off, *qi = q + in.off, *di = dinv + in.off;
    int room = smem_bytes;
    auto place = [&](auto*& v, int cnt) {
      const int bytes = (cnt * (int)sizeof(*v) + 15) & ~15;
      if (bytes > room) return false;
      v = reinterpret_cast<std::remove_reference_t<decltype(v)>>(s_dyn + (smem_bytes - room));
      room -= bytes;
      return true;
    };
    place(pi, n);
    int32_t* rp = nullptr;
    const bool rps = place(rp, nb + 1);
    place(ri, n);
    place(qi, n);
    place(di, n);
    place(xsi, n);
    for (int i = wid; i <= LCLUSTER; i += VNW) {
      const int64_t f = local_first_row(in.rowptr, nb, LCLUSTER, i, BS * BS, BS * row_cost(BS));
      if (lane == 0) S.first[i] = (int)f;
    }
    if (rps)
      for (int i = tid; i <= nb; i += VT) rp[i] = (int32_t)in.rowptr[i];
    for (int i = tid; i < n; i += VT) {
      const int br = i / BS, c = i - br * BS;
      const int64_t pos = (in.rowptr[br] + in.diag[br]) * BS * BS + c * BS + c;
      di[i] = (X)(1.0 / (in.v64 ? in.v64[pos] : (double)in.v32[pos]));
      if (!cont) xi[i] = 0.0;
      xsi[i] = (X)0;
      pi[i] = (X)0;
    }
    if (tid == 0) {
      S.st = cont ? st[job.x] : PState{};
      S.st.done = 0;
    }
    __syncthreads();
    if (tid == 0) {
      int most = 0;
      for (int s = 0; s < LCLUSTER; s++) most = max(most, S.first[s + 1] - S.first[s]);
      const int gpw = BS == 3 ? 2 : 32 / job.y;  // block rows of a warp in the residual's sums
      S.nw = min(LNW, max((most * BS + 31) / 32, (most + gpw - 1) / gpw));
    }
    for (int i = tid; i < 3 * VW; i += VT) (&S.part[0][0])[i] = Fx{0, kFxZero};
    __syncthreads();
    // out = A x over block rows [row0, re), a warp
    auto product = [&](auto jt, auto ut, auto zero, int row0, int re, auto* v, auto&& get, auto&& put) {
      constexpr int J = decltype(jt)::value, U = decltype(ut)::value;
      if (rps) local_group<BS, J, U, decltype(zero)>(row0, re, rp, v, in.colind, get, put);
      else local_group<BS, J, U, decltype(zero)>(row0, re, in.rowptr, v, in.colind, get, put);
    };
    // Sum of K values over the cluster's threads, then ctl(totals) by thread 0.
    // each(share, lo, hi, w, v): adds the values of this lane as lane of warp w
    // of the share with entries [lo, hi)
    auto total = [&](auto kt, auto zero, auto&& each, auto&& ctl) {
      constexpr int K = decltype(kt)::value;
      for (int t = wid; t < LCLUSTER * S.nw; t += VNW) {
        const int s = t % LCLUSTER, w = t / LCLUSTER;
        const int lo = S.first[s] * BS, hi = S.first[s + 1] * BS;
        Fx f[K];
#pragma unroll
        for (int k = 0; k < K; k++) f[k] = Fx{0, kFxZero};
        if (lo + w * (K == 3 ? 1 : 32) < hi) {  // (else no value: zero)
          decltype(zero) v[K];
#pragma unroll
          for (int k = 0; k < K; k++) v[k] = zero;
          each(lo, hi, w, v);
#pragma unroll
          for (int k = 0; k < K; k++) {
            const Fx u[1] = {fx_from(v[k])};
            f[k] = fx_warp_sum<1>(u);
          }
        }
        if (lane == 0)
#pragma unroll
          for (int k = 0; k < K; k++) S.part[k][s * LNW + w] = f[k];
      }
      __syncthreads();
      if (wid == 0) {
        double tot[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
          Fx u[VW / 32];
#pragma unroll
          for (int i = 0; i < VW / 32; i++) u[i] = S.part[k][lane + i * 32];
          tot[k] = fx_double(fx_warp_sum<VW / 32>(u));
        }
        if (lane == 0) ctl(tot);
      }
      __syncthreads();
    };
    auto finish_act = [&] { S.act = (S.st.done || S.st.iters >= rule.maxit) ? 2 : 0; };
    // FP64 residual -> r, with its sums
    auto residual = [&](auto&& ctl) {
      total(std::integral_constant<int, 3>(), 0.0,
            [&](int lo, int hi, int w, double (&v)[3]) {
              with_lanes<BS>(job.y, [&](auto jt) {
                constexpr int J = decltype(jt)::value, GPW = 32 / (BS * J);
                const std::integral_constant<int, 4> ut;
                auto put = [&](int row, int c, double o) {
                  const int i = row * BS + c;
                  cg_residual(bi[i], o, di[i], ri[i], v);
                };
                auto get = [&](int c, int d) { return xi[c * BS + d]; };
                for (int row0 = lo / BS + w * GPW; row0 < hi / BS; row0 += LNW * GPW) {
                  if constexpr (REL) product(jt, ut, 0.0, row0, hi / BS, in.v64, get, put);
                  else product(jt, ut, 0.0, row0, hi / BS, val, get, put);
                }
              });
            },
            ctl);
    };
    residual([&](const double* tot) {
      ctl_start(S.st, tot, rule, cont);
      finish_act();
    });
    while (!(S.act & 2)) {
      const X beta = (X)S.st.beta;
      for (int i = tid; i < n; i += VT) pi[i] = fma(beta, pi[i], times(di[i], ri[i]));
      __syncthreads();
      with_lanes<BS>(job.y, [&](auto jt) {
        constexpr int J = decltype(jt)::value, GPW = 32 / (BS * J);
        auto get = [&](int c, int d) { return pi[c * BS + d]; };
        auto put = [&](int row, int c, X o) { qi[row * BS + c] = o; };
        const std::integral_constant<int, BS == 3 ? 2 : (sizeof(X) == 4 ? 8 : 4)> ut;
        for (int row0 = wid * GPW; row0 < nb; row0 += VNW * GPW) product(jt, ut, (X)0, row0, nb, val, get, put);
      });
      __syncthreads();
      total(std::integral_constant<int, 1>(), (X)0,
            [&](int lo, int hi, int w, X (&v)[1]) {
              for (int i = lo + w * 32 + lane; i < hi; i += LT) v[0] = fma(qi[i], pi[i], v[0]);
            },
            [&](const double* tot) { S.alpha = quick_div(S.st.rz, tot[0]); });
      const X alpha = (X)S.alpha;
      total(std::integral_constant<int, 2>(), (X)0,
            [&](int lo, int hi, int w, X (&v)[2]) {
              for (int i = lo + w * 32 + lane; i < hi; i += LT) cg_step(alpha, qi[i], pi[i], di[i], ri[i], xsi[i], v);
            },
            [&](const double* tot) {
              const int upd = ctl_step<X, REL>(S.st, tot, rule);
              finish_act();
              if (upd) S.act = upd;
            });
      if constexpr (REL) {
        if (S.act & 1) {
          const bool slow = S.act & 4;
          for (int i = tid; i < n; i += VT) {
            xi[i] += (double)xsi[i];
            xsi[i] = (X)0;
          }
          __syncthreads();
          residual([&](const double* tot) {
            ctl_update<X>(S.st, tot, rule, slow);
            finish_act();
          });
        }
      }
    }
    if (!REL && S.st.done)
      for (int i = tid; i < n; i += VT) xi[i] += (double)xsi[i];
    if (tid == 0) st[job.x] = S.st;
  }
}

// fits[j]: the local sets of instance ids[j] fit the CTAs of a cluster, given
// room64 / room32 bytes in the FP64 / FP32 iteration (0: not asked; xl: with
// FP64 residuals) -- the cluster kernel's own test, which sends an instance
// that fails it to a grid.  A CTA per instance, a warp per share of rows.
template <int BS>
__global__ void __launch_bounds__(BT) k_cluster_fits(const BInst* __restrict__ insts, const int32_t* __restrict__ ids,
                                                     int room64, int room32, int xl, int32_t* __restrict__ fits) {
  using namespace pcg;
  __shared__ uint32_t bits[BNW][kSmallRows / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const BInst in = insts[ids[blockIdx.x]];
  const int nwords = (int)((in.nrows + 31) / 32), tail = bitmap_bytes(nwords);
  uint32_t* bit = bits[wid];
  bool ok = true;
  for (int s = wid; s < LCLUSTER; s += BNW) {
    const int64_t r0 = local_first_row(in.rowptr, in.nrows, LCLUSTER, s, BS * BS, BS * row_cost(BS));
    const int64_t r1 = local_first_row(in.rowptr, in.nrows, LCLUSTER, s + 1, BS * BS, BS * row_cost(BS));
    for (int i = lane; i < nwords; i += 32) bit[i] = 0;
    __syncwarp();
    for (int64_t k = in.rowptr[r0] + lane; k < in.rowptr[r1]; k += 32) atomicOr(&bit[in.colind[k] >> 5], 1u << (in.colind[k] & 31));
    for (int64_t i = r0 + lane; i < r1; i += 32) atomicOr(&bit[i >> 5], 1u << (i & 31));
    __syncwarp();
    int nloc = 0;
    for (int i = lane; i < nwords; i += 32) nloc += __popc(bit[i]);
    nloc = __reduce_add_sync(0xffffffffu, nloc);
    const int nr = (int)(r1 - r0), n = nr * BS;
    ok &= nloc < 65535;
    if (room64) ok &= local_bytes<BS, double, false, true, false>(n, nloc, nr) + tail <= (size_t)room64;
    if (room32)
      ok &= (xl ? local_bytes<BS, float, true, true, false>(n, nloc, nr)
                : local_bytes<BS, float, false, true, false>(n, nloc, nr)) + tail <= (size_t)room32;
    __syncwarp();
  }
  ok = __syncthreads_and(ok);
  if (threadIdx.x == 0) fits[blockIdx.x] = ok;
}

}  // namespace gt

struct gt_batch : gt::BatchImpl {};

namespace gt {

template <class V, class X, bool REL>
static int launch_small_g(gt_batch* B, int bs, int G, const std::vector<int>& ids, const double* b, double* x, double rtol,
                          int maxit, double delta, int from_x, std::vector<BRes>& hres) {
  Ctx* ctx = B->ctx;
  cudaStream_t s = ctx->stream;
  if (ids.empty()) return GT_OK;
  const int64_t n = B->ntot;
  X *xs = nullptr, *r = nullptr, *z = nullptr, *p = nullptr, *q = nullptr, *dinv = nullptr;
  int32_t *queue = nullptr, *head = nullptr;
  BRes* res = nullptr;
  GT_TRY(dalloc(ctx, &xs, n));
  GT_TRY(dalloc(ctx, &r, n));
  GT_TRY(dalloc(ctx, &z, n));
  GT_TRY(dalloc(ctx, &p, n));
  GT_TRY(dalloc(ctx, &q, n));
  GT_TRY(dalloc(ctx, &dinv, n));
  GT_TRY(dalloc(ctx, &queue, (int64_t)ids.size()));
  GT_TRY(dalloc(ctx, &head, 1));
  GT_TRY(dalloc(ctx, (unsigned char**)&res, (int64_t)sizeof(BRes) * B->n));
  GT_TRY(copy_in(ctx, queue, ids.data(), (int64_t)ids.size()));
  GT_CUDA(ctx, cudaMemsetAsync(head, 0, sizeof(int32_t), s));
  auto launch = [&](auto kern) -> int {
    int per_sm = 0;
    GT_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, BT, 0));
    int64_t cap = (int64_t)std::max(per_sm, 1) * ctx->num_sms;
    int grid = (int)std::min<int64_t>(cap, (int64_t)ids.size());
    kern<<<GT_KC(ctx, grid), BT, 0, s>>>(B->d_inst, queue, (int)ids.size(), head, b, x, xs, r, z, p, q, dinv, res,
                                         rtol * rtol, delta * delta, maxit, from_x, ctx->ir_stall_ratio,
                                         ctx->ir_stall_count);
    GT_LAUNCH(ctx, "k_bpcg");
    return GT_OK;
  };
  int st;
  if (bs == 3) {
    // block rows of 3-D elasticity: 2 or 4 lanes (inst_lanes)
    st = G == 2 ? launch(k_bpcg<3, 2, V, X, REL>) : launch(k_bpcg<3, 4, V, X, REL>);
  } else {
    switch (G) {
      case 1: st = launch(k_bpcg<1, 1, V, X, REL>); break;
      case 2: st = launch(k_bpcg<1, 2, V, X, REL>); break;
      case 8: st = launch(k_bpcg<1, 8, V, X, REL>); break;
      default: st = launch(k_bpcg<1, 4, V, X, REL>); break;
    }
  }
  if (st == GT_OK) {
    std::vector<BRes> all(B->n);
    GT_CUDA(ctx, cudaMemcpyAsync(all.data(), res, sizeof(BRes) * B->n, cudaMemcpyDeviceToHost, s));
    GT_CUDA(ctx, cudaStreamSynchronize(s));
    for (int i : ids) hres[i] = all[i];
  }
  dfree(ctx, xs);
  dfree(ctx, r);
  dfree(ctx, z);
  dfree(ctx, p);
  dfree(ctx, q);
  dfree(ctx, dinv);
  dfree(ctx, queue);
  dfree(ctx, head);
  pool_free(ctx, res);
  return st;
}

// lanes of instance i in k_bpcg: fixed by set_lanes, else from
// the instance's own mean row length (so the result depends on nothing
// else); block rows of 3 take 2 or 4
static int inst_lanes(const gt_batch* B, int i) {
  const Matrix* A = B->mats[i];
  int g = B->G ? B->G : row_lanes(A->nbrows > 0 ? (double)A->bnnz / (double)A->nbrows : 1.0);
  if (A->bs == 3) g = g <= 2 ? 2 : 4;
  return g;
}

// one launch per block size and lane count (instances keep their
// largest-first order)
template <class V, class X, bool REL>
static int launch_small(gt_batch* B, const std::vector<int>& ids, const double* b, double* x, double rtol, int maxit,
                        double delta, int from_x, std::vector<BRes>& hres) {
  for (int bs : {1, 3})
    for (int g : {1, 2, 4, 8}) {
      std::vector<int> sub;
      for (int i : ids)
        if (B->mats[i]->bs == bs && inst_lanes(B, i) == g) sub.push_back(i);
      if (!sub.empty()) GT_TRY((launch_small_g<V, X, REL>(B, bs, g, sub, b, x, rtol, maxit, delta, from_x, hres)));
    }
  return GT_OK;
}

// The instances ids, of block size BS, by k_bpcg_cluster; from (optional): the
// states of FP32 runs that these continue, by instance
template <int BS, class V, class X, bool REL>
static int launch_shared(gt_batch* B, const std::vector<int>& ids, const double* b, double* x, double rtol, int maxit,
                         double delta, const std::vector<pcg::PState>* from, std::vector<pcg::PState>& st) {
  Ctx* ctx = B->ctx;
  cudaStream_t s = ctx->stream;
  if (ids.empty()) return GT_OK;
  Blocks mem(ctx);
  const int64_t n = B->ntot;
  X *xs, *r, *p, *q, *dinv;
  int2* queue;
  int32_t* head;
  pcg::PState* dst;
  GT_TRY(mem.get(&xs, n));
  GT_TRY(mem.get(&r, n));
  GT_TRY(mem.get(&p, n));
  GT_TRY(mem.get(&q, n));
  GT_TRY(mem.get(&dinv, n));
  GT_TRY(mem.get(&queue, (int64_t)ids.size()));
  GT_TRY(mem.get(&head, 1));
  GT_TRY(mem.get(&dst, B->n));
  std::vector<int2> jobs;
  for (int i : ids) jobs.push_back(make_int2(i, pcg::entry_lanes(B->mats[i], sizeof(X) == sizeof(double))));
  GT_TRY(copy_in(ctx, queue, jobs.data(), (int64_t)jobs.size()));
  if (from) GT_TRY(copy_in(ctx, dst, from->data(), B->n));
  GT_CUDA(ctx, cudaMemsetAsync(head, 0, sizeof(int32_t), s));
  auto kern = k_bpcg_cluster<BS, V, X, REL>;
  // as much shared memory as the largest instance needs, up to 64 KB: beyond,
  // the L1 left for the matrix is worth more (256 instances of 4,096 rows of
  // 24 entries 6.4 ms at 64 KB, 6.9 with none, 9.7 at 100 KB; of 3,969 rows of 9
  // entries 10.0, 11.9 and 9.6)
  constexpr int kMost = 64 * 1024;
  int64_t need = 0;
  for (int i : ids) need = std::max(need, (5 * (int64_t)sizeof(X) * BS + 4) * (B->mats[i]->nbrows + 1) + 128);
  const int smem = (int)std::min<int64_t>(kMost, need) & ~15;
  GT_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
  int per_sm = 0;
  GT_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, vthreads(BS), smem));
  const int grid = (int)std::min<int64_t>((int64_t)std::max(per_sm, 1) * ctx->num_sms, (int64_t)ids.size());
  const pcg::PRule rule{rtol * rtol, delta * delta, maxit, ctx->ir_stall_ratio, ctx->ir_stall_count};
  kern<<<GT_KC(ctx, grid), vthreads(BS), smem, s>>>(B->d_inst, queue, (int)ids.size(), head, b, x, xs, r, p, q, dinv, dst, rule,
                                          from != nullptr, smem);
  GT_LAUNCH(ctx, "k_bpcg_cluster");
  std::vector<pcg::PState> all(B->n);
  GT_CUDA(ctx, cudaMemcpyAsync(all.data(), dst, sizeof(pcg::PState) * B->n, cudaMemcpyDeviceToHost, s));
  GT_CUDA(ctx, cudaStreamSynchronize(s));
  for (int i : ids) st[i] = all[i];
  return GT_OK;
}
template <class V, class X, bool REL>
static int launch_shared(gt_batch* B, const std::vector<int>& ids, const double* b, double* x, double rtol, int maxit,
                         double delta, const std::vector<pcg::PState>* from, std::vector<pcg::PState>& st) {
  std::vector<int> sub[2];
  for (int i : ids) sub[B->mats[i]->bs == 3].push_back(i);
  GT_TRY((launch_shared<1, V, X, REL>(B, sub[0], b, x, rtol, maxit, delta, from, st)));
  return launch_shared<3, V, X, REL>(B, sub[1], b, x, rtol, maxit, delta, from, st);
}

// operations of an iteration: entries and row costs
static int64_t cg_work(const Matrix* A) {
  return A->bnnz * A->bs * A->bs + pcg::row_cost(A->bs) * A->nbrows * A->bs;
}

// Which of the instances ids (largest first) k_bpcg_cluster takes, the others
// being left to the clusters.  Both give the same result, so the choice may
// look at the whole batch: the smallest ones go to single CTAs as long as that
// shortens the estimated time of the clusters (at_once of them side by side)
// and then the CTAs.  An iteration of an instance of w operations takes
// about 5.5 + w / 55,000 us on a cluster and 4 + w / 2,600 us (block
// rows 3,600) on a CTA alone on its SM, SMs gain 15% by a second one, and iterations go
// roughly with rows^0.4.  Measured, mixed solves to 1e-10, ms, cluster / CTA: 1
// instance of 3,969 rows 1.2 / 6.3, 16 3.7 / 6.3, 64 12.3 / 6.8, 256 46 / 10.0; 64
// of 16,129 rows 33 / 62, 256 125 / 86; 512 of 1,225 rows 54 / 4.7.
static void pick_shared(const gt_batch* B, const std::vector<int>& ids, int at_once, std::vector<int>* shared) {
  const int m = (int)ids.size();
  std::vector<double> cl(m), one(m), rest(m + 1, 0.0);
  for (int k = 0; k < m; k++) {
    const Matrix* A = B->mats[ids[k]];
    const double rows = (double)A->nbrows * A->bs, its = pow(rows, 0.4);
    const double w = (double)cg_work(A);
    cl[k] = its * (5.5 + w / 55000.0);
    one[k] = its * (4.0 + w / (A->bs == 1 ? 2600.0 : 3600.0));
  }
  for (int k = m - 1; k >= 0; k--) rest[k] = rest[k + 1] + one[k];
  std::vector<double> slot(std::max(at_once, 1), 0.0);
  double most = 0.0, best = 0.0;
  int first = 0;  // instances from here on go to single CTAs
  for (int k = 0; k <= m; k++) {
    const double t = most + (k < m ? std::max(one[k], rest[k] / (1.15 * B->ctx->num_sms)) : 0.0);
    if (k == 0 || t <= best) {
      best = t;
      first = k;
    }
    if (k < m) {
      double& s = *std::min_element(slot.begin(), slot.end());
      s += cl[k];
      most = std::max(most, s);
    }
  }
  shared->assign(ids.begin() + first, ids.end());
}

// Moves the instances that k_bpcg_cluster solves from clustered to shared: of
// those pick_shared names, the ones that the cluster kernel would not pass on
// to a grid
static int split_clustered(gt_batch* B, std::vector<int>& clustered, int mode, std::vector<int>* shared) {
  Ctx* ctx = B->ctx;
  std::vector<int> passed;
  for (int bs : {1, 3}) {
    std::vector<int> ids, sub;
    for (int i : clustered)
      if (B->mats[i]->bs == bs) ids.push_back(i);
    if (ids.empty()) continue;
    std::stable_sort(ids.begin(), ids.end(), [&](int i, int j) { return cg_work(B->mats[i]) > cg_work(B->mats[j]); });
    pcg::ClusterRoom r64, r32;
    if (mode != GT_SOLVE_FP32) GT_TRY((pcg::cluster_room<double, double, true>(ctx, bs, &r64)));
    if (mode == GT_SOLVE_FP32) GT_TRY((pcg::cluster_room<float, float, false>(ctx, bs, &r32)));
    if (mode == GT_SOLVE_IR) GT_TRY((pcg::cluster_room<float, float, true>(ctx, bs, &r32)));
    const int at_once = mode == GT_SOLVE_FP64 ? r64.at_once : r32.at_once;
    if (at_once >= 1) pick_shared(B, ids, at_once, &sub);
    std::vector<int32_t> fits(sub.size());
    if (!sub.empty()) {
      Blocks mem(ctx);
      int32_t *dids, *dfits;
      GT_TRY(mem.get(&dids, (int64_t)sub.size()));
      GT_TRY(mem.get(&dfits, (int64_t)sub.size()));
      GT_TRY(copy_in(ctx, dids, sub.data(), (int64_t)sub.size()));
      auto kern = bs == 1 ? k_cluster_fits<1> : k_cluster_fits<3>;
      kern<<<GT_KC(ctx, (unsigned)sub.size()), BT, 0, ctx->stream>>>(B->d_inst, dids, r64.smem, r32.smem,
                                                                    mode == GT_SOLVE_IR, dfits);
      GT_LAUNCH(ctx, "k_cluster_fits");
      GT_CUDA(ctx, cudaMemcpyAsync(fits.data(), dfits, sizeof(int32_t) * sub.size(), cudaMemcpyDeviceToHost, ctx->stream));
      GT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    const size_t head = ids.size() - sub.size();
    for (size_t k = 0; k < ids.size(); k++) (k >= head && fits[k - head] ? *shared : passed).push_back(ids[k]);
  }
  clustered = passed;
  return GT_OK;
}

static int batch_solve(gt_batch* B, const double* b, double* x, double rtol, int maxit, int mode, gt_solve_info* infos) {
  Ctx* ctx = B->ctx;
  const int ni = B->n;
  for (auto* A : B->mats) {
    if ((mode == GT_SOLVE_FP64 && !A->val64) || (mode == GT_SOLVE_FP32 && !A->val32))
      return set_error(ctx, GT_ERR_INVALID, "batch solve: matrices lack the values of this mode");
    if (mode == GT_SOLVE_IR && (!A->val64 || !A->val32))
      return set_error(ctx, GT_ERR_INVALID, "batch IR solve needs GT_MIXED matrices");
  }
  if (mode != GT_SOLVE_FP64 && mode != GT_SOLVE_FP32 && mode != GT_SOLVE_IR)
    return set_error(ctx, GT_ERR_INVALID, "unknown solve mode");
  std::vector<gt_solve_info> info(ni);
  std::vector<BRes> hres(ni);
  int status = GT_OK;
  // x = 0 at the instances ids and their addresses, then the shared launches
  // of the persistent solver (clusters: one cluster per instance)
  auto groups = [&](const std::vector<int>& ids, bool clusters) -> int {
    if (ids.empty()) return GT_OK;
    std::vector<Matrix*> As;
    std::vector<const double*> bs;
    std::vector<double*> xs;
    for (int i : ids) {
      const int64_t off = B->h_inst[i].off;
      As.push_back(B->mats[i]);
      bs.push_back(b + off);
      xs.push_back(x + off);
      GT_CUDA(ctx, cudaMemsetAsync(x + off, 0, sizeof(double) * B->mats[i]->nbrows * B->mats[i]->bs, ctx->stream));
    }
    std::vector<gt_solve_info> ginf;
    std::vector<int> gst;
    GT_TRY(pcg_persistent_groups(ctx, As, mode, bs, xs, rtol, maxit, ginf, gst, clusters));
    for (size_t k = 0; k < ids.size(); k++) {
      info[ids[k]] = ginf[k];
      if (gst[k] != GT_OK && gst[k] != GT_ERR_NOT_CONVERGED) return gst[k];
      if (gst[k] == GT_ERR_NOT_CONVERGED) status = gst[k];
    }
    return GT_OK;
  };
  // small instances: one persistent launch ...
  std::vector<int> one, clustered;
  for (int i : B->small) {
    const int64_t rows = B->h_inst[i].nrows * B->h_inst[i].bs;
    (rows <= kOneCtaRows ? one : clustered).push_back(i);
  }
  if (mode == GT_SOLVE_FP64) {
    GT_TRY((launch_small<double, double, true>(B, one, b, x, rtol, maxit, 0.0, 0, hres)));
  } else if (mode == GT_SOLVE_FP32) {
    GT_TRY((launch_small<float, float, false>(B, one, b, x, rtol, maxit, 0.0, 0, hres)));
  } else {
    GT_TRY((launch_small<float, float, true>(B, one, b, x, rtol, maxit, ctx->ir_delta, 0, hres)));
    std::vector<int> stalled;
    for (int i : one)
      if (hres[i].status == 2) stalled.push_back(i);
    if (!stalled.empty()) {
      // FP32 stalled (eps32 * cond ~ 1): these instances go on in FP64 from
      // their current FP64 solution
      std::vector<BRes> h64(ni);
      GT_TRY((launch_small<double, double, true>(B, stalled, b, x, rtol, maxit, 0.0, 1, h64)));
      for (int i : stalled) {
        info[i].fp64_iterations = h64[i].iters;
        h64[i].iters += hres[i].iters;
        h64[i].nupd += hres[i].nupd;
        hres[i] = h64[i];
      }
    }
  }
  for (int i : one) {
    info[i].iterations = hres[i].iters;
    info[i].outer_iterations = mode == GT_SOLVE_FP32 ? 0 : hres[i].nupd;
    info[i].rel_residual = hres[i].bb > 0 ? sqrt(hres[i].rr / hres[i].bb) : 0.0;
    if (mode == GT_SOLVE_FP64) info[i].fp64_iterations = hres[i].iters;
    if (hres[i].status != 0) status = GT_ERR_NOT_CONVERGED;
  }
  // ... then single CTAs with a cluster's arithmetic, then clusters
  std::vector<int> shared;
  GT_TRY(split_clustered(B, clustered, mode, &shared));
  if (!shared.empty()) {
    std::vector<pcg::PState> st(ni), st2(ni);
    if (mode == GT_SOLVE_FP64) {
      GT_TRY((launch_shared<double, double, true>(B, shared, b, x, rtol, maxit, 0.0, nullptr, st)));
      for (int i : shared) info[i].fp64_iterations = st[i].iters;
    } else if (mode == GT_SOLVE_FP32) {
      GT_TRY((launch_shared<float, float, false>(B, shared, b, x, rtol, maxit, 0.0, nullptr, st)));
    } else {
      GT_TRY((launch_shared<float, float, true>(B, shared, b, x, rtol, maxit, ctx->ir_delta, nullptr, st)));
      std::vector<int> stalled;
      for (int i : shared)
        if (st[i].done == 2) stalled.push_back(i);
      GT_TRY((launch_shared<double, double, true>(B, stalled, b, x, rtol, maxit, 0.0, &st, st2)));
      for (int i : stalled) {
        info[i].fp64_iterations = st2[i].iters - st[i].iters;
        st[i] = st2[i];
      }
    }
    for (int i : shared) {
      info[i].iterations = st[i].iters;
      info[i].outer_iterations = mode == GT_SOLVE_FP32 ? 0 : st[i].nupd;
      info[i].rel_residual = st[i].bb > 0 ? sqrt(st[i].rr / st[i].bb) : 0.0;
      if (!(st[i].rr <= st[i].tol2)) status = GT_ERR_NOT_CONVERGED;
    }
  }
  GT_TRY(groups(clustered, true));
  mark(ctx, "batch_small");
  // medium instances of this context: grouped persistent launches
  std::vector<int> rest;
  {
    std::vector<int> grouped;
    for (int i : B->large) {
      Matrix* A = B->mats[i];
      if ((mode == GT_SOLVE_FP64 || mode == GT_SOLVE_IR) && A->ctx == ctx && A->nbrows * A->bs <= kPersistentMaxRows)
        grouped.push_back(i);
      else
        rest.push_back(i);
    }
    GT_TRY(groups(grouped, false));
  }
  mark(ctx, "batch_grouped");
  // large instances: the single-system solver, one after the other (each
  // fills the device by itself)
  for (int i : rest) {
    Matrix* A = B->mats[i];
    const int64_t off = B->h_inst[i].off;
    GT_CUDA(ctx, cudaMemsetAsync(x + off, 0, sizeof(double) * A->nbrows * A->bs, ctx->stream));
    // a matrix of another context solves on that context's stream: b and x
    // (written on this one) are complete first; solve() returns synchronised
    if (A->ctx != ctx) GT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    int s = solve(A, b + off, x + off, rtol, maxit, mode, &info[i]);
    if (s != GT_OK && s != GT_ERR_NOT_CONVERGED) return s;
    if (s == GT_ERR_NOT_CONVERGED) status = s;
  }
  mark(ctx, "batch_large");
  if (infos)
    for (int i = 0; i < ni; i++) infos[i] = info[i];
  if (status == GT_ERR_NOT_CONVERGED) set_error(ctx, status, "batch solve: some instance missed the tolerance");
  return status;
}

}  // namespace gt

using namespace gt;

extern "C" {

int gt_batch_create(gt_ctx* ctx, int n, gt_matrix* const* mats, gt_batch** out) {
  if (!ctx || !out || n <= 0 || !mats) return GT_ERR_INVALID;
  *out = nullptr;
  cudaSetDevice(ctx->device);
  gt_batch* B = new gt_batch();
  B->ctx = ctx;
  B->n = n;
  int64_t off = 0;
  for (int i = 0; i < n; i++) {
    Matrix* A = mats[i];
    if (!A || A->ctx->device != ctx->device || (A->bs != 1 && A->bs != 3)) {
      delete B;
      return set_error(ctx, GT_ERR_INVALID,
                       "batch: matrices must have block size 1 or 3 and be on this context's device");
    }
    int s = find_diag(A);
    // a matrix of another context (assembled on another stream): its
    // diagonal positions are complete before this context's kernels read them
    if (s == GT_OK && A->ctx != ctx && cudaStreamSynchronize(A->ctx->stream) != cudaSuccess)
      s = set_error(ctx, GT_ERR_CUDA, "batch: synchronising a matrix's context failed");
    if (s != GT_OK) {
      delete B;
      return s;
    }
    BInst in{};
    in.rowptr = A->rowptr;
    in.colind = A->colind;
    in.v64 = A->val64;
    in.v32 = A->val32;
    in.diag = A->diag_pos;
    in.nrows = A->nbrows;
    in.off = off;
    in.bs = A->bs;
    off += A->nbrows * A->bs;
    B->h_inst.push_back(in);
    B->mats.push_back(A);
  }
  classify(B);  // largest small instances first: the queue then balances the CTAs
  B->ntot = off;
  int s = dalloc(ctx, &B->d_inst, n);
  if (s == GT_OK) s = copy_in(ctx, B->d_inst, B->h_inst.data(), n);
  if (s == GT_OK && cudaStreamSynchronize(ctx->stream) != cudaSuccess) s = GT_ERR_CUDA;
  if (s != GT_OK) {
    gt_batch_destroy(B);
    return s;
  }
  *out = B;
  return GT_OK;
}

int gt_batch_set_lanes(gt_batch* B, int lanes) {
  if (!B || (lanes != 0 && lanes != 1 && lanes != 2 && lanes != 4 && lanes != 8)) return GT_ERR_INVALID;
  B->G = lanes;
  return GT_OK;
}

int gt_batch_set_small_rows(gt_batch* B, int64_t rows) {
  if (!B || rows < 0 || rows > kSmallRows) return GT_ERR_INVALID;
  B->small_rows = rows;
  classify(B);
  return GT_OK;
}

int gt_batch_info(const gt_batch* B, int64_t* info) {
  if (!B || !info) return GT_ERR_INVALID;
  info[0] = B->n;
  info[1] = B->ntot;
  info[2] = (int64_t)B->small.size();
  info[3] = B->G;
  return GT_OK;
}

int gt_batch_solve(gt_batch* B, const double* b, double* x, double rtol, int maxit, int mode, gt_solve_info* infos) {
  if (!B || !b || !x) return GT_ERR_INVALID;
  Ctx* ctx = B->ctx;
  cudaSetDevice(ctx->device);
  cudaPointerAttributes ab{}, ax{};
  bool bdev = cudaPointerGetAttributes(&ab, b) == cudaSuccess && ab.type == cudaMemoryTypeDevice;
  cudaGetLastError();
  bool xdev = cudaPointerGetAttributes(&ax, x) == cudaSuccess && ax.type == cudaMemoryTypeDevice;
  cudaGetLastError();
  double *bd = (double*)b, *xd = x;
  if (!bdev) {
    GT_TRY(dalloc(ctx, &bd, B->ntot));
    GT_TRY(copy_in(ctx, bd, b, B->ntot));
  }
  if (!xdev) GT_TRY(dalloc(ctx, &xd, B->ntot));
  int s = batch_solve(B, bd, xd, rtol, maxit, mode, infos);
  if (!xdev) {
    int s2 = copy_out(ctx, x, xd, B->ntot);
    cudaStreamSynchronize(ctx->stream);
    if (s == GT_OK) s = s2;
    dfree(ctx, xd);
  }
  if (!bdev) dfree(ctx, bd);
  return s;
}

int gt_batch_destroy(gt_batch* B) {
  if (!B) return GT_ERR_INVALID;
  Ctx* ctx = B->ctx;
  dfree(ctx, B->d_inst);
  delete B;
  return GT_OK;
}

}  // extern "C"
