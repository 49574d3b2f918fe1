// gt_pcg.cu -- entry points of the persistent Jacobi-PCG (gt_pcg_impl.cuh) and
// its FP64 instances.
#include "gt_pcg_impl.cuh"

namespace gt {
namespace pcg {

template int cluster_room<double, double, true>(Ctx*, int, ClusterRoom*);
template int run_sliced<double, double, true>(Ctx*, Matrix*, const double*, const double*, double*, double, int, double,
                                    const PRun*, PRun*, int);
template int run_groups_dispatch<double, double, true>(
    Ctx*, Place, int, const std::vector<Matrix*>&, const std::vector<const double*>&,
    const std::vector<const double*>&, const std::vector<double*>&, double, int, double, const std::vector<const PRun*>&,
    std::vector<PRun>&, std::vector<int>&);

template <class V, class X, bool REL>
int run_dispatch(Matrix* A, const V* val, const double* b, double* x, double rtol, int maxit, double delta,
                 const PRun* from, PRun* out) {
  std::vector<PRun> outs(1);
  std::vector<int> st(1, GT_OK);
  GT_TRY((run_groups_dispatch<V, X, REL>(A->ctx, Place::Auto, A->bs, {A}, {val}, {b}, {x}, rtol, maxit,
                                         delta, {from}, outs, st)));
  *out = outs[0];
  return st[0];
}

// The solver's grid barrier run alone: `ctas` co-resident CTAs wait for
// ctas + missing arrivals.  With missing > 0 the barrier can never complete,
// so each CTA gives up after timeout_ns and sets the error word.
__global__ void __launch_bounds__(PT) k_barrier_probe(uint32_t* bar, uint32_t target, int32_t* err,
                                                      uint64_t timeout_ns) {
  __shared__ int s_abort;
  if (threadIdx.x == 0) s_abort = 0;
  grid_sync(bar, target, err, &s_abort, timeout_ns);
}

// The local kernel's sum run alone: each thread of `gridDim.x` CTAs brings one
// value, and the CTAs wait for nb arrivals.
template <class X>
__global__ void __launch_bounds__(LT) k_sum_probe(const double* __restrict__ values, int nb, double* slots, int32_t* err,
                                                  double* total, uint64_t timeout_ns) {
  __shared__ LShared S;
  if (threadIdx.x == 0) S.abort = 0;
  __syncthreads();
  uint32_t epoch = 0;
  const X v[1] = {(X)values[(size_t)blockIdx.x * LT + threadIdx.x]};
  local_total<1, false>(
      v, LT, nb, blockIdx.x, slots, epoch, err, S, nullptr,
      [&](const double* tot) {
        if (blockIdx.x == 0) *total = tot[0];
      },
      timeout_ns);
}

__global__ void k_divide_probe(const double* __restrict__ a, const double* __restrict__ b, int64_t n,
                               double* __restrict__ q) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) q[i] = quick_div(a[i], b[i]);
}

}  // namespace pcg

using namespace pcg;

int barrier_probe(Ctx* ctx, int ctas, int missing, int64_t timeout_ns) {
  if (ctas < 1 || missing < 0 || timeout_ns <= 0 || timeout_ns > 2000000000ll)
    return set_error(ctx, GT_ERR_INVALID, "barrier probe: 1 <= ctas, 0 <= missing, 0 < timeout <= 2 s");
  int dev = 0, nsm = 0, per_sm = 0;
  GT_CUDA(ctx, cudaGetDevice(&dev));
  GT_CUDA(ctx, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  GT_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_barrier_probe, PT, 0));
  if ((int64_t)ctas > (int64_t)nsm * per_sm) return set_error(ctx, GT_ERR_INVALID, "barrier probe: more CTAs than fit");
  cudaStream_t s = ctx->stream;
  uint32_t* bar = nullptr;
  int32_t* err = nullptr;
  GT_TRY(dalloc(ctx, &bar, 2));
  GT_TRY(dalloc(ctx, &err, 2));
  GT_CUDA(ctx, cudaMemsetAsync(bar, 0, 2 * sizeof(uint32_t), s));
  GT_CUDA(ctx, cudaMemsetAsync(err, 0, 2 * sizeof(int32_t), s));
  uint32_t target = (uint32_t)(ctas + missing);
  uint64_t tns = (uint64_t)timeout_ns;
  void* kargs[] = {&bar, &target, &err, &tns};
  ctx->launches++;
  GT_CUDA(ctx, cudaLaunchCooperativeKernel((const void*)k_barrier_probe, dim3(ctas), dim3(PT), kargs, 0, s));
  GT_CUDA(ctx, cudaMemcpyAsync(ctx->h_scratch, err, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  GT_CUDA(ctx, cudaStreamSynchronize(s));
  int32_t e = 0;
  memcpy(&e, ctx->h_scratch, sizeof(int32_t));
  dfree(ctx, bar);
  dfree(ctx, err);
  return e ? set_error(ctx, GT_ERR_TIMEOUT, "barrier probe: the grid barrier timed out") : GT_OK;
}

int sum_probe(Ctx* ctx, int ctas, int missing, int64_t timeout_ns, int precision, const double* values,
              double* total) {
  if (ctas < 1 || missing < 0 || ctas + missing > LMAXCTA || ctas > ctx->num_sms || timeout_ns <= 0 ||
      timeout_ns > 2000000000ll || !values || !total || (precision != GT_FP64 && precision != GT_FP32))
    return set_error(ctx, GT_ERR_INVALID, "sum probe: 1 <= ctas <= SMs, 0 <= missing, at most 160 CTAs, timeout <= 2 s");
  cudaStream_t s = ctx->stream;
  const int nb = ctas + missing;
  Blocks mem(ctx);
  double *dv, *slots, *dt;
  int32_t* err;
  GT_TRY(mem.get(&dv, (int64_t)ctas * LT));
  GT_TRY(mem.get(&slots, (int64_t)LSLOTS * nb + LCTRS));
  GT_TRY(mem.get(&dt, 1));
  GT_TRY(mem.get(&err, 2));
  GT_TRY(copy_in(ctx, dv, values, (int64_t)ctas * LT));
  GT_CUDA(ctx, cudaMemsetAsync(slots, 0, sizeof(double) * (LSLOTS * nb + LCTRS), s));
  GT_CUDA(ctx, cudaMemsetAsync(err, 0, 2 * sizeof(int32_t), s));
  uint64_t tns = (uint64_t)timeout_ns;
  int n = nb;
  void* kargs[] = {&dv, &n, &slots, &err, &dt, &tns};
  const void* kern = precision == GT_FP64 ? (const void*)k_sum_probe<double> : (const void*)k_sum_probe<float>;
  ctx->launches++;
  GT_CUDA(ctx, cudaLaunchCooperativeKernel(kern, dim3(ctas), dim3(LT), kargs, 0, s));
  GT_CUDA(ctx, cudaMemcpyAsync(ctx->h_scratch, err, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  GT_CUDA(ctx, cudaMemcpyAsync(ctx->h_dscratch, dt, sizeof(double), cudaMemcpyDeviceToHost, s));
  GT_CUDA(ctx, cudaStreamSynchronize(s));
  int32_t e = 0;
  memcpy(&e, ctx->h_scratch, sizeof(int32_t));
  if (e) return set_error(ctx, GT_ERR_TIMEOUT, "sum probe: the sum timed out");
  memcpy(total, ctx->h_dscratch, sizeof(double));
  return GT_OK;
}

int divide_probe(Ctx* ctx, int64_t n, const double* a, const double* b, double* q) {
  if (n < 1 || !a || !b || !q) return set_error(ctx, GT_ERR_INVALID, "divide probe: empty");
  Blocks mem(ctx);
  double *da, *db, *dq;
  GT_TRY(mem.get(&da, n));
  GT_TRY(mem.get(&db, n));
  GT_TRY(mem.get(&dq, n));
  GT_TRY(copy_in(ctx, da, a, n));
  GT_TRY(copy_in(ctx, db, b, n));
  k_divide_probe<<<GT_KC(ctx, grid_for(n, 256)), 256, 0, ctx->stream>>>(da, db, n, dq);
  GT_LAUNCH(ctx, "k_divide_probe");
  GT_TRY(copy_out(ctx, q, dq, n));
  GT_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return GT_OK;
}

// pcg_persistent for several systems on ctx, grouped into shared launches by
// block size; x: start values; per-system infos and statuses.
// Each system's result is bitwise that of pcg_persistent on it alone, or --
// with clusters -- of the same call on it alone: every system on one cluster.
int pcg_persistent_groups(Ctx* ctx, const std::vector<Matrix*>& As, int mode, const std::vector<const double*>& b,
                          const std::vector<double*>& x, double rtol, int maxit, std::vector<gt_solve_info>& infos,
                          std::vector<int>& status, bool clusters) {
  const int n = (int)As.size();
  const Place place = clusters ? Place::Cluster : Place::Auto;
  infos.assign(n, gt_solve_info{});
  status.assign(n, GT_OK);
  std::vector<PRun> runs(n);
  for (int bs : {1, 3}) {
    std::vector<int> ids;
    for (int i = 0; i < n; i++)
      if (As[i]->bs == bs) ids.push_back(i);
    if (ids.empty()) continue;
    std::vector<Matrix*> A;
    std::vector<const double*> bb;
    std::vector<double*> xx;
    std::vector<const PRun*> none(ids.size(), nullptr);
    std::vector<PRun> out(ids.size());
    std::vector<int> st(ids.size(), GT_OK);
    for (int i : ids) {
      A.push_back(As[i]);
      bb.push_back(b[i]);
      xx.push_back(x[i]);
    }
    std::vector<const double*> v64;
    std::vector<const float*> v32;
    for (Matrix* M : A) {
      v64.push_back(M->val64);
      v32.push_back(M->val32);
    }
    if (mode == GT_SOLVE_FP64) {
      GT_TRY((run_groups_dispatch<double, double, true>(ctx, place, bs, A, v64, bb, xx, rtol, maxit, 0.0, none,
                                                        out, st)));
      for (size_t k = 0; k < ids.size(); k++) infos[ids[k]].fp64_iterations = out[k].st.iters;
    } else if (mode == GT_SOLVE_FP32) {
      GT_TRY((run_groups_dispatch<float, float, false>(ctx, place, bs, A, v32, bb, xx, rtol, maxit, 0.0, none, out,
                                                       st)));
    } else {
      GT_TRY((run_groups_dispatch<float, float, true>(ctx, place, bs, A, v32, bb, xx, rtol, maxit, ctx->ir_delta,
                                                      none, out, st)));
      // stalled FP32 runs go on in FP64 from their FP64 solutions, as alone
      std::vector<size_t> sk;
      for (size_t k = 0; k < ids.size(); k++)
        if (st[k] == PCG_STALLED) sk.push_back(k);
      if (!sk.empty()) {
        std::vector<Matrix*> A2;
        std::vector<const double*> v2, b2;
        std::vector<double*> x2;
        std::vector<const PRun*> f2;
        for (size_t k : sk) {
          A2.push_back(A[k]);
          v2.push_back(A[k]->val64);
          b2.push_back(bb[k]);
          x2.push_back(xx[k]);
          f2.push_back(&out[k]);
        }
        std::vector<PRun> o2(sk.size());
        std::vector<int> s2(sk.size(), GT_OK);
        GT_TRY((run_groups_dispatch<double, double, true>(ctx, place, bs, A2, v2, b2, x2, rtol, maxit, 0.0, f2, o2,
                                                          s2)));
        for (size_t j = 0; j < sk.size(); j++) {
          infos[ids[sk[j]]].fp64_iterations = o2[j].st.iters - out[sk[j]].st.iters;
          out[sk[j]] = o2[j];
          st[sk[j]] = s2[j];
        }
      }
    }
    for (size_t k = 0; k < ids.size(); k++) {
      gt_solve_info& inf = infos[ids[k]];
      inf.iterations = out[k].st.iters;
      inf.outer_iterations = mode == GT_SOLVE_FP32 ? 0 : out[k].st.nupd;
      inf.rel_residual = out[k].st.bb > 0 ? sqrt(out[k].st.rr / out[k].st.bb) : 0.0;
      status[ids[k]] = st[k];
    }
    }
  return GT_OK;
}

int pcg_persistent(Matrix* A, int mode, const double* b, double* x, double rtol, int maxit, int32_t* iters,
                   int32_t* nupd, int32_t* iters64, double* relres, bool sliced) {
  PRun run;
  int s;
  *iters64 = 0;
  Ctx* ctx = A->ctx;
  if (mode == GT_SOLVE_FP64) {
    s = sliced ? run_sliced<double, double, true>(ctx, A, A->val64, b, x, rtol, maxit, 0.0, nullptr, &run, 0)
               : run_dispatch<double, double, true>(A, A->val64, b, x, rtol, maxit, 0.0, nullptr, &run);
    *iters64 = run.st.iters;
  } else if (mode == GT_SOLVE_IR) {
    s = sliced ? run_sliced<float, float, true>(ctx, A, A->val32, b, x, rtol, maxit, ctx->ir_delta, nullptr, &run, 0)
               : run_dispatch<float, float, true>(A, A->val32, b, x, rtol, maxit, ctx->ir_delta, nullptr, &run);
    if (s == PCG_STALLED) {
      // the FP32 iteration stalled or lost its rate (eps32 * cond(A) too
      // large): CG goes on in FP64 from the current FP64 solution, its
      // directions restarted (the iteration count and ||b|| carry over)
      PRun r32 = run;
      PRun r64;
      s = sliced ? run_sliced<double, double, true>(ctx, A, A->val64, b, x, rtol, maxit, 0.0, &r32, &r64, 0) : PCG_NOFIT;
      if (s == PCG_NOFIT) s = run_dispatch<double, double, true>(A, A->val64, b, x, rtol, maxit, 0.0, &r32, &r64);
      *iters64 = r64.st.iters - r32.st.iters;
      run = r64;
    }
  } else {
    s = sliced ? run_sliced<float, float, false>(ctx, A, A->val32, b, x, rtol, maxit, 0.0, nullptr, &run, 0)
               : run_dispatch<float, float, false>(A, A->val32, b, x, rtol, maxit, 0.0, nullptr, &run);
  }
  if (s == PCG_NOFIT) return s;
  *iters = run.st.iters;
  *nupd = run.st.nupd;
  *relres = run.st.bb > 0 ? sqrt(run.st.rr / run.st.bb) : 0.0;
  return s;
}

}  // namespace gt
