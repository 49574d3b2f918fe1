// gt_pcg_local.cuh -- the persistent Jacobi-PCG on CTA-local vectors.
//
// Included by gt_pcg_impl.cuh (inside its namespace), which owns the
// state, the launches and the algorithm's description.  CTA c owns a
// contiguous range of block rows and keeps in shared memory
//
//   s_r, s_q, s_xs, s_di   its own rows' vectors (and s_z in a cluster)
//   s_p                    p at every column its rows touch: its own rows and
//                          its halo, the sorted distinct columns (a bitmap
//                          over all columns gives each its local index)
//   s_val, s_lc            the values and local columns of its first rows, as
//                          many as fit; the others stream from L2 with 16-bit
//                          local columns
//
// The direction p = z + beta p is formed by every CTA on its own local set
// (the halo entries are bitwise the owner's: the same operands in the same
// operation), so p never goes through global memory, the SpMV gathers from
// shared memory, and an iteration needs two barriers instead of three:
//
//   P1  p = z + beta p (own + halo), q = A p, p.q   -> sum + barrier, alpha
//   P2  xs += alpha p, r -= alpha q, z = Dinv r     -> sum + barrier, beta
//
// CL: the CTAs are one thread-block cluster.  z is read from its owner's
// shared memory, the partial sums go straight into every CTA's, and the
// barrier is the cluster's: 770 clocks against 2,700 for an arrival counter
// in L2 polled by the CTAs of a grid (and 1,500 more for the partials behind
// it).  Small systems, for which the barriers are the iteration, take it.
//
// SL: systems too large for that (scalar rows).  xs and Dinv stay in global
// memory (a thread only touches its own rows' entries), the matrix streams
// from its sliced copy (32-row slices, a lane per row, coalesced) with 16-bit
// local columns in the same layout, and the bitmap covers only the window of
// columns the CTA touches.
//
// What bounds it.  GB300 issues one FP64 warp instruction per SM sub-partition
// every 63 clocks (measured; 304 clocks for one FP64 add in each of 16 warps,
// 570 for a division), whatever the number of active lanes.  So
//   * the rows are split by cost (entries and rows), not by count: Q2 vertex
//     rows have 125 entries, cell rows 27; and a CTA's warps take row groups
//     from a counter;
//   * the CG scalars are computed by one thread;
//   * sums over threads and CTAs run on the integer pipes (Fx): the partials
//     aligned to their largest exponent and rounded 54 to 57 bits below it,
//     added exactly by redux.sync -- order-independent, with an error below
//     that of an FP64 add chain -- instead of 109 clocks per FP64 butterfly
//     step.
// Large systems are bound by the FP64 pipe (2 FMAs a clock and SM) and the L2
// stream of the rows that are not resident.
#pragma once

constexpr int LT = 512;        // threads per CTA
constexpr int LNW = LT / 32;   // warps per CTA
constexpr int LMAXCTA = 160;   // most CTAs of one system in a grid (five partials per lane)
constexpr int LCLUSTER = 16;   // CTAs of one system in a cluster
constexpr int kLocalRows = 64; // scalar rows per CTA up to a CTA per SM
constexpr int kSliceRowCost = 5;  // a row's cost beside its entries in the sliced form, in entries
constexpr int LOVERFLOW = 3;   // PState::done: a CTA's local set does not fit
// a scalar row's cost beside its entries, in FMAs: the vector updates, the
// combination of its partial sums and its lanes' idle last step
constexpr int row_cost(int bs) { return bs == 1 ? 12 : 32; }
constexpr int LSLOTS = 12;     // doubles per CTA of the partial slots (two sets of three 16-byte slots)
constexpr int LCTRS = 16;      // doubles behind them: the arrival counter's line

// --- exact sums on the integer pipes ----------------------------------------
// A number m * 2^e; m = 0: zero (e = kFxZero); e = kFxNan: infinite or NaN.
// Normalised: |m| in [2^57, 2^58].
struct alignas(16) Fx {  // one 16-byte access
  long long m;
  int e;
};
constexpr int kFxZero = -100000, kFxNan = 100000;

__device__ __forceinline__ Fx fx_from(double v) {
  const long long b = __double_as_longlong(v);
  const int x = (int)((b >> 52) & 0x7ff);
  long long m = b & 0xfffffffffffffll;
  if (x) m |= 0x10000000000000ll;
  Fx f;
  f.e = x == 2047 ? kFxNan : (m ? (x ? x : 1) - 1080 : kFxZero);
  f.m = b < 0 ? -(m << 5) : m << 5;
  return f;
}
__device__ __forceinline__ Fx fx_from(float v) {
  const int b = __float_as_int(v);
  const int x = (b >> 23) & 0xff;
  int m = b & 0x7fffff;
  if (x) m |= 0x800000;
  Fx f;
  f.e = x == 255 ? kFxNan : (m ? (x ? x : 1) - 184 : kFxZero);
  f.m = b < 0 ? -((long long)m << 34) : (long long)m << 34;
  return f;
}
// m * 2^e with |m| in [2^57, 2^58]
__device__ __forceinline__ Fx fx_norm(Fx f) {
  if (f.m == 0 || f.e >= kFxNan) return Fx{f.e >= kFxNan ? 1 : 0, f.e >= kFxNan ? kFxNan : kFxZero};
  const int s = __clzll(f.m < 0 ? -f.m : f.m) - 6;
  if (s >= 0) return Fx{f.m << s, f.e - s};
  return Fx{(f.m + (1ll << (-s - 1))) >> -s, f.e - s};
}
__device__ __forceinline__ double fx_double(Fx f) {  // of a normalised number
  if (f.e >= kFxNan) return __longlong_as_double(0x7ff8000000000000ll);
  if (f.m == 0) return 0.0;
  const unsigned long long m = (unsigned long long)(f.m < 0 ? -f.m : f.m);
  const int x = f.e + 1080;  // biased exponent
  const long long sg = f.m < 0 ? (long long)(1ull << 63) : 0;
  if (__builtin_expect(x <= 0, 0)) {  // below 2^-1022: fewer than 53 bits
    const int sh = min(6 - x, 63);
    return __longlong_as_double(sg | (long long)((m + (1ull << (sh - 1))) >> sh));
  }
  if (x > 2046) return __longlong_as_double(sg | 0x7ff0000000000000ll);
  return __longlong_as_double(sg | (long long)(((unsigned long long)(x - 1) << 52) + ((m + 16) >> 5)));
}
// The sum over the warp of each lane's M numbers (normalised or from fx_from;
// at most 256 in all), in every lane, normalised: aligned to the largest
// exponent, rounded 54 to 57 bits below it, then added exactly, so the result
// does not depend on their order.
template <int M>
__device__ __forceinline__ Fx fx_warp_sum(const Fx (&v)[M]) {
  constexpr int DROP = M == 1 ? 1 : (M <= 4 ? 3 : 4);  // room for M * 32 numbers of 58 bits
  static_assert(M <= 8, "256 numbers");
  int em = kFxZero;
  long long t = 0;
#pragma unroll
  for (int i = 0; i < M; i++) em = max(em, v[i].e);
  em = __reduce_max_sync(0xffffffffu, em) + DROP;
#pragma unroll
  for (int i = 0; i < M; i++) {
    const int sh = min(em - v[i].e, 62);
    t += (v[i].m + ((1ll << sh) >> 1)) >> sh;
  }
  const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)t & 0x7ffffffu);
  const unsigned mi = __reduce_add_sync(0xffffffffu, (unsigned)(t >> 27) & 0x7ffffffu);
  const int hi = __reduce_add_sync(0xffffffffu, (int)(t >> 54));
  return fx_norm(Fx{((long long)hi << 54) + ((long long)mi << 27) + (long long)lo, em});
}

// a / b for one thread: Newton's iteration for the reciprocal and a residual
// correction of the quotient, five dependent FP64 instructions (315 clocks)
// where the library division takes 570; error below an ulp.  Operands near
// the ends of the exponent range, zero and non-finite ones take the division.
__device__ __forceinline__ double quick_div(double a, double b) {
  const int ea = (int)((__double_as_longlong(a) >> 52) & 0x7ff), eb = (int)((__double_as_longlong(b) >> 52) & 0x7ff);
  if (min(ea, eb) < 512 || max(ea, eb) > 1535) return a / b;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
  r = fma(r, fma(-b, r, 1.0), r);
  const double q = a * r;
  return fma(fma(-b, q, a), r, q);
}

__device__ __forceinline__ void slot_store(void* p, Fx f) {
  __stcg(reinterpret_cast<longlong2*>(p), make_longlong2(f.m, (long long)f.e));
}
__device__ __forceinline__ Fx slot_load(const void* p) {
  const longlong2 v = __ldcg(reinterpret_cast<const longlong2*>(p));
  return Fx{v.x, (int)v.y};
}

// --- the CTAs of a cluster --------------------------------------------------
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_store(uint32_t a, Fx f) {
  asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(f.m), "l"((long long)f.e) : "memory");
}
__device__ __forceinline__ double cluster_load(uint32_t a, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float cluster_load(uint32_t a, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// a <= b for values that are not negative (false when a is NaN): an integer
// comparison, which does not wait for the FP64 pipe
__device__ __forceinline__ bool le_pos(double a, double b) {
  return __double_as_longlong(a) <= __double_as_longlong(b) && __double_as_longlong(a) <= 0x7ff0000000000000ll;
}
__device__ __forceinline__ bool is_nan(double a) {
  return (__double_as_longlong(a) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}

// shared state of one CTA
struct LShared {
  Fx part[3][LNW];      // the warps' partials
  PState st;            // thread 0's
  double alpha, beta;   // of the step in hand
  int overflow;
  int act;              // bit 0: reliable update now, bit 1: leave the loop, bit 2: with bit 0, the cycle was slow
  int abort;
  int next;             // next row group of local_rows
  int rsm;              // rows whose matrix part is in shared memory
  int nloc;             // local columns
  int cmin, cmax;       // the columns' range (SL)
  int64_t rows[2];      // the CTA's first row and its end
  int wsum[LNW];
};
// partial sums of every CTA's warps, two sets (CL)
struct LCluster {
  Fx part[2][3][LNW * LCLUSTER];
  int64_t first[LCLUSTER + 1];  // first rows of the cluster's CTAs
};

// Sum of K values over all CTAs of the system, ctl(totals) by thread 0, and a
// barrier: what any thread wrote before it is visible to every
// thread after it.  nth: threads from there on hold zeros.  Two slot sets
// alternate by epoch: a CTA writes epoch e + 2 only after every CTA arrived
// at e + 1, so after every CTA read e.  False when a CTA of a grid did not
// arrive within the time limit (error word set; every CTA returns).
template <int K, bool CL, class T, class F>
__device__ __forceinline__ bool local_total(const T (&v)[K], int nth, int nb, int blk, double* slots, uint32_t& epoch,
                                            int32_t* err, LShared& S, LCluster* C, F&& ctl,
                                            uint64_t timeout_ns = BAR_TIMEOUT_NS) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nw = (min(nth, LT) + 31) >> 5;
  epoch++;
  if constexpr (CL) {
    // every warp's partials to every CTA, the cluster's barrier, one warp sums
    // them all
    auto& set = C->part[epoch & 1];
#pragma unroll
    for (int k = 0; k < K; k++) {
      Fx t{0, kFxZero};
      if (w < nw) {
        const Fx u[1] = {fx_from(v[k])};
        t = fx_warp_sum<1>(u);
      }
      if (lane < nb) cluster_store(cluster_addr(&set[k][blk * LNW + w], lane), t);
    }
    cluster_sync();
    if (w == 0) {
      Fx u[K][LNW * LCLUSTER / 32];
      double tot[K];
#pragma unroll
      for (int k = 0; k < K; k++)
#pragma unroll
        for (int i = 0; i < LNW * LCLUSTER / 32; i++)
          u[k][i] = lane + i * 32 < nb * LNW ? set[k][lane + i * 32] : Fx{0, kFxZero};
#pragma unroll
      for (int k = 0; k < K; k++) tot[k] = fx_double(fx_warp_sum<LNW * LCLUSTER / 32>(u[k]));
      if (lane == 0) ctl(tot);
    }
    __syncthreads();
    return true;
  } else {
    if (w < nw) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        const Fx u[1] = {fx_from(v[k])};
        const Fx t = fx_warp_sum<1>(u);
        if (lane == 0) S.part[k][w] = t;
      }
    }
    __syncthreads();
    if (w == 0) {
      Fx t[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const Fx u1[1] = {lane < nw ? S.part[k][lane] : Fx{0, kFxZero}};
        t[k] = fx_warp_sum<1>(u1);
      }
      if (nb > 1) {
        char* set = reinterpret_cast<char*>(slots) + (size_t)(epoch & 1) * 3 * nb * 16;
        uint32_t* ctr = reinterpret_cast<uint32_t*>(slots + (size_t)LSLOTS * nb);
        if (lane == 0) {
#pragma unroll
          for (int k = 0; k < K; k++) slot_store(set + ((size_t)k * nb + blk) * 16, t[k]);
          __threadfence();  // release: these stores and the CTA's writes before the __syncthreads above
          atomicAdd(ctr, 1u);
        }
        const uint32_t want = epoch * (uint32_t)nb;
        uint64_t t0 = 0;
        bool timed_out = false;
        for (int spin = 0;; spin++) {
          uint32_t n;
          asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(ctr) : "memory");
          if (__all_sync(0xffffffffu, (int32_t)(n - want) >= 0)) break;
          if ((spin & 255) == 255) {
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            timed_out = now - t0 > timeout_ns;
          }
          if (__any_sync(0xffffffffu, timed_out)) {
            if (lane == 0) {
              atomicExch(err, 1);
              S.abort = 1;
            }
            break;
          }
        }
        __threadfence();  // acquire: the other CTAs' writes before their arrivals
        Fx u[K][LMAXCTA / 32];
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
          for (int i = 0; i < LMAXCTA / 32; i++)
            u[k][i] = lane + i * 32 < nb ? slot_load(set + ((size_t)k * nb + lane + i * 32) * 16) : Fx{0, kFxZero};
#pragma unroll
        for (int k = 0; k < K; k++) t[k] = fx_warp_sum<LMAXCTA / 32>(u[k]);
      }
      double tot[K];
#pragma unroll
      for (int k = 0; k < K; k++) tot[k] = fx_double(t[k]);
      if (lane == 0) ctl(tot);
    }
    __syncthreads();
    return S.abort == 0;
  }
}

// combination of a row's J partial sums (lane stride BS) in lanes j = 0
template <int BS, int J, class A>
__device__ __forceinline__ A local_combine(A s, int j) {
  if constexpr (J == 5) {
    const A t = __shfl_down_sync(0xffffffffu, s, 3 * BS);
    if (j < 2) s += t;
    const A t1 = __shfl_down_sync(0xffffffffu, s, BS), t2 = __shfl_down_sync(0xffffffffu, s, 2 * BS);
    if (j == 0) s += t1 + t2;
  } else {
#pragma unroll
    for (int o = J / 2; o; o >>= 1) {
      const A t = __shfl_down_sync(0xffffffffu, s, BS * o);
      if (j < o) s += t;
    }
  }
  return s;
}

// out = A x over one group of the CTA's block rows [row0, re): BS * J lanes
// per block row, lane (j, c) adds component c of the row's entries j, j + J,
// ... in that order, then the J partial sums are combined; put(row, c, sum)
// by lanes j = 0; get(k, d): component d of x at a column.
template <int BS, int J, int U, class A, class R, class V, class C, class GET, class PUT>
__device__ __forceinline__ void local_group(int row0, int re, const R* rp, const V* val, const C* lc, GET&& get,
                                            PUT&& put) {
  constexpr int GL = BS * J, GPW = 32 / GL;
  const int lane = threadIdx.x & 31;
  const int g = lane / GL, l = lane - g * GL, j = l / BS, c = l - j * BS;
  const int row = row0 + g;
  const bool ok = g < GPW && row < re;
  const int k0 = ok ? (int)rp[row] + j : 0, e = ok ? (int)rp[row + 1] : 0;
  const int n = __reduce_max_sync(0xffffffffu, ok && e > k0 ? (e - k0 + J - 1) / J : 0);  // the warp's steps
  A s = (A)0;
  for (int t = 0; t < n; t += U) {
    int cj[U];
    A a[U][BS], xv[U][BS];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int kk = k0 + (t + u) * J;
      const bool in = kk < e;
      cj[u] = in ? (int)lc[kk] : 0;
#pragma unroll
      for (int d = 0; d < BS; d++) a[u][d] = in ? (A)val[(size_t)kk * (BS * BS) + c * BS + d] : (A)0;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int d = 0; d < BS; d++) xv[u][d] = k0 + (t + u) * J < e ? get(cj[u], d) : (A)0;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (t + u < n)  // the same in the whole warp: no FP64 instruction for nothing
#pragma unroll
        for (int d = 0; d < BS; d++) s = fma(a[u][d], xv[u][d], s);
  }
  __syncwarp();
  s = local_combine<BS, J>(s, j);
  if (ok && j == 0) put(row, c, s);
}

// One sweep over the CTA's ns slices, a lane per row, a warp taking its own
// number's slice, then the next one nobody took (*next); sp[i]: first entry of
// slice i (its steps' 32 entries are adjacent).  put(row, sum).  U steps are
// loaded at once: 4 of FP64, where the FP64 pipe is the limit (8 and 16: 6 and
// 13% slower), 16 of FP32 (8: 2% slower); loading ahead of the additions, also
// across slices, gained nothing over the other warps' loads in flight.
template <int U, class A, class V, class GET, class PUT>
__device__ __forceinline__ void local_slices(int ns, const int32_t* sp, const V* __restrict__ val, const uint16_t* lc,
                                             int* next, GET&& get, PUT&& put) {
  const int lane = threadIdx.x & 31;
  int si = threadIdx.x >> 5;
  while (si < ns) {
    const int o = sp[si] + lane, n = (sp[si + 1] - sp[si]) >> 5;
    A s = (A)0;
    V a[U];
    int c[U];
    auto load = [&](int t, V (&v)[U], int (&j)[U]) {
#pragma unroll
      for (int u = 0; u < U; u++)
        if (t + u < n) {
          v[u] = __ldcg(val + o + (t + u) * 32);
          j[u] = __ldcg(lc + o + (t + u) * 32);
        }
    };
    for (int t = 0; t < n; t += U) {
      load(t, a, c);
#pragma unroll
      for (int u = 0; u < U; u++)
        if (t + u < n) s = fma((A)a[u], get(c[u]), s);
    }
    put(si * 32 + lane, s);
    if (lane == 0) si = atomicAdd(next, 1);
    si = __shfl_sync(0xffffffffu, si, 0);
  }
}

// The CTA's row groups, the streamed rows [rsm, nr) first (their loads take
// longest), then the resident ones; a warp takes its own first group, then
// the next one nobody took (S.next, reset by local_total's callers).
template <int BS, int J, class F1, class F2>
__device__ __forceinline__ void local_sweep(int nr, int rsm, LShared& S, F1&& streamed, F2&& resident) {
  constexpr int GPW = 32 / (BS * J);
  const int lane = threadIdx.x & 31;
  const int n1 = (nr - rsm + GPW - 1) / GPW, n2 = (rsm + GPW - 1) / GPW;
  int gi = threadIdx.x >> 5;
  while (gi < n1 + n2) {
    if (gi < n1) streamed(rsm + gi * GPW);
    else resident((gi - n1) * GPW);
    if (n1 + n2 <= LNW) break;
    if (lane == 0) gi = atomicAdd(&S.next, 1);
    gi = __shfl_sync(0xffffffffu, gi, 0);
  }
}

// first row (slice) of CTA blk of nb: the rows are split at equal shares of
// cost(r) = per_entry x the entries before r + per_row x r.  Called by one
// warp (32 probes a step).
__device__ __forceinline__ int64_t local_first_row(const int64_t* __restrict__ rowptr, int64_t n, int nb, int blk,
                                                   int per_entry, int per_row) {
  const int lane = threadIdx.x & 31;
  if (blk <= 0) return 0;
  if (blk >= nb) return n;
  const int64_t total = __ldg(rowptr + n) * per_entry + n * per_row;
  const int64_t want = total / nb * blk + total % nb * blk / nb;
  int64_t lo = 0, hi = n;  // cost(lo) < want <= cost(hi)
  while (hi - lo > 1) {
    const int64_t step = (hi - lo + 32) / 33;
    const int64_t r = lo + step * (lane + 1);
    const bool ge = r >= hi || __ldg(rowptr + r) * per_entry + r * per_row >= want;
    const unsigned m = __ballot_sync(0xffffffffu, ge);
    const int f = m ? __ffs(m) - 1 : 32;
    const int64_t nlo = lo + step * f;
    hi = min(hi, lo + step * (f + 1));
    lo = nlo;
  }
  return hi;
}

// --- the vector updates and the iteration's scalars ---------------------------
// (shared with the kernel that does a cluster's arithmetic on one CTA: products
// and sums are contracted as written here)
template <class X>
__device__ __forceinline__ X times(X a, X b) {
  if constexpr (sizeof(X) == sizeof(double)) return __dmul_rn(a, b);
  else return __fmul_rn(a, b);
}
// r -= alpha q, xs += alpha p, z = Dinv r; v: r.z, r.r.  Returns z
template <class X>
__device__ __forceinline__ X cg_step(X alpha, X q, X p, X di, X& r, X& xs, X (&v)[2]) {
  r = fma(-alpha, q, r);
  const X z = times(di, r);
  xs = fma(alpha, p, xs);
  v[0] = fma(r, z, v[0]);
  v[1] = fma(r, r, v[1]);
  return z;
}
// a row's FP64 residual b - o -> r; v: r.z, ||r||^2, ||b||^2.  Returns z
template <class X>
__device__ __forceinline__ X cg_residual(double b, double o, X di, X& r, double (&v)[3]) {
  const double ri = b - o;
  const X rx = (X)ri, z = times(di, rx);
  r = rx;
  v[0] = fma((double)rx, (double)z, v[0]);
  v[1] = fma(ri, ri, v[1]);
  v[2] = fma(b, b, v[2]);
  return z;
}

// The iteration's scalars, by one thread, from the sums' totals.
// After the residual of the start's x (cont: the continuation of an FP32 run)
__device__ __forceinline__ void ctl_start(PState& T, const double* tot, const PRule& u, bool cont) {
  T.started = 1;
  T.rz = tot[0];
  T.rr = tot[1];
  T.rmax2 = T.rr;
  T.thr = u.delta2 * T.rmax2;
  T.beta = 0.0;
  if (cont) {
    T.it_upd = T.iters;
    T.max_cyc = 0;
    T.stall = 0;
  } else {
    T.bb = tot[2];
    T.tol2 = u.rtol2 * T.bb;
    T.rzold = 0.0;
    T.iters = 0;
    T.nupd = 0;
  }
  T.done = le_pos(T.rr, T.tol2);
}
// After a step: 1 when a reliable update is due, 5 when after a slow cycle
template <class X, bool RELIABLE>
__device__ __forceinline__ int ctl_step(PState& T, const double* tot, const PRule& u) {
  const double rr = tot[1];
  T.iters += 1;
  T.beta = quick_div(tot[0], T.rz);
  T.rzold = T.rz;
  T.rz = tot[0];
  T.rr = rr;
  const bool stop = le_pos(rr, T.tol2) || T.iters >= u.maxit || is_nan(rr);
  if constexpr (RELIABLE) {
    // an FP32 cycle (recurrence residual down by delta) that runs past 2.5x
    // the longest earlier cycle: the FP32 iteration has lost the rate of the
    // exact iteration (eps32 * cond(A) too large); hand over to FP64
    const int cyc = T.iters - T.it_upd;
    const bool slow =
        sizeof(X) < sizeof(double) && (cyc > kSlowCycle || (T.max_cyc > 0 && cyc > (5 * T.max_cyc) / 2 + 16));
    const bool upd = stop || slow || (sizeof(X) < sizeof(double) && le_pos(rr, T.thr));
    return upd ? (slow ? 5 : 1) : 0;
  } else {
    T.done = stop;
    return 0;
  }
}
// After a reliable update's residual
template <class X>
__device__ __forceinline__ void ctl_update(PState& T, const double* tot, const PRule& u, bool slow) {
  const double rzn = tot[0], rrn = tot[1];
  double beta = T.rzold != 0.0 ? rzn / T.rzold : 0.0;
  // the recurrence lost track of the true residual (an FP64 run past its
  // attainable accuracy, or FP32 drift): the next direction restarts from the
  // true residual instead of scaling the old one by the true/recurrence
  // mismatch
  if (rzn > (sizeof(X) == sizeof(double) ? kRestartRatio64 : kRestartRatio) * T.rz) beta = 0.0;
  const double prev = T.rmax2;
  const int cyc = T.iters - T.it_upd;
  T.rz = rzn;
  T.rr = rrn;
  T.rmax2 = rrn;
  T.thr = u.delta2 * rrn;
  T.nupd += 1;
  T.done = rrn <= T.tol2 || T.iters >= u.maxit || !(rrn == rrn);
  if (sizeof(X) == sizeof(double) && !T.done) {
    // FP64: true-residual checks that do not halve ||r||, kStagnation times
    // running -- the tolerance lies below the attainable accuracy
    // (eps64 * cond(A)); the solve ends, not converged
    T.stall = rrn > 0.25 * prev ? T.stall + 1 : 0;
    if (T.stall >= kStagnation) T.done = 1;
  }
  if (sizeof(X) < sizeof(double) && !T.done) {
    // the recurrence fell by delta but the true residual did not halve: the
    // FP32 operator no longer resolves the error (eps32 * cond ~ 1)
    T.stall = rrn > u.stall_ratio * prev ? T.stall + 1 : 0;
    if (T.stall >= u.stall_count || slow) T.done = 2;
  }
  if (cyc > T.max_cyc) T.max_cyc = cyc;
  T.it_upd = T.iters;
  T.beta = beta;
}

// Shared memory of a CTA's local set: its own vectors (n_own entries), p at its
// nloc local columns, their numbers (XL: and FP64 x at them) and nptr row (or
// slice) pointers; the bitmap and the resident part of the matrix come on top.
template <int BS, class X, bool XL, bool CL, bool SL>
__host__ __device__ inline size_t local_bytes(int n_own, int nloc, int nptr) {
  size_t off = ((size_t)n_own * (2 + CL + 2 * !SL) + (size_t)nloc * BS) * sizeof(X);
  off = (off + 7) & ~size_t(7);
  off += (size_t)nloc * ((XL ? BS * sizeof(double) : 0) + sizeof(int32_t) * (XL && CL ? 2 : 1));
  off += ((size_t)nptr + 1) * sizeof(int32_t);
  return (off + 15) & ~size_t(15);
}
__host__ __device__ inline int bitmap_bytes(int nwords) { return (nwords * 6 + 15) & ~15; }  // words + 16-bit prefixes

// The solve of one system by nb CTAs, this CTA being number blk of them;
// smem_bytes: the dynamic shared memory of the launch.
// Entry lanes per block row: every lane of a row costs a step of the
// combination, every entry beyond a multiple of them an idle lane, and fewer
// mean fewer FP64 instructions but longer runs.  Block rows of 3 take 5 (15
// lanes, two rows a warp), of 2 two; scalar rows 1 (FP64, means up to 20
// entries), 2 (up to 40) or 4.
template <int BS, class F>
__device__ __forceinline__ void with_lanes(int j, F&& f) {
  if constexpr (BS == 3) f(std::integral_constant<int, 5>());
  else if constexpr (BS == 2) f(std::integral_constant<int, 2>());
  else if (j == 1) f(std::integral_constant<int, 1>());
  else if (j == 2) f(std::integral_constant<int, 2>());
  else f(std::integral_constant<int, 4>());
}

template <int BS, class V, class X, bool RELIABLE, bool CL, bool SL>
__device__ __forceinline__ void pcg_local_body(const PArgs& a, int nb, int blk, int init, int it_end,
                                               unsigned char* smem, int smem_bytes, LShared& S, LCluster* C) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if constexpr (CL) {
    for (int i = wid; i <= nb; i += LNW) {
      const int64_t r = local_first_row(a.rowptr, a.nrows, nb, i, BS * BS, BS * row_cost(BS));
      if (lane == 0) {
        C->first[i] = r;
        if (i == blk) S.rows[0] = r;
        if (i == blk + 1) S.rows[1] = r;
      }
    }
  } else if (wid < 2) {
    const int64_t r = SL ? local_first_row(a.rowptr, (a.nrows + 31) / 32, nb, blk + wid, 1, 32 * kSliceRowCost)
                         : local_first_row(a.rowptr, a.nrows, nb, blk + wid, BS * BS, BS * row_cost(BS));
    if (lane == 0) S.rows[wid] = r;
  }
  if (tid == 0) {
    S.abort = 0;
    S.cmin = INT_MAX;
    S.cmax = 0;
    S.next = LNW;
    S.st = *a.st;
  }
  uint32_t epoch = a.st->epoch;
  if constexpr (CL) cluster_sync();  // every CTA of the cluster runs: its shared memory may be written
  else __syncthreads();
  // SL: the rows of slices [f0, f1), a.rowptr being the slices' pointers
  const int64_t f0 = S.rows[0], f1 = S.rows[1];
  const int64_t r0 = SL ? min(a.nrows, f0 * 32) : f0, r1 = SL ? min(a.nrows, f1 * 32) : f1;
  const int nr = (int)(r1 - r0);
  const int n_own = nr * BS;
  const int64_t e0 = r0 * BS;
  auto none = [](const double*) {};

  // --- shared memory: own vectors, local p and its columns, row pointers,
  // the resident part of the matrix; the bitmap and its prefix at the end
  X* s_z = reinterpret_cast<X*>(smem);  // CL only, at the same address in every CTA
  X* s_r = s_z + (CL ? n_own : 0);
  X* s_q = s_r + n_own;
  X* s_xs = s_q + n_own;
  X* s_di = s_xs + (SL ? 0 : n_own);
  X* s_p = s_di + (SL ? 0 : n_own);
  X* const w_xs = SL ? (X*)a.xs + e0 : s_xs;
  const X* const w_di = SL ? (const X*)a.dinv + e0 : s_di;
  const int64_t k0 = a.rowptr[f0];
  const int nk = (int)(a.rowptr[f1] - k0);
  // bitmap words [w0, w0 + nwords)
  int w0 = 0, nwords = (int)((a.nrows + 31) / 32);
  if constexpr (SL) {
    int lo = INT_MAX, hi = 0;
    for (int i = tid; i < nk; i += LT) {
      const int c = __ldg(a.colind + k0 + i);
      lo = min(lo, c);
      hi = max(hi, c);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
      atomicMin(&S.cmin, lo);
      atomicMax(&S.cmax, hi);
    }
    __syncthreads();
    lo = min(S.cmin, nr > 0 ? (int)r0 : INT_MAX);
    hi = max(S.cmax, (int)r1 - 1);
    w0 = nr > 0 ? lo >> 5 : 0;
    nwords = nr > 0 ? (hi >> 5) - w0 + 1 : 0;
  }
  const int tail = bitmap_bytes(nwords);
  // (a window beyond the shared memory: no columns are marked, and the local
  // set counts as not fitting below)
  const bool window = !SL || tail + 4096 <= smem_bytes;
  if (!window) nwords = 0;
  uint32_t* s_bit = reinterpret_cast<uint32_t*>(smem + smem_bytes - (window ? tail : 0));
  uint16_t* s_base = reinterpret_cast<uint16_t*>(s_bit + nwords);

  // --- the local columns
  for (int i = tid; i < nwords; i += LT) s_bit[i] = 0;
  __syncthreads();
  if (window) {
    for (int i = tid; i < nk; i += LT) {
      const int c = __ldg(a.colind + k0 + i);
      const uint32_t m = 1u << (c & 31);
      if (!(*(volatile uint32_t*)&s_bit[(c >> 5) - w0] & m)) atomicOr(&s_bit[(c >> 5) - w0], m);
    }
    for (int i = tid; i < nr; i += LT) {
      const int c = (int)r0 + i;
      atomicOr(&s_bit[(c >> 5) - w0], 1u << (c & 31));
    }
  }
  __syncthreads();
  {
    // exclusive prefix of the words' bit counts: a run of words per thread
    const int per = (nwords + LT - 1) / LT;
    const int v0 = min(nwords, tid * per), v1 = min(nwords, v0 + per);
    int t = 0;
    for (int i = v0; i < v1; i++) t += __popc(s_bit[i]);
    int inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += u;
    }
    if (lane == 31) S.wsum[wid] = inc;
    __syncthreads();
    int b = 0, all = 0;
    for (int i = 0; i < LNW; i++) {
      if (i < wid) b += S.wsum[i];
      all += S.wsum[i];
    }
    b += inc - t;
    for (int i = v0; i < v1; i++) {
      s_base[i] = (uint16_t)min(b, 65535);
      b += __popc(s_bit[i]);
    }
    if (tid == 0) S.nloc = all;
  }
  __syncthreads();
  const int nloc = S.nloc;
  // FP32 iteration: FP64 x at the local columns for the residuals, and (CL)
  // the columns' numbers
  constexpr bool XL = RELIABLE && sizeof(X) < sizeof(double);
  size_t off = reinterpret_cast<unsigned char*>(s_p + (size_t)nloc * BS) - smem;
  off = (off + 7) & ~size_t(7);
  double* s_x = reinterpret_cast<double*>(smem + off);
  int32_t* s_g = reinterpret_cast<int32_t*>(s_x + (XL ? (size_t)nloc * BS : 0));
  int32_t* s_gc = XL && CL ? s_g + nloc : s_g;
  int32_t* s_rp = s_gc + nloc;
  const size_t used = local_bytes<BS, X, XL, CL, SL>(n_own, nloc, (int)(f1 - f0));
  {
    const bool fits = window && nloc < 65535 && used + tail <= (size_t)smem_bytes;
    const float v[1] = {fits ? 0.0f : 1.0f};
    if (!local_total<1, CL>(v, 1, nb, blk, a.part, epoch, a.err, S, C,
                            [&](const double* tot) { S.overflow = __double_as_longlong(tot[0]) != 0; }))
      return;
    if (S.overflow) {  // the same in every CTA
      if (blk == 0 && tid == 0) {
        S.st.done = LOVERFLOW;
        S.st.epoch = epoch;
        *a.st = S.st;
      }
      if constexpr (CL) cluster_sync();
      return;
    }
  }
  for (int i = tid; i < nwords; i += LT) {
    uint32_t m = s_bit[i];
    int b = s_base[i], own = 0;
    while (m) {
      const int c = (w0 + i) * 32 + __ffs(m) - 1;
      if constexpr (CL) {
        // the column's z in its owner's shared memory
        while (c >= C->first[own + 1]) own++;
        if constexpr (XL) s_gc[b] = c;
        s_g[b++] = (int32_t)(cluster_addr(s_z, own) + (uint32_t)(c - C->first[own]) * (uint32_t)(BS * sizeof(X)));
      } else {
        s_g[b++] = c;
      }
      m &= m - 1;
    }
  }
  for (int i = tid; i <= (int)(f1 - f0); i += LT) s_rp[i] = (int)(a.rowptr[f0 + i] - k0);
  __syncthreads();
  const int ownb = nr > 0 ? s_base[(r0 >> 5) - w0] + __popc(s_bit[(r0 >> 5) - w0] & ((1u << (r0 & 31)) - 1u)) : 0;
  if (SL) {
    if (tid == 0) S.rsm = 0;
  } else if (tid == 0) {
    // the most rows whose entries fit
    const size_t avail = smem_bytes - tail - used;
    const int cap = (int)min((size_t)nk, avail / (sizeof(V) * BS * BS + sizeof(uint16_t)));
    int lo = 0, hi = nr;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s_rp[mid] <= cap) lo = mid;
      else hi = mid - 1;
    }
    // unless all fit, whole groups of rows (local_group) or, BS = 3, of the
    // warps' rounds over them: residual() goes from resident to other rows there
    if constexpr (XL)
      if (lo < nr)
        with_lanes<BS>(a.lanes, [&](auto jt) { lo -= lo % (32 / (BS * decltype(jt)::value) * (BS == 3 ? LNW : 1)); });
    S.rsm = lo;
  }
  __syncthreads();
  const int rsm = S.rsm, ksm = s_rp[rsm];
  V* s_val = reinterpret_cast<V*>(smem + used);
  uint16_t* s_lc = reinterpret_cast<uint16_t*>(s_val + (size_t)ksm * BS * BS);
  const V* gval = reinterpret_cast<const V*>(a.val) + (size_t)k0 * BS * BS;
  const int32_t* gcol = a.colind + k0;
  uint16_t* glc = a.lcol + k0;
  for (int i = tid; i < ksm * BS * BS; i += LT) s_val[i] = __ldg(gval + i);
  for (int i = tid; i < nk; i += LT) {
    const int c = __ldg(gcol + i);
    const uint16_t lc = (uint16_t)(s_base[(c >> 5) - w0] + __popc(s_bit[(c >> 5) - w0] & ((1u << (c & 31)) - 1u)));
    if (i < ksm) s_lc[i] = lc;
    else glc[i] = lc;  // read back by this CTA only, after the barriers below
  }
  const X* s_po = s_p + (size_t)ownb * BS;
  const int nl = nloc * BS;
  X* xs = (X*)a.xs;
  X* r = (X*)a.r;
  X* z = (X*)a.z;
  X* p = (X*)a.p;
  const X* dinv = (const X*)a.dinv;
  if constexpr (!SL)
    for (int i = tid; i < n_own; i += LT) s_di[i] = dinv[e0 + i];
  // one sweep over the CTA's slices with values v (SL): put(row, sum)
  auto slices = [&](auto* v, auto zero, auto&& get, auto&& put) {
    local_slices<sizeof(*v) == 8 ? 4 : 16, decltype(zero)>((int)(f1 - f0), s_rp, v, glc, &S.next, get,
                                                            [&](int row, auto t) {
                                                              if (row < nr) put(row, t);
                                                            });
  };

  // FP64 residual r = b - A x of the own rows -> s_r, z; v: r.z, ||r||^2, ||b||^2
  auto residual = [&](double (&v)[3]) {
    if constexpr (XL) {
      for (int i = tid; i < nl; i += LT) {
        const int b = i / BS;
        s_x[i] = __ldcg(a.x + (int64_t)s_gc[b] * BS + (i - b * BS));
      }
      __syncthreads();
    }
    auto get = [&](int c, int d) { return __ldcg(a.x + (int64_t)c * BS + d); };
    auto getl = [&](int c, int d) { return s_x[c * BS + d]; };
    auto put = [&](int row, int c, double o) {
      const int i = row * BS + c;
      X rx;
      const X zx = cg_residual(a.b[e0 + i], o, w_di[i], rx, v);
      s_r[i] = rx;
      if constexpr (CL) s_z[i] = zx;
      else __stcg(z + e0 + i, zx);
    };
    if constexpr (SL) {
      // (the rows' sums first: a thread's own rows follow its number alone)
      auto sq = [&](int row, double o) { a.resid[r0 + row] = o; };
      if constexpr (XL) slices(a.val64 + k0, 0.0, [&](int c) { return s_x[c]; }, sq);
      else if constexpr (RELIABLE) slices(a.val64 + k0, 0.0, [&](int c) { return __ldcg(a.x + s_g[c]); }, sq);
      else slices(gval, 0.0, [&](int c) { return __ldcg(a.x + s_g[c]); }, sq);
      __syncthreads();
      if (tid == 0) S.next = LNW;
      for (int i = tid; i < nr; i += LT) put(i, 0, a.resid[r0 + i]);
    } else
    // (a thread's rows follow its number alone, whatever part of the matrix is
    // resident: the sums are the same at any size of shared memory)
    with_lanes<BS>(a.lanes, [&](auto jt) {
      constexpr int J = decltype(jt)::value, GPW = 32 / (BS * J), U = BS == 1 ? 8 : 4;
      if constexpr (XL) {
        // (resident rows end between two of a warp's groups, or with the rows;
        // two loops: the compiler then reads s_lc as shared memory.  BS = 3: the
        // second starts at a round of 32 rows; going on from the first's last
        // row, the same rows, was up to 3.5% slower: 4^3 to 13^3 Q2 elasticity)
        const double* v64 = a.val64 + (size_t)k0 * BS * BS;
        int row0 = wid * GPW;
        for (; row0 < rsm; row0 += LNW * GPW) local_group<BS, J, U, double>(row0, rsm, s_rp, v64, s_lc, getl, put);
        if constexpr (BS == 3) row0 = rsm + wid * GPW;
        for (; row0 < nr; row0 += LNW * GPW) local_group<BS, J, U, double>(row0, nr, s_rp, v64, glc, getl, put);
      } else {
        const auto* v64 = [&] {
          if constexpr (RELIABLE) return a.val64 + (size_t)k0 * BS * BS;
          else return gval;
        }();
        for (int row0 = wid * GPW; row0 < nr; row0 += LNW * GPW)
          local_group<BS, J, U, double>(row0, nr, s_rp, v64, gcol, get, put);
      }
    });
  };
  auto finish_act = [&] {
    S.act = (S.st.done || S.st.iters >= it_end) ? 2 : 0;
  };

  __syncthreads();
  if (init) {
    // init 1: start from x; init 2: the continuation of a stalled FP32 run in
    // FP64 from its solution x (iteration count and ||b|| carry over), with
    // the directions restarted: the FP32 run's direction no longer fits the
    // true residual, and continuing it made the FP64 recurrence stagnate or
    // diverge at tolerances near the attainable accuracy (measured)
    double v[3] = {0.0, 0.0, 0.0};
    residual(v);
    for (int i = tid; i < n_own; i += LT) w_xs[i] = (X)0;
    for (int i = tid; i < nl; i += LT) s_p[i] = (X)0;
    if (!local_total<3, CL>(v, LT, nb, blk, a.part, epoch, a.err, S, C, [&](const double* tot) {
          ctl_start(S.st, tot, a, init == 2);
          S.beta = 0.0;
          finish_act();
        }))
      return;
  } else {
    for (int i = tid; i < n_own; i += LT) {
      s_r[i] = r[e0 + i];
      if constexpr (!SL) s_xs[i] = xs[e0 + i];
    }
    for (int i = tid; i < n_own; i += LT)
      if constexpr (CL) s_z[i] = s_di[i] * s_r[i];
    // p at the local columns: the words of the bitmap in order
    for (int i = tid; i < nwords; i += LT) {
      uint32_t m = s_bit[i];
      int b = s_base[i];
      while (m) {
        const int64_t c = (int64_t)(w0 + i) * 32 + __ffs(m) - 1;
        for (int d = 0; d < BS; d++) s_p[b * BS + d] = __ldcg(p + c * BS + d);
        b++;
        m &= m - 1;
      }
    }
    if constexpr (CL) cluster_sync();
    if (tid == 0) {
      S.beta = S.st.beta;
      finish_act();
    }
    __syncthreads();
  }

  while (!(S.act & 2)) {
    // P1: p = z + beta p on the local set, q = A p, p.q
    {
      const X bx = (X)S.beta;
      constexpr int U = 4;
      for (int i0 = tid; i0 < nl; i0 += U * LT) {
        X zv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int i = i0 + u * LT, b = i / BS;
          if constexpr (CL)
            zv[u] = i < nl ? cluster_load((uint32_t)s_g[b] + (uint32_t)((i - b * BS) * sizeof(X)), X()) : (X)0;
          else
            zv[u] = i < nl ? __ldcg(z + (int64_t)s_g[b] * BS + (i - b * BS)) : (X)0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int i = i0 + u * LT;
          if (i < nl) s_p[i] = fma(bx, s_p[i], zv[u]);
        }
      }
    }
    __syncthreads();
    {
      auto get = [&](int c, int d) { return s_p[c * BS + d]; };
      auto put = [&](int row, int c, X o) { s_q[row * BS + c] = o; };
      if constexpr (SL) slices(gval, (X)0, [&](int c) { return s_p[c]; }, [&](int row, X o) { s_q[row] = o; });
      else with_lanes<BS>(a.lanes, [&](auto jt) {
        constexpr int J = decltype(jt)::value;
        local_sweep<BS, J>(
            nr, rsm, S, [&](int row0) { local_group<BS, J, 4, X>(row0, nr, s_rp, gval, glc, get, put); },
            [&](int row0) { local_group<BS, J, 4, X>(row0, rsm, s_rp, s_val, s_lc, get, put); });
      });
      __syncthreads();
      X acc[1] = {(X)0};
      for (int i = tid; i < n_own; i += LT) acc[0] = fma(s_q[i], s_po[i], acc[0]);
      if (!local_total<1, CL>(acc, n_own, nb, blk, a.part, epoch, a.err, S, C, [&](const double* tot) {
            S.alpha = quick_div(S.st.rz, tot[0]);
            S.next = LNW;
          }))
        return;
    }
    // P2: xs += alpha p, r -= alpha q, z = Dinv r; r.z, r.r
    {
      const X alpha = (X)S.alpha;
      X v[2] = {(X)0, (X)0};
      constexpr int U = SL ? 4 : 1;
      for (int i0 = tid; i0 < n_own; i0 += U * LT) {
        X dv[U], xv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int i = i0 + u * LT;
          dv[u] = i < n_own ? w_di[i] : (X)0;
          xv[u] = i < n_own ? w_xs[i] : (X)0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int i = i0 + u * LT;
          if (i < n_own) {
            X ri = s_r[i];
            const X zi = cg_step(alpha, s_q[i], s_po[i], dv[u], ri, xv[u], v);
            w_xs[i] = xv[u];
            s_r[i] = ri;
            if constexpr (CL) s_z[i] = zi;
            else __stcg(z + e0 + i, zi);
          }
        }
      }
      if (!local_total<2, CL>(v, n_own, nb, blk, a.part, epoch, a.err, S, C, [&](const double* tot) {
            const int upd = ctl_step<X, RELIABLE>(S.st, tot, a);
            S.beta = S.st.beta;
            finish_act();
            if (upd) S.act = upd;
          }))
        return;
    }
    if constexpr (RELIABLE) {
      if (S.act & 1) {
        // x += xs; then the FP64 true residual replaces the recurrence's
        const bool slow = S.act & 4;
        for (int i = tid; i < n_own; i += LT) {
          a.x[e0 + i] += (double)w_xs[i];
          w_xs[i] = (X)0;
        }
        const float w[1] = {0.0f};
        if (!local_total<1, CL>(w, 1, nb, blk, a.part, epoch, a.err, S, C, none)) return;
        double v[3] = {0.0, 0.0, 0.0};
        residual(v);
        if (!local_total<3, CL>(v, LT, nb, blk, a.part, epoch, a.err, S, C, [&](const double* tot) {
              ctl_update<X>(S.st, tot, a, slow);
              S.beta = S.st.beta;
              finish_act();
            }))
          return;
      }
    }
  }
  if (!RELIABLE && S.st.done)
    for (int i = tid; i < n_own; i += LT) {
      a.x[e0 + i] += (double)w_xs[i];
      w_xs[i] = (X)0;
    }
  if (!S.st.done)
    for (int i = tid; i < n_own; i += LT) {
      r[e0 + i] = s_r[i];
      if constexpr (!SL) xs[e0 + i] = s_xs[i];
      p[e0 + i] = s_po[i];
    }
  if (blk == 0 && tid == 0) {
    S.st.epoch = epoch;
    *a.st = S.st;
  }
  if constexpr (CL) cluster_sync();  // no CTA leaves while another may still read its shared memory
}
