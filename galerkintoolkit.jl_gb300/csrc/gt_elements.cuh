// gt_elements.cuh -- element kernels of the scalar Laplacian that do without a
// quadrature loop over node pairs: sum factorisation on general hexahedra
// (Q1, Q2) and closed-form integrals on P2 tetrahedra.
//
// Both are bound by FP64 instructions (GB300: 2 FMAs a clock and SM), so they
// are written to need few of them.
//
// Included by gt_assembly.cu inside namespace gt.
#pragma once

// 1-D Gauss-Legendre points on (0, 1) with n = order + 1 points, their
// weights, and the 1-D Lagrange basis there ([point][node])
struct Line1D {
  double x[3], w[3], L[3][3], dL[3][3];
};
inline Line1D line_1d(int order) {
  Line1D t{};
  if (order == 1) {
    const double s = 0.5 / sqrt(3.0);
    t.x[0] = 0.5 - s;
    t.x[1] = 0.5 + s;
    t.w[0] = t.w[1] = 0.5;
  } else {
    const double s = 0.5 * sqrt(0.6);
    t.x[0] = 0.5 - s;
    t.x[1] = 0.5;
    t.x[2] = 0.5 + s;
    t.w[0] = t.w[2] = 5.0 / 18.0;
    t.w[1] = 8.0 / 18.0;
  }
  for (int q = 0; q <= order; q++) lagrange1d(order, t.x[q], t.L[q], t.dL[q]);
  return t;
}

// the contractions' arithmetic: FP64, FP32 or double-float
template <class C>
__device__ __forceinline__ C arith(double x) {
  if constexpr (std::is_same<C, dfl>::value) return df_from_double(x);
  else return (C)x;
}
__device__ __forceinline__ double mac(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mac(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ dfl mac(dfl a, dfl b, dfl c) { return df_add_sloppy(df_mul(a, b), c); }
template <class T, class C>
__device__ __forceinline__ T rounded(C x) {
  if constexpr (std::is_same<C, dfl>::value) return x.hi;  // the nearest FP32 number: |lo| <= ulp(hi) / 2
  else return (T)x;
}

// Scalar Laplacian on hexahedra with a trilinear map, order M - 1, CPB cells
// per CTA.  With J the Jacobian at a point, the quadrature sum of the
// reference (src/compiler.jl:1865-1917 with src/accessors.jl:1365-1373 and
// dV = |det J| w, src/quadrature.jl:4-6) is
//
//   K_ab = sum_q sum_kl D^kl_q (d_k phi_a)(q) (d_l phi_b)(q),
//   D = coef w |det J| J^-1 J^-T = (coef w / |det J|) adj(J) adj(J)^T
//
// with phi a product of 1-D functions, so the sum over q is taken one
// direction at a time (a = (a1, a2, a3), i = (a2, a3), j = (b2, b3); LL, LD,
// DL, DD: products of the 1-D functions or derivatives of a and b at a point):
//
//   U^kl(q1 q2; a3 b3)  = sum_q3 D^kl F3        F3: DD for 33, LD for 13, 23, else LL
//   X(q1; i j) = sum_q2 LL U33 + DD U22 + LD' ...   the terms without direction 1
//   Y(q1; i j) = sum_q2 LD U12 + LL U13             k = 1, l = 2, 3
//   Z(q1; i j) = sum_q2 LL U11
//   K_ab = sum_q1 LL X(i j) + DD Z(i j) + DL Y(i j) + LD Y(j i)
//
// 11,900 FMAs per Q2 cell instead of the 50,000 of the loop over node pairs
// and points (k_elements), and the Jacobian comes from the eight coefficients
// of the trilinear map (27 FMAs a point instead of 72), which also rounds
// less: against extended precision the 2-norm error of assembled Q1 matrices
// is 1.3e-16 (2.8e-16 before), of Q2 ones 2.6e-16 (3.3e-16).  Measured: 23^3
// Q2 cells FP64 1262 -> 290 us, 25^3 Q1 cells FP64 79 -> 58 us.  FP32 values of
// Q1 cells are contracted in double-float numbers and rounded once: 53 -> 42 us
// at a 2-norm error of 4.6e-8 (the loop's gradients in FP64: 5.5e-8; three FP32
// contractions take 34 us at 9.8e-8).
template <int M>
struct HexSize {
  static constexpr int NP = M * M, NN = M * M * M, NPAIR = NN * (NN + 1) / 2, XP = NP * (NP + 1) / 2;
};
//
// FORM: GT_LAPLACE, GT_MASS (D^00 = coef w |det J| alone, LL in every
// direction) or 0, the element vector without a matrix; T: the matrix's values,
// C: the contractions' arithmetic.  The vector is the same in all of them, so
// assemble_vector is bitwise that of assemble_matrix_and_vector.
template <int M, class T, class C, int CPB, int FORM>
__global__ void __launch_bounds__(256) k_elements_hex(const double* __restrict__ coords,
                                                      const int32_t* __restrict__ cell_nodes,
                                                      const double* __restrict__ coef, Line1D line, int64_t ncells,
                                                      T* __restrict__ Ke, double* __restrict__ be,
                                                      const double* __restrict__ fsrc,
                                                      const double* __restrict__ scoef, uint32_t* err) {
  constexpr int NP = HexSize<M>::NP, NN = HexSize<M>::NN, NPAIR = HexSize<M>::NPAIR, XP = HexSize<M>::XP;
  constexpr int TH = 256;
  constexpr bool LAP = FORM == GT_LAPLACE, MAT = FORM != 0;
  constexpr int ND = LAP ? 6 : 1, CM = MAT ? CPB : 1, CL = LAP ? CPB : 1;
  __shared__ double s_c[CPB][3][8];      // coefficients of the map: 1, x, y, xy, z, xz, yz, xyz
  __shared__ double s_dv[CPB][NN];       // |det J| w
  __shared__ double s_v[2][CPB][NN];     // partial contractions of the element vector
  __shared__ C s_D[CM][ND][NN];          // 11, 22, 33, 12, 13, 23 (or 00) at the points
  __shared__ C s_U[CM][ND][NP][NP];      // [kl][q1 q2][a3 b3]
  __shared__ C s_X[CM][M][NP][NP], s_Y[CL][M][NP][NP], s_Z[CL][M][NP][NP];
  __shared__ C s_LL[M][M][M], s_LD[M][M][M], s_DD[M][M][M];  // [q][a][b]
  __shared__ double s_L[M][M];           // [q][a]
  __shared__ uint16_t s_pair[NPAIR], s_xpair[XP];
  const int tid = threadIdx.x;
  const int64_t c0 = (int64_t)blockIdx.x * CPB;
  for (int i = tid; i < M * M * M; i += TH) {
    const int q = i / (M * M), a = i / M % M, b = i % M;
    (&s_LL[0][0][0])[i] = arith<C>(line.L[q][a] * line.L[q][b]);
    (&s_LD[0][0][0])[i] = arith<C>(line.L[q][a] * line.dL[q][b]);
    (&s_DD[0][0][0])[i] = arith<C>(line.dL[q][a] * line.dL[q][b]);
    if (b == 0) s_L[q][a] = line.L[q][a];
  }
  for (int n = tid; n < NN; n += TH) {
    const int o = n * NN - n * (n - 1) / 2;
    for (int m = n; m < NN; m++) s_pair[o + m - n] = (uint16_t)(n * 32 + m);
  }
  for (int n = tid; n < NP; n += TH) {
    const int o = n * NP - n * (n - 1) / 2;
    for (int m = n; m < NP; m++) s_xpair[o + m - n] = (uint16_t)(n * 32 + m);
  }
  // the map's coefficients: for corner set k, the alternating sum of the
  // corners inside k (differences of nearby coordinates)
  for (int i = tid; i < CPB * 24; i += TH) {
    const int cl = i / 24, d = i % 3, k = i / 3 % 8;
    const int64_t c = min(c0 + cl, ncells - 1);
    double s = 0.0;
    const int32_t* cn = cell_nodes + c * 8;
    auto X = [&](int n) { return coords[(int64_t)cn[n] * 3 + d]; };
    if (k == 0) s = X(0);
    else if (k == 1 || k == 2 || k == 4) s = X(k) - X(0);
    else if (k == 7) s = ((X(7) - X(6)) - (X(5) - X(4))) - ((X(3) - X(2)) - (X(1) - X(0)));
    else {
      const int lo = k & -k, hi = k - lo;
      s = (X(k) - X(hi)) - (X(lo) - X(0));
    }
    s_c[cl][d][k] = s;
  }
  __syncthreads();
  // the points: D and dV
  for (int it = tid; it < CPB * NN; it += TH) {
    const int cl = it / NN, q = it - cl * NN, q1 = q % M, q2 = q / M % M, q3 = q / (M * M);
    const int64_t c = c0 + cl;
    const double x = line.x[q1], y = line.x[q2], z = line.x[q3];
    double J[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double* k = s_c[cl][i];
      const double xz = fma(k[7], y, k[5]), yx = fma(k[7], x, k[6]);
      J[i][0] = fma(xz, z, fma(k[3], y, k[1]));
      J[i][1] = fma(yx, z, fma(k[3], x, k[2]));
      J[i][2] = fma(yx, y, fma(k[5], x, k[4]));
    }
    // rows of adj(J) = det J J^-1 (contracted as written, in every form)
    auto cof = [&](int i, int j, int k, int l) { return fma(J[i][j], J[k][l], -__dmul_rn(J[i][l], J[k][j])); };
    double A[3][3];
    A[0][0] = cof(1, 1, 2, 2);
    A[1][0] = cof(1, 2, 2, 0);
    A[2][0] = cof(1, 0, 2, 1);
    const double det = fma(J[0][2], A[2][0], fma(J[0][1], A[1][0], __dmul_rn(J[0][0], A[0][0])));
    if (c < ncells && !(det != 0.0)) atomicOr(err, DEV_ERR_DEGENERATE);
    const double w = line.w[q1] * line.w[q2] * line.w[q3], adet = fabs(det);
    s_dv[cl][q] = (double)(T)__dmul_rn(adet, w);  // |det J| w is held in T, also for the element vector
    if constexpr (MAT) {
      const double cw = (coef && c < ncells ? coef[c] : 1.0) * w;
      if constexpr (!LAP) {
        s_D[cl][0][q] = arith<C>(cw * adet);
      } else {
        A[0][1] = cof(0, 2, 2, 1);
        A[1][1] = cof(0, 0, 2, 2);
        A[2][1] = cof(0, 1, 2, 0);
        A[0][2] = cof(0, 1, 1, 2);
        A[1][2] = cof(0, 2, 1, 0);
        A[2][2] = cof(0, 0, 1, 1);
        const double cf = cw * recip_nr2(adet);
        auto dot = [&](int k, int l) { return cf * (A[k][0] * A[l][0] + A[k][1] * A[l][1] + A[k][2] * A[l][2]); };
        s_D[cl][0][q] = arith<C>(dot(0, 0));
        s_D[cl][1][q] = arith<C>(dot(1, 1));
        s_D[cl][2][q] = arith<C>(dot(2, 2));
        s_D[cl][3][q] = arith<C>(dot(0, 1));
        s_D[cl][4][q] = arith<C>(dot(0, 2));
        s_D[cl][5][q] = arith<C>(dot(1, 2));
      }
    }
  }
  __syncthreads();
  // contraction over q3 (with the element vector's: NN items a cell)
  const int nv = be ? CPB * NN : 0;
  if constexpr (MAT)
    for (int it = tid; it < CPB * NP * NP; it += TH) {
      const int cl = it / (NP * NP), r = it - cl * (NP * NP), q12 = r / NP, ab = r - q12 * NP, a = ab / M, b = ab % M;
      C u[ND];
#pragma unroll
      for (int k = 0; k < ND; k++) u[k] = C{};
#pragma unroll
      for (int q = 0; q < M; q++) {
        const C ll = s_LL[q][a][b];
        const int p = q * NP + q12;
        u[0] = mac(ll, s_D[cl][0][p], u[0]);
        if constexpr (LAP) {
          const C ld = s_LD[q][a][b], dd = s_DD[q][a][b];
          u[1] = mac(ll, s_D[cl][1][p], u[1]);
          u[2] = mac(dd, s_D[cl][2][p], u[2]);
          u[3] = mac(ll, s_D[cl][3][p], u[3]);
          u[4] = mac(ld, s_D[cl][4][p], u[4]);
          u[5] = mac(ld, s_D[cl][5][p], u[5]);
        }
      }
#pragma unroll
      for (int k = 0; k < ND; k++) s_U[cl][k][q12][ab] = u[k];
    }
  for (int it = tid; it < nv; it += TH) {
    const int cl = it / NN, r = it - cl * NN, q12 = r % NP, a = r / NP;
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < M; q++) s = fma(s_L[q][a], s_dv[cl][q * NP + q12], s);
    s_v[0][cl][r] = s;  // [a3][q2][q1]
  }
  __syncthreads();
  // contraction over q2: X by its pairs i <= j, then Y and Z
  if constexpr (MAT)
    for (int it = tid; it < CPB * M * (XP + (LAP ? NP * NP : 0)); it += TH) {
      if (it < CPB * M * XP) {
        const int cl = it / (M * XP), r = it - cl * (M * XP), q1 = r / XP, p = s_xpair[r - q1 * XP];
        const int i = p >> 5, j = p & 31, a2 = i % M, a3 = i / M, b2 = j % M, b3 = j / M;
        C s{};
#pragma unroll
        for (int q = 0; q < M; q++) {
          const int q12 = q * M + q1;
          s = mac(s_LL[q][a2][b2], s_U[cl][LAP ? 2 : 0][q12][a3 * M + b3], s);
          if constexpr (LAP) {
            s = mac(s_DD[q][a2][b2], s_U[cl][1][q12][a3 * M + b3], s);
            s = mac(s_LD[q][b2][a2], s_U[cl][5][q12][a3 * M + b3], s);  // k = 2, l = 3
            s = mac(s_LD[q][a2][b2], s_U[cl][5][q12][b3 * M + a3], s);  // k = 3, l = 2
          }
        }
        s_X[cl][q1][i][j] = s;
        s_X[cl][q1][j][i] = s;
      } else if constexpr (LAP) {
        const int t = it - CPB * M * XP;
        const int cl = t / (M * NP * NP), r = t - cl * (M * NP * NP), q1 = r / (NP * NP), ij = r - q1 * (NP * NP);
        const int i = ij / NP, j = ij - i * NP, a2 = i % M, a3 = i / M, b2 = j % M, b3 = j / M;
        C y{}, z{};
#pragma unroll
        for (int q = 0; q < M; q++) {
          const int q12 = q * M + q1;
          const C ll = s_LL[q][a2][b2];
          z = mac(ll, s_U[cl][0][q12][a3 * M + b3], z);
          y = mac(s_LD[q][a2][b2], s_U[cl][3][q12][a3 * M + b3], y);
          y = mac(ll, s_U[cl][4][q12][a3 * M + b3], y);
        }
        s_Y[cl][q1][i][j] = y;
        s_Z[cl][q1][i][j] = z;
      }
    }
  for (int it = tid; it < nv; it += TH) {
    const int cl = it / NN, r = it - cl * NN, q1 = r % M, a2 = r / M % M, a3 = r / NP;
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < M; q++) s = fma(s_L[q][a2], s_v[0][cl][a3 * NP + q * M + q1], s);
    s_v[1][cl][r] = s;  // [a3][a2][q1]
  }
  __syncthreads();
  // contraction over q1: the node pairs n <= m
  if constexpr (MAT)
    for (int it = tid; it < CPB * NPAIR; it += TH) {
      const int cl = it / NPAIR, p = s_pair[it - cl * NPAIR];
      const int64_t c = c0 + cl;
      const int n = p >> 5, m = p & 31, a1 = n % M, i = n / M, b1 = m % M, j = m / M;
      C s{};
#pragma unroll
      for (int q = 0; q < M; q++) {
        s = mac(s_LL[q][a1][b1], s_X[cl][q][i][j], s);
        if constexpr (LAP) {
          s = mac(s_DD[q][a1][b1], s_Z[cl][q][i][j], s);
          s = mac(s_LD[q][b1][a1], s_Y[cl][q][i][j], s);
          s = mac(s_LD[q][a1][b1], s_Y[cl][q][j][i], s);
        }
      }
      if (c < ncells) {
        T* K = Ke + c * (NN * NN);
        K[n * NN + m] = K[m * NN + n] = rounded<T>(s);
      }
    }
  for (int it = tid; it < nv; it += TH) {
    const int cl = it / NN, n = it - cl * NN, a1 = n % M;
    const int64_t c = c0 + cl;
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < M; q++) s = fma(s_L[q][a1], s_v[1][cl][n - a1 + q], s);
    if (c < ncells) be[c * NN + n] = (scoef ? scoef[c] : 1.0) * fsrc[0] * s;
  }
}

// Scalar Laplacian on P2 tetrahedra, one thread per cell.  The map is affine,
// so with S_ij = |det J| coef grad l_i . grad l_j (barycentric coordinates l)
// the element matrix is a sum of S entries times exact integrals of l_a l_b
// (1/60 for a = b, 1/120 else, 1/24 of l_a, 1/6 of 1) -- the degree-2
// integrands the reference's degree-4 rule integrates exactly.  With shape
// functions l_i (2 l_i - 1) and 4 l_a l_b and S scaled by 1/30:
//
//   vertex i, vertex j      3 S_ii (i = j), -S_ij
//   vertex i, edge ab       (i = b ? 3 : -1) S_ia + (i = a ? 3 : -1) S_ib
//   edge ab, edge cd        4 [(1 + d_bd) S_ac + (1 + d_bc) S_ad + (1 + d_ad) S_bc + (1 + d_ac) S_bd]
//
// about 230 FP64 instructions per warp of 32 cells instead of 4,200 per cell
// of the loop over points.  The block goes through shared memory (rows of 101
// entries: conflict-free for a thread per row) to coalesced stores.  Measured,
// 21^3 x 6 cells FP64: 445 -> 43 us.
template <class T>
__global__ void __launch_bounds__(128) k_elements_p2(const double* __restrict__ coords,
                                                     const int32_t* __restrict__ cell_nodes,
                                                     const double* __restrict__ coef, int64_t ncells,
                                                     T* __restrict__ Ke, double* __restrict__ be,
                                                     const double* __restrict__ fsrc,
                                                     const double* __restrict__ scoef, int want_matrix, uint32_t* err) {
  constexpr int ROW = 101;
  extern __shared__ __align__(16) unsigned char s_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T* sk = reinterpret_cast<T*>(s_raw) + (size_t)w * 32 * ROW + lane * ROW;
  const int64_t c0 = (int64_t)blockIdx.x * 128 + w * 32, c = c0 + lane;
  if (c0 >= ncells) return;
  const int64_t cc = c < ncells ? c : ncells - 1;
  const int4 nd = __ldg(reinterpret_cast<const int4*>(cell_nodes) + cc);
  double x0[3], J[3][3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    x0[d] = coords[(int64_t)nd.x * 3 + d];
    J[d][0] = coords[(int64_t)nd.y * 3 + d] - x0[d];
    J[d][1] = coords[(int64_t)nd.z * 3 + d] - x0[d];
    J[d][2] = coords[(int64_t)nd.w * 3 + d] - x0[d];
  }
  // det J grad l_i: rows of adj(J), grad l_0 = -(sum)
  double G[4][3];
  G[1][0] = J[1][1] * J[2][2] - J[1][2] * J[2][1];
  G[2][0] = J[1][2] * J[2][0] - J[1][0] * J[2][2];
  G[3][0] = J[1][0] * J[2][1] - J[1][1] * J[2][0];
  G[1][1] = J[0][2] * J[2][1] - J[0][1] * J[2][2];
  G[2][1] = J[0][0] * J[2][2] - J[0][2] * J[2][0];
  G[3][1] = J[0][1] * J[2][0] - J[0][0] * J[2][1];
  G[1][2] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
  G[2][2] = J[0][2] * J[1][0] - J[0][0] * J[1][2];
  G[3][2] = J[0][0] * J[1][1] - J[0][1] * J[1][0];
#pragma unroll
  for (int d = 0; d < 3; d++) G[0][d] = -(G[1][d] + G[2][d] + G[3][d]);
  const double det = J[0][0] * G[1][0] + J[0][1] * G[2][0] + J[0][2] * G[3][0];
  if (c < ncells && !(det != 0.0)) atomicOr(err, DEV_ERR_DEGENERATE);
  const double adet = fabs(det);
  constexpr int V[4] = {0, 2, 5, 9};                                        // node of vertex i
  constexpr int EA[6] = {0, 0, 1, 0, 1, 2}, EB[6] = {1, 2, 2, 3, 3, 3};     // edges
  constexpr int EN[6] = {1, 3, 4, 6, 7, 8};                                 // their nodes
  if (want_matrix) {
    const double cf = (coef ? coef[cc] : 1.0) * recip_nr2(adet) * (1.0 / 30.0);
    T S[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = i; j < 4; j++)
        S[i][j] = S[j][i] = (T)(cf * (G[i][0] * G[j][0] + G[i][1] * G[j][1] + G[i][2] * G[j][2]));
    auto put = [&](int n, int m, T v) {
      sk[n * 10 + m] = v;
      if (n != m) sk[m * 10 + n] = v;
    };
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = i; j < 4; j++) put(V[i], V[j], i == j ? (T)3 * S[i][i] : -S[i][j]);
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int e = 0; e < 6; e++) {
        const int a = EA[e], b = EB[e];
        const T v = i == b ? (T)3 * S[i][a] - S[i][b] : (i == a ? (T)3 * S[i][b] - S[i][a] : -S[i][a] - S[i][b]);
        put(V[i], EN[e], v);
      }
#pragma unroll
    for (int e = 0; e < 6; e++)
#pragma unroll
      for (int f = e; f < 6; f++) {
        const int a = EA[e], b = EB[e], p = EA[f], q = EB[f];
        auto t = [&](bool twice, T s) { return twice ? s + s : s; };
        const T v = (t(b == q, S[a][p]) + t(b == p, S[a][q])) + (t(a == q, S[b][p]) + t(a == p, S[b][q]));
        put(EN[e], EN[f], (T)4 * v);
      }
    __syncwarp();
    const T* sw = reinterpret_cast<const T*>(s_raw) + (size_t)w * 32 * ROW;
    const int nc = (int)min((int64_t)32, ncells - c0);
    T* K = Ke + c0 * 100;
    for (int i = lane; i < nc * 100; i += 32) {
      const int r = i / 100;
      K[i] = sw[r * ROW + i - r * 100];
    }
  }
  if (be && c < ncells) {
    // integrals of the shape functions: -1/120 (vertex), 1/30 (edge).  FP32
    // matrices hold |det J| w at the points of the 11-point rule in FP32, as
    // k_elements does: with its three weights the sums over the points are
    // those of the shape functions over the rule's three orbits
    const double cf = (scoef ? scoef[c] : 1.0) * fsrc[0];
    double s, sv;
    if constexpr (sizeof(T) == 4) {
      const double d0 = (double)(T)(adet * (-74.0 / 5625.0)), d1 = (double)(T)(adet * (343.0 / 45000.0)),
                   d2 = (double)(T)(adet * (56.0 / 2250.0));
      s = cf * (0.25 * d0 + (24.0 / 49.0) * d1 + (37.0 / 28.0) * d2);
      sv = cf * (-0.125 * d0 + (13.0 / 49.0) * d1 - (27.0 / 56.0) * d2);
    } else {
      s = adet * cf * (1.0 / 30.0);
      sv = -0.25 * s;
    }
    double* b = be + c * 10;
#pragma unroll
    for (int i = 0; i < 4; i++) b[V[i]] = sv;
#pragma unroll
    for (int e = 0; e < 6; e++) b[EN[e]] = s;
  }
}
