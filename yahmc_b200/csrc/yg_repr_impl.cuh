// Device code of the representation map and of the clover-term build (included by the
// yg_inst_*_aux.cu units).
//
//   represent_links          repr.cpp:107-263     fund N x N -> fermion-representation D x D
//   AP sign                  bcs.cpp:264-272      U_0(t=0) *= -1 on the represented links
//   clover_repr              wilsonloop.cpp:5-31  four plaquette leaves, each represented
//   _compute_clover_term     clover.cpp:120-168   the blocks A0..A3 with coefficient -csw/16
//   _bcs_clover_term         clover.cpp:93-118    open / SF boundary slices zeroed
#pragma once

#include "yg_kernels.h"

namespace yg {

template <int N>
__device__ __forceinline__ void rk_load(double2 (&m)[N * N], const double2 *base, const Geom &g, int id, int mu) {
#pragma unroll
  for (int k = 0; k < N * N; k++) m[k] = base[fidx(g, id, mu * N * N + k, 4 * N * N)];
}

// X = the link (id, mu) or its dagger
template <int N, bool DAG>
__device__ __forceinline__ void rk_start(double2 (&X)[N * N], const double2 *base, const Geom &g, int id, int mu) {
  double2 m[N * N];
  rk_load<N>(m, base, g, id, mu);
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) X[i * N + j] = DAG ? cconj(m[j * N + i]) : m[i * N + j];
}

// X <- U X (DAG: U^dag X) for the link U = (id, mu), in place column by column
template <int N, bool DAG>
__device__ __forceinline__ void rk_lmul(double2 (&X)[N * N], const double2 *base, const Geom &g, int id, int mu) {
  double2 m[N * N];
  asm volatile("" ::: "memory");     // the loads of a chain stay in order: hoisting them all costs spills
  rk_load<N>(m, base, g, id, mu);
#pragma unroll
  for (int j = 0; j < N; j++) {
    double2 v[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
      double2 t = make_double2(0, 0);
#pragma unroll
      for (int k = 0; k < N; k++) {
        if (DAG) cfmac(t, m[k * N + i], X[k * N + j]);
        else cfma(t, m[i * N + k], X[k * N + j]);
      }
      v[i] = t;
    }
#pragma unroll
    for (int i = 0; i < N; i++) X[i * N + j] = v[i];
  }
}

// Representation map of one fundamental matrix.  Fundamental: copy.  Otherwise
// R_nm = tr(b_n^dag U b_m W) with W = U^T (two-index representations, U acting as
// S -> U S U^T) or W = U^dag (adjoint, X -> U X U^dag), in the orthonormal basis b of
// repr.cpp:25-59; this is the map the explicit formulas of repr.cpp:114-259 evaluate.
// The adjoint map is real and its imaginary part is set to zero, as in the reference.
template <int NC, int D>
__device__ void represent_one(double2 (&r)[D * D], const double2 (&u)[NC * NC], const double2 *basis, int rep) {
  if (rep == YG_REPR_FUNDAMENTAL) {
#pragma unroll
    for (int k = 0; k < D * D; k++) r[k] = (k < NC * NC) ? u[k] : make_double2(0, 0);
    return;
  }
#pragma unroll 1
  for (int m = 0; m < D; m++) {
    double2 ub[NC * NC];                      // U b_m
#pragma unroll
    for (int i = 0; i < NC; i++)
#pragma unroll
      for (int j = 0; j < NC; j++) {
        double2 s = make_double2(0, 0);
#pragma unroll
        for (int k = 0; k < NC; k++) cfma(s, u[i * NC + k], basis[m * NC * NC + k * NC + j]);
        ub[i * NC + j] = s;
      }
#pragma unroll 1
    for (int n = 0; n < D; n++) {
      double2 tr = make_double2(0, 0);
#pragma unroll
      for (int a = 0; a < NC; a++)
#pragma unroll
        for (int b = 0; b < NC; b++) {
          double2 bn = basis[n * NC * NC + a * NC + b];
          if (bn.x == 0.0 && bn.y == 0.0) continue;
          double2 x = make_double2(0, 0);     // (U b_m W)[a][b]
#pragma unroll
          for (int k = 0; k < NC; k++) {
            double2 w = (rep == YG_REPR_ADJOINT) ? cconj(u[b * NC + k]) : u[b * NC + k];
            cfma(x, ub[a * NC + k], w);
          }
          cfmac(tr, bn, x);
        }
      if (rep == YG_REPR_ADJOINT) tr.y = 0.0;
      r[n * D + m] = tr;
    }
  }
}

// REAL: also the real parts alone (adjoint representations).  A kernel of its own: with a test of the
// pointer in the loop the stores of every representation were no longer unrolled (d = 3 16^4: 20.4 us, 13.8
// without it).
template <int NC, int D, bool REAL>
__global__ void k_represent(double2 *links, double *real, const double2 *fund, Geom g, const double2 *basis, int rep) {
  long r = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (r >= 4L * g.V) return;
  int id = (int)(r >> 2), mu = (int)(r & 3);
  double2 u[NC * NC];
  rk_load<NC>(u, fund, g, id, mu);
  double2 R[D * D];
  represent_one<NC, D>(R, u, basis, rep);
  int c[4];
  coords_of(g, id, c);
  double sgn = (g.bc == YG_BC_ANTIPERIODIC && mu == 0 && c[0] == 0) ? -1.0 : 1.0;   // bcs.cpp:264-272
  for (int k = 0; k < D * D; k++) {
    const long ix = fidx(g, id, mu * D * D + k, 4 * D * D);
    links[ix] = cscale(R[k], sgn);
    if (REAL) real[ix] = sgn * R[k].x;
  }
}

// clover_repr(id,mu,nu) (wilsonloop.cpp:5-31) in the fermion representation: each leaf is a chain
// of left multiplications
template <int NC, int D>
__device__ __forceinline__ void clover_leaves(double2 (&out)[D * D], const double2 *fund, const Geom &g, const int c[4],
                                              int id, int mu, int nu, const double2 *basis, int rep) {
  _Pragma(YG_STR(unroll (D <= 4 ? 64 : 8)))
  for (int k = 0; k < D * D; k++) out[k] = make_double2(0, 0);
  int cc[4];
  const int fm = neighbour(g, c, mu, +1), fn = neighbour(g, c, nu, +1);
  const int bm = neighbour(g, c, mu, -1), bn = neighbour(g, c, nu, -1);
  coords_of(g, bm, cc);
  const int bmfn = neighbour(g, cc, nu, +1), bmbn = neighbour(g, cc, nu, -1);
  coords_of(g, fm, cc);
  const int fmbn = neighbour(g, cc, nu, -1);
#pragma unroll 1
  for (int leaf = 0; leaf < 4; leaf++) {
    double2 X[NC * NC];
    if (leaf == 0) {         // U(x,mu) U(x+mu,nu) [U(x,nu) U(x+nu,mu)]^dag
      rk_start<NC, true>(X, fund, g, id, nu);
      rk_lmul<NC, true>(X, fund, g, fn, mu);
      rk_lmul<NC, false>(X, fund, g, fm, nu);
      rk_lmul<NC, false>(X, fund, g, id, mu);
    } else if (leaf == 1) {  // U(x,nu) [U(x-mu,nu) U(x-mu+nu,mu)]^dag U(x-mu,mu)
      rk_start<NC, false>(X, fund, g, bm, mu);
      rk_lmul<NC, true>(X, fund, g, bm, nu);
      rk_lmul<NC, true>(X, fund, g, bmfn, mu);
      rk_lmul<NC, false>(X, fund, g, id, nu);
    } else if (leaf == 2) {  // [U(x-mu-nu,nu) U(x-mu,mu)]^dag U(x-mu-nu,mu) U(x-nu,nu)
      rk_start<NC, false>(X, fund, g, bn, nu);
      rk_lmul<NC, false>(X, fund, g, bmbn, mu);
      rk_lmul<NC, true>(X, fund, g, bmbn, nu);
      rk_lmul<NC, true>(X, fund, g, bm, mu);
    } else {                 // U(x-nu,nu)^dag U(x-nu,mu) U(x-nu+mu,nu) U(x,mu)^dag
      rk_start<NC, true>(X, fund, g, id, mu);
      rk_lmul<NC, false>(X, fund, g, fmbn, nu);
      rk_lmul<NC, false>(X, fund, g, bn, mu);
      rk_lmul<NC, true>(X, fund, g, bn, nu);
    }
    if (NC == D && rep == YG_REPR_FUNDAMENTAL) {
#pragma unroll
      for (int k = 0; k < NC * NC; k++) out[k < D * D ? k : 0] = cadd(out[k < D * D ? k : 0], X[k]);
    } else {
      double2 R[D * D];
      represent_one<NC, D>(R, X, basis, rep);
      _Pragma(YG_STR(unroll (D <= 4 ? 64 : 8)))
      for (int k = 0; k < D * D; k++) out[k] = cadd(out[k], R[k]);
    }
  }
}

template <int N>
__device__ __forceinline__ void rk_mm(double2 (&c)[N * N], const double2 (&a)[N * N], const double2 (&b)[N * N]) {
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) {
      double2 s = make_double2(0, 0);
#pragma unroll
      for (int k = 0; k < N; k++) cfma(s, a[i * N + k], b[k * N + j]);
      c[i * N + j] = s;
    }
}

// c = a b^dag
template <int N>
__device__ __forceinline__ void rk_mmd(double2 (&c)[N * N], const double2 (&a)[N * N], const double2 (&b)[N * N]) {
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) {
      double2 s = make_double2(0, 0);
#pragma unroll
      for (int k = 0; k < N; k++) cfma(s, a[i * N + k], cconj(b[j * N + k]));
      c[i * N + j] = s;
    }
}

// c = a^dag b
template <int N>
__device__ __forceinline__ void rk_mdm(double2 (&c)[N * N], const double2 (&a)[N * N], const double2 (&b)[N * N]) {
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int j = 0; j < N; j++) {
      double2 s = make_double2(0, 0);
#pragma unroll
      for (int k = 0; k < N; k++) cfmac(s, a[k * N + i], b[k * N + j]);
      c[i * N + j] = s;
    }
}

// The same with the links of a leaf multiplied in pairs: for d >= 10, where the leaf sums live in local
// memory either way
template <int NC, int D>
__device__ void clover_leaves_tree(double2 (&out)[D * D], const double2 *fund, const Geom &g, const int c[4], int id,
                              int mu, int nu, const double2 *basis, int rep) {
  double2 A[NC * NC], B[NC * NC], P[NC * NC], Q[NC * NC], R[D * D];
  for (int k = 0; k < D * D; k++) out[k] = make_double2(0, 0);
  int cc[4];
#pragma unroll 1
  for (int leaf = 0; leaf < 4; leaf++) {
    if (leaf == 0) {         // U(x,mu) U(x+mu,nu) [U(x,nu) U(x+nu,mu)]^dag
      int a = neighbour(g, c, mu, +1), b = neighbour(g, c, nu, +1);
      rk_load<NC>(A, fund, g, id, mu); rk_load<NC>(B, fund, g, a, nu); rk_mm<NC>(P, A, B);
      rk_load<NC>(A, fund, g, id, nu); rk_load<NC>(B, fund, g, b, mu); rk_mm<NC>(Q, A, B);
      rk_mmd<NC>(A, P, Q);
    } else if (leaf == 1) {  // U(x,nu) [U(x-mu,nu) U(x-mu+nu,mu)]^dag U(x-mu,mu)
      int a = neighbour(g, c, mu, -1);
      coords_of(g, a, cc);
      int b = neighbour(g, cc, nu, +1);
      rk_load<NC>(A, fund, g, a, nu); rk_load<NC>(B, fund, g, b, mu); rk_mm<NC>(Q, A, B);
      rk_load<NC>(A, fund, g, id, nu); rk_mmd<NC>(P, A, Q);
      rk_load<NC>(B, fund, g, a, mu); rk_mm<NC>(A, P, B);
    } else if (leaf == 2) {  // [U(x-mu-nu,nu) U(x-mu,mu)]^dag U(x-mu-nu,mu) U(x-nu,nu)
      int a = neighbour(g, c, mu, -1), b = neighbour(g, c, nu, -1);
      coords_of(g, a, cc);
      int ci = neighbour(g, cc, nu, -1);
      rk_load<NC>(A, fund, g, ci, nu); rk_load<NC>(B, fund, g, a, mu); rk_mm<NC>(Q, A, B);
      rk_load<NC>(A, fund, g, ci, mu); rk_mdm<NC>(P, Q, A);
      rk_load<NC>(B, fund, g, b, nu); rk_mm<NC>(A, P, B);
    } else {                 // U(x-nu,nu)^dag U(x-nu,mu) U(x-nu+mu,nu) U(x,mu)^dag
      int a = neighbour(g, c, nu, -1);
      coords_of(g, a, cc);
      int b = neighbour(g, cc, mu, +1);
      rk_load<NC>(A, fund, g, a, nu); rk_load<NC>(B, fund, g, a, mu); rk_mdm<NC>(P, A, B);
      rk_load<NC>(B, fund, g, b, nu); rk_mm<NC>(Q, P, B);
      rk_load<NC>(B, fund, g, id, mu); rk_mmd<NC>(A, Q, B);
    }
    represent_one<NC, D>(R, A, basis, rep);
    for (int k = 0; k < D * D; k++) out[k] = cadd(out[k], R[k]);
  }
}

// the slices whose clover term vanishes (_bcs_clover_term, clover.cpp:93-118)
__device__ __forceinline__ bool clover_zeroed(const Geom &g, int t) {
  const int T = g.dim[0];
  return (g.bc == YG_BC_SF && (t == 0 || t == T - 1 || t == T - 2)) || (g.bc == YG_BC_OPEN && (t == 0 || t == T - 1));
}

// entry (i, j) of the blocks A0..A3 from the leaf sums q[plane](i, j) and q[plane](j, i), planes
// (0,1),(0,2),(0,3),(1,2),(1,3),(2,3); _compute_clover_term, clover.cpp:120-168
__device__ __forceinline__ void clover_entry(double2 (&A)[4], const double2 (&ij)[6], const double2 (&ji)[6], double csw) {
  const double a_re = ij[2].y + ji[2].y, a_im = ji[2].x - ij[2].x;
  const double b_re = ij[3].y + ji[3].y, b_im = ij[3].x - ji[3].x;
  const double c_re = ij[0].y + ji[0].y - ij[1].x + ji[1].x, c_im = ji[0].x - ij[0].x - ij[1].y - ji[1].y;
  const double d_re = ij[4].x - ji[4].x + ij[5].y + ji[5].y, d_im = ij[4].y + ji[4].y - ij[5].x + ji[5].x;
  A[0] = make_double2(csw * (a_re - b_re), csw * (a_im + b_im));
  A[1] = make_double2(csw * (c_re - d_re), csw * (c_im - d_im));
  A[2] = make_double2(-csw * (a_re + b_re), csw * (b_im - a_im));
  A[3] = make_double2(-csw * (c_re + d_re), -csw * (c_im + d_im));
}

// The clover term for d <= 8: a block takes 32 sites with one warp per plane, whose leaf sums
// meet in shared memory, where one thread a site kept all six in local memory (1.1 kB a thread
// for d = 3, indexed by the plane).  SU(3) 32 x 16^3: 188 us, 282 before (cold caches).  Represent + clover
// term, a thread a site / this: sextet (d = 6) 8^4 483 / 148 us, 16^4 1267 / 1191; SU(4) antisymmetric
// (d = 6) 8^4 751 / 178, 16^4 2098 / 2064; d = 8 8^4 743 / 196, 12^4 1040 / 788.  SU(4) at d = 6 and
// d = 8 take the registers of one block an SM (with two, d = 6 of SU(4) spilled: 16^4 3775).
template <int NC, int D>
__global__ void __launch_bounds__(192, (D <= 4 || (D == 6 && NC == 3) ? 2 : 1)) k_clover_term_planes(double2 *cl, const double2 *fund, Geom g, const double2 *basis,
                                                            int rep, double csw_in) {
  constexpr int DD = D * D;
  extern __shared__ __align__(16) unsigned char leaf_smem[];
  double2 *sm = reinterpret_cast<double2 *>(leaf_smem);      // [plane][entry][lane]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool live = blockIdx.x * 32 + lane < g.V;
  const int id = live ? blockIdx.x * 32 + lane : g.V - 1;
  int c[4];
  coords_of(g, id, c);
  const int mu = w < 3 ? 0 : w < 5 ? 1 : 2, nu = w < 3 ? w + 1 : w < 5 ? w - 1 : 3;
  double2 q[DD];
  clover_leaves<NC, D>(q, fund, g, c, id, mu, nu, basis, rep);
#pragma unroll
  for (int k = 0; k < DD; k++) sm[(w * DD + k) * 32 + lane] = q[k];
  __syncthreads();
  if (!live) return;
  const double csw = clover_zeroed(g, c[0]) ? 0.0 : -csw_in / 16.0;
  for (int e = w; e < DD; e += 6) {
    const int t = (e % D) * D + e / D;
    double2 ij[6], ji[6], A[4];
#pragma unroll
    for (int p = 0; p < 6; p++) {
      ij[p] = sm[(p * DD + e) * 32 + lane];
      ji[p] = sm[(p * DD + t) * 32 + lane];
    }
    clover_entry(A, ij, ji, csw);
#pragma unroll
    for (int m = 0; m < 4; m++) cl[fidx(g, id, m * DD + e, 4 * DD)] = csw == 0.0 ? make_double2(0, 0) : A[m];
  }
}

// The same for larger d, one thread a site, whose leaf sums (24 kB at d = 15) travel through L2.
// TREE: leaves as pairs of products.  represent + clover term, chains / pairs: d = 10 4^4 1508 / 1677 us,
// 8^4 1540 / 1709, 12^4 2440 / 2303, 16^4 5876 / 5225; d = 15 4^4 3628 / 3415, 12^4 6160 / 5140.
constexpr int kLeafPairSites = 10000;      // d = 10: between 8^4 and 12^4
template <int NC, int D, bool TREE>
__global__ void k_clover_term(double2 *cl, const double2 *fund, Geom g, const double2 *basis, int rep, double csw_in) {
  int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= g.V) return;
  int c[4];
  coords_of(g, id, c);
  if (clover_zeroed(g, c[0])) {
    for (int k = 0; k < 4 * D * D; k++) cl[fidx(g, id, k, 4 * D * D)] = make_double2(0, 0);
    return;
  }
  const double csw = -csw_in / 16.0;
  const int pm[6][2] = {{0, 1}, {0, 2}, {0, 3}, {1, 2}, {1, 3}, {2, 3}};
  double2 tmp[6][D * D];
#pragma unroll 1
  for (int q = 0; q < 6; q++) {
    if constexpr (TREE) clover_leaves_tree<NC, D>(tmp[q], fund, g, c, id, pm[q][0], pm[q][1], basis, rep);
    else clover_leaves<NC, D>(tmp[q], fund, g, c, id, pm[q][0], pm[q][1], basis, rep);
  }
  for (int i = 0; i < D; i++)
    for (int j = 0; j < D; j++) {
      double2 ij[6], ji[6], A[4];
#pragma unroll
      for (int q = 0; q < 6; q++) {
        ij[q] = tmp[q][i * D + j];
        ji[q] = tmp[q][j * D + i];
      }
      clover_entry(A, ij, ji, csw);
#pragma unroll
      for (int m = 0; m < 4; m++) cl[fidx(g, id, m * D * D + i * D + j, 4 * D * D)] = A[m];
    }
}

template <int NC, int D>
void RK<NC, D>::represent(double2 *links, double *real, const double2 *fund, Geom g, const double2 *basis, int rep,
                          cudaStream_t s) {
  if constexpr (D == NC * NC - 1) {
    if (real) {
      k_represent<NC, D, true><<<nblk(4L * g.V, 128), 128, 0, s>>>(links, real, fund, g, basis, rep);
      return;
    }
  }
  k_represent<NC, D, false><<<nblk(4L * g.V, 128), 128, 0, s>>>(links, nullptr, fund, g, basis, rep);
}

template <int NC, int D>
void RK<NC, D>::clover_term(double2 *cl, const double2 *fund, Geom g, const double2 *basis, int rep, double csw,
                            cudaStream_t s) {
  if constexpr (D <= 8) {      // six planes of d x d entries for 32 sites in shared memory: 192 kB at d = 8
    constexpr int smem = sizeof(double2) * 6 * D * D * 32;
    if (smem > 48 * 1024)
      check_cuda(cudaFuncSetAttribute(k_clover_term_planes<NC, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                 "clover term shared memory");
    k_clover_term_planes<NC, D><<<nblk(g.V, 32), 192, smem, s>>>(cl, fund, g, basis, rep, csw);
  } else {
    if (D == 10 && g.V < kLeafPairSites)
      k_clover_term<NC, D, D != 10><<<nblk(g.V, 64), 64, 0, s>>>(cl, fund, g, basis, rep, csw);
    else
      k_clover_term<NC, D, true><<<nblk(g.V, 64), 64, 0, s>>>(cl, fund, g, basis, rep, csw);
  }
}

}  // namespace yg
