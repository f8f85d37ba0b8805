// Device code of the Wilson-clover Dirac operator (included by the yg_inst_*_op.cu units).
//
//  hop (dirac_kernel, dirac.cpp:227-704):
//      out(x) = -sign/2 * sum_mu [ (1-g_mu) U(x,mu) psi(x+mu) + (1+g_mu) U(x-mu,mu)^dag psi(x-mu) ]
//    in the chiral basis of spinor.cpp:191-264, followed by apply_bcs_on_spinor_field
//    (bcs.cpp:139-164).  One thread per output site; each direction spin-projects the
//    neighbour to a half spinor (2 x d), multiplies by the d x d link and reconstructs the
//    other two spin components.  The antiperiodic sign sits in the links (set at upload,
//    bcs.cpp:264-272).
//  Epilogues fused into the hop (the even-odd Schur operator of dirac.cpp:738-765):
//    CLOVINV  tmp_o = A_oo^-1 (hop)           (clover_inv_kernel, dirac.cpp:109-225)
//    CLOVADD  dst_e = A_ee src_e + hop [g5]    (clover_kernel, dirac.cpp:25-107; Hphi :769-773)
//    AXPY     dst   = a*src + hop [g5]         (dirac.cpp:755-765, no clover term)
//  Compute type R = double (the FP64 operator) or float (the inner operator of the
//  mixed-precision solver); storage is cplx<R>.
#pragma once

#include <type_traits>
#include "yg_kernels.h"

namespace yg {

template <typename T>
__device__ __forceinline__ T ld(const T *p, long i) { return __ldg(p + i); }

// a word of a spinor field: through the read-only path, or (NC = false, a kernel that also writes
// the field between its grid barriers) an ordinary load
template <bool NC, typename T>
__device__ __forceinline__ T ldf(const T *p, long i) { return NC ? __ldg(p + i) : p[i]; }

template <int D, typename R, bool NC = true>
__device__ __forceinline__ void load_spinor(cplx<R> (&s)[4][D], const cplx<R> *f, const Geom &g, int id) {
#pragma unroll
  for (int sp = 0; sp < 4; sp++) {
    YG_UNROLL_D
    for (int c = 0; c < D; c++) s[sp][c] = ldf<NC>(f, fidx(g, id, sp * D + c, 4 * D));
  }
}

template <int D, typename R>
__device__ __forceinline__ void store_spinor(cplx<R> *f, const cplx<R> (&s)[4][D], const Geom &g, int id) {
#pragma unroll
  for (int sp = 0; sp < 4; sp++) {
    YG_UNROLL_D
    for (int c = 0; c < D; c++) f[fidx(g, id, sp * D + c, 4 * D)] = s[sp][c];
  }
}

// acc += u h for a real link entry u
template <typename T, typename R>
__device__ __forceinline__ void rfma(T &acc, R u, T h) {
  acc.x = fma(u, h.x, acc.x);
  acc.y = fma(u, h.y, acc.y);
}

// The links a hop reads: complex, or (adjoint representations, FP64) the real copy, half the bytes.
// The product with an imaginary part of zero is the same number.  Hphi_sq, complex / real links: d = 3
// 24^4 295 / 210 us, d = 8 16^4 503 / 422, d = 15 16^4 1416 / 1172.
template <typename R, bool REAL> struct LinkPtr { using t = const cplx<R> *; };
template <typename R> struct LinkPtr<R, true> { using t = const R *; };
template <bool REAL, typename R>
__device__ __forceinline__ typename LinkPtr<R, REAL>::t hop_links(const HopArgs<R> &a) {
  if constexpr (REAL) return a.Ur;
  else return a.U;
}

// chi = U h (DAG=false) or U^dag h (DAG=true), U = link (id, mu)
template <int D, typename R, bool DAG, typename LP>
__device__ __forceinline__ void link_mul(cplx<R> (&chi)[2][D], const cplx<R> (&h)[2][D], LP U, const Geom &g, int id,
                                         int mu) {
  YG_UNROLL_D
  for (int i = 0; i < D; i++) {
    cplx<R> s0 = mk<R>(0, 0), s1 = mk<R>(0, 0);
    YG_UNROLL_D
    for (int j = 0; j < D; j++) {
      const auto u = ld(U, fidx(g, id, mu * D * D + (DAG ? j * D + i : i * D + j), 4 * D * D));
      if constexpr (std::is_same_v<LP, const R *>) { rfma(s0, u, h[0][j]); rfma(s1, u, h[1][j]); }
      else if (DAG) { cfmac(s0, u, h[0][j]); cfmac(s1, u, h[1][j]); }
      else { cfma(s0, u, h[0][j]); cfma(s1, u, h[1][j]); }
    }
    chi[0][i] = s0;
    chi[1][i] = s1;
  }
}

// One direction: SIG = -1 for the forward term (1-g_mu), +1 for the backward term (1+g_mu).
template <int D, typename R, int MU, int SIG, bool NC, typename LP>
__device__ __forceinline__ void hop_dir(cplx<R> (&acc)[4][D], const cplx<R> *src, LP U, const Geom &g, int nid,
                                        int lid) {
  cplx<R> h[2][D];
  YG_UNROLL_D
  for (int c = 0; c < D; c++) {
    cplx<R> p0 = ldf<NC>(src, fidx(g, nid, 0 * D + c, 4 * D));
    cplx<R> p1 = ldf<NC>(src, fidx(g, nid, 1 * D + c, 4 * D));
    cplx<R> p2 = ldf<NC>(src, fidx(g, nid, 2 * D + c, 4 * D));
    cplx<R> p3 = ldf<NC>(src, fidx(g, nid, 3 * D + c, 4 * D));
    if (MU == 0) {
      h[0][c] = SIG < 0 ? cadd(p0, p2) : csub(p0, p2);
      h[1][c] = SIG < 0 ? cadd(p1, p3) : csub(p1, p3);
    } else if (MU == 1) {
      h[0][c] = SIG < 0 ? cadd(p0, ctimesi(p3)) : csub(p0, ctimesi(p3));
      h[1][c] = SIG < 0 ? cadd(p1, ctimesi(p2)) : csub(p1, ctimesi(p2));
    } else if (MU == 2) {
      h[0][c] = SIG < 0 ? cadd(p0, p3) : csub(p0, p3);
      h[1][c] = SIG < 0 ? csub(p1, p2) : cadd(p1, p2);
    } else {
      h[0][c] = SIG < 0 ? cadd(p0, ctimesi(p2)) : csub(p0, ctimesi(p2));
      h[1][c] = SIG < 0 ? csub(p1, ctimesi(p3)) : cadd(p1, ctimesi(p3));
    }
  }
  cplx<R> chi[2][D];
  link_mul<D, R, (SIG > 0)>(chi, h, U, g, lid, MU);
  YG_UNROLL_D
  for (int c = 0; c < D; c++) {
    acc[0][c] = cadd(acc[0][c], chi[0][c]);
    acc[1][c] = cadd(acc[1][c], chi[1][c]);
    if (MU == 0) {
      acc[2][c] = SIG < 0 ? cadd(acc[2][c], chi[0][c]) : csub(acc[2][c], chi[0][c]);
      acc[3][c] = SIG < 0 ? cadd(acc[3][c], chi[1][c]) : csub(acc[3][c], chi[1][c]);
    } else if (MU == 1) {
      acc[2][c] = SIG < 0 ? cadd(acc[2][c], ctimesmi(chi[1][c])) : cadd(acc[2][c], ctimesi(chi[1][c]));
      acc[3][c] = SIG < 0 ? cadd(acc[3][c], ctimesmi(chi[0][c])) : cadd(acc[3][c], ctimesi(chi[0][c]));
    } else if (MU == 2) {
      acc[2][c] = SIG < 0 ? csub(acc[2][c], chi[1][c]) : cadd(acc[2][c], chi[1][c]);
      acc[3][c] = SIG < 0 ? cadd(acc[3][c], chi[0][c]) : csub(acc[3][c], chi[0][c]);
    } else {
      acc[2][c] = SIG < 0 ? cadd(acc[2][c], ctimesmi(chi[0][c])) : cadd(acc[2][c], ctimesi(chi[0][c]));
      acc[3][c] = SIG < 0 ? cadd(acc[3][c], ctimesi(chi[1][c])) : cadd(acc[3][c], ctimesmi(chi[1][c]));
    }
  }
}

template <int D, typename R, bool NC, typename LP>
__device__ __forceinline__ void hop_site(cplx<R> (&acc)[4][D], const cplx<R> *src, LP U, const Geom &g, int id,
                                         const int c[4]) {
#pragma unroll
  for (int s = 0; s < 4; s++) {
    YG_UNROLL_D
    for (int k = 0; k < D; k++) acc[s][k] = mk<R>(0, 0);
  }
  int f, b;
  f = neighbour(g, c, 0, +1); hop_dir<D, R, 0, -1, NC>(acc, src, U, g, f, id);
  b = neighbour(g, c, 0, -1); hop_dir<D, R, 0, +1, NC>(acc, src, U, g, b, b);
  f = neighbour(g, c, 1, +1); hop_dir<D, R, 1, -1, NC>(acc, src, U, g, f, id);
  b = neighbour(g, c, 1, -1); hop_dir<D, R, 1, +1, NC>(acc, src, U, g, b, b);
  f = neighbour(g, c, 2, +1); hop_dir<D, R, 2, -1, NC>(acc, src, U, g, f, id);
  b = neighbour(g, c, 2, -1); hop_dir<D, R, 2, +1, NC>(acc, src, U, g, b, b);
  f = neighbour(g, c, 3, +1); hop_dir<D, R, 3, -1, NC>(acc, src, U, g, f, id);
  b = neighbour(g, c, 3, -1); hop_dir<D, R, 3, +1, NC>(acc, src, U, g, b, b);
}

// (4+m+cf) psi + [[A0,A1],[A1^dag,-A0]] (psi0,psi1) (+) [[A2,A3],[A3^dag,-A2]] (psi2,psi3)
template <int D, typename R>
__device__ __forceinline__ void clover_site(cplx<R> (&out)[4][D], const cplx<R> (&s)[4][D], const cplx<R> *cl,
                                            const Geom &g, int id, R diag) {
#pragma unroll
  for (int blk = 0; blk < 2; blk++) {
    const int s0 = 2 * blk, s1 = 2 * blk + 1;
    const int m0 = 2 * blk, m1 = 2 * blk + 1;
    YG_UNROLL_D
    for (int i = 0; i < D; i++) {
      cplx<R> o0 = cscale(s[s0][i], diag), o1 = cscale(s[s1][i], diag);
      YG_UNROLL_D
      for (int j = 0; j < D; j++) {
        // A0 and A2 are Hermitian to the last bit: only their lower triangles are read
        cplx<R> a0 = ld(cl, fidx(g, id, m0 * D * D + (i >= j ? i * D + j : j * D + i), 4 * D * D));
        if (i < j) a0.y = -a0.y;
        cplx<R> a1 = ld(cl, fidx(g, id, m1 * D * D + i * D + j, 4 * D * D));
        cplx<R> a1t = ld(cl, fidx(g, id, m1 * D * D + j * D + i, 4 * D * D));
        cfma(o0, a0, s[s0][j]);
        cfma(o0, a1, s[s1][j]);
        cfmac(o1, a1t, s[s0][j]);
        o1 = csub(o1, cmul(a0, s[s1][j]));
      }
      out[s0][i] = o0;
      out[s1][i] = o1;
    }
  }
}

// acc += A psi for the psi stored at src2 (A as in clover_site), one spin block at a time
// so that only two spins of psi are live next to the accumulator
template <int D, typename R, bool NC>
__device__ __forceinline__ void clover_add_site(cplx<R> (&acc)[4][D], const cplx<R> *src2, const cplx<R> *cl,
                                                const Geom &g, int id, R diag) {
#pragma unroll
  for (int blk = 0; blk < 2; blk++) {
    const int s0 = 2 * blk, s1 = 2 * blk + 1;
    const int m0 = 2 * blk, m1 = 2 * blk + 1;
    cplx<R> p0[D], p1[D];
#pragma unroll
    for (int c = 0; c < D; c++) {
      p0[c] = ldf<NC>(src2, fidx(g, id, s0 * D + c, 4 * D));
      p1[c] = ldf<NC>(src2, fidx(g, id, s1 * D + c, 4 * D));
    }
    // each entry is loaded once: A0 is Hermitian to the last bit, so its lower triangle serves both
    // triangles and, negated, the lower spin; A1 serves the upper spin and, daggered, the lower one
    // (step 2 on 32^4, d = 3: 204 us, 247 with an entry loaded for each use)
#pragma unroll
    for (int i = 0; i < D; i++) {
      acc[s0][i] = cadd(acc[s0][i], cscale(p0[i], diag));
      acc[s1][i] = cadd(acc[s1][i], cscale(p1[i], diag));
    }
#pragma unroll
    for (int i = 0; i < D; i++)
#pragma unroll
      for (int j = 0; j <= i; j++) {
        const cplx<R> e = ld(cl, fidx(g, id, m0 * D * D + i * D + j, 4 * D * D)), ne = mk<R>(-e.x, -e.y);
        cfma(acc[s0][i], e, p0[j]);
        cfma(acc[s1][i], ne, p1[j]);
        if (j < i) {
          cfmac(acc[s0][j], e, p0[i]);
          cfmac(acc[s1][j], ne, p1[i]);
        }
      }
#pragma unroll
    for (int i = 0; i < D; i++)
#pragma unroll
      for (int j = 0; j < D; j++) {
        const cplx<R> w = ld(cl, fidx(g, id, m1 * D * D + i * D + j, 4 * D * D));
        cfma(acc[s0][i], w, p1[j]);
        cfmac(acc[s1][j], w, p0[i]);
      }
  }
}

// A^-1 psi through the packed LDL factors of the site: forward substitution, D^-1, back
// substitution with conj(L) (clover_inv_kernel, dirac.cpp:135-212)
template <int D, typename R>
__device__ __forceinline__ void ldl_site(cplx<R> (&out)[4][D], const cplx<R> (&s)[4][D], const double2 *ldl,
                                         int h, int Vh) {
  constexpr int N = 2 * D, P = D * (2 * D + 1);
#pragma unroll
  for (int blk = 0; blk < 2; blk++) {
    const double2 *Lb = ldl + (long)blk * P * Vh + h;
    double2 x[N];
    #pragma unroll
    for (int i = 0; i < D; i++) {
      x[i] = make_double2((double)s[2 * blk][i].x, (double)s[2 * blk][i].y);
      x[i + D] = make_double2((double)s[2 * blk + 1][i].x, (double)s[2 * blk + 1][i].y);
    }
    #pragma unroll
    for (int i = 1; i < N; i++) {
      #pragma unroll
      for (int k = 0; k < i; k++) x[i] = csub(x[i], cmul(__ldg(Lb + (long)(i * (i + 1) / 2 + k) * Vh), x[k]));
    }
    #pragma unroll
    for (int i = N - 1; i >= 0; i--) {
      double dii = __ldg(Lb + (long)(i * (i + 1) / 2 + i) * Vh).x;
      x[i] = cscale(x[i], 1.0 / dii);
      #pragma unroll
      for (int k = i + 1; k < N; k++) x[i] = csub(x[i], cmulc(__ldg(Lb + (long)(k * (k + 1) / 2 + i) * Vh), x[k]));
    }
    #pragma unroll
    for (int i = 0; i < D; i++) {
      out[2 * blk][i] = mk<R>((R)x[i].x, (R)x[i].y);
      out[2 * blk + 1][i] = mk<R>((R)x[i + D].x, (R)x[i + D].y);
    }
  }
}

// A^-1 psi with explicit (2d x 2d) inverse blocks per site (FP32 inner operator)
template <int D, typename R>
__device__ __forceinline__ void cinv_site(cplx<R> (&out)[4][D], const cplx<R> (&s)[4][D], const cplx<R> *cinv,
                                          int h, int Vh) {
  constexpr int N = 2 * D;
#pragma unroll
  for (int blk = 0; blk < 2; blk++) {
    YG_UNROLL_D
    for (int i = 0; i < N; i++) {
      cplx<R> acc = mk<R>(0, 0);
      YG_UNROLL_D
      for (int j = 0; j < N; j++) {
        cplx<R> a = ld(cinv, ((long)blk * N * N + i * N + j) * Vh + h);
        cplx<R> v = j < D ? s[2 * blk][j] : s[2 * blk + 1][j - D];
        cfma(acc, a, v);
      }
      if (i < D) out[2 * blk][i] = acc;
      else out[2 * blk + 1][i - D] = acc;
    }
  }
}

// A^-1 psi with the packed Hermitian inverse blocks of the FP64 path: per block of
// N = 2d rows, N real diagonal entries (two per double2 word) then the N(N-1)/2 complex
// lower-triangle entries (1,0),(2,0),(2,1),... one per word; word w of block b of the
// site h lives at (b*2d^2 + w)*Vh + h.  The upper triangle is the conjugate transpose.
template <int D, typename R>
__device__ __forceinline__ void cpk_site(cplx<R> (&out)[4][D], const cplx<R> (&s)[4][D], const double2 *cpk,
                                         int h, int Vh) {
  constexpr int N = 2 * D, W = 2 * D * D;
#pragma unroll
  for (int blk = 0; blk < 2; blk++) {
    const double2 *Cb = cpk + (long)blk * W * Vh + h;
    double2 x[N], y[N];
    #pragma unroll
    for (int i = 0; i < D; i++) {
      x[i] = make_double2((double)s[2 * blk][i].x, (double)s[2 * blk][i].y);
      x[i + D] = make_double2((double)s[2 * blk + 1][i].x, (double)s[2 * blk + 1][i].y);
    }
    #pragma unroll
    for (int w = 0; w < D; w++) {
      double2 dd = __ldg(Cb + (long)w * Vh);
      y[2 * w] = cscale(x[2 * w], dd.x);
      y[2 * w + 1] = cscale(x[2 * w + 1], dd.y);
    }
    #pragma unroll
    for (int i = 1; i < N; i++) {
      #pragma unroll
      for (int j = 0; j < i; j++) {
        double2 m = __ldg(Cb + (long)(D + i * (i - 1) / 2 + j) * Vh);
        cfma(y[i], m, x[j]);
        cfmac(y[j], m, x[i]);
      }
    }
    #pragma unroll
    for (int i = 0; i < D; i++) {
      out[2 * blk][i] = mk<R>((R)y[i].x, (R)y[i].y);
      out[2 * blk + 1][i] = mk<R>((R)y[i + D].x, (R)y[i + D].y);
    }
  }
}

// One output site of the launch's range: its four spins in acc, for the caller to store
template <int D, typename R, int EPI, bool NC, bool REAL = false>
__device__ __forceinline__ void hop_values(const HopArgs<R> &a, int t, cplx<R> (&acc)[4][D]) {
  const Geom &g = a.g;
  int id = a.lo + t;
  int c[4];
  coords_of(g, id, c);
  bool bnd = spinor_zeroed(g, c[0]);
  hop_site<D, R, NC>(acc, a.src, hop_links<REAL>(a), g, id, c);
#pragma unroll
  for (int s = 0; s < 4; s++) {
    YG_UNROLL_D
    for (int k = 0; k < D; k++) acc[s][k] = bnd ? mk<R>(0, 0) : cscale(acc[s][k], a.coeff);
  }

  if (EPI == EPI_PLAIN) {
    if (a.assign && !bnd) {
      cplx<R> old[4][D];
      load_spinor<D, R>(old, a.dst, g, id);
#pragma unroll
      for (int s = 0; s < 4; s++) {
        YG_UNROLL_D
        for (int k = 0; k < D; k++) acc[s][k] = cadd(acc[s][k], old[s][k]);
      }
    }
  } else if (EPI == EPI_CLOVINV || EPI == EPI_CLOVPK) {
    if (a.dst2) store_spinor<D, R>(a.dst2, acc, g, id);
    cplx<R> out[4][D];
    if (EPI == EPI_CLOVPK) cpk_site<D, R>(out, acc, a.cpk, id - g.Vh, g.Vh);
    else cinv_site<D, R>(out, acc, a.cinv, id - g.Vh, g.Vh);
#pragma unroll
    for (int s = 0; s < 4; s++) {
      YG_UNROLL_D
      for (int k = 0; k < D; k++) acc[s][k] = out[s][k];
    }
  } else {
    bool zero_add = bnd && a.zero_add_at_boundary;
    if (EPI == EPI_CLOVADD) {
      R diag = a.diag + ((c[0] == g.Ta || c[0] == g.Tb) ? a.cfm1 : (R)0);
      if (!zero_add) clover_add_site<D, R, NC>(acc, a.src2, a.cl, g, id, diag);
    } else {
      cplx<R> s2[4][D];
      load_spinor<D, R, NC>(s2, a.src2, g, id);
#pragma unroll
      for (int s = 0; s < 4; s++) {
        YG_UNROLL_D
        for (int k = 0; k < D; k++) acc[s][k] = zero_add ? acc[s][k] : cadd(acc[s][k], cscale(s2[s][k], a.diag));
      }
    }
    if (a.g5) {
      YG_UNROLL_D
      for (int k = 0; k < D; k++) {
        acc[2][k] = cscale(acc[2][k], (R)-1);
        acc[3][k] = cscale(acc[3][k], (R)-1);
      }
    }
  }
}

template <int D, typename R, int EPI, bool REAL>
__global__ void __launch_bounds__(128) k_hop(HopArgs<R> a) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n) return;
  cplx<R> acc[4][D];
  hop_values<D, R, EPI, true, REAL>(a, t, acc);
  store_spinor<D, R>(a.dst, acc, a.g, a.lo + t);
}

// ------------------------------------------------------------------ four lanes a site
// The same operator with four neighbouring lanes per output site: lane q takes the directions +mu and
// -mu of mu = q, and a reduce-scatter of the four partial spinors leaves it spin q of the sum.  Each
// lane has one direction's links and neighbours in flight instead of eight in a row, a quarter of the
// accumulators, and its half of a clover block in the epilogue.
//
// The lanes of a warp carry different mu, so the projections are written with per-lane phases.  With
// (X, Y) the lower spins that (1 -+ g_mu) adds to spins 0 and 1: h0 = p0 +- ph0 pX, h1 = p1 +- ph1 pY,
// and the lower components of the result are conj(ph0) chi0 at X and conj(ph1) chi1 at Y (+-).
//   mu = 0: X,Y = 2,3, ph = 1, 1;  1: 3,2, i, i;  2: 3,2, 1, -1;  3: 2,3, i, -i
//
// Taken up to one block of 32 sites per SM.  There a thread per site is a chain of eight rounds of
// loads on a few SMs; on a full GPU the lanes' shuffles and shorter runs (8 sites, 128 bytes a load) lose.
// Hphi_sq, us, a thread per site / four lanes, at 2048, 3840, 4800, 6912, 10368, 16800 and 32768 outputs:
//   d = 2  28.7/24.6  31.3/24.6  30.9/24.6  32.8/24.6  32.7/29.4  32.8/32.8  36.3/49.8
//   d = 3  35.9/27.7  37.5/27.7  37.9/32.8  37.3/32.8  39.2/41.0  41.0/45.0  53.4/88.1   (32^4: 810 / 1127)
//   d = 4  48.4/32.8  49.2/32.8  49.2/40.6  49.2/41.0  49.2/49.2  54.1/73.3  111/149
//   d = 6  83.7/45.1  87.0/45.1  85.9/59.4  89.2/65.4  129/116    186/150    226/292
// The line is the one at which no d loses; d = 3 crosses at about 8000 outputs, d = 6 not before 16800.
constexpr int kQuadSites = 148 * 32;

template <typename C>
__device__ __forceinline__ C shfl_c(C v, int m) {
  v.x = __shfl_xor_sync(0xffffffffu, v.x, m);
  v.y = __shfl_xor_sync(0xffffffffu, v.y, m);
  return v;
}
template <typename C>
__device__ __forceinline__ C sel(bool p, C a, C b) { C c; c.x = p ? a.x : b.x; c.y = p ? a.y : b.y; return c; }

// half spinor of the neighbour nid times the link lid: chi0, chi1
template <int D, typename R, bool NC, bool DAG, typename LP>
__device__ __forceinline__ void quad_dir(cplx<R> (&chi)[2][D], const cplx<R> *src, LP U, const Geom &g, int mu,
                                          bool swap, cplx<R> ph0, cplx<R> ph1, int nid, int lid) {
  const int nb = nid >= g.Vh, lb = lid >= g.Vh;
  const cplx<R> *f = src + (long)nb * 4 * D * g.Vh + (nid - nb * g.Vh);
  const LP u = U + (long)(lb * 4 + mu) * D * D * g.Vh + (lid - lb * g.Vh);
  const long st = g.Vh;
  const long ox = (swap ? 3L * D : 2L * D) * st, oy = (swap ? 2L * D : 3L * D) * st;
  cplx<R> h[2][D];
#pragma unroll
  for (int c = 0; c < D; c++) {
    h[0][c] = ldf<NC>(f, c * st);
    h[1][c] = ldf<NC>(f, (D + c) * st);
    cfma(h[0][c], ph0, ldf<NC>(f, ox + c * st));
    cfma(h[1][c], ph1, ldf<NC>(f, oy + c * st));
  }
#pragma unroll
  for (int i = 0; i < D; i++) {
    cplx<R> c0 = mk<R>(0, 0), c1 = mk<R>(0, 0);
#pragma unroll
    for (int j = 0; j < D; j++) {
      const auto w = ld(u, (DAG ? j * D + i : i * D + j) * st);
      if constexpr (std::is_same_v<LP, const R *>) { rfma(c0, w, h[0][j]); rfma(c1, w, h[1][j]); }
      else if (DAG) { cfmac(c0, w, h[0][j]); cfmac(c1, w, h[1][j]); }
      else { cfma(c0, w, h[0][j]); cfma(c1, w, h[1][j]); }
    }
    chi[0][i] = c0;
    chi[1][i] = c1;
  }
}

// spin q of A^-1 w for the packed Hermitian inverse: w is the lane's spin, its partner (lane ^ 1)
// holds the block's other spin
template <int D, typename R>
__device__ __forceinline__ void quad_cpk(cplx<R> (&w)[D], const double2 *cpk, int h, int Vh, int q) {
  constexpr int W = 2 * D * D;
  const double2 *C = cpk + (long)(q >> 1) * W * Vh + h;
  const bool up = !(q & 1);
  const int r0 = up ? 0 : D;
  cplx<R> z[D], o[D];
#pragma unroll
  for (int c = 0; c < D; c++) z[c] = shfl_c(w[c], 1);
#pragma unroll
  for (int i = 0; i < D; i++) {
    const int r = r0 + i;
    const double d = __ldg(reinterpret_cast<const double *>(C + (long)(r >> 1) * Vh) + (r & 1));
    o[i] = cscale(w[i], (R)d);
  }
#pragma unroll
  for (int i = 1; i < D; i++)
#pragma unroll
    for (int j = 0; j < i; j++) {
      const double2 m = __ldg(C + (long)(D + (r0 + i) * (r0 + i - 1) / 2 + r0 + j) * Vh);
      const cplx<R> e = mk<R>((R)m.x, (R)m.y);
      cfma(o[i], e, w[j]);
      cfmac(o[j], e, w[i]);
    }
  const double sg = up ? -1.0 : 1.0;                    // the upper right block is the conjugate transpose
#pragma unroll
  for (int i = 0; i < D; i++)
#pragma unroll
    for (int j = 0; j < D; j++) {
      const int a = up ? j : i, b = up ? i : j;
      const double2 m = __ldg(C + (long)(D + (D + a) * (D + a - 1) / 2 + b) * Vh);
      cfma(o[i], mk<R>((R)m.x, (R)(sg * m.y)), z[j]);
    }
#pragma unroll
  for (int i = 0; i < D; i++) w[i] = o[i];
}

// the same for the explicit FP32 inverse blocks
template <int D, typename R>
__device__ __forceinline__ void quad_cinv(cplx<R> (&w)[D], const cplx<R> *cinv, int h, int Vh, int q) {
  constexpr int N = 2 * D;
  const int own = (q & 1) * D, oth = D - own;
  const cplx<R> *C = cinv + ((long)(q >> 1) * N * N + (long)own * N) * Vh + h;
  cplx<R> z[D], o[D];
#pragma unroll
  for (int c = 0; c < D; c++) z[c] = shfl_c(w[c], 1);
#pragma unroll
  for (int i = 0; i < D; i++) {
    o[i] = mk<R>(0, 0);
#pragma unroll
    for (int j = 0; j < D; j++) {
      cfma(o[i], ld(C, (long)(i * N + own + j) * Vh), w[j]);
      cfma(o[i], ld(C, (long)(i * N + oth + j) * Vh), z[j]);
    }
  }
#pragma unroll
  for (int i = 0; i < D; i++) w[i] = o[i];
}

// w += spin q of A p for the lane's spin p of the site (A as in clover_site; A0 and A2 are Hermitian to
// the last bit, so only their lower triangles are read)
template <int D, typename R>
__device__ __forceinline__ void quad_clover_add(cplx<R> (&w)[D], const cplx<R> (&p)[D], bool add, const cplx<R> *cl,
                                                const Geom &g, int id, R diag, int q) {
  const int blk = id >= g.Vh;
  const cplx<R> *A = cl + ((long)blk * 4 + (q & 2)) * D * D * g.Vh + (id - blk * g.Vh);
  const cplx<R> *B = A + (long)D * D * g.Vh;
  const bool up = !(q & 1);
  const R sa = up ? (R)1 : (R)-1;
  cplx<R> z[D];
#pragma unroll
  for (int c = 0; c < D; c++) z[c] = shfl_c(p[c], 1);
  if (!add) return;
#pragma unroll
  for (int i = 0; i < D; i++) {
    w[i].x = fma(diag, p[i].x, w[i].x);
    w[i].y = fma(diag, p[i].y, w[i].y);
  }
#pragma unroll
  for (int i = 0; i < D; i++)
#pragma unroll
    for (int j = 0; j <= i; j++) {
      const cplx<R> e = cscale(ld(A, (long)(i * D + j) * g.Vh), sa);
      cfma(w[i], e, p[j]);
      if (j < i) cfmac(w[j], e, p[i]);
    }
#pragma unroll
  for (int i = 0; i < D; i++)
#pragma unroll
    for (int j = 0; j < D; j++) {
      cplx<R> e = ld(B, (long)(up ? i * D + j : j * D + i) * g.Vh);
      e.y = up ? e.y : -e.y;
      cfma(w[i], e, z[j]);
    }
}

// Spin q = threadIdx.x & 3 of output site t (clamped to the range by the caller; the four lanes of a
// site and the other sites of the warp all take part): the result in w, `at` the index of its first
// word (the others follow at Vh).
template <int D, typename R, int EPI, bool NC, bool REAL = false>
__device__ __forceinline__ void hop_quad(const HopArgs<R> &a, int t, bool live, cplx<R> (&w)[D], long &at) {
  const Geom &g = a.g;
  const int q = threadIdx.x & 3, id = a.lo + t;
  int c[4];
  coords_of(g, id, c);
  const bool bnd = spinor_zeroed(g, c[0]);
  const bool swap = q == 1 || q == 2, im = q & 1;
  const cplx<R> ph0 = im ? mk<R>(0, 1) : mk<R>(1, 0);
  const cplx<R> ph1 = im ? mk<R>(0, q == 1 ? (R)1 : (R)-1) : mk<R>(q == 0 ? (R)1 : (R)-1, 0);
  cplx<R> v[4][D];
  {
    cplx<R> cf[2][D], cb[2][D];
    int n[4] = {c[0], c[1], c[2], c[3]};
#pragma unroll
    for (int mu = 0; mu < 4; mu++)
      if (mu == q) n[mu] = n[mu] + 1 == g.dim[mu] ? 0 : n[mu] + 1;
    quad_dir<D, R, NC, false>(cf, a.src, hop_links<REAL>(a), g, q, swap, ph0, ph1, id_of(g, n[0], n[1], n[2], n[3]), id);
#pragma unroll
    for (int mu = 0; mu < 4; mu++) n[mu] = mu == q ? (c[mu] == 0 ? g.dim[mu] - 1 : c[mu] - 1) : c[mu];
    const int b = id_of(g, n[0], n[1], n[2], n[3]);
    quad_dir<D, R, NC, true>(cb, a.src, hop_links<REAL>(a), g, q, swap, mk<R>(-ph0.x, -ph0.y), mk<R>(-ph1.x, -ph1.y), b, b);
#pragma unroll
    for (int k = 0; k < D; k++) {
      v[0][k] = cadd(cf[0][k], cb[0][k]);
      v[1][k] = cadd(cf[1][k], cb[1][k]);
      const cplx<R> e0 = cmulc(ph0, csub(cf[0][k], cb[0][k])), e1 = cmulc(ph1, csub(cf[1][k], cb[1][k]));
      v[2][k] = sel(swap, e1, e0);
      v[3][k] = sel(swap, e0, e1);
    }
  }
  // reduce-scatter: lanes 0, 1 keep the upper spins, then even lanes the first of their two
  const bool lo2 = q & 2, od = q & 1;
#pragma unroll
  for (int k = 0; k < D; k++) {
    const cplx<R> a0 = cadd(sel(lo2, v[2][k], v[0][k]), shfl_c(sel(lo2, v[0][k], v[2][k]), 2));
    const cplx<R> a1 = cadd(sel(lo2, v[3][k], v[1][k]), shfl_c(sel(lo2, v[1][k], v[3][k]), 2));
    const cplx<R> s = cadd(sel(od, a1, a0), shfl_c(sel(od, a0, a1), 1));
    w[k] = bnd ? mk<R>(0, 0) : cscale(s, a.coeff);
  }
  const int blk = id >= g.Vh, h = id - blk * g.Vh;
  at = ((long)blk * 4 + q) * D * g.Vh + h;
  if (EPI == EPI_PLAIN) {
    if (a.assign && !bnd) {
#pragma unroll
      for (int k = 0; k < D; k++) w[k] = cadd(w[k], a.dst[at + (long)k * g.Vh]);
    }
  } else if (EPI == EPI_CLOVINV || EPI == EPI_CLOVPK) {
    if (a.dst2 && live) {
#pragma unroll
      for (int k = 0; k < D; k++) a.dst2[at + (long)k * g.Vh] = w[k];
    }
    if (EPI == EPI_CLOVPK) quad_cpk<D, R>(w, a.cpk, id - g.Vh, g.Vh, q);
    else quad_cinv<D, R>(w, a.cinv, id - g.Vh, g.Vh, q);
  } else {
    const bool add = !(bnd && a.zero_add_at_boundary);
    cplx<R> p[D];
#pragma unroll
    for (int k = 0; k < D; k++) p[k] = ldf<NC>(a.src2, at + (long)k * g.Vh);
    if (EPI == EPI_CLOVADD) {
      const R diag = a.diag + ((c[0] == g.Ta || c[0] == g.Tb) ? a.cfm1 : (R)0);
      quad_clover_add<D, R>(w, p, add, a.cl, g, id, diag, q);
    } else {
#pragma unroll
      for (int k = 0; k < D; k++)
        if (add) w[k] = cadd(w[k], cscale(p[k], a.diag));
    }
    if (a.g5 && q >= 2) {
#pragma unroll
      for (int k = 0; k < D; k++) w[k] = cscale(w[k], (R)-1);
    }
  }
}

template <int D, typename R, int EPI, bool REAL>
__global__ void __launch_bounds__(128) k_hop_quad(HopArgs<R> a) {
  const int t = (blockIdx.x * 128 + threadIdx.x) >> 2;
  const bool live = t < a.n;
  cplx<R> w[D];
  long at;
  hop_quad<D, R, EPI, true, REAL>(a, live ? t : a.n - 1, live, w, at);
  if (live) {
#pragma unroll
    for (int k = 0; k < D; k++) a.dst[at + (long)k * a.g.Vh] = w[k];
  }
}

// ------------------------------------------------------------------ colour-row hop
// The same operator with one warp per output colour: a block takes 32 sites, lane = site, warp i =
// colour i.  Each warp projects colour i of the eight neighbours into shared memory (2 spins x d
// colours per direction), then forms row i of the eight link products, so a thread keeps 4 complex
// accumulators where a thread per site keeps 4 d.  For d >= 8, where a thread per site lives in local
// memory: Hphi_sq, a thread per site / a warp per colour, d = 8 8^4 211 / 66 us, 16^4 562 / 503 us;
// d = 10 16^4 989 / 766 us; d = 15 8^4 1653 / 168 us, 16^4 2822 / 1416 us.  Up to d = 6 a thread per site
// is bound by HBM and faster (d = 3 32^4, before either loaded the clover entries once: 907 / 1126 us; d = 6
// 32 x 16^3: 423 / 532 us).
template <int D, typename R> struct RowTile {
  static constexpr int threads = 32 * D;
  // half spinors of four directions at a time (eight would leave one block per SM), later the 4 d words of a site
  static constexpr int words = 4 * 2 * D;
  static constexpr size_t smem = sizeof(cplx<R>) * 32 * words;
};

// half spinor (1 -+ g_mu) psi of one colour: SIG = -1 forward, +1 backward
template <int MU, int SIG, typename C>
__device__ __forceinline__ void row_project(C &h0, C &h1, C p0, C p1, C p2, C p3) {
  if (MU == 0) {
    h0 = SIG < 0 ? cadd(p0, p2) : csub(p0, p2);
    h1 = SIG < 0 ? cadd(p1, p3) : csub(p1, p3);
  } else if (MU == 1) {
    h0 = SIG < 0 ? cadd(p0, ctimesi(p3)) : csub(p0, ctimesi(p3));
    h1 = SIG < 0 ? cadd(p1, ctimesi(p2)) : csub(p1, ctimesi(p2));
  } else if (MU == 2) {
    h0 = SIG < 0 ? cadd(p0, p3) : csub(p0, p3);
    h1 = SIG < 0 ? csub(p1, p2) : cadd(p1, p2);
  } else {
    h0 = SIG < 0 ? cadd(p0, ctimesi(p2)) : csub(p0, ctimesi(p2));
    h1 = SIG < 0 ? csub(p1, ctimesi(p3)) : cadd(p1, ctimesi(p3));
  }
}

template <int D, typename R, int MU, int SIG>
__device__ __forceinline__ void row_gather(cplx<R> *sm, int slot, int i, int lane, const cplx<R> *src, const Geom &g,
                                           int nid) {
  const int blk = nid >= g.Vh;
  const cplx<R> *f = src + ((long)blk * 4 * D + i) * g.Vh + (nid - blk * g.Vh);
  const long st = (long)D * g.Vh;
  cplx<R> h0, h1;
  row_project<MU, SIG>(h0, h1, __ldg(f), __ldg(f + st), __ldg(f + 2 * st), __ldg(f + 3 * st));
  sm[((slot * 2 + 0) * D + i) * 32 + lane] = h0;
  sm[((slot * 2 + 1) * D + i) * 32 + lane] = h1;
}

// row i of U h (forward, link of the site) or U^dag h (backward, link of the neighbour), added
// to the four spin components
template <int D, typename R, int MU, int SIG, typename LP>
__device__ __forceinline__ void row_apply(cplx<R> (&acc)[4], const cplx<R> *sm, int slot, int i, int lane, LP U,
                                          const Geom &g, int lid) {
  const int blk = lid >= g.Vh;
  const LP u = U + ((long)(blk * 4 + MU) * D * D + (SIG < 0 ? i * D : i)) * g.Vh + (lid - blk * g.Vh);
  const long st = (long)(SIG < 0 ? 1 : D) * g.Vh;
  const cplx<R> *h = sm + slot * 2 * D * 32 + lane;
  cplx<R> c0 = mk<R>(0, 0), c1 = mk<R>(0, 0);
#pragma unroll
  for (int j = 0; j < D; j++) {
    const auto w = __ldg(u + j * st);
    const cplx<R> h0 = h[j * 32], h1 = h[(D + j) * 32];
    if constexpr (std::is_same_v<LP, const R *>) { rfma(c0, w, h0); rfma(c1, w, h1); }
    else if (SIG < 0) { cfma(c0, w, h0); cfma(c1, w, h1); }
    else { cfmac(c0, w, h0); cfmac(c1, w, h1); }
  }
  acc[0] = cadd(acc[0], c0);
  acc[1] = cadd(acc[1], c1);
  if (MU == 0) {
    acc[2] = SIG < 0 ? cadd(acc[2], c0) : csub(acc[2], c0);
    acc[3] = SIG < 0 ? cadd(acc[3], c1) : csub(acc[3], c1);
  } else if (MU == 1) {
    acc[2] = SIG < 0 ? cadd(acc[2], ctimesmi(c1)) : cadd(acc[2], ctimesi(c1));
    acc[3] = SIG < 0 ? cadd(acc[3], ctimesmi(c0)) : cadd(acc[3], ctimesi(c0));
  } else if (MU == 2) {
    acc[2] = SIG < 0 ? csub(acc[2], c1) : cadd(acc[2], c1);
    acc[3] = SIG < 0 ? cadd(acc[3], c0) : csub(acc[3], c0);
  } else {
    acc[2] = SIG < 0 ? cadd(acc[2], ctimesmi(c0)) : cadd(acc[2], ctimesi(c0));
    acc[3] = SIG < 0 ? cadd(acc[3], ctimesi(c1)) : cadd(acc[3], ctimesmi(c1));
  }
}

// Rows (spin 2b, colour i) and (spin 2b+1, colour i) of the packed Hermitian inverse blocks (layout of
// cpk_site) applied to the 4 D words x[(s * D + c) * 32]
template <int D, typename R>
__device__ __forceinline__ void row_cpk(cplx<R> (&out)[4], const cplx<R> *x, int i, const double2 *cpk, int h,
                                        int Vh) {
  constexpr int W = 2 * D * D;
#pragma unroll
  for (int b = 0; b < 2; b++) {
    const double2 *C = cpk + (long)b * W * Vh + h;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int r = q * D + i;
      const double2 dd = __ldg(C + (long)(r >> 1) * Vh);
      const cplx<R> xr = x[((2 * b + q) * D + i) * 32];
      cplx<R> y = cscale(xr, (R)((r & 1) ? dd.y : dd.x));
#pragma unroll
      for (int c = 0; c < 2 * D; c++) {
        if (c == r) continue;
        const int hi = c < r ? r : c, lo = c < r ? c : r;
        double2 m = __ldg(C + (long)(D + hi * (hi - 1) / 2 + lo) * Vh);
        if (c > r) m.y = -m.y;
        const cplx<R> v = x[(2 * b * D + c) * 32];
        cfma(y, mk<R>((R)m.x, (R)m.y), v);
      }
      out[2 * b + q] = y;
    }
  }
}

// row i of both explicit inverse blocks (FP32 inner operator)
template <int D, typename R>
__device__ __forceinline__ void row_cinv(cplx<R> (&out)[4], const cplx<R> *x, int i, const cplx<R> *cinv, int h,
                                         int Vh) {
  constexpr int N = 2 * D;
#pragma unroll
  for (int b = 0; b < 2; b++)
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const cplx<R> *C = cinv + ((long)b * N * N + (q * D + i) * N) * Vh + h;
      cplx<R> y = mk<R>(0, 0);
#pragma unroll
      for (int c = 0; c < N; c++) cfma(y, __ldg(C + (long)c * Vh), x[(2 * b * D + c) * 32]);
      out[2 * b + q] = y;
    }
}

// row i of the clover term (clover_site) applied to the 4 D words x, diag included; A0 and A2
// are Hermitian, so only their lower triangles are read
template <int D, typename R>
__device__ __forceinline__ void row_clover(cplx<R> (&out)[4], const cplx<R> *x, int i, const cplx<R> *cl,
                                           const Geom &g, int id, R diag) {
  const int blk = id >= g.Vh;
  const cplx<R> *C0 = cl + (long)blk * 4 * D * D * g.Vh + (id - blk * g.Vh);
#pragma unroll
  for (int b = 0; b < 2; b++) {
    const cplx<R> *A = C0 + (long)(2 * b) * D * D * g.Vh, *B = A + (long)D * D * g.Vh;
    cplx<R> o0 = cscale(x[(2 * b * D + i) * 32], diag), o1 = cscale(x[((2 * b + 1) * D + i) * 32], diag);
#pragma unroll
    for (int j = 0; j < D; j++) {
      const cplx<R> p0 = x[(2 * b * D + j) * 32], p1 = x[((2 * b + 1) * D + j) * 32];
      cplx<R> a = __ldg(A + (long)(j <= i ? i * D + j : j * D + i) * g.Vh);
      if (j > i) a.y = -a.y;
      const cplx<R> w = __ldg(B + (long)(i * D + j) * g.Vh), wt = __ldg(B + (long)(j * D + i) * g.Vh);
      cfma(o0, a, p0);
      cfma(o0, w, p1);
      cfmac(o1, wt, p0);
      o1 = csub(o1, cmul(a, p1));
    }
    out[2 * b] = o0;
    out[2 * b + 1] = o1;
  }
}

// One tile of 32 output sites [32 tile, 32 tile + 32) of the launch's range; every thread of the
// block takes part (lanes beyond the range work on its last site).  acc receives the four spins of
// the thread's colour, `at` the index of the first of them (the others follow at D Vh); false for a
// lane beyond the range, whose result the caller drops.
template <int D, typename R, int EPI, bool REAL>
__device__ __forceinline__ bool hop_rows(const HopArgs<R> &a, int tile, cplx<R> *sm, cplx<R> (&acc)[4], long &at) {
  const Geom &g = a.g;
  const auto U = hop_links<REAL>(a);
  const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
  const int t = tile * 32 + lane;
  const bool live = t < a.n;
  const int id = a.lo + (live ? t : a.n - 1);
  int c[4];
  coords_of(g, id, c);
  const bool bnd = spinor_zeroed(g, c[0]);
#pragma unroll
  for (int s = 0; s < 4; s++) acc[s] = mk<R>(0, 0);
  int f[4], b[4];
#pragma unroll
  for (int mu = 0; mu < 4; mu++) {
    f[mu] = neighbour(g, c, mu, +1);
    b[mu] = neighbour(g, c, mu, -1);
  }
  row_gather<D, R, 0, -1>(sm, 0, i, lane, a.src, g, f[0]);
  row_gather<D, R, 0, +1>(sm, 1, i, lane, a.src, g, b[0]);
  row_gather<D, R, 1, -1>(sm, 2, i, lane, a.src, g, f[1]);
  row_gather<D, R, 1, +1>(sm, 3, i, lane, a.src, g, b[1]);
  __syncthreads();
  row_apply<D, R, 0, -1>(acc, sm, 0, i, lane, U, g, id);
  row_apply<D, R, 0, +1>(acc, sm, 1, i, lane, U, g, b[0]);
  row_apply<D, R, 1, -1>(acc, sm, 2, i, lane, U, g, id);
  row_apply<D, R, 1, +1>(acc, sm, 3, i, lane, U, g, b[1]);
  __syncthreads();
  row_gather<D, R, 2, -1>(sm, 0, i, lane, a.src, g, f[2]);
  row_gather<D, R, 2, +1>(sm, 1, i, lane, a.src, g, b[2]);
  row_gather<D, R, 3, -1>(sm, 2, i, lane, a.src, g, f[3]);
  row_gather<D, R, 3, +1>(sm, 3, i, lane, a.src, g, b[3]);
  __syncthreads();
  row_apply<D, R, 2, -1>(acc, sm, 0, i, lane, U, g, id);
  row_apply<D, R, 2, +1>(acc, sm, 1, i, lane, U, g, b[2]);
  row_apply<D, R, 3, -1>(acc, sm, 2, i, lane, U, g, id);
  row_apply<D, R, 3, +1>(acc, sm, 3, i, lane, U, g, b[3]);
#pragma unroll
  for (int s = 0; s < 4; s++) acc[s] = bnd ? mk<R>(0, 0) : cscale(acc[s], a.coeff);

  const int blk = id >= g.Vh;
  const long st = (long)D * g.Vh;
  at = ((long)blk * 4 * D + i) * g.Vh + (id - blk * g.Vh);
  if (EPI == EPI_PLAIN) {
    if (a.assign && !bnd) {
#pragma unroll
      for (int s = 0; s < 4; s++) acc[s] = cadd(acc[s], a.dst[at + s * st]);
    }
    return live;
  }
  cplx<R> *x = sm + lane;                            // 4 D words per lane, after the last use of the half spinors
  if (EPI == EPI_CLOVINV || EPI == EPI_CLOVPK) {
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 4; s++) {
      if (a.dst2 && live) a.dst2[at + s * st] = acc[s];
      x[(s * D + i) * 32] = acc[s];
    }
    __syncthreads();
    if (EPI == EPI_CLOVPK) row_cpk<D, R>(acc, x, i, a.cpk, id - g.Vh, g.Vh);
    else row_cinv<D, R>(acc, x, i, a.cinv, id - g.Vh, g.Vh);
  } else {
    const bool zero_add = bnd && a.zero_add_at_boundary;
    cplx<R> p[4];
#pragma unroll
    for (int s = 0; s < 4; s++) p[s] = __ldg(a.src2 + at + s * st);
    if (EPI == EPI_CLOVADD) {
      const R diag = a.diag + ((c[0] == g.Ta || c[0] == g.Tb) ? a.cfm1 : (R)0);
      __syncthreads();
#pragma unroll
      for (int s = 0; s < 4; s++) x[(s * D + i) * 32] = p[s];
      __syncthreads();
      row_clover<D, R>(p, x, i, a.cl, g, id, diag);
    } else {
#pragma unroll
      for (int s = 0; s < 4; s++) p[s] = cscale(p[s], a.diag);
    }
#pragma unroll
    for (int s = 0; s < 4; s++) {
      if (!zero_add) acc[s] = cadd(acc[s], p[s]);
      if (a.g5 && s >= 2) acc[s] = cscale(acc[s], (R)-1);
    }
  }
  return live;
}

template <int D, typename R, int EPI, bool REAL>
__global__ void __launch_bounds__(32 * D) k_hop_rows(HopArgs<R> a) {
  extern __shared__ __align__(16) unsigned char hop_smem[];
  cplx<R> acc[4];
  long at;
  if (hop_rows<D, R, EPI, REAL>(a, blockIdx.x, reinterpret_cast<cplx<R> *>(hop_smem), acc, at)) {
#pragma unroll
    for (int s = 0; s < 4; s++) a.dst[at + s * (long)D * a.g.Vh] = acc[s];
  }
}

// clover_kernel (dirac.cpp:25-107) standalone: dst (=|+=) A psi over [lo, lo+n)
template <int D>
__global__ void __launch_bounds__(128) k_clover(double2 *dst, const double2 *src, const double2 *cl, Geom g,
                                                double mass4, double cfm1, int lo, int n, int assign) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  int id = lo + t;
  int c[4];
  coords_of(g, id, c);
  double diag = mass4 + ((c[0] == g.Ta || c[0] == g.Tb) ? cfm1 : 0.0);
  double2 s[4][D], o[4][D];
  load_spinor<D, double>(s, src, g, id);
  clover_site<D, double>(o, s, cl, g, id, diag);
  if (assign) {
    double2 old[4][D];
    load_spinor<D, double>(old, dst, g, id);
#pragma unroll
    for (int a = 0; a < 4; a++) {
      YG_UNROLL_D
      for (int k = 0; k < D; k++) o[a][k] = cadd(o[a][k], old[a][k]);
    }
  }
  store_spinor<D, double>(dst, o, g, id);
}

// clover_inv_kernel (dirac.cpp:109-225) standalone, sites of block 1
template <int D>
__global__ void __launch_bounds__(128) k_clover_inv(double2 *dst, const double2 *src, const double2 *ldl, Geom g,
                                                    int assign) {
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= g.Vh) return;
  int id = g.Vh + h;
  double2 s[4][D], o[4][D];
  load_spinor<D, double>(s, src, g, id);
  ldl_site<D, double>(o, s, ldl, h, g.Vh);
  if (assign) {
    double2 old[4][D];
    load_spinor<D, double>(old, dst, g, id);
#pragma unroll
    for (int a = 0; a < 4; a++) {
      YG_UNROLL_D
      for (int k = 0; k < D; k++) o[a][k] = cadd(o[a][k], old[a][k]);
    }
  }
  store_spinor<D, double>(dst, o, g, id);
}

// _compute_ldl_decomp (clover.cpp:25-91) with ldl() of solver.cpp:97-117, one thread per
// site of block 1 (the odd sites with even-odd ordering; odd_sites_for in geometry.h:18-19) and
// spin block (blockIdx.y)
template <int D>
__global__ void k_ldl(double2 *ldl, const double2 *cl, Geom g, double sigma, double cf_in, int boundary_term) {
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= g.Vh) return;
  int id = g.Vh + h;
  constexpr int N = 2 * D;
  constexpr int P = D * (2 * D + 1);
  double cf = 0;
  if (boundary_term) {
    int c[4];
    coords_of(g, id, c);
    if (c[0] == g.Ta || c[0] == g.Tb) cf = cf_in - 1.0;
  }
  {
    const int blk = blockIdx.y;
    double2 A[N * N];
    for (int k = 0; k < N * N; k++) A[k] = make_double2(0, 0);
    int m0 = blk ? 2 : 0, m1 = blk ? 3 : 1;
    for (int i = 0; i < D; i++)
      for (int j = 0; j < D; j++) {
        A[(i + D) * N + j] = cconj(cl[fidx(g, id, m1 * D * D + j * D + i, 4 * D * D)]);
        if (i >= j) {
          double2 a = cl[fidx(g, id, m0 * D * D + i * D + j, 4 * D * D)];
          A[i * N + j] = a;
          A[(i + D) * N + D + j] = make_double2(-a.x, -a.y);
          if (i == j) {
            A[i * N + j].x += sigma + cf;
            A[(i + D) * N + D + j].x += sigma + cf;
          }
        }
      }
    for (int i = 0; i < N; i++) {
      for (int k = 0; k < i; k++)
        A[i * N + i].x -= (A[i * N + k].x * A[i * N + k].x + A[i * N + k].y * A[i * N + k].y) * A[k * N + k].x;
      for (int j = i + 1; j < N; j++) {
        for (int k = 0; k < i; k++) {
          double2 t = cmul(A[j * N + k], cconj(A[i * N + k]));
          A[j * N + i] = csub(A[j * N + i], cscale(t, A[k * N + k].x));
        }
        A[j * N + i] = cscale(A[j * N + i], 1.0 / A[i * N + i].x);
      }
    }
    int k = 0;
    for (int i = 0; i < N; i++)
      for (int j = 0; j <= i; j++, k++) ldl[((long)blk * P + k) * g.Vh + h] = A[i * N + j];
  }
}

// LDL factors and packed inverse (layout of cpk_site) of one clover block in one pass for d <= 3:
// a thread takes one of the two blocks of a site with everything in registers.  With A = L D L^dag,
// M = L^-1 replaces L and A^-1(i, j) = sum_{k >= i} conj(M(k, i)) M(k, j) / D_k for i >= j.
// Bound by its 1.8 kB a site.  32 x 16^3: 16 us; factors and inverse column by column in local memory
// took 37 + 84 us.
template <int D>
__global__ void __launch_bounds__(128) k_ldl_inverse(double2 *ldl, double2 *cpk, const double2 *cl, Geom g, double sigma,
                                                     double cf_in, int boundary_term) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x, blk = blockIdx.y;
  if (h >= g.Vh) return;
  const int id = g.Vh + h;
  constexpr int N = 2 * D, P = D * (2 * D + 1), W = 2 * D * D;
  double shift = sigma;
  if (boundary_term) {
    int c[4];
    coords_of(g, id, c);
    if (c[0] == g.Ta || c[0] == g.Tb) shift += cf_in - 1.0;
  }
  double dg[N];              // the diagonal, then D
  double2 A[N * (N - 1) / 2];   // strict lower triangle, row by row
#pragma unroll
  for (int i = 0; i < D; i++) {
#pragma unroll
    for (int j = 0; j <= i; j++) {
      const double2 a = __ldg(cl + fidx(g, id, 2 * blk * D * D + i * D + j, 4 * D * D));
      if (i == j) {
        dg[i] = a.x + shift;
        dg[i + D] = shift - a.x;
      } else {
        A[i * (i - 1) / 2 + j] = a;
        A[(i + D) * (i + D - 1) / 2 + D + j] = make_double2(-a.x, -a.y);
      }
    }
#pragma unroll
    for (int j = 0; j < D; j++)
      A[(i + D) * (i + D - 1) / 2 + j] = cconj(__ldg(cl + fidx(g, id, (2 * blk + 1) * D * D + j * D + i, 4 * D * D)));
  }
#pragma unroll
  for (int i = 0; i < N; i++) {
#pragma unroll
    for (int k = 0; k < i; k++) {
      const double2 l = A[i * (i - 1) / 2 + k];
      dg[i] -= (l.x * l.x + l.y * l.y) * dg[k];
    }
    const double r = 1.0 / dg[i];
#pragma unroll
    for (int j = i + 1; j < N; j++) {
      double2 v = A[j * (j - 1) / 2 + i];
#pragma unroll
      for (int k = 0; k < i; k++)
        v = csub(v, cscale(cmul(A[j * (j - 1) / 2 + k], cconj(A[i * (i - 1) / 2 + k])), dg[k]));
      A[j * (j - 1) / 2 + i] = cscale(v, r);
    }
  }
  double2 *Lb = ldl + (long)blk * P * g.Vh + h;
#pragma unroll
  for (int i = 0; i < N; i++) {
#pragma unroll
    for (int j = 0; j < i; j++) Lb[(long)(i * (i + 1) / 2 + j) * g.Vh] = A[i * (i - 1) / 2 + j];
    Lb[(long)(i * (i + 1) / 2 + i) * g.Vh] = make_double2(dg[i], 0.0);
  }
  // M = L^-1, row by row in place: M(i, j) = -L(i, j) - sum_{j < k < i} L(i, k) M(k, j)
#pragma unroll
  for (int i = 1; i < N; i++) {
    double2 row[N];
#pragma unroll
    for (int j = 0; j < i; j++) {
      double2 v = A[i * (i - 1) / 2 + j];
#pragma unroll
      for (int k = j + 1; k < i; k++) cfma(v, A[i * (i - 1) / 2 + k], A[k * (k - 1) / 2 + j]);
      row[j] = make_double2(-v.x, -v.y);
    }
#pragma unroll
    for (int j = 0; j < i; j++) A[i * (i - 1) / 2 + j] = row[j];
  }
#pragma unroll
  for (int i = 0; i < N; i++) dg[i] = 1.0 / dg[i];
  double2 *Cb = cpk + (long)blk * W * g.Vh + h;
#pragma unroll
  for (int w = 0; w < D; w++) {
    double2 dd;
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int i = 2 * w + q;
      double v = dg[i];
#pragma unroll
      for (int k = i + 1; k < N; k++) {
        const double2 m = A[k * (k - 1) / 2 + i];
        v = fma(m.x * m.x + m.y * m.y, dg[k], v);
      }
      if (q) dd.y = v; else dd.x = v;
    }
    Cb[(long)w * g.Vh] = dd;
  }
#pragma unroll
  for (int i = 1; i < N; i++)
#pragma unroll
    for (int j = 0; j < i; j++) {
      double2 v = cscale(A[i * (i - 1) / 2 + j], dg[i]);          // k = i: M(i, i) = 1
#pragma unroll
      for (int k = i + 1; k < N; k++)
        v = cadd(v, cscale(cmulc(A[k * (k - 1) / 2 + i], A[k * (k - 1) / 2 + j]), dg[k]));
      Cb[(long)(D + i * (i - 1) / 2 + j) * g.Vh] = v;
    }
}

// explicit inverse of both clover blocks in FP32, from the FP64 LDL factors
template <int D>
__global__ void k_cinv_float(float2 *cinv, const double2 *ldl, int Vh) {
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= Vh) return;
  constexpr int N = 2 * D, P = D * (2 * D + 1);
  for (int blk = 0; blk < 2; blk++) {
    const double2 *Lb = ldl + (long)blk * P * Vh + h;
    for (int col = 0; col < N; col++) {
      double2 x[N];
      for (int i = 0; i < N; i++) x[i] = make_double2(i == col ? 1.0 : 0.0, 0.0);
      for (int i = 1; i < N; i++)
        for (int k = 0; k < i; k++) x[i] = csub(x[i], cmul(Lb[(long)(i * (i + 1) / 2 + k) * Vh], x[k]));
      for (int i = N - 1; i >= 0; i--) {
        x[i] = cscale(x[i], 1.0 / Lb[(long)(i * (i + 1) / 2 + i) * Vh].x);
        for (int k = i + 1; k < N; k++) x[i] = csub(x[i], cmulc(Lb[(long)(k * (k + 1) / 2 + i) * Vh], x[k]));
      }
      for (int i = 0; i < N; i++)
        cinv[((long)blk * N * N + i * N + col) * Vh + h] = make_float2((float)x[i].x, (float)x[i].y);
    }
  }
}

// packed Hermitian FP64 inverse of both clover blocks (layout of cpk_site) from the LDL factors, for
// d > 3: a thread per site, block and column (blockIdx.y = block * 2d + column) solves by forward
// substitution, D^-1 and back substitution
template <int D>
__global__ void __launch_bounds__(64) k_cinv_packed64(double2 *cpk, const double2 *ldl, int Vh) {
  const int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= Vh) return;
  constexpr int N = 2 * D, P = D * (2 * D + 1), W = 2 * D * D;
  const int blk = blockIdx.y / N, col = blockIdx.y % N;
  const double2 *Lb = ldl + (long)blk * P * Vh + h;
  double2 *Cb = cpk + (long)blk * W * Vh + h;
  double2 x[N];
  x[col] = make_double2(1.0, 0.0);
  for (int i = col + 1; i < N; i++) {
    double2 v = make_double2(0.0, 0.0);
    for (int k = col; k < i; k++) v = csub(v, cmul(Lb[(long)(i * (i + 1) / 2 + k) * Vh], x[k]));
    x[i] = v;
  }
  for (int i = N - 1; i >= col; i--) {
    double2 v = cscale(x[i], 1.0 / Lb[(long)(i * (i + 1) / 2 + i) * Vh].x);
    for (int k = i + 1; k < N; k++) v = csub(v, cmulc(Lb[(long)(k * (k + 1) / 2 + i) * Vh], x[k]));
    x[i] = v;
  }
  // diagonal entry (col, col): real part into its half of word col/2
  double *dw = reinterpret_cast<double *>(Cb + (long)(col / 2) * Vh);
  dw[col & 1] = x[col].x;
  for (int i = col + 1; i < N; i++) Cb[(long)(D + i * (i - 1) / 2 + col) * Vh] = x[i];
}

// log prod_n D_nn of both blocks per site (clover_logdet, clover.cpp:281-305)
template <int D>
__global__ void k_logdet(double *out, const double2 *ldl, int Vh) {
  int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= Vh) return;
  constexpr int N = 2 * D, P = D * (2 * D + 1);
  double prod = 1;
  for (int n = 0; n < N; n++) {
    prod *= ldl[((long)0 * P + n * (n + 1) / 2 + n) * Vh + h].x;
    prod *= ldl[((long)1 * P + n * (n + 1) / 2 + n) * Vh + h].x;
  }
  out[h] = log(prod);
}

// ------------------------------------------------------------------ DK<D> launchers
template <int D, typename R, int EPI, bool REAL>
static void launch_hop_links(const HopArgs<R> &a, cudaStream_t s) {
  if constexpr (D <= 6) {
    if (a.n <= kQuadSites) k_hop_quad<D, R, EPI, REAL><<<nblk(4L * a.n, 128), 128, 0, s>>>(a);
    else k_hop<D, R, EPI, REAL><<<nblk(a.n, 128), 128, 0, s>>>(a);
  } else {
    using T = RowTile<D, R>;
    if (T::smem > 48 * 1024)
      check_cuda(cudaFuncSetAttribute(k_hop_rows<D, R, EPI, REAL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)T::smem), "operator shared memory");
    k_hop_rows<D, R, EPI, REAL><<<nblk(a.n, 32), T::threads, T::smem, s>>>(a);
  }
}

// d = 3, 8 and 15 are the adjoint dimensions of SU(2), SU(3) and SU(4); d = 8 and 15 are nothing else
template <int D, typename R, int EPI>
static void launch_hop(const HopArgs<R> &a, cudaStream_t s) {
  constexpr bool fp64 = sizeof(R) == sizeof(double);
  if constexpr (fp64 && (D == 8 || D == 15)) {
    launch_hop_links<D, R, EPI, true>(a, s);
  } else {
    if constexpr (fp64 && D == 3) {
      if (a.Ur) {
        launch_hop_links<D, R, EPI, true>(a, s);
        return;
      }
    }
    launch_hop_links<D, R, EPI, false>(a, s);
  }
}

template <int D, typename R>
static void launch_hop_epi(const HopArgs<R> &a, int epi, cudaStream_t s) {
  constexpr int kInverse = sizeof(R) == sizeof(double) ? EPI_CLOVPK : EPI_CLOVINV;
  switch (epi) {
    case EPI_PLAIN: launch_hop<D, R, EPI_PLAIN>(a, s); break;
    case kInverse: launch_hop<D, R, kInverse>(a, s); break;
    case EPI_CLOVADD: launch_hop<D, R, EPI_CLOVADD>(a, s); break;
    default: launch_hop<D, R, EPI_AXPY>(a, s); break;
  }
}

template <int D>
void DK<D>::hop(const HopArgs<double> &a, int epi, cudaStream_t s) { launch_hop_epi<D, double>(a, epi, s); }

template <int D>
void DK<D>::hop(const HopArgs<float> &a, int epi, cudaStream_t s) { launch_hop_epi<D, float>(a, epi, s); }

template <int D>
void DK<D>::clover(double2 *dst, const double2 *src, const double2 *cl, Geom g, double mass4, double cfm1, int lo,
                   int n, int assign, cudaStream_t s) {
  k_clover<D><<<nblk(n, 128), 128, 0, s>>>(dst, src, cl, g, mass4, cfm1, lo, n, assign);
}

template <int D>
void DK<D>::clover_inv(double2 *dst, const double2 *src, const double2 *ldl, Geom g, int assign, cudaStream_t s) {
  k_clover_inv<D><<<nblk(g.Vh, 128), 128, 0, s>>>(dst, src, ldl, g, assign);
}

template <int D>
void DK<D>::ldl_inverse(double2 *ldl, double2 *cpk, const double2 *cl, Geom g, double sigma, double cf, int boundary_term,
                        cudaStream_t s) {
  if constexpr (D <= 3) {      // the 6 x 6 block and its inverse fit one thread's registers
    k_ldl_inverse<D><<<dim3(nblk(g.Vh, 128), 2), 128, 0, s>>>(ldl, cpk, cl, g, sigma, cf, boundary_term);
  } else {
    k_ldl<D><<<dim3(nblk(g.Vh, 64), 2), 64, 0, s>>>(ldl, cl, g, sigma, cf, boundary_term);
    k_cinv_packed64<D><<<dim3(nblk(g.Vh, 64), 4 * D), 64, 0, s>>>(cpk, ldl, g.Vh);
  }
}

template <int D>
void DK<D>::cinv_float(float2 *cinv, const double2 *ldl, int Vh, cudaStream_t s) {
  k_cinv_float<D><<<nblk(Vh, 64), 64, 0, s>>>(cinv, ldl, Vh);
}

template <int D>
void DK<D>::logdet(double *out, const double2 *ldl, int Vh, cudaStream_t s) {
  k_logdet<D><<<nblk(Vh, 128), 128, 0, s>>>(out, ldl, Vh);
}

}  // namespace yg
