// Device code of the fermion forces and the gauge-side support kernels (included by the
// yg_inst_*_aux.cu units).
//
//   clover_fermion_force   forces.cpp:122-172   sigma_{mu nu} gamma5 outer products -> cl_force
//   hopping force          forces.cpp:175-227   Proj_TA[ U(x,mu) fmat ] -> momenta
//   compute_clover_force   clover.cpp:170-279   coeff * A_oo^-1 from the packed inverse -> cl_force
//   clover_force_core      forces.cpp:33-106    6-link assembly of cl_force -> momenta
//   wilson_gauge_force     forces.cpp:262-283   plaquette staples -> momenta
//   avr_wilson(1,1)        wilsonloop.cpp:116-133
// Momenta keep the reference's host layout afield_momenta[4*id+mu].av[NG]; FP64 throughout.
#pragma once

#include "yg_kernels.h"

namespace yg {

template <int D>
__device__ __forceinline__ void ld_spinor64(double2 (&s)[4][D], const double2 *f, const Geom &g, int id) {
#pragma unroll
  for (int sp = 0; sp < 4; sp++) {
    YG_UNROLL_DF
    for (int c = 0; c < D; c++) s[sp][c] = f[fidx(g, id, sp * D + c, 4 * D)];
  }
}

// Spinor::g5_sigma(mu,nu) for the clover-force slot order (0,1),(0,2),(1,2),(0,3),(1,3),(2,3)
// (spinor.cpp:266-438, forces.cpp:130-170)
template <int D>
__device__ __forceinline__ void g5_sigma(double2 (&o)[4][D], const double2 (&s)[4][D], int slot) {
  YG_UNROLL_DF
  for (int c = 0; c < D; c++) {
    switch (slot) {
      case 0: o[0][c] = ctimesmi(s[1][c]); o[1][c] = ctimesmi(s[0][c]); o[2][c] = ctimesmi(s[3][c]); o[3][c] = ctimesmi(s[2][c]); break;
      case 1: o[0][c] = cscale(s[1][c], -1.0); o[1][c] = s[0][c]; o[2][c] = cscale(s[3][c], -1.0); o[3][c] = s[2][c]; break;
      case 2: o[0][c] = ctimesi(s[0][c]); o[1][c] = ctimesmi(s[1][c]); o[2][c] = ctimesmi(s[2][c]); o[3][c] = ctimesi(s[3][c]); break;
      case 3: o[0][c] = ctimesmi(s[0][c]); o[1][c] = ctimesi(s[1][c]); o[2][c] = ctimesmi(s[2][c]); o[3][c] = ctimesi(s[3][c]); break;
      case 4: o[0][c] = cscale(s[1][c], -1.0); o[1][c] = s[0][c]; o[2][c] = s[3][c]; o[3][c] = cscale(s[2][c], -1.0); break;
      default: o[0][c] = ctimesi(s[1][c]); o[1][c] = ctimesi(s[0][c]); o[2][c] = ctimesmi(s[3][c]); o[3][c] = ctimesmi(s[2][c]); break;
    }
  }
}

// gamma5 (1 - gamma_mu) (Spinor::g5_one_minus_gamma, spinor.cpp:440-500)
template <int D>
__device__ __forceinline__ void g5_omg(double2 (&o)[4][D], const double2 (&s)[4][D], int mu) {
  YG_UNROLL_DF
  for (int c = 0; c < D; c++) {
    double2 a, b;
    switch (mu) {
      case 0: a = cadd(s[0][c], s[2][c]); b = cadd(s[1][c], s[3][c]);
        o[0][c] = a; o[1][c] = b; o[2][c] = cscale(a, -1.0); o[3][c] = cscale(b, -1.0); break;
      case 1: o[0][c] = cadd(s[0][c], ctimesi(s[3][c])); o[1][c] = cadd(s[1][c], ctimesi(s[2][c]));
        o[2][c] = csub(ctimesi(s[1][c]), s[2][c]); o[3][c] = csub(ctimesi(s[0][c]), s[3][c]); break;
      case 2: o[0][c] = cadd(s[0][c], s[3][c]); o[1][c] = csub(s[1][c], s[2][c]);
        o[2][c] = csub(s[1][c], s[2][c]); o[3][c] = cscale(cadd(s[3][c], s[0][c]), -1.0); break;
      default: o[0][c] = cadd(s[0][c], ctimesi(s[2][c])); o[1][c] = csub(s[1][c], ctimesi(s[3][c]));
        o[2][c] = csub(ctimesi(s[0][c]), s[2][c]); o[3][c] = cscale(cadd(s[3][c], ctimesi(s[1][c])), -1.0); break;
    }
  }
}

template <int D>
__device__ __forceinline__ void scale_spinor(double2 (&s)[4][D], double w) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    YG_UNROLL_DF
    for (int c = 0; c < D; c++) s[k][c] = cscale(s[k][c], w);
  }
}

// fmat[i][j] += sum_k a[k][i] conj(b[k][j])  (fmat_create, forces.cpp:13-30)
template <int D>
__device__ __forceinline__ void outer_acc(double2 (&f)[D * D], const double2 (&a)[4][D], const double2 (&b)[4][D]) {
  YG_UNROLL_DF
  for (int i = 0; i < D; i++) {
    YG_UNROLL_DF
    for (int j = 0; j < D; j++) {
#pragma unroll
      for (int k = 0; k < 4; k++) cfma(f[i * D + j], a[k][i], cconj(b[k][j]));
    }
  }
}

// Re tr(iT[a] m).  The colour loops are unrolled for d <= 6, so that m stays in registers, and rolled above;
// every lane reads the same generator entries.
template <int D>
__device__ __forceinline__ double gen_trace(const double2 (&m)[D * D], const double2 *gens, int a) {
  const double2 *t = gens + a * D * D;
  double tr = 0;
  YG_UNROLL_DF
  for (int i = 0; i < D; i++) {
    YG_UNROLL_DF
    for (int k = 0; k < D; k++) {
      const double2 w = __ldg(t + i * D + k), v = m[k * D + i];
      tr = fma(w.x, v.x, fma(-w.y, v.y, tr));
    }
  }
  return tr;
}

// av[a] += coeff/(-TF) * Re tr(iT[a] m)   (algebra_project, suNa.cpp:91-111), TF = 2.  TRACE = false
// leaves the unrolling to the compiler, which is faster for large matrices in local memory: clover force of
// d = 8 12^4 28.6 ms, 30.0 with rolled loops; d = 15 8^4 60.6, 66.5 (the hopping force of d = 8, and of
// d = 10 with several poles, is faster with them: 12^4 12 poles d = 8 4.0 ms / 5.2, d = 10 7.7 / 10.6)
template <int D, bool TRACE = (D <= 6)>
__device__ __forceinline__ void project_add(double *mom, const double2 (&m)[D * D], const double2 *gens, int ng,
                                            double coeff) {
  const double c = coeff / -2.0;
  if constexpr (TRACE) {
#pragma unroll 1
    for (int a = 0; a < ng; a++) mom[a] += c * gen_trace<D>(m, gens, a);
  } else {
    for (int a = 0; a < ng; a++) {
      double tr = 0;
      for (int i = 0; i < D; i++)
        for (int k = 0; k < D; k++) {
          const double2 t = gens[(a * D + i) * D + k], v = m[k * D + i];
          tr = fma(t.x, v.x, fma(-t.y, v.y, tr));
        }
      mom[a] += c * tr;
    }
  }
}

template <int D>
__device__ __forceinline__ void ld_mat(double2 (&m)[D * D], const double2 *base, const Geom &g, int id, int slot,
                                       int nslots) {
  YG_UNROLL_DF
  for (int k = 0; k < D * D; k++) m[k] = base[fidx(g, id, slot * D * D + k, nslots * D * D)];
}

template <int D>
__device__ __forceinline__ void mat_mul(double2 (&c)[D * D], const double2 (&a)[D * D], const double2 (&b)[D * D]) {
  YG_UNROLL_DF
  for (int i = 0; i < D; i++) {
    YG_UNROLL_DF
    for (int j = 0; j < D; j++) {
      double2 s = make_double2(0, 0);
      YG_UNROLL_DF
      for (int k = 0; k < D; k++) cfma(s, a[i * D + k], b[k * D + j]);
      c[i * D + j] = s;
    }
  }
}

template <int D>
__device__ __forceinline__ void dag(double2 (&c)[D * D], const double2 (&a)[D * D]) {
  YG_UNROLL_DF
  for (int i = 0; i < D; i++) {
    YG_UNROLL_DF
    for (int j = 0; j < D; j++) c[i * D + j] = cconj(a[j * D + i]);
  }
}

// X <- M X (DAG: M^dag X) for the matrix M of record (id, slot), in place column by column: the
// chains of products below are written as such left multiplications, so that a thread holds the
// running product, one sum and one loaded matrix (d = 3: 168 registers and 0.3 to 0.6 kB of spills).
// Only with the colour loops unrolled: with rolled loops (d >= 8) nvcc 12.9 compiles a chain that
// alternates lmul and lmul_add (lmul, lmul_add, lmul on one running product) to wrong results, while
// each alone, the same source on the host (under the address and undefined-behaviour sanitizers) and a
// build without the front end's optimizations are right.
template <int D, bool DAG>
__device__ __forceinline__ void lmul(double2 (&X)[D * D], const double2 *base, const Geom &g, int id, int slot,
                                     int nslots) {
  static_assert(D <= 6, "unrolled colour loops only");
  double2 M[D * D];
  asm volatile("" ::: "memory");     // M's loads stay behind the previous product: hoisting them all costs spills
  ld_mat<D>(M, base, g, id, slot, nslots);
  YG_UNROLL_DF
  for (int j = 0; j < D; j++) {
    double2 v[D];
    YG_UNROLL_DF
    for (int i = 0; i < D; i++) {
      double2 t = make_double2(0, 0);
      YG_UNROLL_DF
      for (int k = 0; k < D; k++) {
        if (DAG) cfmac(t, M[k * D + i], X[k * D + j]);
        else cfma(t, M[i * D + k], X[k * D + j]);
      }
      v[i] = t;
    }
    YG_UNROLL_DF
    for (int i = 0; i < D; i++) X[i * D + j] = v[i];
  }
}

// t += M X
template <int D>
__device__ __forceinline__ void lmul_add(double2 (&t)[D * D], const double2 (&X)[D * D], const double2 *base,
                                         const Geom &g, int id, int slot, int nslots) {
  static_assert(D <= 6, "unrolled colour loops only");
  double2 M[D * D];
  asm volatile("" ::: "memory");
  ld_mat<D>(M, base, g, id, slot, nslots);
  YG_UNROLL_DF
  for (int i = 0; i < D; i++) {
    YG_UNROLL_DF
    for (int j = 0; j < D; j++) {
      YG_UNROLL_DF
      for (int k = 0; k < D; k++) cfma(t[i * D + j], M[i * D + k], X[k * D + j]);
    }
  }
}

// the same into shared memory: out[a * OST] = coeff/(-TF) * Re tr(iT[a] m)
template <int D, int OST>
__device__ __forceinline__ void project_store(double *out, const double2 (&m)[D * D], const double2 *gens, int ng,
                                              double coeff) {
  const double c = coeff / -2.0;
#pragma unroll 1
  for (int a = 0; a < ng; a++) out[a * OST] = c * gen_trace<D>(m, gens, a);
}

// Force kernels take 32 consecutive sites per block, lane = site, so that every field, link and
// cl_force access of a warp is a contiguous run, with one warp per direction (and plane).  The
// per-link algebra components go through shared memory: acc[(warp * ng + a) * 33 + lane]
// (a stride of 33 doubles), NW warps per direction summed in order, then the block adds its
// 32 sites x NMU directions of momenta (the AoS records [site][mu][a]) in one coalesced pass.
template <int NMU, int NW>
__device__ __forceinline__ void add_momenta(double *mom, const double *acc, const Geom &g, int site0, int mu0, int ng) {
  __syncthreads();
  for (int e = threadIdx.x; e < 32 * NMU * ng; e += blockDim.x) {
    const int a = e % ng, mu = (e / ng) % NMU, lane = e / (ng * NMU);
    if (site0 + lane >= g.V) continue;
    double v = 0;
#pragma unroll
    for (int w = 0; w < NW; w++) v += acc[((mu * NW + w) * ng + a) * 33 + lane];
    mom[((long)(site0 + lane) * 4 + mu0 + mu) * ng + a] += v;
  }
}

constexpr size_t momenta_smem(int warps, int ng) { return sizeof(double) * 33 * warps * ng; }

// ---- clover_fermion_force, forces.cpp:122-172 (all sites), summed over the poles of a
// rational approximation (rhmc.cpp:86-106 calls wilson_fermion_force_q once per pole; one pole
// is the plain force): cl_force is read and written once, 1728 B a site for d = 3, which bounds it.
// fmat of one slot and the poles, added to cl_force
template <int D>
__device__ __forceinline__ void clover_slot_force(double2 *clf, const PoleSet &ps, const Geom &g, int id, int slot) {
  double2 f[D * D];
  YG_UNROLL_DF
  for (int k = 0; k < D * D; k++) f[k] = make_double2(0, 0);
#pragma unroll 1
  for (int n = 0; n < ps.n; n++) {
    double2 l[4][D], r[4][D], s[4][D];
    ld_spinor64<D>(l, ps.lhs[n], g, id);
    ld_spinor64<D>(r, ps.rhs[n], g, id);
    g5_sigma<D>(s, l, slot);
    scale_spinor<D>(s, ps.w[n]);
    outer_acc<D>(f, s, r);
    g5_sigma<D>(s, r, slot);
    scale_spinor<D>(s, ps.w[n]);
    outer_acc<D>(f, s, l);
  }
  YG_UNROLL_DF
  for (int k = 0; k < D * D; k++) {
    long ix = fidx(g, id, slot * D * D + k, 6 * D * D);
    double2 o = clf[ix];
    o.x += f[k].x;
    o.y += f[k].y;
    clf[ix] = o;
  }
}

// row i of the same, in d registers: the spinors come from L1
template <int D>
__device__ __forceinline__ void clover_slot_row(double2 *clf, const PoleSet &ps, const Geom &g, int id, int i, int slot) {
  double2 f[D];
  YG_UNROLL_DF
  for (int j = 0; j < D; j++) f[j] = make_double2(0, 0);
#pragma unroll 1
  for (int n = 0; n < ps.n; n++) {
    double2 l[4][1], r[4][1], sl[4][1], sr[4][1];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      l[k][0] = cscale(ps.lhs[n][fidx(g, id, k * D + i, 4 * D)], ps.w[n]);
      r[k][0] = cscale(ps.rhs[n][fidx(g, id, k * D + i, 4 * D)], ps.w[n]);
    }
    g5_sigma<1>(sl, l, slot);
    g5_sigma<1>(sr, r, slot);
    YG_UNROLL_DF
    for (int j = 0; j < D; j++) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        cfma(f[j], sl[k][0], cconj(ps.rhs[n][fidx(g, id, k * D + j, 4 * D)]));
        cfma(f[j], sr[k][0], cconj(ps.lhs[n][fidx(g, id, k * D + j, 4 * D)]));
      }
    }
  }
  YG_UNROLL_DF
  for (int j = 0; j < D; j++) {
    const long ix = fidx(g, id, slot * D * D + i * D + j, 6 * D * D);
    clf[ix] = cadd(clf[ix], f[j]);
  }
}

// Three splits.  Small lattices, and d >= 8 always: d <= 3 a warp per slot of 32 sites with a constant slot
// (sigma psi is a renaming of psi's registers), d >= 4, where that spills, a warp per slot and row
// (blockIdx.y).  Larger lattices, one pole: a thread a site, slot after slot (k_clover_fermion_site).
// Larger lattices, several poles: as on small ones, d = 4 and 6 a thread per site and slot
// (k_clover_fermion_slots).  One pole, warps / a thread a site, us with the operands in L2 where they fit,
// and from DRAM:
//   d = 1 16^4 9.2/9.0 and 13.2/12.3, 20 x 16^3 10.2/9.0 and 13.1/13.1, 24^4 20.8/16.2;
//   d = 2 12^4 10.1/12.3 and 15.2/21.4, 16^4 17.3/20.5 and 27.6/37.7, 32 x 16^3 33.7/31.4 and 50.1/56.3, 24^4 112/111;
//   d = 3 8^4 11/31, 16 x 12^3 23.5/19.4 and 33.8/39.9, 16^4 52.0/41.9 and 70.6/74.7, 20 x 16^3 86/93 and 89/103,
//         32 x 16^3 132/139, 32 x 20^2 x 16 204/207, 32 x 20^3 250/246, 24^4 320/312, 32 x 24^3 427/414;
//   d = 4 8^4 12.4/52.7, 16^4 116/123, 24 x 16^3 205/183;
//   d = 6 8^4 23/119, 12^4 96/121, 16 x 12^3 145/144, 16^4 419/292;  d = 8 12^4 125/665.
// At d = 3 a thread a site, which reads the spinors once instead of six times, wins where everything stays in
// L2 (1.25 kB a site, up to 16^4) and, by 2 to 3 %, on the largest lattices; within a whole force the two
// are equal on 16^4 (operator, this and the hopping force together 194 us).
// 12 poles, warps / a thread per site and slot: d = 4 8^4 58/68, 12^4 240/253, 16^4 970/702; d = 6 4^4 40/143,
// 8^4 134/198, 12^4 887/861, 16^4 2790/2350 (pole after pole a thread a site 3350).
template <int D> constexpr bool clf_site_one(int V) {
  if (D == 3) return (V > 25000 && V < 75000) || V > 250000;
  return V > (D == 1 ? 75000 : D == 4 ? 80000 : 25000) && D != 2;
}
constexpr int kClfSlotsMany = 30000;        // sites from which several poles take a thread per site and slot
template <int D>
__global__ void __launch_bounds__(192) k_clover_fermion_force(double2 *clf, const __grid_constant__ PoleSet ps, Geom g) {
  const int id = blockIdx.x * 32 + (threadIdx.x & 31), i = blockIdx.y;
  if (id >= g.V) return;
  auto slot = [&](int sl) {
    if (D <= 3) clover_slot_force<D>(clf, ps, g, id, sl);
    else clover_slot_row<D>(clf, ps, g, id, i, sl);
  };
  switch (threadIdx.x >> 5) {
    case 0: slot(0); break;
    case 1: slot(1); break;
    case 2: slot(2); break;
    case 3: slot(3); break;
    case 4: slot(4); break;
    default: slot(5); break;
  }
}

template <int D>
__global__ void k_clover_fermion_slots(double2 *clf, const __grid_constant__ PoleSet ps, Geom g) {
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t < 6L * g.V) clover_slot_force<D>(clf, ps, g, (int)(t / 6), (int)(t % 6));
}

template <int D>
__global__ void k_clover_fermion_site(double2 *clf, const double2 *lhs, const double2 *rhs, Geom g, double residue) {
  int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= g.V) return;
  double2 l[4][D], r[4][D];
  ld_spinor64<D>(l, lhs, g, id);
  ld_spinor64<D>(r, rhs, g, id);
#pragma unroll 1
  for (int slot = 0; slot < 6; slot++) {
    double2 sl[4][D], sr[4][D];
    g5_sigma<D>(sl, l, slot);
    g5_sigma<D>(sr, r, slot);
    double2 f[D * D];
    YG_UNROLL_DF
    for (int k = 0; k < D * D; k++) f[k] = make_double2(0, 0);
    outer_acc<D>(f, sl, r);
    outer_acc<D>(f, sr, l);
    YG_UNROLL_DF
    for (int k = 0; k < D * D; k++) {
      long ix = fidx(g, id, slot * D * D + k, 6 * D * D);
      double2 o = clf[ix];
      o.x += residue * f[k].x;
      o.y += residue * f[k].y;
      clf[ix] = o;
    }
  }
}

// ---- hopping force, forces.cpp:200-223 (all sites, all mu), summed over the poles as above: one
// thread per (site, mu) accumulates sum_n c_n fmat_n, multiplies by U once and projects once (the
// projection is linear, so the result equals the sum of the per-pole forces up to rounding).  The
// four directions of a site sit in neighbouring lanes and share the loads of its spinors; a warp per
// direction reads them once each and was 5 to 15 % slower.
//
// ONE: a single pole needs no loop and no weights, which cost 10 to 28 % of it (us, with the loop / this:
// d = 3 16^4 56.6 / 49.0, d = 4 16^4 129 / 111, d = 10 8^4 575 / 440).  WIDE loads the four spinors of a pole
// at once, which hides their latency but takes registers: us for 12 poles, narrow / wide: d = 3 8^4 40.2 /
// 36.7, 12^4 98 / 117, 16^4 290 / 329; d = 4 8^4 58 / 51, 16^4 541 / 479; d = 6 8^4 97 / 108, 16^4 932 / 1054;
// d = 10 8^4 1620 / 1900; for one pole d = 3 16^4 49 / 53, d = 6 16^4 175 / 169.
constexpr int kHopWideSites = 10000;        // d <= 3, several poles
template <int D, bool ONE, bool WIDE>
__global__ void k_hopping_force(double *mom, const __grid_constant__ PoleSet ps, const double2 *U, Geom g,
                                const double2 *itrepr, int ng) {
  long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= 4L * g.V) return;
  int id = (int)(t >> 2), mu = (int)(t & 3);
  int c[4];
  coords_of(g, id, c);
  int fw = neighbour(g, c, mu, +1);
  double2 f[D * D];
  YG_UNROLL_DF
  for (int k = 0; k < D * D; k++) f[k] = make_double2(0, 0);
#pragma unroll 1
  for (int n = 0; n < (ONE ? 1 : ps.n); n++) {
    double2 a[4][D], s[4][D];
    ld_spinor64<D>(a, ps.lhs[n], g, fw);
    g5_omg<D>(s, a, mu);
    if constexpr (WIDE) {
      double2 b[4][D], q[4][D];
      ld_spinor64<D>(a, ps.rhs[n], g, fw);
      g5_omg<D>(q, a, mu);
      ld_spinor64<D>(a, ps.rhs[n], g, id);
      ld_spinor64<D>(b, ps.lhs[n], g, id);
      if (!ONE) {
        scale_spinor<D>(a, ps.w[n]);
        scale_spinor<D>(b, ps.w[n]);
      }
      outer_acc<D>(f, s, a);
      outer_acc<D>(f, q, b);
    } else {
      ld_spinor64<D>(a, ps.rhs[n], g, id);
      if (!ONE) scale_spinor<D>(a, ps.w[n]);
      outer_acc<D>(f, s, a);
      ld_spinor64<D>(a, ps.rhs[n], g, fw);
      g5_omg<D>(s, a, mu);
      ld_spinor64<D>(a, ps.lhs[n], g, id);
      if (!ONE) scale_spinor<D>(a, ps.w[n]);
      outer_acc<D>(f, s, a);
    }
  }
  mom += (4L * id + mu) * ng;
  const double coeff = ONE ? ps.w[0] : 1.0;
  if constexpr (D <= 6) {
    lmul<D, false>(f, U, g, id, mu, 4);
    project_add<D>(mom, f, itrepr, ng, coeff);
  } else {
    double2 u[D * D], m[D * D];
    ld_mat<D>(u, U, g, id, mu, 4);
    mat_mul<D>(m, u, f);
    project_add<D, D == 8 || (D == 10 && !ONE)>(mom, m, itrepr, ng, coeff);
  }
}

// ---- _compute_clover_force, clover.cpp:170-262 (sites of block 1): coeff times the entries of
// A_oo^-1 combined into the six planes, from the packed Hermitian inverse the Schur operator
// uses (layout of cpk_site).  Lane = site, one (i, j) colour pair per warp: each entry of the
// inverse is read as it is needed and each word of cl_force updated once, which bounds it.
// SU(3) 32 x 16^3: 25 us, 89 with a thread a site solving for its columns from the LDL factors.
template <int D>
__device__ __forceinline__ double2 cpk_entry(const double2 *Cb, int Vh, int r, int c) {
  if (r == c) {
    const double2 d = __ldg(Cb + (long)(r >> 1) * Vh);
    return make_double2((r & 1) ? d.y : d.x, 0.0);
  }
  const int hi = r > c ? r : c, lo = r > c ? c : r;
  const double2 m = __ldg(Cb + (long)(D + hi * (hi - 1) / 2 + lo) * Vh);
  return r > c ? m : cconj(m);
}

template <int D>
__global__ void __launch_bounds__(256) k_clover_ldl_force(double2 *clf, const double2 *cpk, Geom g, double coeff) {
  const int h = blockIdx.x * 32 + (threadIdx.x & 31);
  const int ij = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (h >= g.Vh || ij >= D * D) return;
  const int id = g.Vh + h, i = ij / D, j = ij % D;
  const double2 *A = cpk + h, *B = A + 2L * D * D * g.Vh;
  const double2 a21 = cscale(cpk_entry<D>(A, g.Vh, i + D, j), coeff), a12 = cscale(cpk_entry<D>(A, g.Vh, i, j + D), coeff);
  const double2 a43 = cscale(cpk_entry<D>(B, g.Vh, i + D, j), coeff), a34 = cscale(cpk_entry<D>(B, g.Vh, i, j + D), coeff);
  const double2 a11 = cscale(cpk_entry<D>(A, g.Vh, i, j), coeff), a22 = cscale(cpk_entry<D>(A, g.Vh, i + D, j + D), coeff);
  const double2 a33 = cscale(cpk_entry<D>(B, g.Vh, i, j), coeff), a44 = cscale(cpk_entry<D>(B, g.Vh, i + D, j + D), coeff);
  double2 F[6];
  F[0] = make_double2(a12.y + a21.y - a34.y - a43.y, -a12.x - a21.x + a34.x + a43.x);   // X_01
  F[1] = make_double2(a12.x - a21.x + a43.x - a34.x, a12.y - a21.y + a43.y - a34.y);    // X_02
  F[2] = make_double2(a22.y - a11.y + a44.y - a33.y, a11.x - a22.x + a33.x - a44.x);    // X_12
  F[3] = make_double2(a11.y - a22.y + a44.y - a33.y, a22.x - a11.x + a33.x - a44.x);    // X_03
  F[4] = make_double2(a12.x - a21.x + a34.x - a43.x, a12.y - a21.y + a34.y - a43.y);    // X_13
  F[5] = make_double2(-a12.y - a21.y - a34.y - a43.y, a12.x + a21.x + a34.x + a43.x);   // X_23
#pragma unroll
  for (int s = 0; s < 6; s++) {
    const long ix = fidx(g, id, s * D * D + ij, 6 * D * D);
    clf[ix] = cadd(clf[ix], F[s]);
  }
}

// ---- clover_force_core, forces.cpp:33-106.  For each plane the eight terms of its two loops
// through the link are, with A the side link at x (or its dagger), S the opposite link, C the far
// side link and Z_a..Z_c the cl_force of the corners,
//     C [ Z_s (S A) + S (Z_a A + A Z_0) ] + Z_1 (C S A),
// up (A = U(x,nu)^dag, S = U(x+nu,mu)^dag, C = U(x+mu,nu)) minus down (A = U(x-nu,nu),
// S = U(x-nu,mu)^dag, C = U(x-nu+mu,nu)^dag).  A block takes 32 sites and one direction mu, one
// warp per nu != mu, and the projected planes are summed in shared memory.  Bound by FP64 latency at
// 12 warps an SM (168 registers).  SU(3) 32 x 16^3: 459 us, 647 with a thread a link and 13 matrices;
// d = 6 16^4: 7.9 ms, 14.0, at 255 registers with 26 kB of spill stores a thread.
template <int D, bool UP>
__device__ __forceinline__ void clover_loop(double2 (&t)[D * D], const double2 *clf, const double2 *U, const Geom &g,
                                            int num, int mu, int nu, int x0, int x1, int aid, int sid, int cid, int za,
                                            int zs) {
  double2 p[D * D];
  ld_mat<D>(t, clf, g, x0, num, 6);
  lmul<D, UP>(t, U, g, aid, nu, 4);                       // A Z_0
  ld_mat<D>(p, U, g, aid, nu, 4);
  if (UP) {
    double2 q[D * D];
    dag<D>(q, p);
    YG_UNROLL_DF
    for (int k = 0; k < D * D; k++) p[k] = q[k];          // A
  }
  lmul_add<D>(t, p, clf, g, za, num, 6);                  // + Z_a A
  lmul<D, true>(t, U, g, sid, mu, 4);                     // S (...)
  lmul<D, true>(p, U, g, sid, mu, 4);                     // S A
  lmul_add<D>(t, p, clf, g, zs, num, 6);                  // + Z_s (S A)
  lmul<D, !UP>(t, U, g, cid, nu, 4);                      // C [...]
  lmul<D, !UP>(p, U, g, cid, nu, 4);                      // C S A
  lmul_add<D>(t, p, clf, g, x1, num, 6);                  // + Z_1 (C S A)
}

template <int D>
__global__ void __launch_bounds__(96, (D <= 3 ? 4 : 2))
    k_clover_force_core(double *mom, const double2 *clf, const double2 *U, Geom g, const double2 *itrepr, int ng,
                        double coeff) {
  extern __shared__ double mom_acc[];
  const int site0 = (blockIdx.x >> 2) * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5, mu = blockIdx.x & 3;
  const int id = min(site0 + lane, g.V - 1);
  const int nu = w + (w >= mu);
  int c[4], cc[4];
  coords_of(g, id, c);
  const int o1 = neighbour(g, c, mu, +1), o2 = neighbour(g, c, nu, +1), o3 = neighbour(g, c, nu, -1);
  coords_of(g, o3, cc);
  const int o4 = neighbour(g, cc, mu, +1);
  coords_of(g, o2, cc);
  const int o5 = neighbour(g, cc, mu, +1);
  int num, sign;
  if (mu < nu) { num = nu * (nu - 1) / 2 + mu; sign = 1; }
  else { num = mu * (mu - 1) / 2 + nu; sign = -1; }
  double2 F[D * D], t[D * D];
  clover_loop<D, true>(F, clf, U, g, num, mu, nu, id, o1, id, o2, o1, o2, o5);
  clover_loop<D, false>(t, clf, U, g, num, mu, nu, id, o1, o3, o3, o4, o3, o4);
  YG_UNROLL_DF
  for (int k = 0; k < D * D; k++) F[k] = csub(F[k], t[k]);
  lmul<D, false>(F, U, g, id, mu, 4);
  project_store<D, 33>(mom_acc + w * ng * 33 + lane, F, itrepr, ng, sign * coeff);
  add_momenta<1, 3>(mom, mom_acc, g, site0, mu, ng);
}

// The same for larger d, one thread a link (the matrices live in local memory either way)
template <int D>
__global__ void k_clover_force_core_link(double *mom, const double2 *clf, const double2 *U, Geom g, const double2 *itrepr,
                                    int ng, double coeff) {
  long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= 4L * g.V) return;
  int id = (int)(t >> 2), mu = (int)(t & 3);
  int c[4], cc[4];
  coords_of(g, id, c);
#pragma unroll 1
  for (int nu = 0; nu < 4; nu++) {
    if (nu == mu) continue;
    int o1 = neighbour(g, c, mu, +1);
    int o2 = neighbour(g, c, nu, +1);
    int o3 = neighbour(g, c, nu, -1);
    coords_of(g, o3, cc);
    int o4 = neighbour(g, cc, mu, +1);
    coords_of(g, o2, cc);
    int o5 = neighbour(g, cc, mu, +1);
    int num, sign;
    if (mu < nu) { num = nu * (nu - 1) / 2 + mu; sign = 1; }
    else { num = mu * (mu - 1) / 2 + nu; sign = -1; }
    double2 W0[D * D], W1[D * D], W2[D * D], W3[D * D], W4[D * D], W5[D * D], W6[D * D], W7[D * D], W8[D * D];
    double2 X[D * D], Y[D * D], Z[D * D], F[D * D];
    ld_mat<D>(X, U, g, o3, mu, 4); dag<D>(W0, X);
    ld_mat<D>(W1, U, g, o3, nu, 4);
    ld_mat<D>(W2, U, g, o1, nu, 4);
    ld_mat<D>(X, U, g, o2, mu, 4); dag<D>(W3, X);
    ld_mat<D>(X, U, g, id, nu, 4); dag<D>(W4, X);
    ld_mat<D>(X, U, g, o4, nu, 4); dag<D>(W5, X);
    mat_mul<D>(W6, W0, W1);
    mat_mul<D>(W7, W2, W3);
    mat_mul<D>(X, W7, W4);
    mat_mul<D>(Y, W5, W6);
    for (int k = 0; k < D * D; k++) W8[k] = csub(X[k], Y[k]);
    // F = W8 Z0 + Z1 W8
    ld_mat<D>(Z, clf, g, id, num, 6); mat_mul<D>(F, W8, Z);
    ld_mat<D>(Z, clf, g, o1, num, 6); mat_mul<D>(X, Z, W8);
    for (int k = 0; k < D * D; k++) F[k] = cadd(F[k], X[k]);
    // F -= W5 (W0 Z2 W1 + Z3 W6)
    ld_mat<D>(Z, clf, g, o3, num, 6); mat_mul<D>(X, W0, Z); mat_mul<D>(Y, X, W1);
    ld_mat<D>(Z, clf, g, o4, num, 6); mat_mul<D>(X, Z, W6);
    for (int k = 0; k < D * D; k++) Y[k] = cadd(Y[k], X[k]);
    mat_mul<D>(X, W5, Y);
    for (int k = 0; k < D * D; k++) F[k] = csub(F[k], X[k]);
    // F += (W2 Z4 W3 + W7 Z5) W4
    ld_mat<D>(Z, clf, g, o5, num, 6); mat_mul<D>(X, W2, Z); mat_mul<D>(Y, X, W3);
    ld_mat<D>(Z, clf, g, o2, num, 6); mat_mul<D>(X, W7, Z);
    for (int k = 0; k < D * D; k++) Y[k] = cadd(Y[k], X[k]);
    mat_mul<D>(X, Y, W4);
    for (int k = 0; k < D * D; k++) F[k] = cadd(F[k], X[k]);
    ld_mat<D>(X, U, g, id, mu, 4);
    mat_mul<D>(Y, X, F);
    project_add<D>(mom + (4L * id + mu) * ng, Y, itrepr, ng, sign * coeff);
  }
}

// ------------------------------------------------------------------ launchers
template <int D>
void DK<D>::clover_fermion_force(double2 *clf, const PoleSet &ps, Geom g, cudaStream_t s) {
  if constexpr (D <= 6) {
    if (ps.n == 1 && clf_site_one<D>(g.V)) {
      k_clover_fermion_site<D><<<nblk(g.V, 64), 64, 0, s>>>(clf, ps.lhs[0], ps.rhs[0], g, ps.w[0]);
      return;
    }
  }
  if constexpr (D == 4 || D == 6) {
    if (ps.n > 1 && g.V > kClfSlotsMany) {
      k_clover_fermion_slots<D><<<nblk(6L * g.V, 64), 64, 0, s>>>(clf, ps, g);
      return;
    }
  }
  k_clover_fermion_force<D><<<dim3(nblk(g.V, 32), D <= 3 ? 1 : D), 192, 0, s>>>(clf, ps, g);
}

template <int D>
void DK<D>::hopping_force(double *mom, const PoleSet &ps, const double2 *U, Geom g, const double2 *itrepr, int ng,
                          cudaStream_t s) {
  const int grid = nblk(4L * g.V, 64);
  if (ps.n == 1)
    k_hopping_force<D, true, D == 6><<<grid, 64, 0, s>>>(mom, ps, U, g, itrepr, ng);
  else if (D == 4 || (D <= 3 && g.V <= kHopWideSites))
    k_hopping_force<D, false, D <= 4><<<grid, 64, 0, s>>>(mom, ps, U, g, itrepr, ng);
  else
    k_hopping_force<D, false, false><<<grid, 64, 0, s>>>(mom, ps, U, g, itrepr, ng);
}

template <int D>
void DK<D>::clover_ldl_force(double2 *clf, const double2 *cpk, Geom g, double coeff, cudaStream_t s) {
  const int warps = D * D < 8 ? D * D : 8;
  k_clover_ldl_force<D><<<dim3(nblk(g.Vh, 32), nblk(D * D, warps)), 32 * warps, 0, s>>>(clf, cpk, g, coeff);
}

template <int D>
void DK<D>::clover_force_core(double *mom, const double2 *clf, const double2 *U, Geom g, const double2 *itrepr, int ng,
                              double coeff, cudaStream_t s) {
  if constexpr (D <= 6)
    k_clover_force_core<D><<<4 * nblk(g.V, 32), 96, momenta_smem(3, ng), s>>>(mom, clf, U, g, itrepr, ng, coeff);
  else
    k_clover_force_core_link<D><<<nblk(4L * g.V, 64), 64, 0, s>>>(mom, clf, U, g, itrepr, ng, coeff);
}

}  // namespace yg
