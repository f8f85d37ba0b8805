// Persistent uneven-volume batch: independent cg_inverter solves (cg.cpp:132-202) of Hphi_sq on
// several even-odd lattices of different sizes in ONE cooperative kernel launch.
//
// A small lattice's CG is bound by launch and reduction latency: a 8^4 or 12^4 operator step
// fills a few SMs for a few microseconds, and the reference's recurrence needs two host
// round trips per iteration (<p,q> for alpha, |r|^2 for beta and the stopping test).  Here
// the grid is split into one group of blocks per lattice, sized in proportion to the
// lattice's even volume (at least one block each), and every group runs its lattice's whole
// CG loop on the device:
//
//   P1  o = A_oo^-1 (1/2 H p)              (odd sites)
//   P2  t = g5 (A_ee p - 1/2 H o), |t|^2   (even sites)          t = Hphi p
//   P3  o = A_oo^-1 (1/2 H t)
//   P4  q = g5 (A_ee t - 1/2 H o)          (even sites)          q = Hphi_sq p, never stored:
//       r -= alpha q, |r|^2
//   P5  x += alpha p, p = beta p + r
//
// with a barrier of the group after each phase.  Hphi is Hermitian on these lattices (no open or
// SF slices), so <p, Hphi_sq p> = |Hphi p|^2 and alpha is known before the second Hphi ends, which
// leaves five barriers an iteration and no pass over q.  The operator steps are the FP64 Schur
// steps of the single-lattice path (yg_dirac_impl.cuh: a thread or four lanes a site) with
// ordinary loads for the fields, which the kernel also writes.  The scalars are the reference's:
// alpha = rr / <p,q>, beta = rr_new / rr, stop when rr_new < prec |b|^2, iteration count as
// cg_inverter's.  Reductions are deterministic: one partial per block, which every block of the
// group adds in block order after the barrier, so all blocks of a group hold the same alpha and
// beta.  Groups never wait for each other: a lattice that converges early just ends its blocks.
//
// Barriers: one arrival counter per group, on a line of its own, that only grows; a block
// releases its writes with its arrival and acquires the others' by polling the counter up to the
// group's next multiple, one round trip each.  Every wait is bounded by a cycle limit; a block whose
// wait runs out sets the launch's error flag and returns, every other block meets the flag in its
// next wait (the missing arrival keeps it there) and returns too, and the host reports YG_TIMEOUT.
// The launch is cooperative, so all blocks are resident and in a healthy run every barrier
// completes; the limit is the guard against anything else.  The iterations of one launch are bounded
// too (launch_iters): a solve that needs more, or never converges, goes on in further launches from the
// fields and scalars the last one left, so the device and the host get their turn.
#include <algorithm>
#include <cmath>
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <vector>
#include "yg_lattice.h"
#include "yg_kernels.h"
#include "yg_dirac_impl.cuh"

namespace yg {

namespace {

constexpr int kThreads = 128;
constexpr int kPerSM = 3;                           // blocks an SM has room for, whatever the instantiation

// Persistent grids that run at once must all fit the device together, or each could hold
// multiprocessors that another one's blocks need.  So, as far as this process goes, a launch takes a slot
// for each of its blocks, kPerSM for each SM of the device, and waits, in order of arrival, until enough
// are free: an SM with fewer than kPerSM blocks has room for one more of any instantiation, so while the
// blocks of all launches are no more than the slots, each finds a place.  A launch of more blocks than
// slots (small d) runs alone.  Solves of host threads on lattices of their own, one call each, us for all
// of them, one launch at a time / sharing the device (cg_launches before this kernel took them):
//   d = 3, 60 iterations: 8^4 x 4 4962 / 1767 (5533), x 16 19336 / 6370 (11152);
//   12^4 x 2 5691 / 3196 (6538), x 8 22459 / 11295 (11910), x 16 44696 / 21953 (20651);
//   16^4 fills the device: x 4 18872 / 18881 (16470), where one alone takes 4935 (8083).
constexpr int kMaxDevices = 64;
struct Slots {
  std::mutex m;
  std::condition_variable cv;
  long used = 0;
  unsigned long next = 0, serving = 0;
} g_slots[kMaxDevices];

class SlotHold {
 public:
  SlotHold(int device, long blocks, long cap) : s(g_slots[device % kMaxDevices]), held(std::min(blocks, cap)) {
    std::unique_lock<std::mutex> lk(s.m);
    const unsigned long mine = s.next++;
    s.cv.wait(lk, [&] { return s.serving == mine && s.used + held <= cap; });
    s.serving++;
    s.used += held;
    s.cv.notify_all();
  }
  ~SlotHold() {
    std::lock_guard<std::mutex> lk(s.m);
    s.used -= held;
    s.cv.notify_all();
  }

 private:
  Slots &s;
  const long held;
};

constexpr int kSyncStride = 32;                     // words between the groups' counters: 128 bytes

constexpr long long kDefaultWait = 20000000000LL;   // cycles (about 10 s at 2 GHz)

constexpr int kMaxLattices = 64;

constexpr int kMore = -1;                           // status of a lattice that goes on in the next launch

// iterations of one launch: at most about 0.1 s of them (3 ns a site and iteration at d = 3, 25 us the
// least), against some 20 us for another launch
int launch_iters(long sites) { return (int)std::max(16L, std::min(1000L, 40000000L / sites)); }

// d = 6 always takes four lanes a site, which spill 0.7 kB under 168 registers (d = 4: 0.6 kB, d = 3: 0.1 kB).
// Batches of 60 iterations, the kernel's first form with a thread a site at all sizes / this: d = 6 8^4 + 12^4
// 15.6 / 4.6 ms, 8^4 + 12^4 + 16^4 20.6 / 16.5 ms, 8 x 6^4 8.6 / 3.2 ms; d = 4 8^4 + 12^4 + 16^4 13.5 / 10.4 ms.
constexpr int kSiteMaxD = 4;

struct BLat {
  Geom g;
  const double2 *U, *cl, *cpk;
  double2 *x, *r, *p, *t, *o;          // whole-field layout; x, r, p, t even sites, o odd
  int b0, nb;                          // the group's blocks [b0, b0 + nb)
  int quad;                            // four lanes a site instead of one thread
  int it0, it1;                        // iterations it0 + 1 .. it1 of this launch; it0 = -1: none, the solve has ended
  double diag, target, rr0;            // diagonal of A_ee, prec |b|^2, |r|^2 after it0 iterations
};

// A kernel parameter: geometry and pointers stay in the constant bank.  Read from global memory they
// are loaded again after every store, which doubled the time of a step on 16^4.
struct BArgs {
  BLat l[kMaxLattices];
  int n;
};

struct BOut {
  int iters, status;
  double rr;
};

__device__ __forceinline__ double block_sum(double v) {
  __shared__ double sh[kThreads / 32];
  __syncthreads();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; w++) s += sh[w];
  return s;
}

// sum of the group's partials in block order (the same value in every block of the group)
__device__ __forceinline__ double group_total(const double *part, int b0, int nb) {
  double acc = 0.0;
  for (int i = threadIdx.x; i < nb; i += kThreads) acc += part[b0 + i];
  return block_sum(acc);
}

// barrier of the nb blocks of a group: `due` counts the arrivals of all barriers so far.  False
// when this block's wait ran out or another block of the launch gave up: the block returns.
__device__ __forceinline__ bool group_sync(unsigned *cnt, unsigned &due, unsigned nb, int *err, long long limit) {
  __shared__ int ok;
  due += nb;
  __syncthreads();
  if (threadIdx.x == 0) {
    int good = 1;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");
    const long long t0 = clock64();
    while (true) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
      if ((int)(v - due) >= 0) break;
      if (*reinterpret_cast<volatile int *>(err)) { good = 0; break; }
      if (clock64() - t0 > limit) { atomicExch(err, 1); good = 0; break; }
    }
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// One word of a Schur step's result: stored as t (second = false) with its square, or taken as q,
// r -= alpha q, with the square of the new r.
__device__ __forceinline__ double finish(double2 v, bool second, double2 *t, double2 *r, double alpha, long i) {
  if (!second) {
    t[i] = v;
  } else {
    const double2 rv = r[i];
    v = make_double2(fma(-alpha, v.x, rv.x), fma(-alpha, v.y, rv.y));
    r[i] = v;
  }
  return fma(v.x, v.x, v.y * v.y);
}

// The whole CG loop of one lattice's group.  QUAD: four lanes a site (dead lanes, beyond the lattice,
// take part), else a site per thread.  Both Hphi of an iteration run through the same two step bodies.
template <int D, int CLOV, bool QUAD>
__device__ __forceinline__ void group_cg(const BLat &L, double *part_pq, double *part_rr, unsigned *cnt, int *err,
                                         BOut *out, long long limit) {
  constexpr int E1 = CLOV ? EPI_CLOVPK : EPI_PLAIN, E2 = CLOV ? EPI_CLOVADD : EPI_AXPY;
  constexpr int kSites = QUAD ? kThreads / 4 : kThreads;              // sites per block and pass
  const int lb = blockIdx.x - L.b0, nb = L.nb, Vh = L.g.Vh;
  const int stride = nb * kSites, passes = (Vh + stride - 1) / stride;
  const int first = lb * kSites + (QUAD ? threadIdx.x >> 2 : threadIdx.x);
  HopArgs<double> a{}, e{};
  a.g = L.g; a.U = L.U; a.cpk = L.cpk; a.dst = L.o; a.lo = Vh; a.n = Vh; a.coeff = 0.5;
  e.g = L.g; e.U = L.U; e.cl = L.cl; e.src = L.o; e.lo = 0; e.n = Vh; e.coeff = -0.5; e.diag = L.diag; e.g5 = 1;
  e.zero_add_at_boundary = 1;
  unsigned due = 0;
  double rr = L.rr0, alpha = 0.0;
  const int it1 = L.it1;
  int it = L.it0, status = L.it0 >= 0 ? kMore : YG_OK;
  // cg.cpp:151-153: a system solved by its initial guess returns 0 iterations
  while (status == kMore) {
    ++it;
#pragma unroll 1
    for (int half = 0; half < 2; half++) {
      a.src = half ? L.t : L.p;
      e.src2 = a.src;
      for (int k = 0; k < passes; k++) {
        const int t = first + k * stride;
        const bool live = t < Vh;
        if (QUAD) {
          double2 w[D];
          long at;
          hop_quad<D, double, E1, false>(a, live ? t : Vh - 1, live, w, at);
          if (live) {
#pragma unroll
            for (int c = 0; c < D; c++) L.o[at + (long)c * Vh] = w[c];
          }
        } else if (live) {
          double2 w[4][D];
          hop_values<D, double, E1, false>(a, t, w);
          store_spinor<D, double>(L.o, w, L.g, Vh + t);
        }
      }
      if (!group_sync(cnt, due, nb, err, limit)) { status = YG_TIMEOUT; break; }
      double acc = 0.0;
      for (int k = 0; k < passes; k++) {
        const int t = first + k * stride;
        const bool live = t < Vh;
        if (QUAD) {
          double2 w[D];
          long at;
          hop_quad<D, double, E2, false>(e, live ? t : Vh - 1, live, w, at);
          if (live) {
#pragma unroll
            for (int c = 0; c < D; c++) acc += finish(w[c], half, L.t, L.r, alpha, at + (long)c * Vh);
          }
        } else if (live) {
          double2 w[4][D];
          hop_values<D, double, E2, false>(e, t, w);
#pragma unroll
          for (int sp = 0; sp < 4; sp++)
#pragma unroll
            for (int c = 0; c < D; c++) acc += finish(w[sp][c], half, L.t, L.r, alpha, (long)(sp * D + c) * Vh + t);
        }
      }
      double *part = half ? part_rr : part_pq;
      acc = block_sum(acc);
      if (threadIdx.x == 0) part[blockIdx.x] = acc;
      if (!group_sync(cnt, due, nb, err, limit)) { status = YG_TIMEOUT; break; }
      const double total = group_total(part, L.b0, nb);
      if (!isfinite(total)) { status = YG_NONFINITE; break; }
      if (half == 0) {
        alpha = rr / total;
      } else {
        const double beta = total / rr;
        rr = total;
        for (int k = 0; k < passes; k++) {
          const int t = first + k * stride;
          if (t >= Vh) break;
          const long at = (long)(QUAD ? (threadIdx.x & 3) * D : 0) * Vh + t;
#pragma unroll
          for (int c = 0; c < (QUAD ? D : 4 * D); c++) {
            const long i = at + (long)c * Vh;
            const double2 pv = L.p[i], rv = L.r[i];
            double2 xv = L.x[i];
            xv.x = fma(alpha, pv.x, xv.x);
            xv.y = fma(alpha, pv.y, xv.y);
            L.x[i] = xv;
            L.p[i] = make_double2(fma(beta, pv.x, rv.x), fma(beta, pv.y, rv.y));
          }
        }
      }
    }
    if (status != kMore) break;
    if (rr < L.target) { status = YG_OK; break; }
    if (it >= it1) break;
    if (!group_sync(cnt, due, nb, err, limit)) status = YG_TIMEOUT;
  }
  if (lb == 0 && threadIdx.x == 0) {
    out->iters = it;
    out->status = status;
    out->rr = rr;
  }
}

// CLOV = 1: A_oo^-1 from the packed inverse blocks and A_ee from the clover term (d <= 6);
// CLOV = 0: no clover term, A_oo = 1 and the (4+m)^2 diagonal.
template <int D, int CLOV>
__global__ void __launch_bounds__(kThreads, kPerSM) k_cg_batch(const __grid_constant__ BArgs args, double *part_pq,
                                                       double *part_rr, unsigned *sync, int *err, BOut *out,
                                                       long long limit) {
  int li = 0;
  while (li + 1 < args.n && (int)blockIdx.x >= args.l[li + 1].b0) li++;
  const BLat &L = args.l[li];
  unsigned *cnt = sync + kSyncStride * li;
  if constexpr (D <= kSiteMaxD) {
    if (!L.quad) {
      group_cg<D, CLOV, false>(L, part_pq, part_rr, cnt, err, out + li, limit);
      return;
    }
  }
  group_cg<D, CLOV, true>(L, part_pq, part_rr, cnt, err, out + li, limit);
}

template <int D, int CLOV>
void launch_batch(int grid, cudaStream_t s, const BArgs &a, double *part_pq, double *part_rr, unsigned *sync, int *err,
                  BOut *out, long long limit) {
  void *args[] = {(void *)&a, (void *)&part_pq, (void *)&part_rr, (void *)&sync, (void *)&err, (void *)&out,
                  (void *)&limit};
  YG_CUDA(cudaLaunchCooperativeKernel((const void *)k_cg_batch<D, CLOV>, dim3(grid), dim3(kThreads), args, 0, s));
  YG_LAUNCHED();
}

int sm_count() {
  int dev = 0, sms = 0;
  YG_CUDA(cudaGetDevice(&dev));
  YG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return sms;
}

template <int D, int CLOV>
int resident_blocks() {
  int per = 0;
  YG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cg_batch<D, CLOV>, kThreads, 0));
  return sm_count() * per;
}

// one device buffer: partials, barrier counters, error flag, results
struct WorkLayout {
  size_t sync, err, out, bytes;
  WorkLayout(int n, int grid) {
    sync = (2 * sizeof(double) * grid + 127) / 128 * 128;
    err = sync + sizeof(unsigned) * kSyncStride * n;
    out = err + 16;
    bytes = out + sizeof(BOut) * n;
  }
};

// the representation dimensions of the persistent batch: SU(2) fundamental (2), SU(3)
// fundamental and SU(2) adjoint (3), SU(4) fundamental (4), SU(3) sextet and SU(4)
// antisymmetric (6)
#define YG_BATCH_D(DV, CV, ...)                                                                                    \
  do {                                                                                                            \
    const bool cv_ = (CV);                                                                                        \
    switch (DV) {                                                                                                 \
      case 2: if (cv_) { constexpr int BD = 2, BC = 1; __VA_ARGS__; } else { constexpr int BD = 2, BC = 0; __VA_ARGS__; } break; \
      case 3: if (cv_) { constexpr int BD = 3, BC = 1; __VA_ARGS__; } else { constexpr int BD = 3, BC = 0; __VA_ARGS__; } break; \
      case 4: if (cv_) { constexpr int BD = 4, BC = 1; __VA_ARGS__; } else { constexpr int BD = 4, BC = 0; __VA_ARGS__; } break; \
      case 6: if (cv_) { constexpr int BD = 6, BC = 1; __VA_ARGS__; } else { constexpr int BD = 6, BC = 0; __VA_ARGS__; } break; \
      default: throw Error(YG_ERR_ARG, "the persistent batch exists for d = 2, 3, 4, 6");                        \
    }                                                                                                             \
  } while (0)

}  // namespace

bool batch_eligible(int n, Lattice *const *L, const yg_inv_par *par) {
  const int d = L[0]->d;
  if (d != 2 && d != 3 && d != 4 && d != 6) return false;
  for (int i = 0; i < n; i++) {
    const Lattice &l = *L[i];
    if (par[i].op != YG_OP_HPHI_SQ || !l.p.eo || l.d != d || l.p.clover != L[0]->p.clover) return false;
    if (l.p.bc == YG_BC_OPEN || l.p.bc == YG_BC_SF) return false;   // spinor boundary slices
  }
  return true;
}

void persistent_prepare(Lattice &L) {
  int grid_max = 0;
  YG_BATCH_D(L.d, L.p.clover, grid_max = resident_blocks<BD, BC>());
  L.cg_work.alloc(WorkLayout(1, grid_max).bytes);
}

// The cg_inverter prologue on every lattice (cg.cpp:134-150: r = b - A x, p = r, |b|^2, |r|^2)
// with the engine's ordinary launches, then one persistent launch for all iterations.
int cg_lattices_persistent(int n, Lattice *const *L, const yg_inv_par *par, double *const *xs, double *const *bs,
                           int *iters, long long wait_cycles) {
  if (n < 1 || n > kMaxLattices) throw Error(YG_ERR_ARG, "1..64 lattices");
  if (!batch_eligible(n, L, par))
    throw Error(YG_ERR_ARG, "the persistent batch solves Hphi_sq on even-odd lattices of one d (2, 3, 4 or 6), "
                            "all with or all without a clover term, without open/SF boundaries");
  const int d = L[0]->d;
  const bool clov = L[0]->p.clover;
  BArgs args{};
  args.n = n;
  BLat *h = args.l;
  // Four lanes a site only where every lattice is small: beside a larger one, whose group decides the time,
  // they take multiprocessors from it.  8^4 + 12^4 + 16^4, 60 iterations, four lanes at 8^4 / a thread a
  // site: d = 2 4190 / 2885 us, d = 3 7450 / 6790, d = 4 11230 / 10375; all small: 16 x 4^4 d = 3 2163 /
  // 2935, 4 x 8^4 d = 4 2150 / 3500.
  long vol = 0, largest = 0;
  for (int i = 0; i < n; i++) {
    vol += L[i]->Vh;
    largest = std::max(largest, (long)L[i]->Vh);
  }
  int grid_max = 0;
  YG_BATCH_D(d, clov, grid_max = resident_blocks<BD, BC>());
  if (grid_max < n) throw Error(YG_ERR_ARG, "more lattices than resident blocks");
  int b0 = 0;
  std::vector<BOut> fin(n);
  for (int i = 0; i < n; i++) {
    Lattice &l = *L[i];
    const double mass = par[i].mass;
    double *r = l.scratch_field(3), *p = l.scratch_field(4), *q = l.scratch_field(5);
    double *t = l.scratch_field(2), *o = l.scratch_field(1);
    long lo, cnt;
    l.view_range(YG_VIEW_DEFAULT, lo, cnt);
    const double rr = true_residual(l, mass, r, q, p, xs[i], bs[i], lo, cnt);   // also builds the clover inverse
    blas_copy_range(l, p, r, lo, cnt);
    const double norm = blas_sqnorm(l, bs[i], lo, cnt);
    BLat &b = h[i];
    b.g = l.g;
    b.U = l.links.as<double2>();
    b.cl = l.clover.as<double2>();
    b.cpk = l.cpk64.as<double2>();
    b.diag = clov ? 4.0 + mass : (4.0 + mass) * (4.0 + mass);
    b.t = (double2 *)t;
    b.o = (double2 *)o;
    b.x = (double2 *)xs[i];
    b.r = (double2 *)r;
    b.p = (double2 *)p;
    b.target = norm * par[i].prec;
    b.rr0 = rr;
    b.it0 = rr < b.target ? -1 : 0;
    fin[i] = BOut{0, YG_OK, rr};
    // one block each, the others in proportion to the even volume (so that all shares together fit the
    // resident grid), and no more than the passes over the sites need (fewer blocks make a cheaper barrier)
    const long share = 1 + (grid_max - n) * (long)l.Vh / vol;
    b.quad = d > kSiteMaxD || largest <= kQuadSites;
    const long tiles = nblk(l.Vh, b.quad ? kThreads / 4 : kThreads), passes = (tiles + share - 1) / share;
    b.nb = (int)((tiles + passes - 1) / passes);
    b.b0 = b0;
    b0 += b.nb;
    YG_CUDA(cudaStreamSynchronize(l.stream));
  }
  const int grid = b0;
  if (grid > grid_max) throw Error(YG_ERR_ARG, "block groups exceed the resident grid");
  const WorkLayout lay(n, grid);
  L[0]->cg_work.alloc(lay.bytes);        // kept: an allocation would synchronise the device on every solve
  char *base = L[0]->cg_work.as<char>();
  cudaStream_t s = L[0]->stream;
  int err = 0, step = launch_iters(vol);
  bool more = true;
  std::vector<BOut> res(n);
  try {
    const long long limit = wait_cycles > 0 ? wait_cycles : kDefaultWait;
    double *part = reinterpret_cast<double *>(base);
    while (more && !err) {
      for (int i = 0; i < n; i++) {
        h[i].it1 = h[i].it0 + step;
        if (par[i].maxiter > 0) h[i].it1 = std::min(h[i].it1, par[i].maxiter);
      }
      SlotHold hold(L[0]->device, grid, (long)kPerSM * sm_count());
      YG_CUDA(cudaMemsetAsync(base, 0, lay.bytes, s));
      YG_BATCH_D(d, clov, launch_batch<BD, BC>(grid, s, args, part, part + grid,
                                               reinterpret_cast<unsigned *>(base + lay.sync),
                                               reinterpret_cast<int *>(base + lay.err),
                                               reinterpret_cast<BOut *>(base + lay.out), limit));
      YG_CUDA(cudaMemcpyAsync(res.data(), base + lay.out, sizeof(BOut) * n, cudaMemcpyDeviceToHost, s));
      YG_CUDA(cudaMemcpyAsync(&err, base + lay.err, sizeof(int), cudaMemcpyDeviceToHost, s));
      YG_CUDA(cudaStreamSynchronize(s));
      more = false;
      for (int i = 0; i < n; i++) {
        if (h[i].it0 < 0) continue;
        fin[i] = res[i];
        if (fin[i].status == kMore && fin[i].iters == par[i].maxiter) fin[i].status = YG_MAXITER;
        h[i].rr0 = res[i].rr;
        h[i].it0 = fin[i].status == kMore ? fin[i].iters : -1;
        more = more || h[i].it0 >= 0;
      }
    }
  } catch (...) {
    cudaStreamSynchronize(s);
    throw;
  }
  int worst = YG_OK;
  for (int i = 0; i < n; i++) {
    iters[i] = fin[i].iters;
    L[i]->mvm += 4 * fin[i].iters;
    if (par[i].log)
      fprintf(stderr, "[INVERTER][30]cg: iterations = %d, precision = %1.4e\n", fin[i].iters,
              fin[i].rr / (h[i].target / par[i].prec));
    if (fin[i].status > YG_OK && worst == YG_OK) worst = fin[i].status;
  }
  if (err) return YG_TIMEOUT;
  return worst;
}

}  // namespace yg
