// krylov.cu -- batched, persistent Krylov solvers with the Jacobi
// preconditioner and FP64 reliable updates on the SELL-32 pattern (sm_100a):
// the velocity systems (prediction, mass) by CG or BiCGStab, and the pressure
// systems where the multigrid (mgcg.cu) is not used.
//
// One cooperative launch solves every system of a solve phase (components x
// instances) to the reference's stopping rule: the absolute 2-norm of the
// unpreconditioned residual b - A x <= tol within max_iter iterations
// (deal.II SolverControl(max_iter, tol), cylinder2D/cylinder2D.cc:736-779).
//
// The work between two synchronisation points is a "phase". A phase ends
// with every block publishing its partial sums and a release add on the
// counters of its systems; the next phase starts once the counters of the
// block's running systems show every block of those systems done (a
// per-system barrier: the instances of a batch do not wait for each other).
// Every block computes its systems' scalars itself, from the partial sums of
// the previous phase in a fixed order: no block publishes scalars and no
// phase waits for a finalizer.
//
// BiCGStab (right-preconditioned, van der Vorst 1992) takes two phases per
// iteration, CG one (single reduction, Chronopoulos and Gear 1989). A
// restart costs one phase more: the FP64 residual r64 = b - A64 (x + e) is
// formed with BiCGStab's pending e += omega K^-1 s on the fly, and the first
// phase of the next cycle reads its start vector from r64 at the columns.
// The vectors that a product gathers are packed four to a row (V4), so that
// an entry costs one vector load instead of two to four.
//
// What bounds it: on the 52k-row channel the wait for the slowest block and
// the dependent loads after it (a phase is about 2.5 us of waiting, sums and
// publishing and 2 us of work), on the 131k-cell pipe the gathers and the
// matrix from L2. A block owns a contiguous run of slices with all their
// components, cut to equal lengths, and a warp takes one (slice, component)
// at a time (where warps would be left over, several share one). Measured against tiles of 8 slices per component (some blocks
// held two, others one), separate vectors, generic pointers and three phases
// per restart, prediction and correction take per step: 52k channel FP32 0.45
// ms instead of 0.86, FP64 0.59 instead of 1.03; 16 channels 1.38 instead of
// 2.43; 10k pipe FP64 1.63 instead of 2.39; 131k pipe 3.6 instead of 7.7.
//
// The iterate is split x + e: e accumulates in the inner type R (FP32 for
// the mixed path, FP64 for the plain path); once the recurrence residual
// has dropped below max(eta * res, tol / 2) a reliable update runs in FP64
// (r64 = b - A64 (x + e), then x += e, e = 0, r = r64) and the solver restarts
// from the true residual. A system is done when the FP64 residual is <= tol.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "krylov_ws.h"

namespace pfem2 {

// entries of a SELL row whose loads are issued together: a Q1 row of 9 (2D)
// in one round, one of 27 (3D) in three; with FP64 the registers hold five
template <typename R> struct Chunk { static constexpr int value = sizeof(R) == 8 ? 5 : 9; };

template <int MINB> struct SolveThreads { static constexpr int value = MINB == 1 ? 768 : 384; };
static int solve_threads(int minb) { return minb == 1 ? SolveThreads<1>::value : SolveThreads<2>::value; }

enum { S_OUT_A = 0, S_OUT_B, S_A, S_B, S_C1, S_DONE };
enum {
  ACT_NONE = 0,
  ACT_OUT_A = 1,   // FP64 residual
  ACT_FINISH = 2,  // x += e
  ACT_P1 = 3,      // BiCGStab: finish the previous step, y = K^-1 p, v = A y
  ACT_P2 = 4,      // BiCGStab: e += alpha y, s = r - alpha v, t = A K^-1 s
  ACT_C0 = 5,      // CG: restart, w = A u
  ACT_C1 = 6       // CG: one iteration in one phase (single reduction)
};
// partial sums per block and system: CG uses 3, BiCGStab 5 (and the FP64
// residual phase |r|^2 and |b|^2)
constexpr int kMaxSums = 5;
constexpr int kClusterMax = 16;  // blocks of a cluster
// systems (components x instances) a block may own parts of: a run of slices
// that cuts an instance at either end touches up to two instances more than
// its length holds, so that 1,570 instances in 3D and 2,360 in 2D, the smallest
// at one slice each, fit two blocks on each of 148 SMs
constexpr int kMaxRunSys = 24;
// Items (slices x components) up to which one cluster solves: above, the 16
// SMs' work outweighs the cheaper barrier. Prediction and correction of uniform
// channels, cluster / grid, ms per step:
//   items            70          150         240         300         350         400         520
//   FP64 BiCGStab  .38 / .47   .42 / .45   .41 / .42   .44 / .41   .45 / .41   .56 / .40   .57 / .38
//   FP64 CG        .33 / .41   .35 / .40   .36 / .39   .38 / .38   .40 / .37   .51 / .37   .51 / .36
//   FP32 BiCGStab  .31 / .39   .32 / .38   .32 / .36   .33 / .37   .35 / .37   .42 / .34   .43 / .34
//   FP32 CG        .40 / .49   .39 / .49   .38 / .46   .38 / .45   .39 / .46   .51 / .44   .52 / .44
// (from 385 items on a warp takes two). One line for all: FP64 crosses between
// 270 and 300, FP32 at 385.
constexpr int kClusterItems = 300;

// What a block keeps in shared memory (template parameter SM, the most that
// fits; every phase start's GPU-scope acquire invalidates L1, so what is read
// from global memory costs an L2 round trip per phase). Known at compile time:
// generic pointers made the solves 15-20% slower.
//   -1 nothing, the items' partial sums in global memory: their pointer alone,
//      left generic, cost the 1.05M-cell pipe 3 to 6% of its velocity solves
//   0  those sums
//   1  the own rows of the vectors that no product gathers, the slices' pointers
//   2  and the SELL columns
//   3  and the SELL values of every component (once where they share a matrix)

// the gathered vectors of a row: BiCGStab zr = K^-1 r, w = K^-1 v, y, kt =
// K^-1 t; CG u = K^-1 r, wh = K^-1 w, sh = K^-1 s
template <typename R> struct V4;
template <> struct __align__(16) V4<float> { float a, b, c, d; };
template <> struct __align__(32) V4<double> { double a, b, c, d; };

__device__ __forceinline__ V4<float> ld4(const V4<float>* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return V4<float>{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ V4<double> ld4(const V4<double>* p) {
  const double2 v = reinterpret_cast<const double2*>(p)[0], w = reinterpret_cast<const double2*>(p)[1];
  return V4<double>{v.x, v.y, w.x, w.y};
}
__device__ __forceinline__ void ld2(const V4<float>* p, float& a, float& b) {
  const float2 v = *reinterpret_cast<const float2*>(p);
  a = v.x;
  b = v.y;
}
__device__ __forceinline__ void ld2(const V4<double>* p, double& a, double& b) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  a = v.x;
  b = v.y;
}

template <typename R> struct SolveArgs {
  int ncomp, ninst, nv;
  const int *blk_inst, *blk_inst_off;  // instances of each block, at blk_inst_off[b]
  const int *blk_slot;                 // per blk_inst entry: the block's partial slot (component 0)
  const int *sys_slot0;                // [nsys+1] partial slots of each system
  const int *blk_sl;                   // [grid+1] first slice
  const int *slk;                      // [nslices] local instance of each slice (in its block)
  const int *sl_ptr, *sl_len, *sl_col;
  const double* A64[3];
  const R* Ain[3];
  const R* dinv[3];
  int share;              // the components share one matrix
  int items_max;
  int split;              // warps that share an item's entries
  double* x[3];
  const double* b[3];
  const unsigned char* isd[3];
  const double* g[3];    // Dirichlet values preset in x (nullptr -> 0)
  const double* tol_i;   // per instance
  const double* rtol_i;  // per instance: stop at max(tol, rtol |b|)
  const int* maxit_i;    // per instance
  int bicg;              // BiCGStab instead of CG
  V4<R>* pk;             // [2 parities][ncomp][nv]
  // own rows only, [ncomp][nv]: BiCGStab shadow residual, s, t, v; CG w, s, p
  R *rh, *s, *t, *v;
  R *e, *r;
  double* r64;
  double* part;          // [2 parities][kMaxSums][nslots]
  double* item_part;     // [blocks][items_max][sums] where they do not fit shared memory
  int nslots;
  unsigned* scount;      // [nsys][32]: per-system count of block phases published (one 128-byte line each, zeroed per launch)
  int* active;
  int* out_it;           // [nsys] iterations
  double* out_res;       // [nsys] final residual norm
  double* out_tol;       // [nsys] tolerance the system was solved to
  int* out_outer;        // [nsys] FP64 residual evaluations
  double eta;
  int floor;             // CG: a residual at the rounding of b - A x counts as converged (decide)
  int iter_cap;
  GridBarrier gb;
};

struct LocalSys {
  int sys, state, act, it, outer, par, first, pend, met, maxit, slot;
  int s0, s1;                       // partial slots of the system
  int j0, j1;                       // its slices in the block
  double tol, rtol, intol, res, rz_prev, alpha, beta, omega, irv;
  double sum[kMaxSums];
};

// sum of a partial array over the slots [t0, t1) by one warp, in a fixed order
__device__ __forceinline__ double slot_sum(const double* part, int t0, int t1, int lane) {
  double s = 0.0;
  for (int tb = t0; tb < t1; tb += 320) {
    double v[10];
#pragma unroll
    for (int u = 0; u < 10; ++u) {
      const int t = tb + u * 32 + lane;
      v[u] = t < t1 ? __ldcg(part + t) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 10; ++u) s += v[u];
  }
  return warp_sum(s);
}

// partial sums that a step needs from its system's previous phase
__device__ __forceinline__ int sums_of(int state) {
  return state == S_A ? 5 : state == S_C1 ? 3 : state == S_OUT_B ? 2 : state == S_B ? 1 : 0;
}

// the next step of a system from the sums of its previous phase (one thread;
// identical in every block of the system). at_floor: a CG cycle that reached
// its goal by the recurrences without halving the FP64 residual has come to
// the rounding of b - A x, which no further cycle lowers: the system is
// finished, and that residual is the tolerance it was solved to.
__device__ __forceinline__ void decide(LocalSys& L, bool bicg, bool at_floor, double eta) {
  const double* s = L.sum;
  switch (L.state) {
    case S_OUT_A:
      L.act = ACT_OUT_A;
      L.state = S_OUT_B;
      break;
    case S_OUT_B: {
      const double before = L.res;
      L.res = sqrt(s[0]);
      // the first FP64 residual also summed |b|^2: the relative tolerance
      if (L.outer == 0) L.tol = fmax(L.tol, L.rtol * sqrt(s[1]));
      L.outer += 1;
      if (at_floor && L.met && (L.it >= L.maxit ? L.intol <= L.tol : L.res > 0.5 * before)) L.tol = fmax(L.tol, L.res);
      if (L.res <= L.tol || L.it >= L.maxit || (bicg && L.outer > L.maxit) || !(L.res == L.res)) {
        L.act = ACT_FINISH;
        L.state = S_DONE;
      } else {
        L.intol = fmax(eta * L.res, at_floor ? L.tol : 0.5 * L.tol);
        L.first = 1;
        L.met = 0;
        L.beta = 0.0;
        L.rz_prev = L.res * L.res;  // BiCGStab: rho = (rh, r) with rh = r
        L.act = bicg ? ACT_P1 : ACT_C0;
        L.state = bicg ? S_B : S_C1;
      }
      break;
    }
    case S_A: {
      // BiCGStab after P2: (t,s), (t,t), (rh,s), (rh,t), (s,s)
      // (one division deep: beta = (rho / rho_prev) (alpha / omega) with
      // alpha / rho_prev = 1 / (rh, v))
      const double om = s[1] > 0.0 ? s[0] / s[1] : 0.0, iom = s[1] / s[0];
      const double rr = s[4] - 2.0 * om * s[0] + om * om * s[1];  // |s - omega t|^2
      const double rho = s[2] - om * s[3];
      L.omega = om;
      L.it += 1;
      // a rho that is mostly the rounding of its sum is no direction: the solve
      // would wander, up to max_iter on the rounding-sized cross components of a
      // pipe, so the next cycle takes a new shadow residual (1e-12 |rh| |r|: at
      // most 83 iterations over 8 steps of the 442k-cell pipe, FP64, where 1e-13
      // had 163, an exact zero 10,000)
      if (!(om != 0.0) || !(fabs(rho) > 1e-12 * L.res * sqrt(rr)) || rr <= L.intol * L.intol || L.it >= L.maxit || !(rr == rr)) {
        L.pend = 1;  // x += omega K^-1 s is folded into the FP64 residual
        L.act = ACT_OUT_A;
        L.state = S_OUT_B;
      } else {
        L.beta = rho * L.irv * iom;
        L.rz_prev = rho;
        L.act = ACT_P1;
        L.state = S_B;
      }
      break;
    }
    case S_B: {
      const double rv = s[0];  // (rh, v)
      L.first = 0;
      L.pend = 0;
      if (!(rv != 0.0) || !(rv == rv)) {
        L.act = ACT_OUT_A;  // breakdown: restart from the FP64 residual
        L.state = S_OUT_B;
      } else {
        L.irv = 1.0 / rv;
        L.alpha = L.rz_prev / rv;
        L.act = ACT_P2;
        L.state = S_A;
      }
      break;
    }
    case S_C1: {
      // CG: (r, u), (w, u), (r, r) of the previous phase; beta = gamma /
      // gamma_old, alpha = gamma / (delta - beta gamma / alpha_old)
      const double g = s[0], dl = s[1], rr = s[2];
      if (L.first == 1) {
        L.first = 2;
        L.alpha = dl != 0.0 ? g / dl : 0.0;
        L.beta = 0.0;
        L.rz_prev = g;
        L.act = ACT_C1;
      } else {
        L.first = 0;
        L.it += 1;
        const double be = L.rz_prev != 0.0 ? g / L.rz_prev : 0.0;
        const double den = dl - (L.alpha != 0.0 ? be * g / L.alpha : 0.0);
        if (rr <= L.intol * L.intol || L.it >= L.maxit || !(rr == rr) || !(den > 0.0)) {
          L.met = rr <= L.intol * L.intol;
          L.act = ACT_OUT_A;  // reliable update in FP64
          L.state = S_OUT_B;
        } else {
          L.beta = be;
          L.alpha = g / den;
          L.rz_prev = g;
          L.act = ACT_C1;
        }
      }
      break;
    }
    default:
      L.act = ACT_NONE;
      break;
  }
}

// CL: the grid is one thread-block cluster. The blocks then exchange their
// partial sums through each other's shared memory and meet at the cluster's
// hardware barrier (about 0.5 us) instead of publishing to and polling
// counters in L2 (about 2 us a phase): small systems, whose phases are short.
__device__ __forceinline__ void cluster_sync_ra() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// stores v at the address that p has in the shared memory of block `rank` of the cluster
__device__ __forceinline__ void st_cluster(double* p, unsigned rank, double v) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(p);
  unsigned remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(v) : "memory");
}

template <typename R, int MINB, int SM, bool CL>
__global__ void __launch_bounds__(SolveThreads<MINB>::value, MINB) k_krylov(SolveArgs<R> a) {
  constexpr int kSolveThreads = SolveThreads<MINB>::value, kWarps = kSolveThreads / 32;
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  constexpr int CH = Chunk<R>::value;
  __shared__ LocalSys ls[kMaxRunSys];
  __shared__ int s_err;
  __shared__ double s_pub[CL ? 2 * 3 * kMaxSums * kClusterMax : 1];  // [parity][system][sum][block]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t nv = (size_t)a.nv;
  const int NC = a.ncomp;
  const int io = a.blk_inst_off[blockIdx.x];
  const int nls = min((a.blk_inst_off[blockIdx.x + 1] - io) * NC, kMaxRunSys);
  const int bs0 = a.blk_sl[blockIdx.x], bs1 = a.blk_sl[blockIdx.x + 1];
  const int nitems = (bs1 - bs0) * NC, own0 = bs0 * 32;
  const int NS = a.bicg ? kMaxSums : 3;
  const int split = a.split, group = warp / split, part = warp - group * split, ngroups = kWarps / split;
  unsigned bar_gen = 0;

  // ---- shared memory: partial products of split items, the items' partial
  // sums, then the staged static data
  double* const s_dot = reinterpret_cast<double*>(dyn_smem);
  double* spart;
  unsigned char* cur = dyn_smem;
  if constexpr (SM < 0) {
    spart = a.item_part + (size_t)blockIdx.x * a.items_max * NS;
  } else {
    spart = s_dot + (split > 1 ? kWarps * 32 : 0);
    cur = reinterpret_cast<unsigned char*>(spart) + al16_dev((size_t)a.items_max * NS * sizeof(double));
  }
  // own rows of the vectors that no product gathers: by item in shared memory
  R *ve, *vr, *vs, *vt, *vv, *vh;
  const int *SLp, *SLl, *SLk, *SLc;  // by slice - bs0; columns by entry - e0
  const R *A0, *A1, *A2;
  const int e0 = a.sl_ptr[bs0], ne = a.sl_ptr[bs1] - e0;
  if constexpr (SM >= 1) {
    const int n = a.items_max * 32;
    ve = reinterpret_cast<R*>(cur);
    vr = ve + n;
    vs = ve + 2 * n;
    vt = ve + 3 * n;
    vv = ve + 4 * n;
    vh = ve + 5 * n;
    cur += al16_dev((size_t)6 * n * sizeof(R));
    SLp = stage_copy(cur, a.sl_ptr + bs0, bs1 - bs0);
    SLl = stage_copy(cur, a.sl_len + bs0, bs1 - bs0);
    SLk = stage_copy(cur, a.slk + bs0, bs1 - bs0);
  } else {
    ve = a.e;
    vr = a.r;
    vs = a.s;
    vt = a.t;
    vv = a.v;
    vh = a.rh;
    SLp = a.sl_ptr + bs0;
    SLl = a.sl_len + bs0;
    SLk = a.slk + bs0;
  }
  if constexpr (SM >= 2) SLc = stage_copy(cur, a.sl_col + e0, ne);
  else SLc = a.sl_col + e0;
  if constexpr (SM >= 3) {
    A0 = stage_copy(cur, a.Ain[0] + e0, ne);
    A1 = a.share || NC < 2 ? A0 : stage_copy(cur, a.Ain[1] + e0, ne);
    A2 = a.share || NC < 3 ? A0 : stage_copy(cur, a.Ain[2] + e0, ne);
  } else {
    A0 = a.Ain[0] + e0;
    A1 = a.Ain[1] + e0;
    A2 = a.Ain[2] + e0;
  }

  // ---- local systems: component k of local instance i is system i NC + k
  if (threadIdx.x == 0) s_err = 0;
  for (int l = threadIdx.x; l < nls; l += kSolveThreads) {
    LocalSys& L = ls[l];
    const int inst = a.blk_inst[io + l / NC], s = (l % NC) * a.ninst + inst;
    L.sys = s;
    L.state = S_OUT_A;
    L.act = ACT_NONE;
    L.it = L.outer = L.par = L.pend = L.met = 0;
    L.first = 1;
    L.s0 = a.sys_slot0[s];
    L.s1 = a.sys_slot0[s + 1];
    L.slot = L.s0 + a.blk_slot[io + l / NC];
    L.j0 = 0;
    while (L.j0 < bs1 - bs0 && a.slk[bs0 + L.j0] != l / NC) ++L.j0;
    L.j1 = L.j0;
    while (L.j1 < bs1 - bs0 && a.slk[bs0 + L.j1] == l / NC) ++L.j1;
    L.maxit = a.maxit_i[inst];
    L.tol = a.tol_i[inst];
    L.rtol = a.rtol_i[inst];
    L.intol = 0.5 * L.tol;
    L.res = L.rz_prev = L.alpha = L.beta = L.omega = L.irv = 0.0;
  }
  // ---- init: Dirichlet values preset in x, e = 0
  for (int k = 0; k < NC; ++k)
    for (int i = threadIdx.x; i < (bs1 - bs0) * 32; i += kSolveThreads) {
      const int row = own0 + i;
      if (a.isd[k][row]) a.x[k][row] = a.g[k] ? a.g[k][row] : 0.0;
      a.e[k * nv + row] = R(0);
    }
  if (SM >= 1)
    for (int i = threadIdx.x; i < nitems * 32; i += kSolveThreads) ve[i] = R(0);
  if constexpr (CL) cluster_sync_ra();
  else if (!grid_sync_ra(a.gb, bar_gen)) return;

  for (int iter = 0;; ++iter) {
    if (iter >= a.iter_cap) {
      if (threadIdx.x == 0) atomicCAS(a.gb.err, 0, 2);
      break;
    }
    // ---- phase start: every block of a system adds 1 to its counter once
    // its phase is written, so iter x (blocks of the system) means that all
    // have finished phase iter - 1; the acquire orders what they wrote before
    // this phase's reads. A warp per (local system, sum) waits and sums that
    // phase's partials, then a thread per system takes the next step.
    if constexpr (CL) {
      for (int l = warp; l < nls; l += kWarps) {
        LocalSys& L = ls[l];
        if (iter > 0 && lane < sums_of(L.state)) {
          const double* v = s_pub + ((((iter + 1) & 1) * 3 + l) * kMaxSums + lane) * kClusterMax;
          double t = 0.0;
          for (int b = 0; b < (int)gridDim.x; ++b) t += v[b];
          L.sum[lane] = t;
        }
        __syncwarp();
        if (lane == 0) decide(L, a.bicg != 0, a.floor != 0, a.eta);
      }
      __syncthreads();
    } else {
      const double* prev = a.part + (size_t)((iter + 1) & 1) * kMaxSums * a.nslots;
      for (int t = warp; t < nls * kMaxSums; t += kWarps) {
        // (the first sums of all systems first)
        const int q = t / nls, l = t - q * nls;
        const LocalSys& L = ls[l];
        if (L.state == S_DONE || iter == 0 || (q > 0 && q >= sums_of(L.state))) continue;
        if (!wait_count(a.scount + (size_t)L.sys * 32, (unsigned)iter * (unsigned)(L.s1 - L.s0), a.gb)) {
          if (lane == 0) {
            atomicCAS(a.gb.err, 0, 1);
            s_err = 1;
          }
          break;
        }
        if (q < sums_of(L.state)) {
          const double s = slot_sum(prev + (size_t)q * a.nslots, L.s0, L.s1, lane);
          if (lane == 0) ls[l].sum[q] = s;
        }
      }
      __syncthreads();
      if (threadIdx.x < nls) decide(ls[threadIdx.x], a.bicg != 0, a.floor != 0, a.eta);
      __syncthreads();
    }
    if (s_err) break;
    bool any = false;
    for (int l = 0; l < nls; ++l) any |= ls[l].act != ACT_NONE;
    if (!any) break;  // every local system is done
    // ---- the block's (slice, component) items, `split` warps per item: each
    // takes a run of the row's entries, the first adds up their products
    for (int it = group < ngroups ? group : nitems; it < nitems; it += ngroups) {
      const int sl = bs0 + it / NC, k = it % NC;
      const LocalSys& L = ls[SLk[sl - bs0] * NC + k];
      const int act = L.act;
      if (act == ACT_NONE) continue;
      double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0, v4 = 0.0;
      const int row = sl * 32 + lane;
      const size_t g0 = k * nv + row, o = SM >= 1 ? (size_t)(it * 32 + lane) : g0;
      int nj = SLl[sl - bs0], p0 = SLp[sl - bs0] - e0;
      if (split > 1) {
        const int j0 = nj * part / split;
        nj = nj * (part + 1) / split - j0;
        p0 += 32 * j0;
      }
      const auto row_dot = [&](auto zero, const auto& val, const auto& gx) {
        using T = decltype(zero);
        T acc = sell_dot<T, CH>(zero, SLc, p0, nj, lane, val, gx);
        if (split > 1) {  // (a group has one item per phase: its slots are free)
          T* const d = reinterpret_cast<T*>(s_dot + 32 * warp);
          d[lane] = acc;
          asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(32 * split) : "memory");
          if (part == 0)
            for (int u = 1; u < split; ++u) acc += reinterpret_cast<const T*>(s_dot + 32 * (warp + u))[lane];
        }
        return acc;
      };
      const R* dinv = a.dinv[k];
      const R* A = k == 0 ? A0 : (k == 1 ? A1 : A2);
      const auto aval = [&](int ei) { return A[ei]; };
      const double* r64 = a.r64 + k * nv;
      const V4<R>* pk = a.pk + (size_t)(L.par * NC + k) * nv;
      V4<R>* pn = a.pk + (size_t)((L.par ^ 1) * NC + k) * nv;
      if (act == ACT_OUT_A) {
        const double* A64 = a.A64[k] + e0;
        const double* xk = a.x[k];
        const R* e = a.e + k * nv;
        const bool pend = L.pend != 0;
        const R al = R(L.alpha), om = R(L.omega);
        const double bb = a.b[k][row];
        const double acc = row_dot(0.0, [&](int ei) { return A64[ei]; }, [&](int j) {
          R ee = __ldcg(e + j);
          if (pend) {
            R zr, w;
            ld2(pk + j, zr, w);
            ee = fma_r(om, fma_r(-al, w, zr), ee);  // the last step's omega K^-1 s
          }
          return __ldcg(xk + j) + (double)ee;
        });
        if (part) continue;
        const double rr = bb - acc;
        a.r64[g0] = rr;
        v0 = rr * rr;
        v1 = bb * bb;
      } else if (act == ACT_FINISH) {
        if (part) continue;
        R ee = ve[o];
        if (L.pend) {
          R zr, w;
          ld2(pk + row, zr, w);
          ee = fma_r(R(L.omega), fma_r(-R(L.alpha), w, zr), ee);
        }
        a.x[k][row] += (double)ee;
        continue;
      } else if (act == ACT_P1) {
        // y' = zr' + beta (y - omega w), zr' = zr - alpha w - omega kt the
        // preconditioned new residual (after a restart y' = zr' = K^-1 r64),
        // v = A y' with y' formed on the fly at the columns, w' = K^-1 v
        // (own-row loads first: a warp issues in order, so that their round
        // trip and the gathers' are one)
        R yrow, zr_row, acc;
        const R di = dinv[row];
        const R e_old = ve[o];
        if (L.first) {
          const R rr = R(__ldcg(r64 + row));
          const double xo = a.x[k][row];
          R zr = R(0), w = R(0);
          if (L.pend) ld2(pk + row, zr, w);
          acc = row_dot(R(0), aval, [&](int j) { return R(__ldcg(r64 + j)) * dinv[j]; });
          if (part) continue;
          const R ee = L.pend ? fma_r(R(L.omega), fma_r(-R(L.alpha), w, zr), e_old) : e_old;
          a.x[k][row] = xo + (double)ee;
          ve[o] = R(0);
          if (SM >= 1) a.e[g0] = R(0);
          vr[o] = rr;
          vh[o] = rr;
          yrow = zr_row = rr * di;
          v0 = (double)rr * (double)acc;
        } else {
          const R al = R(L.alpha), om = R(L.omega), be = R(L.beta);
          const auto ynew = [&](const V4<R>& g) {
            const R zr = fma_r(-om, g.d, fma_r(-al, g.b, g.a));
            return fma_r(be, fma_r(-om, g.b, g.c), zr);
          };
          const V4<R> g = ld4(pk + row);
          const R t_old = vt[o], s_old = vs[o], rh = vh[o];
          acc = row_dot(R(0), aval, [&](int j) { return ynew(ld4(pk + j)); });
          if (part) continue;
          const R zs = fma_r(-al, g.b, g.a);
          const R ee = fma_r(om, zs, e_old);
          ve[o] = ee;
          if (SM >= 1) a.e[g0] = ee;  // read by the FP64 residual at its columns
          vr[o] = fma_r(-om, t_old, s_old);
          zr_row = fma_r(-om, g.d, zs);
          yrow = ynew(g);
          v0 = (double)rh * (double)acc;
        }
        pn[row] = V4<R>{zr_row, acc * di, yrow, R(0)};
        vv[o] = acc;
      } else if (act == ACT_P2) {
        // e += alpha y, s = r - alpha v, t = A K^-1 s (K^-1 s = zr - alpha w
        // formed on the fly), kt = K^-1 t; sums (t,s) (t,t) (rh,s) (rh,t) (s,s)
        const R al = R(L.alpha);
        const R y = pk[row].c, e_old = ve[o], v_old = vv[o], r_old = vr[o], di = dinv[row];
        const double rh = (double)vh[o];
        const R tv = row_dot(R(0), aval, [&](int j) {
          R zr, w;
          ld2(pk + j, zr, w);
          return fma_r(-al, w, zr);
        });
        if (part) continue;
        const R sv = fma_r(-al, v_old, r_old);
        const R ee = fma_r(al, y, e_old);
        ve[o] = ee;
        if (SM >= 1) a.e[g0] = ee;
        vs[o] = sv;
        vt[o] = tv;
        const_cast<V4<R>*>(pk)[row].d = tv * di;
        v0 = (double)tv * (double)sv;
        v1 = (double)tv * (double)tv;
        v2 = rh * (double)sv;
        v3 = rh * (double)tv;
        v4 = (double)sv * (double)sv;
      } else if (act == ACT_C0) {
        // restart: u = K^-1 r64, w = A u, wh = K^-1 w; (r, u), (w, u), (r, r)
        const R e_old = ve[o], rr = R(__ldcg(r64 + row)), di = dinv[row], u = rr * di;
        const double xo = a.x[k][row];
        const R w = row_dot(R(0), aval, [&](int j) { return R(__ldcg(r64 + j)) * dinv[j]; });
        if (part) continue;
        a.x[k][row] = xo + (double)e_old;
        ve[o] = R(0);
        if (SM >= 1) a.e[g0] = R(0);
        vr[o] = rr;
        vv[o] = w;
        pn[row] = V4<R>{u, w * di, R(0), R(0)};
        v0 = (double)rr * (double)u;
        v1 = (double)w * (double)u;
        v2 = (double)rr * (double)rr;
      } else {
        // C1: p = u + beta p, s = w + beta s, sh = wh + beta sh, e += alpha p,
        // r -= alpha s, u' = u - alpha sh (= K^-1 r'), w' = A u' with u'
        // formed on the fly at the columns, wh' = K^-1 w'; (r', u'), (w', u'),
        // (r', r'). The first iteration after a restart has p = u, s = w, sh = wh.
        const bool first = L.first != 0;
        const R al = R(L.alpha), be = R(L.beta);
        const auto shn = [&](const V4<R>& g) { return first ? g.b : fma_r(be, g.c, g.b); };
        const V4<R> g = ld4(pk + row);
        const R p_old = vt[o], s_old = vs[o], w_old = vv[o], e_old = ve[o], r_old = vr[o], di = dinv[row];
        const R w = row_dot(R(0), aval, [&](int j) {
          const V4<R> h = ld4(pk + j);
          return fma_r(-al, shn(h), h.a);
        });
        if (part) continue;
        const R sh = shn(g), un = fma_r(-al, sh, g.a);
        const R pp = first ? g.a : fma_r(be, p_old, g.a);
        const R ss = first ? w_old : fma_r(be, s_old, w_old);
        const R rn = fma_r(-al, ss, r_old);
        vt[o] = pp;
        vs[o] = ss;
        const R ee = fma_r(al, pp, e_old);
        ve[o] = ee;
        if (SM >= 1) a.e[g0] = ee;
        vr[o] = rn;
        pn[row] = V4<R>{un, w * di, sh, R(0)};
        vv[o] = w;
        v0 = (double)rn * (double)un;
        v1 = (double)w * (double)un;
        v2 = (double)rn * (double)rn;
      }
      // the item's partial sums (warp order is fixed: deterministic)
      double* sp = spart + (size_t)NS * it;
      if (act == ACT_P2) {
        double v[8] = {v0, v1, v2, v3, v4, 0.0, 0.0, 0.0};
        const double tot = warp_sum_many<8, double>(v, lane);
        const int q = warp_sum_many_index<8>(lane);
        if ((lane & 3) == 0 && q < kMaxSums) sp[q] = tot;
      } else if (act == ACT_P1) {
        v0 = warp_sum(v0);
        if (lane == 0) sp[0] = v0;
      } else {
        double v[4] = {v0, v1, v2, 0.0};
        const double tot = warp_sum_many<4, double>(v, lane);
        const int q = warp_sum_many_index<4>(lane);
        if ((lane & 7) == 0 && q < 3) sp[q] = tot;
      }
    }
    __syncthreads();
    // ---- publish, a warp per local system: the block's partial sums (items
    // in a fixed order) into this phase's parity, then a release add on the
    // system's counter, which after the block barrier above covers every
    // write of the block's phase
    for (int l = warp; l < nls; l += kWarps) {
      LocalSys& L = ls[l];
      const int act = L.act, k = l % NC;
      const int ns = act == ACT_P2 ? kMaxSums : act == ACT_P1 ? 1 : act == ACT_NONE || act == ACT_FINISH ? 0 : 3;
      double s = 0.0;
      {
        // lanes q, q + 8, q + 16 and q + 24 add up sum q
        const int q = lane & 7;
        if (q < ns)
#pragma unroll 4
          for (int j = L.j0 + (lane >> 3); j < L.j1; j += 4) s += spart[NS * (j * NC + k) + q];
        s += __shfl_xor_sync(PFEM2_FULL_MASK, s, 8);
        s += __shfl_xor_sync(PFEM2_FULL_MASK, s, 16);
      }
      if constexpr (CL) {
        for (int q = 0; q < ns; ++q) {
          const double v = __shfl_sync(PFEM2_FULL_MASK, s, q);
          if (lane < (int)gridDim.x)
            st_cluster(s_pub + (((iter & 1) * 3 + l) * kMaxSums + q) * kClusterMax + blockIdx.x, lane, v);
        }
      } else if (lane < ns) {
        a.part[((size_t)(iter & 1) * kMaxSums + lane) * a.nslots + L.slot] = s;
      }
      __syncwarp();
      if (lane == 0) {
        if (!CL) red_release_add_u32(a.scount + (size_t)L.sys * 32, 1u);
        if (act == ACT_P1 || act == ACT_C0 || act == ACT_C1) L.par ^= 1;
        if (act == ACT_FINISH && L.slot == L.s0) {
          a.out_it[L.sys] = L.it;
          a.out_res[L.sys] = L.res;
          a.out_tol[L.sys] = L.tol;
          a.out_outer[L.sys] = L.outer;
          atomicSub(a.active, 1);
        }
      }
    }
    if constexpr (CL) cluster_sync_ra();
  }
}

// ------------------------------------------------------------------ host
template <typename R, int MINB>
static const void* kernel_of(int sm) {
  return sm < 0    ? (const void*)k_krylov<R, MINB, -1, false>
         : sm == 0 ? (const void*)k_krylov<R, MINB, 0, false>
         : sm == 1 ? (const void*)k_krylov<R, MINB, 1, false>
         : sm == 2 ? (const void*)k_krylov<R, MINB, 2, false>
                   : (const void*)k_krylov<R, MINB, 3, false>;
}

template <typename R>
static const void* kernel_of(int minb, int sm, bool cluster) {
  if (cluster) return sm == 2 ? (const void*)k_krylov<R, 1, 2, true> : (const void*)k_krylov<R, 1, 3, true>;
  return minb == 1 ? kernel_of<R, 1>(sm) : kernel_of<R, 2>(sm);
}

static const void* kernel_of(bool mixed, int minb, int sm, bool cluster) {
  return mixed ? kernel_of<float>(minb, sm, cluster) : kernel_of<double>(minb, sm, cluster);
}

static int occupancy(bool mixed, int minb, int sm, size_t smem) {
  const void* k = kernel_of(mixed, minb, sm, false);
  int occ = 0;
  // one process-wide upper bound, so contexts with different systems coexist
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_budget(minb));
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, solve_threads(minb), smem) != cudaSuccess) return 0;
  return occ;
}

static void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at, int grid, size_t smem, cudaStream_t st) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(solve_threads(1));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = grid;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
}

// whether the device can hold one cluster of `grid` such blocks
static bool cluster_fits(bool mixed, int sm, int grid, size_t smem) {
  const void* k = kernel_of(mixed, 1, sm, true);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  cluster_config(cfg, at, grid, smem, 0);
  int n = 0;
  const bool ok =
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_budget(1)) == cudaSuccess &&
      cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
      cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n >= 1;
  if (!ok) cudaGetLastError();
  return ok;
}

// the items' partial sums of a block
static size_t plan_partials(const JacobiPlan& P) {
  return al16(sizeof(double) * (P.bicg ? kMaxSums : 3) * (size_t)P.items_max);
}

// shared memory of a block and what it holds
static size_t plan_smem(const JacobiPlan& P, size_t rs, int minb, int nmat, int& sm) {
  sm = P.item_part ? -1 : 0;
  if (sm < 0) return 0;
  size_t smem = plan_partials(P) + (P.split > 1 ? sizeof(double) * solve_threads(minb) : 0);
  const size_t level[3] = {al16(6 * 32 * rs * (size_t)P.items_max) + P.st_meta, al16(4 * P.st_entries),
                           nmat * al16(rs * P.st_entries)};
  while (sm < 3 && smem + level[sm] <= smem_budget(minb)) smem += level[sm++];
  return smem;
}

// the blocks' slice runs: G equal runs of the slices, whose instances are
// given by their slice offsets ioff (ascending, ioff.back() = all)
static pfem2_status plan_runs(JacobiPlan& P, std::vector<int> (&up)[6], const std::vector<int>& ioff,
                              const std::vector<int>& slp, int ncomp, int G) {
  const int ni = (int)ioff.size() - 1, ns = ioff.back();
  std::vector<int>&bsl = up[0], &binst = up[1], &binst_off = up[2], &bslot = up[3], &slot0 = up[4], &slk = up[5];
  std::vector<int> cnt(ni, 0);
  bsl.assign(G + 1, 0);
  binst.clear();
  bslot.clear();
  binst_off.assign(1, 0);
  slot0.assign(ncomp * ni + 1, 0);
  slk.assign(ns, 0);
  for (int b = 0; b <= G; ++b) bsl[b] = (int)((long long)ns * b / G);
  P.grid = G;
  P.items_max = P.sys_max = 0;
  P.st_meta = P.st_entries = 0;
  for (int b = 0, i = 0; b < G; ++b) {
    const int s0 = bsl[b], s1 = bsl[b + 1];
    while (ioff[i + 1] <= s0) ++i;
    int last = i - 1;
    for (int sl = s0, j = i; sl < s1; ++sl) {
      while (ioff[j + 1] <= sl) ++j;
      for (; last < j; ++last) {
        binst.push_back(last + 1);
        bslot.push_back(cnt[last + 1]++);
      }
      slk[sl] = j - i;
    }
    binst_off.push_back((int)binst.size());
    if ((binst_off[b + 1] - binst_off[b]) * ncomp > kMaxRunSys) {
      set_error("krylov: more than 24 systems would share one block (instances too small for the batch)");
      return PFEM2_INVALID_ARG;
    }
    P.items_max = std::max(P.items_max, (s1 - s0) * ncomp);
    P.sys_max = std::max(P.sys_max, (binst_off[b + 1] - binst_off[b]) * ncomp);
    P.st_meta = std::max(P.st_meta, 3 * al16(4 * (size_t)(s1 - s0)));
    P.st_entries = std::max(P.st_entries, (size_t)(slp[s1] - slp[s0]));
  }
  for (int k = 0; k < ncomp; ++k)
    for (int i = 0; i < ni; ++i) slot0[k * ni + i + 1] = slot0[k * ni + i] + cnt[i];
  P.nslots = slot0.back();
  return PFEM2_OK;
}

// Partition of a solve: one cluster where the systems are small, else blocks
// of at least `ts` slices, minb to an SM (0: by size). mixed: the inner type.
static pfem2_status plan_build(Ctx& c, KrylovWs* w, JacobiPlan& P, bool mixed, const std::vector<int>& ioff,
                               const std::vector<int>& slp, int ncomp, int nmat, int minb, int ts, bool try_cluster) {
  const int ni = (int)ioff.size() - 1, ns = ioff.back();
  const size_t rs = mixed ? sizeof(float) : sizeof(double);
  std::vector<int> up[6];
  int len = 0;  // the longest row, and the rounds of loads it takes
  for (int sl = 0; sl < ns; ++sl) len = std::max(len, (slp[sl + 1] - slp[sl]) / kSlice);
  const int ch = mixed ? Chunk<float>::value : Chunk<double>::value, rounds = (len + ch - 1) / ch;
  // warps that would have no item share the others': as many as shorten a row's
  // rounds of loads, each group of warps with one item at most. An iteration of
  // the mesh elasticity (17k rows of 18 entries, FP64) takes 6.0 us instead of
  // 8.5 with four warps to an item; 10k-cell pipe (27 entries, FP64), prediction
  // and correction 1.42 ms instead of 1.65 with two; 13k-cell channel, FP64,
  // 0.41 instead of 0.45.
  const auto set_split = [&] {
    const auto rounds_of = [&](int n) { return ((len + n - 1) / n + ch - 1) / ch; };
    const int most = std::min(solve_threads(P.minb) / 32 / std::max(1, P.items_max), rounds);
    P.split = 1;
    for (int k = 2; k <= most; ++k)
      if (rounds_of(k) < rounds_of(P.split)) P.split = k;
  };
  P.cluster = false;
  if (try_cluster && ni == 1 && ns * ncomp <= kClusterItems) {
    int G = 1;
    while (2 * G <= kClusterMax && 4 * G <= ns) G *= 2;
    PFEM2_TRY(plan_runs(P, up, ioff, slp, ncomp, G));
    P.minb = 1;
    set_split();
    const size_t smem = plan_smem(P, rs, 1, nmat, P.sm);
    if (P.sm >= 2 && cluster_fits(mixed, P.sm, G, smem)) {
      P.cluster = true;
    }
  }
  if (!P.cluster) {
    // one block per SM, but at least four slices in each where a row is one
    // round of loads (13k rows, FP32: 0.39 ms per step with four, 0.40 with
    // two, 0.42 with six), three with two rounds (FP64: 0.41 with three, 0.42
    // with four, 0.46 with six), two with more (10k-cell pipe, FP64: 1.42 with
    // two, 1.46 with three, 1.57 with four)
    const int ts_auto = std::max(std::max(2, 5 - rounds), (ns + c.num_sms - 1) / c.num_sms);
    // one system: a block of 768 threads per SM, so that few blocks are waited
    // for (52k channel: prediction and correction 0.45 ms per step against
    // 0.55 with two blocks of 384; 131k pipe 3.58 against 3.77), unless 12
    // warps hold its items in one round of loads (13k rows: one round, FP32; two,
    // FP64, where 768 threads take 0.42 ms and 384 take 0.45); a batch takes two of 384, whose
    // instances wait less for each other (16 channels: 1.38 against 1.44 ms)
    P.minb = minb ? minb : (ni > 1 || ts_auto * ncomp * rounds <= 12 ? 2 : 1);
    if (!ts) ts = ni > 1 ? 4 : ts_auto;
    P.ts = ts;
    const int occ = std::min(P.minb, occupancy(mixed, P.minb, 0, 0));
    if (occ < 1) {
      set_error("krylov: the solver kernel cannot be resident");
      return PFEM2_CUDA_ERROR;
    }
    // (more blocks than ts asks for where such a run would touch too many instances)
    const int most = std::max(1, std::min(occ * c.num_sms, ns));
    int G = std::max(1, std::min(most, (ns + ts - 1) / ts));
    pfem2_status st;
    while ((st = plan_runs(P, up, ioff, slp, ncomp, G)) != PFEM2_OK && G < most) G = std::min(most, 2 * G);
    PFEM2_TRY(st);
    set_split();
  }
  // Blocks of very long runs (3D BiCGStab from 8M rows on, 13M with CG) keep
  // their items' partial sums in global memory: 40 of the some 10,000 bytes
  // that a phase moves per item. Such a block has more items than warps (split 1).
  if (!P.cluster && plan_partials(P) > std::min((size_t)c.partials_max, smem_budget(P.minb)) && P.split == 1)
    PFEM2_TRY(ws_alloc(w, &P.item_part, (size_t)P.grid * plan_partials(P) / sizeof(double)));
  int** dst[6] = {&P.blk_sl, &P.blk_inst, &P.blk_inst_off, &P.blk_slot, &P.sys_slot0, &P.slk};
  for (int k = 0; k < 6; ++k) PFEM2_TRY(ws_upload(w, dst[k], up[k]));
  return PFEM2_OK;
}

template <typename R>
static void plan_args(const KrylovWs* w, const JacobiPlan& P, SolveArgs<R>& a) {
  a.blk_inst = P.blk_inst;
  a.blk_inst_off = P.blk_inst_off;
  a.blk_slot = P.blk_slot;
  a.sys_slot0 = P.sys_slot0;
  a.blk_sl = P.blk_sl;
  a.slk = P.slk;
  a.items_max = P.items_max;
  a.item_part = P.item_part;
  a.split = P.split;
  a.nslots = P.nslots;
  a.bicg = P.bicg;
  a.scount = w->scount;
  a.active = w->active;
}

template <typename R>
static pfem2_status plan_launch(Ctx& c, const JacobiPlan& P, SolveArgs<R>& a, int nmat) {
  a.gb.count = c.barrier;
  a.gb.gen = c.barrier + 1;
  a.gb.err = c.d_err;
  a.gb.spin_limit = c.spin_limit;
  int sm = 0;
  const size_t smem = plan_smem(P, sizeof(R), P.minb, nmat, sm);
  const void* kern = kernel_of<R>(P.minb, sm, P.cluster);
  void* args[] = {&a};
  if (P.cluster) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    cluster_config(cfg, at, P.grid, smem, c.stream);
    PFEM2_CUDA(cudaLaunchKernelExC(&cfg, kern, args));
  } else {
    PFEM2_CUDA(cudaLaunchCooperativeKernel(kern, dim3(P.grid), dim3(solve_threads(P.minb)), args, smem, c.stream));
  }
  c.launches++;
  return PFEM2_OK;
}

void krylov_free(Ctx& c) {
  KrylovWs* w = (KrylovWs*)c.kws;
  if (!w) return;
  mg_free(w);
  for (void* p : w->allocs) cudaFree(p);
  delete w;
  c.kws = nullptr;
}

// whether the grid of a flow solve is resident with its shared memory (a
// cluster's is checked with its plan)
static pfem2_status plan_resident(Ctx& c, int which) {
  const KrylovWs* w = (const KrylovWs*)c.kws;
  const JacobiPlan& P = w->plan[which == 1 ? 0 : 1];
  if (P.cluster) return PFEM2_OK;
  int sm = 0;
  const size_t smem = plan_smem(P, c.kmixed ? sizeof(float) : sizeof(double), P.minb,
                                which == 1 || (which == 2 && w->mass_share) ? 1 : c.dim, sm);
  if (occupancy(c.kmixed, P.minb, sm, smem) * c.num_sms < P.grid) {
    set_error("krylov: the solver grid cannot be resident");
    return PFEM2_CUDA_ERROR;
  }
  return PFEM2_OK;
}

pfem2_status krylov_setup(Ctx& c) {
  KrylovWs* w = new KrylovWs();
  c.kws = w;
  const int dim = c.dim, ni = (int)c.inst.size();
  const size_t nv = c.nv, rs = c.kmixed ? sizeof(float) : sizeof(double);
  std::vector<int> ioff(1, 0);
  for (const HostInst& in : c.inst) ioff.push_back((in.v_off + in.nv_pad) / kSlice);
  int maxslots = 0;
  // plan 0: the pressure systems where the multigrid is not used, or may turn
  // out not to be (moving meshes)
  for (int ph = c.two_level && !c.moving ? 1 : 0; ph < 2; ++ph) {
    JacobiPlan& P = w->plan[ph];
    P.bicg = ph == 0 ? c.p_bicg : c.vel_bicg;
    const bool tuned = ph == 1 && (c.tune.vel_blocks_per_sm || c.tune.vel_tile_slices);
    PFEM2_TRY(plan_build(c, w, P, c.kmixed, ioff, c.h_sl_ptr, ph == 0 ? 1 : dim, ph == 0 ? 1 : dim,
                         ph == 0 ? 0 : c.tune.vel_blocks_per_sm, ph == 0 ? 0 : c.tune.vel_tile_slices, !tuned));
    maxslots = std::max(maxslots, P.nslots);
    // (the shape that makes this partition again when it is set; with a cluster
    // both fields stay automatic: any value would rule it out)
    if (ph == 1 && !P.cluster) {
      if (!c.tune.vel_blocks_per_sm) c.tune.vel_blocks_per_sm = P.minb;
      if (!c.tune.vel_tile_slices) c.tune.vel_tile_slices = P.ts;
    }
  }
  // systems whose components have the same Dirichlet rows share the mass matrix
  w->mass_share = true;
  {
    std::vector<unsigned char> d0(nv), dk(nv);
    PFEM2_CUDA(cudaMemcpy(d0.data(), c.isdir[0], nv, cudaMemcpyDeviceToHost));
    for (int k = 1; k < dim; ++k) {
      PFEM2_CUDA(cudaMemcpy(dk.data(), c.isdir[k], nv, cudaMemcpyDeviceToHost));
      w->mass_share = w->mass_share && d0 == dk;
    }
  }
  unsigned char* b[7];
  const size_t n[7] = {2 * 4 * nv * dim, nv * dim, nv * dim, nv * dim, nv * dim, nv * dim, nv * dim};
  for (int k = 0; k < 7; ++k) PFEM2_TRY(ws_alloc(w, &b[k], n[k] * rs));
  w->pk = b[0]; w->e = b[1]; w->r = b[2]; w->v = b[3]; w->s = b[4]; w->t = b[5]; w->rh = b[6];
  PFEM2_TRY(ws_alloc(w, &w->r64, nv * dim));
  PFEM2_TRY(ws_alloc(w, &w->part, 2 * (size_t)kMaxSums * maxslots));
  PFEM2_TRY(ws_alloc(w, &w->scount, 32 * (size_t)dim * ni));
  PFEM2_TRY(ws_alloc(w, &w->active, 1));
  for (int k = 0; k < 3; ++k) {
    PFEM2_TRY(ws_alloc(w, &w->out_it[k], dim * ni));
    PFEM2_TRY(ws_alloc(w, &w->out_res[k], dim * ni));
    PFEM2_TRY(ws_alloc(w, &w->out_tol[k], dim * ni));
    PFEM2_TRY(ws_alloc(w, &w->out_outer[k], dim * ni));
  }
  // (a cluster keeps the same operands in shared memory in every solve)
  for (int which = 0; which < 3; ++which)
    if (which != 1 || !c.two_level) PFEM2_TRY(plan_resident(c, which));
  return PFEM2_OK;
}

// Plan and vectors of the mesh elasticity (moving contexts, first use): one
// FP64 system of dim x nv rows whose components follow each other, on slices
// of its own (ale.cu).
static pfem2_status elastic_setup(Ctx& c, const std::vector<int>& slp) {
  KrylovWs* w = (KrylovWs*)c.kws;
  JacobiPlan& P = w->elastic;
  const std::vector<int> ioff = {0, (int)slp.size() - 1};
  const size_t n = (size_t)c.nv * c.dim;
  P.bicg = false;
  PFEM2_TRY(plan_build(c, w, P, false, ioff, slp, 1, 1, 0, 0, true));
  double** v[] = {&w->el_pk, &w->el_e, &w->el_r, &w->el_v, &w->el_s, &w->el_t, &w->el_r64, &w->el_part, &w->el_res};
  const size_t m[] = {2 * 4 * n, n, n, n, n, n, n, 2 * (size_t)kMaxSums * P.nslots, 4};
  for (int k = 0; k < 9; ++k) PFEM2_TRY(ws_alloc(w, v[k], m[k]));
  PFEM2_TRY(ws_alloc(w, &w->el_int, 3));
  int sm = 0;
  const size_t smem = plan_smem(P, sizeof(double), P.minb, 1, sm);
  if (!P.cluster && occupancy(false, P.minb, sm, smem) * c.num_sms < P.grid) {
    set_error("moving mesh: the elasticity solver cannot be resident");
    return PFEM2_CUDA_ERROR;
  }
  return PFEM2_OK;
}

pfem2_status krylov_elastic_setup(Ctx& c, const std::vector<int>& slp) {
  KrylovWs* w = (KrylovWs*)c.kws;
  const size_t before = w->allocs.size();
  const pfem2_status st = elastic_setup(c, slp);
  if (st != PFEM2_OK) {  // another call starts over
    for (size_t k = before; k < w->allocs.size(); ++k) cudaFree(w->allocs[k]);
    w->allocs.resize(before);
    w->elastic = JacobiPlan();
  }
  return st;
}

// CG (Jacobi, FP64) on that system. Its residual, s and u all follow by
// recurrence and drift from b - A x (mesh of 30k cells: by 30% at 1e-14 |b|, and
// at 1e-16 |b| it stalled with b - A x at 6e-15 where CG with two reductions came
// to 7e-16), so a cycle lowers the residual by 1e12 at most before it is formed
// anew, and a solve ends on b - A x: two phases more of some 400. el_res: tol,
// rtol, residual, tolerance; el_int: max_iter, iterations, spare.
pfem2_status krylov_elastic_solve(Ctx& c, const ElasticSystem& E, double tol, double rtol, int maxit) {
  KrylovWs* w = (KrylovWs*)c.kws;
  const JacobiPlan& P = w->elastic;
  const double tr[4] = {tol, rtol, 0.0, 0.0};
  const int mi[3] = {maxit, 0, 0};
  PFEM2_CUDA(cudaMemcpyAsync(w->el_res, tr, sizeof(tr), cudaMemcpyHostToDevice, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(w->el_int, mi, sizeof(mi), cudaMemcpyHostToDevice, c.stream));
  SolveArgs<double> a{};
  plan_args(w, P, a);
  a.ncomp = a.ninst = 1;
  a.nv = c.nv * c.dim;
  a.sl_ptr = E.sl_ptr;
  a.sl_len = E.sl_len;
  a.sl_col = E.sl_col;
  a.share = 1;
  for (int k = 0; k < 3; ++k) {
    a.A64[k] = a.Ain[k] = E.A;
    a.dinv[k] = E.dinv;
    a.x[k] = E.x;
    a.b[k] = E.rhs;
    a.isd[k] = E.isd;
    a.g[k] = E.g;
  }
  a.tol_i = w->el_res;
  a.rtol_i = w->el_res + 1;
  a.maxit_i = w->el_int;
  a.pk = (V4<double>*)w->el_pk;
  a.e = w->el_e;
  a.r = w->el_r;
  a.v = w->el_v;
  a.s = w->el_s;
  a.t = a.rh = w->el_t;
  a.r64 = w->el_r64;
  a.part = w->el_part;
  a.out_it = w->el_int + 1;
  a.out_outer = w->el_int + 2;
  a.out_res = w->el_res + 2;
  a.out_tol = w->el_res + 3;
  a.floor = 1;
  a.eta = 1e-12;
  a.iter_cap = 4 * maxit + 256;  // a phase per iteration, and the restarts (two more, at most one per iteration)
  PFEM2_TRY(krylov_init_solve(c, 1));
  return plan_launch(c, P, a, 1);
}

pfem2_status krylov_elastic_read(Ctx& c, int* it, double* res, double* tol) {
  KrylovWs* w = (KrylovWs*)c.kws;
  int mi[3];
  double tr[4];
  PFEM2_CUDA(cudaMemcpyAsync(mi, w->el_int, sizeof(mi), cudaMemcpyDeviceToHost, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(tr, w->el_res, sizeof(tr), cudaMemcpyDeviceToHost, c.stream));
  PFEM2_CUDA(cudaStreamSynchronize(c.stream));
  *it = mi[1];
  *res = tr[2];
  *tol = tr[3];
  return PFEM2_OK;
}

// The multigrid of the pressure matrix (after Dirichlet elimination). A moving
// mesh that has none (too small to coarsen, or a pressure without a Dirichlet
// boundary) is solved by the Jacobi CG.
pfem2_status krylov_setup_precond(Ctx& c) {
  if (!c.two_level) return PFEM2_OK;
  const pfem2_status st = mg_setup(c);
  if (st == PFEM2_OK || st == PFEM2_CUDA_ERROR || !c.moving) return st;
  mg_free((KrylovWs*)c.kws);
  c.two_level = false;
  return plan_resident(c, 1);
}

// resets the solve's state; the previous solve's exit code (1 timeout,
// 2 iteration cap) is kept as bit (1 << code) in *sticky until the host
// reads it, so that the stats read after a whole step see every solve
__global__ void k_init_solve(int nsys, int* __restrict__ active, unsigned* __restrict__ barrier,
                             int* __restrict__ err, int* __restrict__ sticky, unsigned* __restrict__ scount,
                             int ncount) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    *active = nsys;
    barrier[0] = 0;
    barrier[1] = 0;
    const int e = *err;
    if (e > 0 && e < 8) *sticky |= 1 << e;
    *err = 0;
  }
  for (int j = i; j < ncount; j += gridDim.x * blockDim.x) scount[j] = 0u;
}

pfem2_status krylov_init_solve(Ctx& c, int nsys) {
  KrylovWs* w = (KrylovWs*)c.kws;
  k_init_solve<<<std::max(1, std::min(64, (32 * nsys + 255) / 256)), 256, 0, c.stream>>>(
      nsys, w->active, c.barrier, c.d_err, c.d_err_sticky, w->scount, 32 * nsys);
  c.launches++;
  return PFEM2_OK;
}

int krylov_max_iter(const Ctx& c) {
  int mx = 0;
  for (auto& in : c.inst) mx = std::max(mx, in.cs.max_iter > 0 ? in.cs.max_iter : 10000);
  return mx;
}

template <typename R>
static pfem2_status solve_impl(Ctx& c, int which) {
  KrylovWs* w = (KrylovWs*)c.kws;
  const JacobiPlan& P = w->plan[which == 1 ? 0 : 1];
  const int ncomp = which == 1 ? 1 : c.dim;
  const int ni = (int)c.inst.size();
  SolveArgs<R> a{};
  a.ncomp = ncomp;
  a.ninst = ni;
  a.nv = c.nv;
  plan_args(w, P, a);
  a.sl_ptr = c.sl_ptr;
  a.sl_len = c.sl_len;
  a.sl_col = c.sl_col;
  a.share = which == 2 && w->mass_share;
  for (int k = 0; k < 3; ++k) {
    const int kk = k < ncomp ? k : 0;
    const int mtx = which == 0 ? kk : (which == 1 ? 3 : 4 + (a.share ? 0 : kk));
    a.A64[k] = c.A64[mtx];
    a.Ain[k] = c.kmixed ? (const R*)c.A32[mtx] : (const R*)c.A64[mtx];
    a.dinv[k] = c.kmixed ? (const R*)c.dinv32[mtx] : (const R*)c.dinv64[mtx];
    if (which == 0) {
      a.x[k] = c.F[PFEM2_FIELD_PRED_VX + kk];
      a.b[k] = c.rhs[kk];
      a.isd[k] = c.isdir[kk];
      a.g[k] = c.dirval[kk];
    } else if (which == 1) {
      a.x[k] = c.F[PFEM2_FIELD_P];
      a.b[k] = c.rhs[0];
      a.isd[k] = c.isdir[3];
      a.g[k] = c.dirval[3];
    } else {
      a.x[k] = c.corr[kk];
      a.b[k] = c.rhs[kk];
      a.isd[k] = c.isdir[kk];
      a.g[k] = nullptr;
    }
  }
  a.tol_i = (const double*)c.sys_scalars + (which == 1 ? ni : 0);
  a.rtol_i = (const double*)c.sys_scalars + 2 * ni + (which == 1 ? ni : 0);
  a.pk = (V4<R>*)w->pk;
  a.rh = (R*)w->rh; a.s = (R*)w->s; a.t = (R*)w->t; a.v = (R*)w->v;
  a.maxit_i = c.d_sysinfo;
  a.e = (R*)w->e; a.r = (R*)w->r;
  a.r64 = w->r64;
  a.part = w->part;
  a.out_it = w->out_it[which];
  a.out_res = w->out_res[which];
  a.out_tol = w->out_tol[which];
  a.out_outer = w->out_outer[which];
  a.eta = c.kmixed ? c.refine_eta : 0.0;
  // CG: a phase per iteration, and the restarts (two more, at most one per
  // iteration); BiCGStab: two, and the same
  a.iter_cap = (a.bicg ? 5 : 4) * krylov_max_iter(c) + 256;
  PFEM2_TRY(krylov_init_solve(c, ncomp * ni));
  return plan_launch(c, P, a, P.cluster || !a.share ? ncomp : 1);
}

pfem2_status krylov_solve(Ctx& c, int which) {
  if (which == 1 && ((KrylovWs*)c.kws)->mg) return mg_solve(c);
  return c.kmixed ? solve_impl<float>(c, which) : solve_impl<double>(c, which);
}

// per-system iteration counts / residuals into c.stats (max over
// instances); NOT_CONVERGED if a system ended above its tolerance
static pfem2_status read_stats_phase(Ctx& c, int which) {
  KrylovWs* w = (KrylovWs*)c.kws;
  const int ns = (which == 1 ? 1 : c.dim) * (int)c.inst.size();
  std::vector<int> it(ns), outer(ns);
  std::vector<double> res(ns), tolv(ns);
  PFEM2_CUDA(cudaMemcpyAsync(it.data(), w->out_it[which], sizeof(int) * ns, cudaMemcpyDeviceToHost, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(res.data(), w->out_res[which], sizeof(double) * ns, cudaMemcpyDeviceToHost, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(tolv.data(), w->out_tol[which], sizeof(double) * ns, cudaMemcpyDeviceToHost, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(outer.data(), w->out_outer[which], sizeof(int) * ns, cudaMemcpyDeviceToHost, c.stream));
  PFEM2_CUDA(cudaStreamSynchronize(c.stream));
  const int ni = (int)c.inst.size();
  const int ncomp = which == 1 ? 1 : c.dim;
  bool notconv = false;
  for (int k = 0; k < ncomp; ++k) {
    const int slot = which == 0 ? k : (which == 1 ? 3 : 4 + k);
    int mit = 0, mo = 0;
    double mres = 0.0;
    for (int i = 0; i < ni; ++i) {
      const int s = k * ni + i;
      mit = std::max(mit, it[s]);
      mo = std::max(mo, outer[s]);
      mres = std::max(mres, res[s]);
      // (the tolerance the kernel applied: max(tol, rtol |b|))
      if (!(res[s] <= tolv[s])) notconv = true;
    }
    c.stats.iters[slot] = mit;
    c.stats.residual[slot] = mres;
    if (which == 1) c.stats.refinements_p = mo;
  }
  return notconv ? PFEM2_NOT_CONVERGED : PFEM2_OK;
}

void krylov_sizes(Ctx& c, long long* out12) {
  for (int k = 0; k < 12; ++k) out12[k] = 0;
  if (c.kws) mg_sizes((KrylovWs*)c.kws, out12);
}

void krylov_forms(const Ctx& c, int* out12) {
  for (int k = 0; k < 12; ++k) out12[k] = 0;
  const KrylovWs* w = (const KrylovWs*)c.kws;
  if (!w) return;
  const JacobiPlan& P = w->plan[1];
  int sm = 0;
  plan_smem(P, c.kmixed ? sizeof(float) : sizeof(double), P.minb, c.dim, sm);
  const int f[6] = {P.grid, P.minb, P.cluster, P.split, sm, P.sys_max};
  std::copy(f, f + 6, out12);
  mg_forms(w, out12 + 6);
}

pfem2_status krylov_read_stats(Ctx& c) {
  pfem2_status worst = PFEM2_OK;
  for (int wch = 0; wch < 3; ++wch) {
    pfem2_status s = read_stats_phase(c, wch);
    if (s != PFEM2_OK && worst == PFEM2_OK) worst = s;
  }
  // the last solve's exit code and those of the solves before it
  int err = 0, sticky = 0;
  PFEM2_CUDA(cudaMemcpy(&err, c.d_err, sizeof(int), cudaMemcpyDeviceToHost));
  PFEM2_CUDA(cudaMemcpy(&sticky, c.d_err_sticky, sizeof(int), cudaMemcpyDeviceToHost));
  if (err > 0 && err < 8) sticky |= 1 << err;
  if (sticky) {
    PFEM2_CUDA(cudaMemsetAsync(c.d_err_sticky, 0, sizeof(int), c.stream));
    PFEM2_CUDA(cudaMemsetAsync(c.d_err, 0, sizeof(int), c.stream));
  }
  if (sticky & 2) {
    set_error("krylov: a wait for the other blocks timed out");
    c.failed = true;
    return PFEM2_TIMEOUT;
  }
  if (sticky & 4) {
    set_error("krylov: iteration cap reached");
    return PFEM2_NOT_CONVERGED;
  }
  return worst;
}

}  // namespace pfem2
