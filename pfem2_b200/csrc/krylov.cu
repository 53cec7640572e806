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
// with every tile publishing its partial sums and a release add on its
// system's counter; the next phase starts once the counters of the block's
// running systems show every tile of those systems done (a per-system
// barrier: the instances of a batch do not wait for each other). Every
// block that owns tiles of a system computes that system's scalars itself,
// from the per-tile partial sums of the previous phase, in a fixed order:
// no block publishes scalars and no phase waits for a finalizer.
//
// CG takes one phase per iteration (one reduction), BiCGStab two; see the
// decisions below.
//
// The iterate is split x + e: e accumulates in the inner type R (FP32 for
// the mixed path, FP64 for the plain path); once the recurrence residual
// has dropped below max(eta * res, tol / 2) a reliable update runs in FP64
// (r64 = b - A64 (x + e), then x += e, e = 0, r = r64) and the solver restarts
// from the true residual. A system is done when the FP64 residual is <= tol.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstdio>
#include <vector>

#include "krylov_ws.h"

namespace pfem2 {

constexpr int kSolveThreads = 384;  // 12 warps
constexpr int kWarps = kSolveThreads / 32;

enum { S_OUT_A = 0, S_OUT_B = 1, S_A = 2, S_B = 3, S_DONE = 4, S_C0 = 5, S_C1 = 6 };
enum {
  ACT_NONE = 0, ACT_OUT_A = 1, ACT_OUT_B = 2, ACT_OUT_DONE = 3,
  ACT_P1 = 4,  // BiCGStab: finish the previous step, y = K^-1 p, v = A y
  ACT_P2 = 5,  // BiCGStab: e += alpha y, s = r - alpha v, t = A K^-1 s
  ACT_BF = 6,  // BiCGStab: e += omega K^-1 s before a reliable update
  ACT_C0 = 7,  // CG: w = A u after a restart
  ACT_C1 = 8   // CG: one iteration in one phase (single reduction)
};
// partial sums per tile: CG uses 3, BiCGStab 5 (and the FP64 residual
// phase |r|^2 and |b|^2)
constexpr int kMaxSums = 5;

constexpr int kMaxBlockTiles = 64;

// categories of per-block static data copied into shared memory at kernel
// start (every phase start's GPU-scope acquire invalidates L1, so static
// indices read from global memory would cost an L2 round trip per phase)
enum {
  ST_L0META = 1,  // slice pointers / lengths of the block's slice range
  ST_L0COL = 2    // SELL columns of that range
};

template <typename R> struct SolveArgs {
  int ncomp, ninst, nsys, ntiles, nv;
  const Tile* tiles;
  const int* sys_slot0;   // [nsys+1] first partial slot of each system
  const int* sys_owner;   // [nsys] block that reports the system's result
  const int* blk_t0;      // [grid+1] first tile of each block
  const int* blk_sys;     // systems of each block, at blk_sys_off[b]
  const int* blk_sys_off;
  const int* blk_sl;      // [2 grid] slice range [s0, s1) of each block's tiles
  const int* sl_ptr;
  const int* sl_len;
  const int* sl_col;
  const double* A64[3];
  const R* Ain[3];
  const R* dinv[3];
  int stage;              // ST_* categories staged in shared memory
  int ntl_max, items_max; // per block: tiles, (tile, slice) work items
  double* x[3];
  const double* b[3];
  const unsigned char* isd[3];
  const double* g[3];    // Dirichlet values preset in x (nullptr -> 0)
  const double* tol_i;   // per instance
  const double* rtol_i;  // per instance: stop at max(tol, rtol |b|)
  const int* maxit_i;    // per instance
  int nsum;              // partial sums per tile (3, or kMaxSums for BiCGStab)
  int bicg;              // BiCGStab instead of CG
  // BiCGStab vectors (nv entries per component slot): zr = K^-1 r, y and
  // w = K^-1 v double buffered (parity L.par; y in p), the shadow residual
  // rh, s, t and kt = K^-1 t; v in q, r in r's first buffer
  R *bz, *bw, *rh, *bs, *bt, *bkt;
  // CG with one reduction per iteration: u = D^-1 r, wh = D^-1 w and
  // sh = D^-1 s double buffered (parity L.par), w = A u and s = A p on the
  // own rows only; p in p's first buffer, r in r's first buffer
  R *cu, *cwh, *csh, *cw, *cs;
  // workspace per component slot, nv entries each; r and p: 2 buffers
  R *e, *r, *p, *q;
  double* r64;
  double* part;          // [2 parities][2 sums][ntiles slots]
  unsigned* scount;      // [nsys][32]: per-system count of tile phases published (one 128-byte line each, zeroed per launch)
  int* active;
  int* out_it;           // [nsys] iterations
  double* out_res;       // [nsys] final residual norm
  double* out_tol;       // [nsys] tolerance the system was solved to
  int* out_outer;        // [nsys] FP64 residual evaluations
  double eta;
  int iter_cap;
  GridBarrier gb;
};

struct LocalSys {
  int sys, state, it, outer, par, first, owner, maxit, act, chk;
  int t0, t1;                       // partial slots of the system
  double tol, rtol, intol, res, rz_prev, alpha, beta;
  double omega;                     // BiCGStab (rz_prev holds rho = (rh, r))
  double sum[kMaxSums];
};

template <typename R, int MINB>
__global__ void __launch_bounds__(kSolveThreads, MINB) k_krylov(SolveArgs<R> a) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  // entries of a SELL row (and of a long restriction row) whose loads are
  // issued together: more with one block per SM, which has the registers;
  // with two, nine: a Q1 row of 9 entries (2D) in one round of loads and one
  // of 27 (3D) in three (eight took two and four: channel velocity solves
  // 0.64 -> 0.61 ms, pipe 31.0 -> 26.9 ms per step)
  constexpr int CH = MINB == 1 ? 16 : 9;
  constexpr int NSMAX = kMaxSums;
  const int NS = a.nsum;
  __shared__ LocalSys ls[kMaxLocalSys];
  __shared__ Tile stile[kMaxBlockTiles];
  __shared__ int s_nls;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t nv = (size_t)a.nv;
  const int t_lo = a.blk_t0[blockIdx.x], t_hi = a.blk_t0[blockIdx.x + 1];
  const int ntl = t_hi - t_lo;
  const bool tiles_staged = ntl <= kMaxBlockTiles;
  unsigned bar_gen = 0;

  // ---- local systems of this block
  if (threadIdx.x == 0) {
    const int o = a.blk_sys_off[blockIdx.x];
    int n = a.blk_sys_off[blockIdx.x + 1] - o;
    if (n > kMaxLocalSys) n = kMaxLocalSys;  // the host guarantees n <= kMaxLocalSys
    s_nls = n;
    for (int k = 0; k < n; ++k) {
      LocalSys& L = ls[k];
      const int s = a.blk_sys[o + k], inst = s % a.ninst;
      L.sys = s;
      L.state = S_OUT_A;
      L.it = L.outer = L.par = L.chk = 0;
      L.first = 1;
      L.owner = a.sys_owner[s] == (int)blockIdx.x;
      L.t0 = a.sys_slot0[s];
      L.t1 = a.sys_slot0[s + 1];
      L.maxit = a.maxit_i[inst];
      L.tol = a.tol_i[inst];
      L.rtol = a.rtol_i[inst];
      L.intol = 0.5 * L.tol;
      L.res = L.rz_prev = L.alpha = L.beta = L.omega = 0.0;
      for (int q = 0; q < kMaxSums; ++q) L.sum[q] = 0.0;
      L.act = ACT_NONE;
    }
  }
  if (tiles_staged)
    for (int i = threadIdx.x; i < ntl; i += kSolveThreads) stile[i] = a.tiles[t_lo + i];
  __syncthreads();
  const int nls = s_nls;
  auto tile_at = [&](int t) -> Tile { return tiles_staged ? stile[t - t_lo] : a.tiles[t]; };

  // ---- level-0 work items: (tile, slice) pairs in tile order; item0[t] is
  // the first item of local tile t. Every item's partial sums go to spart,
  // then each tile sums its items in order (deterministic).
  double* spart = reinterpret_cast<double*>(dyn_smem);
  int* item0 = reinterpret_cast<int*>(dyn_smem + al16_dev((size_t)a.items_max * NS * sizeof(double)));
  if (threadIdx.x == 0) {
    int n = 0;
    for (int t = 0; t < ntl; ++t) {
      item0[t] = n;
      const Tile T = tile_at(t_lo + t);
      n += T.s1 - T.s0;
    }
    item0[ntl] = n;
  }
  __syncthreads();
  const int nitems = item0[ntl];
  // local tile of item `it` (binary search; tiles are few)
  auto item_tile = [&](int it) -> int {
    int lo = 0, hi = ntl - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (item0[mid] <= it) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  };
  unsigned char* dyn_rest =
      dyn_smem + al16_dev((size_t)a.items_max * NS * sizeof(double)) + al16_dev((size_t)(a.ntl_max + 1) * sizeof(int));

  // ---- shared memory: the staged static data
  unsigned char* cur = dyn_rest;
  const int bs0 = a.blk_sl[2 * blockIdx.x], bs1 = a.blk_sl[2 * blockIdx.x + 1];
  const SV<int> SLp = maybe_stage<int>(a.stage & ST_L0META, cur, a.sl_ptr, bs0, bs1 + 1);
  const SV<int> SLl = maybe_stage<int>(a.stage & ST_L0META, cur, a.sl_len, bs0, bs1);
  const SV<int> SLc = maybe_stage<int>(a.stage & ST_L0COL, cur, a.sl_col, a.sl_ptr[bs0], a.sl_ptr[bs1]);
  // ---- init: Dirichlet values preset in x, e = 0, p = 0
  for (int it = warp; it < nitems; it += kWarps) {
    const int tl = item_tile(it);
    const Tile T = tile_at(t_lo + tl);
    const int k = T.comp;
    {
      const int sl = T.s0 + (it - item0[tl]);
      const int row = sl * 32 + lane;
      if (a.isd[k][row]) a.x[k][row] = a.g[k] ? a.g[k][row] : 0.0;
      a.e[k * nv + row] = R(0);
      a.p[(2 * k) * nv + row] = R(0);
      a.p[(2 * k + 1) * nv + row] = R(0);
    }
  }
  __shared__ int s_stop;
  if (!grid_sync_ra(a.gb, bar_gen)) return;

  for (int iter = 0;; ++iter) {
    if (iter >= a.iter_cap) {
      if (threadIdx.x == 0) atomicCAS(a.gb.err, 0, 2);
      break;
    }
    const double* prev = a.part + (size_t)((iter + 1) & 1) * a.ntiles * NS;
    // ---- wait for the previous phase of the block's running systems: every
    // tile adds 1 to its system's counter with a release add once its phase
    // is written, so iter x (tiles of the system) means that every tile of
    // the system has finished phase iter - 1; lane k of warp 0 polls local
    // system k, then an acquire fence (and the block barrier) orders
    // everything those blocks wrote before this phase's reads. Blocks of
    // other systems are not waited for.
    if (warp == 0) {
      bool stop = true;
      for (int k = 0; k < nls; ++k) stop &= ls[k].state == S_DONE;
      if (!stop && iter > 0) {
        const bool mine = lane < nls && ls[lane].state != S_DONE;
        const unsigned target = mine ? (unsigned)iter * (unsigned)(ls[lane].t1 - ls[lane].t0) : 0u;
        const unsigned* cnt = a.scount + (size_t)(mine ? ls[lane].sys : 0) * 32;
        unsigned spins = 0;
        for (;;) {
          const bool ok = !mine || (int)(ld_relaxed_u32(cnt) - target) >= 0;
          if (__all_sync(PFEM2_FULL_MASK, ok)) {
            fence_acq_rel_gpu();
            break;
          }
          if (__any_sync(PFEM2_FULL_MASK, ++spins > a.gb.spin_limit || *(volatile int*)a.gb.err != 0)) {
            if (lane == 0) atomicCAS(a.gb.err, 0, 1);
            stop = true;
            break;
          }
          __nanosleep(20);
        }
      }
      if (lane == 0) s_stop = stop;
    }
    __syncthreads();
    if (s_stop) break;
    // the sums of the previous phase's partials: warp q sums partial q of
    // every local system over its tiles in a fixed order (lane l adds tiles
    // l, l + 32, ..., then the warp sum), all sums in one round of loads
    if (warp < NS) {
      const int q = warp;
      for (int k = 0; k < nls; ++k) {
        const int st = ls[k].state;
        if (st == S_DONE || st == S_OUT_A) continue;
        const int t0 = ls[k].t0, t1 = ls[k].t1;
        const double* pq = prev + (size_t)q * a.ntiles;
        double sq = 0.0;
        for (int tb = t0; tb < t1; tb += 256) {
          double v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int t = tb + u * 32 + lane;
            v[u] = t < t1 ? __ldcg(pq + t) : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) sq += v[u];
        }
        sq = warp_sum(sq);
        if (lane == 0) ls[k].sum[q] = sq;
      }
    }
    __syncthreads();
    // ---- decisions (thread 0; identical in every block owning the system)
    if (threadIdx.x == 0) {
      for (int k = 0; k < nls; ++k) {
        LocalSys& L = ls[k];
        int act = ACT_NONE;
        // the first FP64 residual phase also summed |b|^2: the relative tolerance
        if (L.state == S_OUT_B && L.outer == 0) L.tol = fmax(L.tol, L.rtol * sqrt(L.sum[1]));
        if (a.bicg) {
          // BiCGStab with the Jacobi preconditioner K (right-preconditioned,
          // van der Vorst 1992) over the phases OUT_A (FP64 residual),
          // OUT_B (restart: r = rh = r64, zr = K^-1 r), then P1 / P2 per
          // iteration; BF completes the iterate before a reliable update
          switch (L.state) {
            case S_OUT_A:
              act = ACT_OUT_A;
              L.state = S_OUT_B;
              break;
            case S_OUT_B:
              L.res = sqrt(L.sum[0]);
              L.outer += 1;
              if (L.res <= L.tol || L.it >= L.maxit || L.outer > L.maxit || !(L.res == L.res)) {
                act = ACT_OUT_DONE;
                L.state = S_DONE;
              } else {
                L.intol = fmax(a.eta * L.res, 0.5 * L.tol);
                L.first = 1;
                L.rz_prev = L.res * L.res;  // rho = (rh, r) with rh = r
                act = ACT_OUT_B;
                L.state = S_A;
              }
              break;
            case S_A:
              if (L.first) {
                L.beta = 0.0;
                act = ACT_P1;
                L.state = S_B;
              } else {
                // sums of P2: (t,s), (t,t), (rh,s), (rh,t), (s,s)
                const double ts = L.sum[0], tt = L.sum[1], rs = L.sum[2], rt = L.sum[3], ss = L.sum[4];
                const double om = tt > 0.0 ? ts / tt : 0.0;
                const double rr = sqrt(fmax(ss - 2.0 * om * ts + om * om * tt, 0.0));
                const double rho = rs - om * rt;
                L.omega = om;
                L.it += 1;
                if (!(om != 0.0) || !(rho != 0.0) || rr <= L.intol || L.it >= L.maxit || !(rr == rr)) {
                  act = ACT_BF;  // x += omega K^-1 s, then a reliable update
                  L.state = S_OUT_A;
                } else {
                  L.beta = (rho / L.rz_prev) * (L.alpha / om);
                  L.rz_prev = rho;
                  act = ACT_P1;
                  L.state = S_B;
                }
              }
              break;
            case S_B: {
              const double rv = L.sum[0];  // (rh, v)
              L.first = 0;
              if (!(rv != 0.0) || !(rv == rv)) {
                act = ACT_OUT_A;  // breakdown: restart from the FP64 residual
                L.state = S_OUT_B;
              } else {
                L.alpha = L.rz_prev / rv;
                act = ACT_P2;
                L.state = S_A;
              }
              break;
            }
            default:
              break;
          }
        } else {
          // CG with one reduction per iteration (Chronopoulos and
          // Gear 1989): u = D^-1 r, w = A u, gamma = (r, u), delta = (w, u);
          // beta = gamma / gamma_old, alpha = gamma / (delta - beta gamma /
          // alpha_old); p = u + beta p, s = w + beta s (= A p), x += alpha p,
          // r -= alpha s. One phase per iteration (C1), the w = A u of a
          // restart in a phase of its own (C0).
          switch (L.state) {
            case S_OUT_A:
              act = ACT_OUT_A;
              L.state = S_OUT_B;
              break;
            case S_OUT_B:
              L.res = sqrt(L.sum[0]);
              L.outer += 1;
              if (L.res <= L.tol || L.it >= L.maxit || !(L.res == L.res)) {
                act = ACT_OUT_DONE;
                L.state = S_DONE;
              } else {
                L.intol = fmax(a.eta * L.res, 0.5 * L.tol);
                L.chk = 0;
                act = ACT_OUT_B;
                L.state = S_C0;
              }
              break;
            case S_C0:
              act = ACT_C0;
              L.state = S_C1;
              break;
            case S_C1: {
              // sums of the previous phase: (r, u), (w, u), (r, r)
              const double g = L.sum[0], dl = L.sum[1], rr = sqrt(L.sum[2]);
              if (!L.chk) {
                L.alpha = dl != 0.0 ? g / dl : 0.0;
                L.beta = 0.0;
                L.rz_prev = g;
                act = ACT_C1;
              } else {
                L.it += 1;
                const double be = L.rz_prev != 0.0 ? g / L.rz_prev : 0.0;
                const double den = dl - (L.alpha != 0.0 ? be * g / L.alpha : 0.0);
                if (rr <= L.intol || L.it >= L.maxit || !(rr == rr) || !(den > 0.0)) {
                  act = ACT_OUT_A;  // reliable update in FP64
                  L.state = S_OUT_B;
                } else {
                  L.beta = be;
                  L.alpha = g / den;
                  L.rz_prev = g;
                  act = ACT_C1;
                }
              }
              break;
            }
            default:
              break;
          }
        }
        L.act = act;
      }
    }
    __syncthreads();
    // ---- level-0 work on the own (tile, slice) items, a warp per item
    for (int it = warp; it < nitems; it += kWarps) {
      const int tl = item_tile(it);
      const Tile T = tile_at(t_lo + tl);
      const int sl = T.s0 + (it - item0[tl]);
      const int k = T.comp;
      const LocalSys& L = ls[T.lk];
      const int act = L.act;
      if (act == ACT_NONE) continue;
      double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0, v4 = 0.0;
      const R* dinv = a.dinv[k];
      R* e = a.e + k * nv;
      R* r = a.r + (2 * k) * nv;
      R* q = a.q + k * nv;
      double* r64 = a.r64 + k * nv;
      if (act == ACT_OUT_A) {
        const double* A = a.A64[k];
        const double* xk = a.x[k];
        {
          const int row = sl * 32 + lane;
          const double acc = sell_dot<double, CH>(
              0.0, SLc, SLp[sl], SLl[sl], lane, [&](int ei) { return A[ei]; },
              [&](int col) { return __ldcg(xk + col) + (double)__ldcg(e + col); });
          const double bb = a.b[k][row];
          const double rr = bb - acc;
          r64[row] = rr;
          v0 += rr * rr;
          v1 += bb * bb;
        }
      } else if (act == ACT_OUT_B || act == ACT_OUT_DONE) {
        {
          const int row = sl * 32 + lane;
          a.x[k][row] += (double)e[row];
          e[row] = R(0);
          if (act == ACT_OUT_B) {
            const R rr = R(r64[row]);
            r[row] = rr;
            if (a.bicg) {
              a.rh[k * nv + row] = rr;
              a.bz[(2 * k + L.par) * nv + row] = rr * dinv[row];
            } else {
              a.cu[(2 * k + L.par) * nv + row] = rr * dinv[row];
            }
          }
        }
      } else if (act == ACT_C0) {
        // w = A u, wh = D^-1 w after a restart; (r, u), (w, u), (r, r)
        const int row = sl * 32 + lane;
        const R* u = a.cu + (2 * k + L.par) * nv;
        const R* A = a.Ain[k];
        const R w = sell_dot<R, CH>(R(0), SLc, SLp[sl], SLl[sl], lane, [&](int ei) { return A[ei]; },
                                    [&](int j) { return u[j]; });
        a.cw[k * nv + row] = w;
        a.cwh[(2 * k + L.par) * nv + row] = w * dinv[row];
        const double rr = (double)r[row], uu = (double)u[row];
        v0 += rr * uu;
        v1 += (double)w * uu;
        v2 += rr * rr;
      } else if (act == ACT_C1) {
        // p = u + beta p, s = w + beta s, sh = wh + beta sh, e += alpha p,
        // r -= alpha s, u' = u - alpha sh (= D^-1 r'), w' = A u' with u'
        // formed on the fly at the columns from u, wh and the old sh, wh' =
        // D^-1 w'; (r', u'), (w', u'), (r', r'). The first iteration after a
        // restart has p = u, s = w, sh = wh.
        const int row = sl * 32 + lane;
        const bool first = L.chk == 0;
        const R al = R(L.alpha), be = R(L.beta);
        const R* uo = a.cu + (2 * k + L.par) * nv;
        const R* who = a.cwh + (2 * k + L.par) * nv;
        const R* sho = a.csh + (2 * k + L.par) * nv;
        const auto unew = [&](int j) -> R {
          const R sh = first ? who[j] : fma_r(be, sho[j], who[j]);
          return fma_r(-al, sh, uo[j]);
        };
        R* pk = a.p + (2 * k) * nv;
        R* sk = a.cs + k * nv;
        const R sh = first ? who[row] : fma_r(be, sho[row], who[row]);
        const R pp = first ? uo[row] : fma_r(be, pk[row], uo[row]);
        const R ss = first ? a.cw[k * nv + row] : fma_r(be, sk[row], a.cw[k * nv + row]);
        pk[row] = pp;
        sk[row] = ss;
        e[row] = fma_r(al, pp, e[row]);
        const R rn = fma_r(-al, ss, r[row]);
        r[row] = rn;
        const R un = unew(row);
        const R* A = a.Ain[k];
        const R w = sell_dot<R, CH>(R(0), SLc, SLp[sl], SLl[sl], lane, [&](int ei) { return A[ei]; }, unew);
        a.csh[(2 * k + (L.par ^ 1)) * nv + row] = sh;
        a.cu[(2 * k + (L.par ^ 1)) * nv + row] = un;
        a.cwh[(2 * k + (L.par ^ 1)) * nv + row] = w * dinv[row];
        a.cw[k * nv + row] = w;
        v0 += (double)rn * (double)un;
        v1 += (double)w * (double)un;
        v2 += (double)rn * (double)rn;
      } else if (act == ACT_P1) {
        // y' = zr' + beta (y - omega w), zr' = zr - alpha w - omega kt the
        // preconditioned new residual (first step after a restart: y' = zr),
        // v = A y' with y' formed on the fly at the columns, w' = K^-1 v
        const int row = sl * 32 + lane;
        const bool first = L.first != 0;
        const R al = R(L.alpha), om = R(L.omega), be = R(L.beta);
        const R* zo = a.bz + (2 * k + L.par) * nv;
        const R* wo = a.bw + (2 * k + L.par) * nv;
        const R* yo = a.p + (2 * k + L.par) * nv;
        const R* kt = a.bkt + k * nv;
        const auto ynew = [&](int j) -> R {
          if (first) return zo[j];
          const R zr = fma_r(-om, kt[j], fma_r(-al, wo[j], zo[j]));
          return fma_r(be, fma_r(-om, wo[j], yo[j]), zr);
        };
        R zr_row = zo[row];
        if (!first) {
          const R zs = fma_r(-al, wo[row], zo[row]);
          e[row] = fma_r(om, zs, e[row]);
          r[row] = fma_r(-om, a.bt[k * nv + row], a.bs[k * nv + row]);
          zr_row = fma_r(-om, kt[row], zs);
        }
        const R yrow = ynew(row);
        const R* A = a.Ain[k];
        const R acc = sell_dot<R, CH>(R(0), SLc, SLp[sl], SLl[sl], lane, [&](int ei) { return A[ei]; }, ynew);
        a.bz[(2 * k + (L.par ^ 1)) * nv + row] = zr_row;
        a.p[(2 * k + (L.par ^ 1)) * nv + row] = yrow;
        a.bw[(2 * k + (L.par ^ 1)) * nv + row] = acc * dinv[row];
        q[row] = acc;
        v0 += (double)a.rh[k * nv + row] * (double)acc;
      } else if (act == ACT_P2) {
        // e += alpha y, s = r - alpha v, t = A K^-1 s (K^-1 s = zr - alpha w
        // formed on the fly), kt = K^-1 t; sums (t,s) (t,t) (rh,s) (rh,t) (s,s)
        const int row = sl * 32 + lane;
        const R al = R(L.alpha);
        const R* zc = a.bz + (2 * k + L.par) * nv;
        const R* wc = a.bw + (2 * k + L.par) * nv;
        e[row] = fma_r(al, a.p[(2 * k + L.par) * nv + row], e[row]);
        const R sv = fma_r(-al, q[row], r[row]);
        const R* A = a.Ain[k];
        const R tv = sell_dot<R, CH>(R(0), SLc, SLp[sl], SLl[sl], lane, [&](int ei) { return A[ei]; },
                                     [&](int j) { return fma_r(-al, wc[j], zc[j]); });
        a.bs[k * nv + row] = sv;
        a.bt[k * nv + row] = tv;
        a.bkt[k * nv + row] = tv * dinv[row];
        const double rh = (double)a.rh[k * nv + row];
        v0 += (double)tv * (double)sv;
        v1 += (double)tv * (double)tv;
        v2 += rh * (double)sv;
        v3 += rh * (double)tv;
        v4 += (double)sv * (double)sv;
      } else if (act == ACT_BF) {
        // the last step's x += omega K^-1 s (K^-1 s = zr - alpha w)
        const int row = sl * 32 + lane;
        const R zs = fma_r(-R(L.alpha), a.bw[(2 * k + L.par) * nv + row], a.bz[(2 * k + L.par) * nv + row]);
        e[row] = fma_r(R(L.omega), zs, e[row]);
      }
      // the item's partial sums (warp order is fixed: deterministic)
      v0 = warp_sum(v0);
      v1 = warp_sum(v1);
      if (lane == 0) {
        spart[NS * it] = v0;
        spart[NS * it + 1] = v1;
      }
      if (NSMAX > 2 && NS > 2) {
        const double vx[3] = {warp_sum(v2), NS > 3 ? warp_sum(v3) : 0.0, NS > 4 ? warp_sum(v4) : 0.0};
        if (lane == 0)
#pragma unroll
          for (int q = 2; q < NSMAX; ++q)
            if (q < NS) spart[NS * it + q] = vx[q - 2];
      }
    }
    __syncthreads();
    // per tile: its items' partials in order, into this phase's parity buffer
    // and the tile's count on its system's counter (a release add: after
    // the block barrier above it publishes every write of the block in this
    // phase)
    for (int tl = threadIdx.x; tl < ntl; tl += kSolveThreads) {
      const Tile T = tile_at(t_lo + tl);
      if (ls[T.lk].act != ACT_NONE) {
        double sm[NSMAX];
#pragma unroll
        for (int q = 0; q < NSMAX; ++q) sm[q] = 0.0;
        for (int it = item0[tl]; it < item0[tl + 1]; ++it) {
#pragma unroll
          for (int q = 0; q < NSMAX; ++q)
            if (q < NS) sm[q] += spart[NS * it + q];
        }
        double* dst = a.part + (size_t)(iter & 1) * a.ntiles * NS + T.slot;
#pragma unroll
        for (int q = 0; q < NSMAX; ++q)
          if (q < NS) dst[(size_t)q * a.ntiles] = sm[q];
      }
      red_release_add_u32(a.scount + (size_t)T.sys * 32, 1u);
    }
    // ---- bookkeeping
    if (threadIdx.x == 0) {
      for (int k = 0; k < nls; ++k) {
        LocalSys& L = ls[k];
        if (L.act == ACT_P1) L.par ^= 1;
        if (L.act == ACT_C1) {
          L.par ^= 1;
          L.chk = 1;
        }
        if (L.act == ACT_OUT_DONE && L.owner) {
          a.out_it[L.sys] = L.it;
          a.out_res[L.sys] = L.res;
          a.out_tol[L.sys] = L.tol;
          a.out_outer[L.sys] = L.outer;
          atomicSub(a.active, 1);
        }
        L.act = ACT_NONE;
      }
    }
  }
}

// ------------------------------------------------------------------ host
template <typename R, int MINB>
static int occupancy(size_t smem) {
  int occ = 0;
  // one process-wide upper bound, so contexts with different systems coexist
  cudaFuncSetAttribute((const void*)k_krylov<R, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)smem_budget(MINB));
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_krylov<R, MINB>, kSolveThreads, smem) != cudaSuccess)
    return 0;
  return occ;
}

static int occupancy_any(bool mixed, int minb, size_t smem) {
  if (minb == 1) return mixed ? occupancy<float, 1>(smem) : occupancy<double, 1>(smem);
  return mixed ? occupancy<float, 2>(smem) : occupancy<double, 2>(smem);
}

void krylov_free(Ctx& c) {
  KrylovWs* w = (KrylovWs*)c.kws;
  if (!w) return;
  mg_free(w);
  for (void* p : w->allocs) cudaFree(p);
  delete w;
  c.kws = nullptr;
}

pfem2_status krylov_setup(Ctx& c) {
  KrylovWs* w = new KrylovWs();
  c.kws = w;
  // the velocity solves: two blocks per SM hide more latency, one has fewer
  // blocks to wait for at every phase and the registers of the SM share
  w->vel_minb = c.tune.vel_blocks_per_sm ? c.tune.vel_blocks_per_sm : 2;
  c.tune.vel_blocks_per_sm = w->vel_minb;
  const int dim = c.dim, ni = (int)c.inst.size();
  const size_t nv = c.nv;
  const int bps = std::max(1, c.solve_blocks_per_sm);
  int maxtiles = 0, maxsys = 0;
  // phase 0: the pressure systems where the multigrid is not used
  for (int ph = c.two_level ? 1 : 0; ph < 2; ++ph) {
    const int ncomp = ph == 0 ? 1 : dim;
    const int nsys = ncomp * ni;
    std::vector<Tile> tiles;
    if (ph == 0) {
      // pressure: about one tile per SM for a single system, tiles of about
      // 8 slices in a batch
      const int dcap = ni == 1 ? 160 : 96;
      const int nb = c.num_sms;
      long long tot_sl = 0;
      for (int i = 0; i < ni; ++i) tot_sl += c.inst[i].nv_pad / kSlice;
      for (int i = 0; i < ni; ++i) {
        const int sl0 = c.inst[i].v_off / kSlice, nsl = c.inst[i].nv_pad / kSlice;
        const long long share = ni == 1 ? std::max<long long>(1, (long long)nb * nsl / tot_sl) : (nsl + 7) / 8;
        int D = (int)std::min<long long>(std::min<long long>(share, dcap), nsl);
        const int sps = (nsl + D - 1) / D;
        for (int a = 0; a < nsl; a += sps) tiles.push_back(Tile{i, 0, sl0 + a, sl0 + std::min(nsl, a + sps), 0, 0});
      }
    } else {
      // velocity components: tiles ordered (instance, slice run, component)
      // so that the slices of a block form one contiguous range
      const long long slices = (long long)c.nslices * ncomp;
      const long long target = 4LL * bps * c.num_sms;
      int ts = (int)std::max<long long>(8, (slices + target - 1) / target);
      if (c.tune.vel_tile_slices > 0) ts = c.tune.vel_tile_slices;
      c.tune.vel_tile_slices = ts;
      for (int i = 0; i < ni; ++i) {
        const int sl0 = c.inst[i].v_off / kSlice, sl1 = (c.inst[i].v_off + c.inst[i].nv_pad) / kSlice;
        for (int a = sl0; a < sl1; a += ts)
          for (int k = 0; k < ncomp; ++k) tiles.push_back(Tile{k * ni + i, k, a, std::min(sl1, a + ts), 0, 0});
      }
    }
    const int T = (int)tiles.size();
    // partial slots: the tiles of a system, contiguous
    std::vector<int> slot0(nsys + 1, 0), cnt(nsys, 0);
    for (const Tile& t : tiles) slot0[t.sys + 1]++;
    for (int s = 0; s < nsys; ++s) slot0[s + 1] += slot0[s];
    std::vector<int> owner(nsys, -1);
    const int minb = ph == 0 ? 2 : w->vel_minb;
    const int occ = std::min(minb, occupancy_any(c.kmixed, minb, 0));
    if (occ < 1) {
      set_error("krylov: the solver kernel cannot be resident");
      return PFEM2_CUDA_ERROR;
    }
    const int G = std::min(T, occ * c.num_sms);
    std::vector<int> bt0(G + 1), bsys_off(1, 0), bsys, bsl(2 * G, 0);
    // split the tile sequence where the running slice count crosses
    // b / G of the total (a tile goes to the block holding its midpoint):
    // blocks get equal work when tiles differ in size
    {
      std::vector<long long> pre(T + 1, 0);
      for (int u = 0; u < T; ++u) pre[u + 1] = pre[u] + (tiles[u].s1 - tiles[u].s0);
      bt0[0] = 0;
      int t = 0;
      for (int b = 1; b < G; ++b) {
        const long long goal = pre[T] * b / G;
        while (t < T && 2 * pre[t] + (pre[t + 1] - pre[t]) < 2 * goal) ++t;
        // every block keeps at least one tile and leaves one for each later block
        t = std::min(std::max(t, bt0[b - 1] + 1), T - (G - b));
        bt0[b] = t;
      }
      bt0[G] = T;
    }
    size_t meta = 0, col = 0;
    int ntl_max = 0, items_max = 0;
    for (int b = 0; b < G; ++b) {
      std::vector<int> lst;
      int s0 = 1 << 30, s1 = -1, items = 0;
      ntl_max = std::max(ntl_max, bt0[b + 1] - bt0[b]);
      for (int t = bt0[b]; t < bt0[b + 1]; ++t) items += tiles[t].s1 - tiles[t].s0;
      items_max = std::max(items_max, items);
      for (int t = bt0[b]; t < bt0[b + 1]; ++t) {
        Tile& tl = tiles[t];
        int k = (int)(std::find(lst.begin(), lst.end(), tl.sys) - lst.begin());
        if (k == (int)lst.size()) lst.push_back(tl.sys);
        tl.lk = k;
        tl.slot = slot0[tl.sys] + cnt[tl.sys]++;
        if (owner[tl.sys] < 0) owner[tl.sys] = b;
        s0 = std::min(s0, tl.s0);
        s1 = std::max(s1, tl.s1);
      }
      if ((int)lst.size() > kMaxLocalSys) {
        set_error("krylov: more than 16 systems would share one block (instances too small for the batch)");
        return PFEM2_INVALID_ARG;
      }
      bsys.insert(bsys.end(), lst.begin(), lst.end());
      bsys_off.push_back((int)bsys.size());
      if (s1 < s0) s0 = s1 = 0;
      // the block's tiles are ordered so that their slices form one range
      bsl[2 * b] = s0;
      bsl[2 * b + 1] = s1;
      meta = std::max(meta, al16(4 * (size_t)(s1 - s0 + 1)) + al16(4 * (size_t)(s1 - s0)));
      col = std::max(col, al16(4 * (size_t)(c.h_sl_ptr[s1] - c.h_sl_ptr[s0])));
    }
    w->ntl_max[ph] = ntl_max;
    w->items_max[ph] = items_max;
    w->bicg[ph] = ph == 0 ? c.p_bicg : c.vel_bicg;
    // BiCGStab 5 sums, CG 3 (one reduction per iteration)
    w->nsum[ph] = w->bicg[ph] ? kMaxSums : 3;
    w->items_bytes[ph] =
        al16(sizeof(double) * w->nsum[ph] * (size_t)items_max) + al16(sizeof(int) * (size_t)(ntl_max + 1));
    w->smem[ph] = w->items_bytes[ph];
    if (w->smem[ph] + meta <= smem_budget(minb)) {
      w->stage[ph] |= ST_L0META;
      w->smem[ph] += meta;
    }
    if (w->smem[ph] + col <= smem_budget(minb)) {
      w->stage[ph] |= ST_L0COL;
      w->smem[ph] += col;
    }
    if (occupancy_any(c.kmixed, minb, w->smem[ph]) * c.num_sms < G) {
      w->stage[ph] = 0;
      w->smem[ph] = w->items_bytes[ph];
    }
    w->ntiles[ph] = T;
    w->nsys[ph] = nsys;
    w->grid[ph] = G;
    PFEM2_TRY(ws_upload(w, &w->tiles[ph], tiles));
    PFEM2_TRY(ws_upload(w, &w->sys_slot0[ph], slot0));
    PFEM2_TRY(ws_upload(w, &w->sys_owner[ph], owner));
    PFEM2_TRY(ws_upload(w, &w->blk_t0[ph], bt0));
    PFEM2_TRY(ws_upload(w, &w->blk_sys[ph], bsys));
    PFEM2_TRY(ws_upload(w, &w->blk_sys_off[ph], bsys_off));
    PFEM2_TRY(ws_upload(w, &w->blk_sl[ph], bsl));
    maxtiles = std::max(maxtiles, T);
    maxsys = std::max(maxsys, nsys);
  }
  if (c.kmixed) {
    float *e, *r, *q, *p;
    PFEM2_TRY(ws_alloc(w, &e, nv * dim));
    PFEM2_TRY(ws_alloc(w, &r, 2 * nv * dim));
    PFEM2_TRY(ws_alloc(w, &q, nv * dim));
    PFEM2_TRY(ws_alloc(w, &p, 2 * nv * dim));
    w->e = e; w->r = r; w->q = q; w->p = p;
  } else {
    double *e, *r, *q, *p;
    PFEM2_TRY(ws_alloc(w, &e, nv * dim));
    PFEM2_TRY(ws_alloc(w, &r, 2 * nv * dim));
    PFEM2_TRY(ws_alloc(w, &q, nv * dim));
    PFEM2_TRY(ws_alloc(w, &p, 2 * nv * dim));
    w->e = e; w->r = r; w->q = q; w->p = p;
  }
  PFEM2_TRY(ws_alloc(w, &w->r64, nv * dim));
  PFEM2_TRY(ws_alloc(w, &w->part, 2 * (size_t)kMaxSums * maxtiles));
  {
    // single-reduction Jacobi CG vectors: u, wh, sh double buffered, w, s
    const size_t rs = c.kmixed ? sizeof(float) : sizeof(double);
    unsigned char* b[5];
    const size_t n[5] = {2 * nv * dim, 2 * nv * dim, 2 * nv * dim, nv * dim, nv * dim};
    for (int k = 0; k < 5; ++k) PFEM2_TRY(ws_alloc(w, &b[k], n[k] * rs));
    w->cu = b[0]; w->cwh = b[1]; w->csh = b[2]; w->cw = b[3]; w->cs = b[4];
  }
  if (c.vel_bicg || c.p_bicg) {
    // BiCGStab vectors: zr and w double buffered, rh, s, t, kt
    const size_t rs = c.kmixed ? sizeof(float) : sizeof(double);
    unsigned char* b[6];
    const size_t n[6] = {2 * nv * dim, 2 * nv * dim, nv * dim, nv * dim, nv * dim, nv * dim};
    for (int k = 0; k < 6; ++k) PFEM2_TRY(ws_alloc(w, &b[k], n[k] * rs));
    w->bz = b[0]; w->bw = b[1]; w->rh = b[2]; w->bs = b[3]; w->bt = b[4]; w->bkt = b[5];
  }
  PFEM2_TRY(ws_alloc(w, &w->scount, 32 * (size_t)maxsys));
  PFEM2_TRY(ws_alloc(w, &w->active, 1));
  for (int k = 0; k < 3; ++k) {
    PFEM2_TRY(ws_alloc(w, &w->out_it[k], maxsys));
    PFEM2_TRY(ws_alloc(w, &w->out_res[k], maxsys));
    PFEM2_TRY(ws_alloc(w, &w->out_tol[k], maxsys));
    PFEM2_TRY(ws_alloc(w, &w->out_outer[k], maxsys));
  }
  return PFEM2_OK;
}

// The multigrid of the pressure matrix (after Dirichlet elimination).
pfem2_status krylov_setup_precond(Ctx& c) { return c.two_level ? mg_setup(c) : PFEM2_OK; }

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
  const int ph = which == 1 ? 0 : 1;
  const int ncomp = which == 1 ? 1 : c.dim;
  const int ni = (int)c.inst.size();
  SolveArgs<R> a{};
  a.ncomp = ncomp;
  a.ninst = ni;
  a.nsys = w->nsys[ph];
  a.ntiles = w->ntiles[ph];
  a.nv = c.nv;
  a.tiles = w->tiles[ph];
  a.sys_slot0 = w->sys_slot0[ph];
  a.sys_owner = w->sys_owner[ph];
  a.blk_t0 = w->blk_t0[ph];
  a.blk_sys = w->blk_sys[ph];
  a.blk_sys_off = w->blk_sys_off[ph];
  a.blk_sl = w->blk_sl[ph];
  a.stage = w->stage[ph];
  a.ntl_max = w->ntl_max[ph];
  a.items_max = w->items_max[ph];
  a.sl_ptr = c.sl_ptr;
  a.sl_len = c.sl_len;
  a.sl_col = c.sl_col;
  for (int k = 0; k < 3; ++k) {
    const int kk = k < ncomp ? k : 0;
    const int mtx = which == 0 ? kk : (which == 1 ? 3 : 4 + kk);
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
  a.bicg = w->bicg[ph] ? 1 : 0;
  a.nsum = w->nsum[ph];
  a.bz = (R*)w->bz; a.bw = (R*)w->bw; a.rh = (R*)w->rh; a.bs = (R*)w->bs; a.bt = (R*)w->bt; a.bkt = (R*)w->bkt;
  a.cu = (R*)w->cu; a.cwh = (R*)w->cwh; a.csh = (R*)w->csh; a.cw = (R*)w->cw; a.cs = (R*)w->cs;
  a.maxit_i = c.d_sysinfo;
  a.e = (R*)w->e; a.r = (R*)w->r; a.q = (R*)w->q; a.p = (R*)w->p;
  a.r64 = w->r64;
  a.part = w->part;
  a.scount = w->scount;
  a.active = w->active;
  a.out_it = w->out_it[which];
  a.out_res = w->out_res[which];
  a.out_tol = w->out_tol[which];
  a.out_outer = w->out_outer[which];
  a.eta = c.kmixed ? c.refine_eta : 0.0;
  // phases per iteration, and BiCGStab's restarts (three phases each, at most max_iter)
  a.iter_cap = (a.bicg ? 5 : 4) * krylov_max_iter(c) + 256;
  a.gb.count = c.barrier;
  a.gb.gen = c.barrier + 1;
  a.gb.err = c.d_err;
  a.gb.spin_limit = c.spin_limit;
  PFEM2_TRY(krylov_init_solve(c, a.nsys));
  void* args[] = {&a};
  // the velocity solves at vel_minb blocks per SM, a pressure solve at two
  const void* kern = (ph == 1 && w->vel_minb == 1) ? (const void*)k_krylov<R, 1> : (const void*)k_krylov<R, 2>;
  PFEM2_CUDA(cudaLaunchCooperativeKernel(kern, dim3(w->grid[ph]), dim3(kSolveThreads), args, w->smem[ph], c.stream));
  c.launches++;
  return PFEM2_OK;
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
    PFEM2_CUDA(cudaMemset(c.d_err_sticky, 0, sizeof(int)));
    PFEM2_CUDA(cudaMemset(c.d_err, 0, sizeof(int)));
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
