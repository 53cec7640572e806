// mgcg.cu -- batched, persistent multigrid-preconditioned CG of the pressure
// systems with FP64 reliable updates on the SELL-32 pattern (sm_100a).
//
// One cooperative launch solves the pressure system of every instance to
// |b - A x| <= max(tol, rtol |b|) within max_iter iterations (deal.II
// SolverControl, cylinder2D/cylinder2D.cc:760-779; the Trilinos cases use CG
// with an AMG preconditioner, TurekBenchmarkCuda/TurekBenchmark.cc:731-797).
// The preconditioner is one V(1,1) cycle in additive form (amg.h):
//   z = J0 r + Pt0 (J1 b1 + Pt1 M2 b2),  b1 = Pt0^T r,  b2 = Pt1^T b1,
// with M2 = J2 + Pt2 E^-1 Pt2^T the two coarsest levels as one dense matrix
// per system (n2 x n2).
//
// What bounds it: at 50k rows an iteration is a chain of grid-wide phases,
// each a wait for values other blocks wrote and one or two dependent rounds
// of loads; from 100k rows in 3D the operators stream from L2. So q = A p,
// its restrictions and J0 q are formed without waiting for a scalar, and the
// residual-like quantities r, b1, b2 and J0 r follow by recurrence from the
// same q (z itself does not: its smooth part is large, and what a recurrence
// of it rounds is amplified by the condition number; nor may Pt0^T q come
// from z as (Pt0^T A) z, which saved a phase: in FP32 its cancellation left
// b1 inconsistent with r and the 34k-cell channel diverged):
//   A   q = A z + beta q, p = z + beta p, dq = D^-1 q  | (p, q), (r, q), (q, q), (r, r)
//   B   c1 = Pt0^T q, as (Pt0^T D) dq
//   B2  alpha; e += alpha p, r -= alpha q, b1 -= alpha c1, b2 -= alpha Pt1^T c1
//       then, while the others arrive: J0 r -= alpha J0 q,
//       J0 q = 2 w dq - w^2 D^-1 A dq
//   X2  x2 = M2 b2 on the own level-2 rows
//       then, while the others arrive: J1 b1 on the level-1 list
//   UZ  x1 = J1 b1 + Pt1 x2 on the level-1 list (own dofs and the halo the
//       own rows prolong from); z = J0 r + Pt0 x1                     | (r, z)
// Where the halo is a large multiple of the own dofs (3D), the list holds the
// own dofs only and x1 is published in a phase X1 of its own before UZ.
// The recurrences restart from the FP64 residual (r64 = b - A64 (x + e)) once
// |r| has dropped below max(eta res, tol / 2); |r - alpha q|^2 follows from
// the sums of phase A, so a finished cycle stops before its coarse phases.
//
// On a moving mesh the hierarchy is that of the mesh at setup, the level-0
// matrix and smoother are the current ones: the preconditioner stays symmetric
// (Pt0^T acts on q itself) and positive (w <= 0.49, below 2 / lambda_max(D^-1
// A) <= 2 / 4 of any 2D Q1 mesh), only its quality follows the mesh. Channel of
// 8k cells, FP32: 30 iterations in 0.56 ms where the Jacobi CG took 1,130 in
// 6.9 ms.
//
// Against the form before it (r' = r - alpha q restricted on the fly from two
// gathered vectors, J2, E^-1 and Pt2 evaluated by every block for its whole
// halo, barriers between the levels of one phase) an iteration takes 17 us
// instead of 40 on the channel with disk (52k rows, FP32), 24 instead of 270
// on a 10k-cell pipe (FP64), 47 instead of 420 on a 131k-cell pipe and 53
// instead of 147 on a batch of 16 channels (282k rows).
#include <algorithm>
#include <cmath>

#include "amg.h"
#include "krylov_ws.h"

namespace pfem2 {

namespace {

constexpr int kMgSums = 4;  // partial sums of a phase at most

enum { T_OUT_A = 0, T_OUT_B, T_B, T_B2, T_X2, T_X1, T_UZ, T_A, T_DONE };
enum { DO_NONE = 0, DO_OUT_A, DO_OUT_B, DO_FINISH, DO_B, DO_B2, DO_X2, DO_X1, DO_UZ, DO_A };

// What a block keeps in shared memory: bits of the template parameter SM (every
// phase start's acquire invalidates L1, so static operands read from global
// memory cost an L2 round trip per phase). Known at compile time: through
// generic pointers a solve took 0.92 ms instead of 0.78 on the 52k channel and
// 3.4 instead of 2.2 on the 131k pipe.
enum {
  SG_OWN = 1,    // the block's own rows of z, p, q, r, e, dq, J0 r, 1 / D; row pointers and local systems
  SG_COL = 2,    // SELL columns
  SG_M2 = 4,     // rows of M2
  SG_Q2 = 8,     // Pt1^T
  SG_A = 16,     // SELL values
  SG_P0 = 32,    // Pt0
  SG_P1 = 64,    // Pt1 of the level-1 list
  SG_J1 = 128,   // J1 of the level-1 list
  SG_R1 = 256    // Pt0^T D
};
// the combinations compiled, largest first: everything (52k rows FP32), all but
// the restriction (FP64), the vectors and small operators, nothing
constexpr int kMgMask[] = {511, 255, 15, 0};

template <typename R> struct MgArgs {
  int nv, nsys, ninst;
  const int *blk_sys, *blk_sys_off;  // systems of each block
  const int *blk_sl;                 // [2 grid] slice range
  const int *blk_slot;               // per blk_sys entry: the block's partial slot of that system
  const int *sys_slot0;              // [nsys+1] partial slots of each system
  const int *blk_o1, *blk_o2;        // [grid+1] own level-1 / level-2 dofs
  const int *slk;                    // [nslices] local system of each slice (in its block)
  const int *lk1, *lk2;              // the same for level-1 / level-2 dofs
  const int *sl_ptr, *sl_len, *sl_col;
  const double* A64;
  const R *A, *dinv;
  int r1_wide;                       // a warp per row of r1 (else 8 lanes)
  int raw;                           // moving mesh: dq holds q, r1 is Pt0^T (D changes under the hierarchy)
  const int *r1_ptr, *r1_col;        // Pt0^T D, global columns
  const R* r1_val;
  const int *q2_ptr, *q2_col;        // Pt1^T, global level-1 columns
  const R* q2_val;
  const R* m2;                       // rows of M2 in level-2 order
  const long long* blk_m2;           // [grid+1] where a block's rows start
  const int* m2_off;                 // per level-2 dof: its row's offset among its block's
  const int *p0_ptr, *p0_len, *p0_col;  // SELL per slice, columns into the block's level-1 list (global with xsplit)
  const R* p0_val;
  int xsplit;                        // the level-1 lists hold own dofs only: phase X1
  const int *blk_s1, *s1_lk, *j1_ptr, *j1_col, *p1_ptr, *p1_col;
  const R *j1_val, *p1_val;
  const int *sys_n2, *sys_off2;
  const double* sys_w;               // level-0 smoother weight
  int items_max, s1max, b2max;
  double* x;
  const double *b, *g;
  const unsigned char* isd;
  const double *tol_i, *rtol_i;
  const int* maxit_i;
  R *z, *p, *q, *r, *e, *dq, *jr, *c1, *b1, *x1, *b2, *x2;
  double *r64, *part;                // part: [7][slots]: OUT 2, A 4, UZ 1
  int nslots;
  unsigned* scount;
  int *active, *out_it, *out_outer;
  double *out_res, *out_tol;
  double eta;
  int iter_cap;
  GridBarrier gb;
};

// what a local system does in a phase, written by the warp that decides it:
// double buffered by phase parity, since the work after publishing still
// reads it while the next phase is being decided
struct MgAct {
  int act, first, restart, stop;
  double alpha, beta;
};

struct MgSys {
  int sys, state, it, outer, first, restart, owner, maxit;
  int s0, s1, slot;                 // partial slots of the system, the block's own
  int it0, it1;                     // the block's items (slices) of the system
  int n2, off2, b2off;
  double tol, rtol, intol, res, rz_prev, alpha, w;
};

// sums of n partial arrays over the slots [t0, t1) by one warp, in a fixed order
template <int N>
__device__ __forceinline__ void slot_sums(const double* part, int stride, int t0, int t1, int lane, double (&s)[N]) {
#pragma unroll
  for (int q = 0; q < N; ++q) s[q] = 0.0;
  for (int tb = t0; tb < t1; tb += 160) {
    double v[N][5];
#pragma unroll
    for (int q = 0; q < N; ++q)
#pragma unroll
      for (int u = 0; u < 5; ++u) {
        const int t = tb + u * 32 + lane;
        v[q][u] = t < t1 ? __ldcg(part + (size_t)q * stride + t) : 0.0;
      }
#pragma unroll
    for (int q = 0; q < N; ++q)
#pragma unroll
      for (int u = 0; u < 5; ++u) s[q] += v[q][u];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < N; ++q) s[q] += __shfl_xor_sync(PFEM2_FULL_MASK, s[q], o);
}

template <bool ON, typename T>
__device__ __forceinline__ const T* place(unsigned char*& cur, const T* src, int n) {
  if constexpr (ON) return stage_copy(cur, src, n);
  else return src;
}

template <typename R, int NT, int MINB, int SM>
__global__ void __launch_bounds__(NT, MINB) k_mgcg(MgArgs<R> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int NW = NT / 32;
  // SELL entries whose loads are issued together: a Q1 row of 9 (2D) in one
  // round, one of 27 (3D) in three
  constexpr int CH = 9;
  __shared__ MgSys ls[kMaxLocalSys];
  __shared__ MgAct sact[2][kMaxLocalSys];
  __shared__ int s_err;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int so = a.blk_sys_off[blockIdx.x];
  const int nls = min(a.blk_sys_off[blockIdx.x + 1] - so, kMaxLocalSys);
  const int bs0 = a.blk_sl[2 * blockIdx.x], bs1 = a.blk_sl[2 * blockIdx.x + 1];
  const int nitems = bs1 - bs0, own0 = bs0 * 32, nown = nitems * 32;
  unsigned bar_gen = 0;

  // ---- shared memory: item partials, level-1 vector, b2, then the staged data
  unsigned char* cur = smem;
  double* spart = reinterpret_cast<double*>(cur);
  cur += al16_dev((size_t)a.items_max * kMgSums * sizeof(double));
  R* sx1 = reinterpret_cast<R*>(cur);
  cur += al16_dev((size_t)a.s1max * sizeof(R));
  R* sb2 = reinterpret_cast<R*>(cur);
  cur += al16_dev((size_t)a.b2max * sizeof(R));
  const int o1lo = a.blk_o1[blockIdx.x], o1hi = a.blk_o1[blockIdx.x + 1];
  const int o2lo = a.blk_o2[blockIdx.x], o2hi = a.blk_o2[blockIdx.x + 1];
  const int s1lo = a.blk_s1[blockIdx.x], s1hi = a.blk_s1[blockIdx.x + 1];
  // (pointers by slice - bs0, level-1 dof - o1lo, level-2 dof - o2lo, level-1
  // list entry - s1lo; columns and values by entry - first entry)
  constexpr bool OWN = SM & SG_OWN;
  const int no1 = o1hi - o1lo, no2 = o2hi - o2lo, ns1 = s1hi - s1lo;
  const int* const SLp = place<OWN>(cur, a.sl_ptr + bs0, nitems + 1);
  const int* const SLl = place<OWN>(cur, a.sl_len + bs0, nitems);
  const int* const SLk = place<OWN>(cur, a.slk + bs0, nitems);
  const int* const P0p = place<OWN>(cur, a.p0_ptr + bs0, nitems + 1);
  const int* const P0l = place<OWN>(cur, a.p0_len + bs0, nitems);
  const int* const K1 = place<OWN>(cur, a.lk1 + o1lo, no1);
  const int* const R1p = place<OWN>(cur, a.r1_ptr + o1lo, no1 + 1);
  const int* const K2 = place<OWN>(cur, a.lk2 + o2lo, no2);
  const int* const Q2p = place<OWN>(cur, a.q2_ptr + o2lo, no2 + 1);
  const int* const M2o = place<OWN>(cur, a.m2_off + o2lo, no2);
  const int* const S1k = place<OWN>(cur, a.s1_lk + s1lo, ns1);
  const int* const J1p = place<OWN>(cur, a.j1_ptr + s1lo, ns1 + 1);
  const int* const P1p = place<OWN>(cur, a.p1_ptr + s1lo, ns1 + 1);
  const R* const di0 = place<OWN>(cur, a.dinv + own0, nown);
  R *lz, *mp, *mq, *mr, *le, *ldq, *mj;
  if constexpr (OWN) {
    lz = reinterpret_cast<R*>(cur);
    mp = lz + nown;
    mq = lz + 2 * nown;
    mr = lz + 3 * nown;
    le = lz + 4 * nown;
    ldq = lz + 5 * nown;
    mj = lz + 6 * nown;
    cur += al16_dev((size_t)7 * nown * sizeof(R));
  } else {
    lz = a.z + own0;
    mp = a.p + own0;
    mq = a.q + own0;
    mr = a.r + own0;
    le = a.e + own0;
    ldq = a.dq + own0;
    mj = a.jr + own0;
  }
  const int e0 = a.sl_ptr[bs0], ne = a.sl_ptr[bs1] - e0;
  const int* const SLc = place<(SM & SG_COL) != 0>(cur, a.sl_col + e0, ne);
  const long long m2lo = a.blk_m2[blockIdx.x];
  const R* const M2 = place<(SM & SG_M2) != 0>(cur, a.m2 + m2lo, (int)(a.blk_m2[blockIdx.x + 1] - m2lo));
  const int q20 = a.q2_ptr[o2lo], nq2 = a.q2_ptr[o2hi] - q20;
  const int* const Q2c = place<(SM & SG_Q2) != 0>(cur, a.q2_col + q20, nq2);
  const R* const Q2v = place<(SM & SG_Q2) != 0>(cur, a.q2_val + q20, nq2);
  const R* const SLa = place<(SM & SG_A) != 0>(cur, a.A + e0, ne);
  const int p00 = a.p0_ptr[bs0], np0 = a.p0_ptr[bs1] - p00;
  const int* const P0c = place<(SM & SG_P0) != 0>(cur, a.p0_col + p00, np0);
  const R* const P0v = place<(SM & SG_P0) != 0>(cur, a.p0_val + p00, np0);
  const int p10 = a.p1_ptr[s1lo], np1 = a.p1_ptr[s1hi] - p10;
  const int* const P1c = place<(SM & SG_P1) != 0>(cur, a.p1_col + p10, np1);
  const R* const P1v = place<(SM & SG_P1) != 0>(cur, a.p1_val + p10, np1);
  const int j10 = a.j1_ptr[s1lo], nj1 = a.j1_ptr[s1hi] - j10;
  const int* const J1c = place<(SM & SG_J1) != 0>(cur, a.j1_col + j10, nj1);
  const R* const J1v = place<(SM & SG_J1) != 0>(cur, a.j1_val + j10, nj1);
  const int r10 = a.r1_ptr[o1lo], nr1 = a.r1_ptr[o1hi] - r10;
  const int* const R1c = place<(SM & SG_R1) != 0>(cur, a.r1_col + r10, nr1);
  const R* const R1v = place<(SM & SG_R1) != 0>(cur, a.r1_val + r10, nr1);

  // ---- local systems (consecutive), their items, own level-2 offsets
  if (threadIdx.x == 0) {
    s_err = 0;
    int b2off = 0, it = 0;
    for (int k = 0; k < nls; ++k) {
      MgSys& L = ls[k];
      const int s = a.blk_sys[so + k], inst = s;
      L.sys = s;
      L.state = T_OUT_A;
      L.it = L.outer = L.first = L.restart = 0;
      L.s0 = a.sys_slot0[s];
      L.s1 = a.sys_slot0[s + 1];
      L.slot = a.blk_slot[so + k];
      L.owner = L.slot == L.s0;
      L.maxit = a.maxit_i[inst];
      L.tol = a.tol_i[inst];
      L.rtol = a.rtol_i[inst];
      L.intol = 0.5 * L.tol;
      L.res = L.rz_prev = L.alpha = 0.0;
      L.w = a.sys_w[s];
      L.n2 = a.sys_n2[s];
      L.off2 = a.sys_off2[s];
      L.b2off = b2off;
      b2off += L.n2;
      L.it0 = it;
      while (it < nitems && a.slk[bs0 + it] == k) ++it;
      L.it1 = it;
    }
  }
  // ---- init: Dirichlet values preset in x, e = 0
  for (int i = threadIdx.x; i < nown; i += NT) {
    const int row = own0 + i;
    if (a.isd[row]) a.x[row] = a.g ? a.g[row] : 0.0;
    a.e[row] = R(0);
    if (OWN) le[i] = R(0);
  }
  if (!grid_sync_ra(a.gb, bar_gen)) return;

  for (int iter = 0;; ++iter) {
    if (iter >= a.iter_cap) {
      if (threadIdx.x == 0) atomicCAS(a.gb.err, 0, 2);
      break;
    }
    // ---- phase start, a warp per local system: every block that owns part
    // of the system adds 1 to its counter once its phase is written, so iter
    // x (blocks of the system) means that all have finished phase iter - 1;
    // the acquire (and the block barrier) orders what they wrote before this
    // phase's reads. Then the sums the next step needs, and the step
    // itself (identical in every block that owns part of the system). Warps
    // without a system come here from the work after publishing.
    MgAct* const sa = sact[iter & 1];
    for (int k = warp; k < nls; k += NW) {
      MgSys& L = ls[k];
      const int st = L.state;
      MgAct d{DO_NONE, L.first, L.restart, 0, L.alpha, 0.0};
      if (st == T_DONE) {
        if (lane == 0) sa[k] = d;
        continue;
      }
      if (iter > 0) {
        const bool ok = wait_count(a.scount + (size_t)L.sys * 32, (unsigned)iter * (unsigned)(L.s1 - L.s0), a.gb);
        if (!ok) {
          if (lane == 0) {
            atomicCAS(a.gb.err, 0, 1);
            s_err = 1;
          }
          continue;
        }
      }
      int next = st + 1;  // T_B .. T_A are in phase order
      switch (st) {
        case T_OUT_A:
          d.act = DO_OUT_A;
          break;
        case T_OUT_B: {
          double s[2];
          slot_sums<2>(a.part, a.nslots, L.s0, L.s1, lane, s);
          const double res = sqrt(s[0]);
          // the first FP64 residual also summed |b|^2: the relative tolerance
          const double tol = L.outer == 0 ? fmax(L.tol, L.rtol * sqrt(s[1])) : L.tol;
          const bool done = res <= tol || L.it >= L.maxit || !(res == res);
          d.act = done ? DO_FINISH : DO_OUT_B;
          next = done ? T_DONE : T_B;
          __syncwarp();
          if (lane == 0) {
            L.res = res;
            L.tol = tol;
            L.outer += 1;
            L.intol = fmax(a.eta * res, 0.5 * tol);
            L.first = L.restart = 1;
          }
          break;
        }
        case T_B:
          d.act = DO_B;
          break;
        case T_B2:
          d.act = DO_B2;
          if (!L.restart) {
            double s[kMgSums];
            slot_sums<kMgSums>(a.part + 2 * (size_t)a.nslots, a.nslots, L.s0, L.s1, lane, s);
            const double al = s[0] != 0.0 ? L.rz_prev / s[0] : 0.0;
            const double rr = sqrt(fmax(s[3] - 2.0 * al * s[1] + al * al * s[2], 0.0));  // |r - alpha q|
            d.alpha = al;
            d.stop = rr <= L.intol || L.it + 1 >= L.maxit || !(rr == rr);
            if (d.stop) next = T_OUT_A;
            __syncwarp();
            if (lane == 0) {
              L.alpha = al;
              L.it += 1;
              L.first = 0;
            }
          }
          break;
        case T_X2:
          d.act = DO_X2;
          if (!a.xsplit) next = T_UZ;
          break;
        case T_X1:
          d.act = DO_X1;
          break;
        case T_UZ:
          d.act = DO_UZ;
          break;
        default: {  // T_A
          double s[1];
          slot_sums<1>(a.part + 6 * (size_t)a.nslots, a.nslots, L.s0, L.s1, lane, s);
          d.act = DO_A;
          d.beta = L.first || L.rz_prev == 0.0 ? 0.0 : s[0] / L.rz_prev;
          next = T_B;
          __syncwarp();
          if (lane == 0) {
            L.rz_prev = s[0];
            L.restart = 0;
          }
          break;
        }
      }
      __syncwarp();
      if (lane == 0) {
        L.state = next;
        sa[k] = d;
      }
    }
    __syncthreads();
    if (s_err) break;
    unsigned acts = 0;
    for (int k = 0; k < nls; ++k) acts |= 1u << sa[k].act;
    if (acts == 1u) break;  // every local system is done
    // ---- coarse rows of the phase
    if (acts & (1u << DO_B)) {
      auto rows = [&](auto gl) {
        constexpr int GL = decltype(gl)::value, NG = NT / GL;
        const int sub = threadIdx.x % GL, grp = threadIdx.x / GL;
        for (int base = o1lo; base < o1hi; base += NG) {
          const int i = base + grp;
          const bool on = i < o1hi && sa[K1[i - o1lo]].act == DO_B;
          R acc = R(0);
          if (on)
            acc = csr_dot<GL, 8, R>(acc, R1p[i - o1lo] - r10, R1p[i - o1lo + 1] - r10, sub, R1c, R1v,
                                    [&](int j) { return a.dq[j]; });
          acc = group_sum<GL>(acc);
          if (on && sub == 0) a.c1[i] = acc;
        }
      };
      if (a.r1_wide) rows(std::integral_constant<int, 32>{});
      else rows(std::integral_constant<int, 8>{});
    }
    if (acts & (1u << DO_B2)) {
      for (int i = o2lo + warp; i < o2hi; i += NW) {
        const MgAct& L = sa[K2[i - o2lo]];
        if (L.act != DO_B2 || L.stop) continue;
        R acc = csr_dot<32, CH, R>(R(0), Q2p[i - o2lo] - q20, Q2p[i - o2lo + 1] - q20, lane, Q2c, Q2v, [&](int c) { return __ldcg(a.c1 + c); });
        acc = warp_sum(acc);
        if (lane == 0) a.b2[i] = L.restart ? acc : fma_r(-R(L.alpha), acc, a.b2[i]);
      }
      for (int i = o1hi - 1 - (int)threadIdx.x; i >= o1lo; i -= NT) {
        const MgAct& L = sa[K1[i - o1lo]];
        if (L.act != DO_B2 || L.stop) continue;
        a.b1[i] = L.restart ? a.c1[i] : fma_r(-R(L.alpha), a.c1[i], a.b1[i]);
      }
    }
    if (acts & (1u << DO_X2)) {
      for (int k = 0; k < nls; ++k) {
        if (sa[k].act != DO_X2) continue;
        for (int d = threadIdx.x; d < ls[k].n2; d += NT) sb2[ls[k].b2off + d] = __ldcg(a.b2 + ls[k].off2 + d);
      }
      __syncthreads();
      for (int i = o2lo + warp; i < o2hi; i += NW) {
        const MgSys& L = ls[K2[i - o2lo]];
        if (sa[K2[i - o2lo]].act != DO_X2) continue;
        const R* bb = sb2 + L.b2off;
        const int m0 = M2o[i - o2lo], n2 = L.n2;
        R acc = R(0);
        for (int d0 = lane; d0 < n2; d0 += 256) {
          R mv[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) mv[u] = d0 + 32 * u < n2 ? M2[m0 + d0 + 32 * u] : R(0);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (d0 + 32 * u < n2) acc = fma_r(mv[u], bb[d0 + 32 * u], acc);
        }
        acc = warp_sum(acc);
        if (lane == 0) a.x2[i] = acc;
      }
    }
    if (acts & ((1u << DO_UZ) | (1u << DO_X1))) {
      const int want = a.xsplit ? DO_X1 : DO_UZ;
      constexpr int GL = 4, NG = NT / GL;
      const int sub = threadIdx.x % GL, grp = threadIdx.x / GL;
      for (int base = s1lo; base < s1hi; base += NG) {
        const int j = base + grp;
        R acc = R(0);
        const bool on = j < s1hi && sa[S1k[j - s1lo]].act == want;
        if (on) acc = csr_dot<GL, 8, R>(acc, P1p[j - s1lo] - p10, P1p[j - s1lo + 1] - p10, sub, P1c, P1v, [&](int c) { return __ldcg(a.x2 + c); });
        acc = group_sum<GL>(acc);
        if (on && sub == 0) {
          acc += sx1[j - s1lo];
          if (a.xsplit) a.x1[o1lo + (j - s1lo)] = acc;
          else sx1[j - s1lo] = acc;
        }
      }
      if (!a.xsplit) __syncthreads();
    }
    // ---- level-0 rows, a warp per slice
    for (int it = warp; it < nitems; it += NW) {
      const MgAct& L = sa[SLk[it]];
      const int act = L.act;
      if (act == DO_NONE || act == DO_B || act == DO_X2 || act == DO_X1) continue;
      const int o = it * 32 + lane, row = own0 + o, c0 = SLp[it] - e0, len = SLl[it];
      double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
      if (act == DO_A) {
        const R di = di0[o];
        const R acc = sell_dot<R, CH>(R(0), SLc, c0, len, lane, [&](int ei) { return SLa[ei]; },
                                      [&](int col) { return a.z[col]; });
        const R be = R(L.beta);
        R qq = acc, pp = lz[o];
        if (!L.first) {
          qq = fma_r(be, mq[o], qq);
          pp = fma_r(be, mp[o], pp);
        }
        mq[o] = qq;
        mp[o] = pp;
        const R dd = di * qq;
        a.dq[row] = a.raw ? qq : dd;
        if (OWN) ldq[o] = dd;
        v0 = (double)pp * (double)qq;
        v1 = (double)mr[o] * (double)qq;
        v2 = (double)qq * (double)qq;
        v3 = (double)mr[o] * (double)mr[o];
      } else if (act == DO_B2) {
        if (!L.restart) {
          const R al = R(L.alpha);
          const R ee = fma_r(al, mp[o], le[o]);
          le[o] = ee;
          mr[o] = fma_r(-al, mq[o], mr[o]);
          if (OWN && L.stop) a.e[row] = ee;
        }
        continue;
      } else if (act == DO_UZ) {
        const int p0 = P0p[it] - p00, pl = P0l[it];
        const R acc = a.xsplit ? sell_dot<R, CH>(mj[o], P0c, p0, pl, lane, [&](int ei) { return P0v[ei]; },
                                                 [&](int col) { return a.x1[col]; })
                               : sell_dot<R, CH>(mj[o], P0c, p0, pl, lane, [&](int ei) { return P0v[ei]; },
                                                 [&](int col) { return sx1[col]; });
        a.z[row] = acc;
        if (OWN) lz[o] = acc;
        v0 = (double)mr[o] * (double)acc;
      } else if (act == DO_OUT_A) {
        const double bb = a.b[row];
        const double acc = sell_dot<double, CH>(
            0.0, SLc, c0, len, lane, [&](int ei) { return a.A64[e0 + ei]; },
            [&](int col) { return __ldcg(a.x + col) + (double)__ldcg(a.e + col); });
        const double rr = bb - acc;
        a.r64[row] = rr;
        v0 = rr * rr;
        v1 = bb * bb;
      } else {  // DO_OUT_B, DO_FINISH
        a.x[row] += (double)le[o];
        le[o] = R(0);
        if (act == DO_OUT_B) {
          const R rr = R(a.r64[row]);
          mr[o] = rr;
          const R dd = di0[o] * rr;
          a.dq[row] = a.raw ? rr : dd;
          if (OWN) ldq[o] = dd;
        }
        continue;
      }
      if (act == DO_UZ) {
        v0 = warp_sum(v0);
        if (lane == 0) spart[kMgSums * it] = v0;
      } else {
        double v[4] = {v0, v1, v2, v3};
        const double tot = warp_sum_many<4, double>(v, lane);
        const int q = warp_sum_many_index<4>(lane);
        if ((lane & 7) == 0) spart[kMgSums * it + q] = tot;
      }
    }
    __syncthreads();
    // ---- publish, a warp per local system: the block's partial sums (items
    // in a fixed order), then a release add on the system's counter, which
    // after the block barrier above covers every write of the block's phase
    for (int k = warp; k < nls; k += NW) {
      const MgSys& L = ls[k];
      const int act = sa[k].act;
      const int ns = act == DO_A ? 4 : act == DO_OUT_A ? 2 : act == DO_UZ ? 1 : 0;
      if (lane < ns) {  // lane q adds up sum q
        double s = 0.0;
        for (int it = L.it0; it < L.it1; ++it) s += spart[kMgSums * it + lane];
        const int row = (act == DO_A ? 2 : act == DO_UZ ? 6 : 0) + lane;
        a.part[(size_t)row * a.nslots + L.slot] = s;
      }
      __syncwarp();
      if (lane == 0) {
        red_release_add_u32(a.scount + (size_t)L.sys * 32, 1u);
        if (act == DO_FINISH && L.owner) {
          a.out_it[L.sys] = L.it;
          a.out_res[L.sys] = L.res;
          a.out_tol[L.sys] = L.tol;
          a.out_outer[L.sys] = L.outer;
          atomicSub(a.active, 1);
        }
      }
    }
    // ---- work that no other block waits for, done while they arrive (with
    // few systems the warps that poll for them skip it)
    const int w0 = nls < NW / 4 ? nls : 0;
    if ((acts & (1u << DO_B2)) && warp >= w0) {
      for (int it = warp - w0; it < nitems; it += NW - w0) {
        const MgAct& L = sa[SLk[it]];
        if (L.act != DO_B2 || L.stop) continue;
        const int o = it * 32 + lane;
        const R di = di0[o], w = R(ls[SLk[it]].w);
        const R acc = sell_dot<R, CH>(R(0), SLc, SLp[it] - e0, SLl[it], lane, [&](int ei) { return SLa[ei]; },
                                      [&](int col) { return a.raw ? a.dq[col] * a.dinv[col] : a.dq[col]; });
        const R jq = w * fma_r(-w * di, acc, R(2) * (OWN || !a.raw ? ldq[o] : ldq[o] * di));
        mj[o] = L.restart ? jq : fma_r(-R(L.alpha), jq, mj[o]);
      }
    }
    if ((acts & (1u << DO_X2)) && warp >= w0) {
      constexpr int GL = 4, GPW = 32 / GL;
      const int NG = (NW - w0) * GPW;
      const int sub = lane % GL, grp = (warp - w0) * GPW + lane / GL;
      for (int base = s1lo; base < s1hi; base += NG) {
        const int j = base + grp;
        R acc = R(0);
        const bool on = j < s1hi && sa[S1k[j - s1lo]].act == DO_X2;
        if (on) acc = csr_dot<GL, 8, R>(acc, J1p[j - s1lo] - j10, J1p[j - s1lo + 1] - j10, sub, J1c, J1v, [&](int c) { return __ldcg(a.b1 + c); });
        acc = group_sum<GL>(acc);
        if (on && sub == 0) sx1[j - s1lo] = acc;
      }
    }
  }
}

}  // namespace

// ------------------------------------------------------------------ host
struct MgWs {
  int minb = 1, grid = 0, nsys = 0, nslots = 0, mask = 0;  // mask: index into kMgMask
  size_t smem = 0;
  bool wide = false, xsplit = false;
  int items_max = 0, s1max = 0, b2max = 0, sys_max = 0;
  long long sizes[12] = {};
  int *blk_sys, *blk_sys_off, *blk_sl, *blk_slot, *sys_slot0, *blk_o1, *blk_o2, *slk, *lk1, *lk2;
  int *r1_ptr, *r1_col, *q2_ptr, *q2_col, *m2_off, *p0_ptr, *p0_len, *p0_col;
  int *blk_s1, *s1_lk, *j1_ptr, *j1_col, *p1_ptr, *p1_col, *sys_n2, *sys_off2;
  double* sys_w;
  void* d0 = nullptr;  // level-0 smoother diagonal (fixed mesh)
  long long* blk_m2;
  void *r1_val, *q2_val, *m2, *p0_val, *j1_val, *p1_val;
  void *z, *dq, *jr, *c1, *b1, *x1, *b2, *x2;
  double* part;
};

void mg_free(KrylovWs* w) {
  delete w->mg;
  w->mg = nullptr;
}

void mg_sizes(const KrylovWs* w, long long* out12) {
  for (int k = 0; k < 12; ++k) out12[k] = w->mg ? w->mg->sizes[k] : 0;
}

void mg_forms(const KrylovWs* w, int* out6) {
  const MgWs* m = w->mg;
  const int f[6] = {m ? m->grid : 0, m ? m->minb : 0,         m ? m->mask : 0,
                    m ? (m->wide ? 32 : 8) : 0, m ? m->xsplit : 0, m ? m->sys_max : 0};
  std::copy(f, f + 6, out6);
}

namespace {

constexpr int mg_threads(int minb) { return minb == 1 ? 512 : 384; }

template <typename R, int MINB>
const void* mg_kernel(int mask) {
  constexpr int NT = mg_threads(MINB);
  return mask == 0   ? (const void*)k_mgcg<R, NT, MINB, kMgMask[0]>
         : mask == 1 ? (const void*)k_mgcg<R, NT, MINB, kMgMask[1]>
         : mask == 2 ? (const void*)k_mgcg<R, NT, MINB, kMgMask[2]>
                     : (const void*)k_mgcg<R, NT, MINB, kMgMask[3]>;
}

template <typename R>
const void* mg_kernel(int minb, int mask) {
  return minb == 1 ? mg_kernel<R, 1>(mask) : mg_kernel<R, 2>(mask);
}

}  // namespace

pfem2_status mg_setup(Ctx& c) {
  KrylovWs* w = (KrylovWs*)c.kws;
  MgWs* m = new MgWs();
  w->mg = m;
  // one system of moderate size: one block per SM (its level-1 halo lists are
  // replicated per block); a batch, or one system from mg_wide_min rows on
  // (bound by memory parallelism, not by latency): two
  m->minb = (c.inst.size() > 1 || (long long)c.nv >= c.mg_wide_min) ? 2 : 1;
  if (c.inst.size() == 1 && c.tune.p_blocks_per_sm) m->minb = c.tune.p_blocks_per_sm;
  c.tune.p_blocks_per_sm = m->minb;
  const int ni = (int)c.inst.size();
  m->nsys = ni;
  // tiles = the aggregation domains of the hierarchy: one per block of the
  // grid for a single system (at most 160), in a batch tiles of about 8
  // slices, at most 96 per system
  const int nb = m->minb * c.num_sms;
  const int dcap = ni == 1 ? (m->minb == 2 ? 2 * c.num_sms : 160) : 96;
  std::vector<Tile> tiles;
  std::vector<int> st0(1, 0);
  for (int i = 0; i < ni; ++i) {
    const int sl0 = c.inst[i].v_off / kSlice, nsl = c.inst[i].nv_pad / kSlice;
    const long long share = ni == 1 ? std::max(1, nb) : (nsl + 7) / 8;
    const int D = (int)std::min<long long>(std::min<long long>(share, dcap), nsl);
    const int sps = (nsl + D - 1) / D;
    for (int t = 0; t < nsl; t += sps) tiles.push_back(Tile{i, sl0 + t, sl0 + std::min(nsl, t + sps)});
    st0.push_back((int)tiles.size());
  }
  const int T = (int)tiles.size(), G = std::min(T, nb);
  m->grid = G;
  // contiguous tiles per block, split where the running slice count crosses
  // b / G of the total (a tile goes to the block that holds its midpoint)
  std::vector<int> bt0(G + 1, 0), bsys, bsys_off(1, 0), bsl(2 * G), bslot, slot0(ni + 1, 0), cnt(ni, 0);
  std::vector<int> slk(c.nslices, 0);
  {
    std::vector<long long> pre(T + 1, 0);
    for (int u = 0; u < T; ++u) pre[u + 1] = pre[u] + (tiles[u].s1 - tiles[u].s0);
    int t = 0;
    for (int b = 1; b < G; ++b) {
      const long long goal = pre[T] * b / G;
      while (t < T && 2 * pre[t] + (pre[t + 1] - pre[t]) < 2 * goal) ++t;
      t = std::min(std::max(t, bt0[b - 1] + 1), T - (G - b));
      bt0[b] = t;
    }
    bt0[G] = T;
  }
  for (int b = 0; b < G; ++b) {
    const int s0 = tiles[bt0[b]].sys, s1 = tiles[bt0[b + 1] - 1].sys;
    if (s1 - s0 + 1 > kMaxLocalSys) {
      set_error("krylov: more than 16 systems would share one block (instances too small for the batch)");
      return PFEM2_INVALID_ARG;
    }
    m->sys_max = std::max(m->sys_max, s1 - s0 + 1);
    for (int s = s0; s <= s1; ++s) bsys.push_back(s);
    bsys_off.push_back((int)bsys.size());
    bsl[2 * b] = tiles[bt0[b]].s0;
    bsl[2 * b + 1] = tiles[bt0[b + 1] - 1].s1;
    for (int t = bt0[b]; t < bt0[b + 1]; ++t)
      for (int sl = tiles[t].s0; sl < tiles[t].s1; ++sl) slk[sl] = tiles[t].sys - s0;
    m->items_max = std::max(m->items_max, bsl[2 * b + 1] - bsl[2 * b]);
  }
  for (int s : bsys) slot0[s + 1]++;
  for (int s = 0; s < ni; ++s) slot0[s + 1] += slot0[s];
  for (int s : bsys) bslot.push_back(slot0[s] + cnt[s]++);
  m->nslots = slot0[ni];
  // ---- the hierarchy
  std::vector<double> A(c.nell);
  std::vector<int> col(c.nell), len(c.nslices);
  PFEM2_CUDA(cudaMemcpy(A.data(), c.A64[3], sizeof(double) * c.nell, cudaMemcpyDeviceToHost));
  PFEM2_CUDA(cudaMemcpy(col.data(), c.sl_col, sizeof(int) * c.nell, cudaMemcpyDeviceToHost));
  PFEM2_CUDA(cudaMemcpy(len.data(), c.sl_len, sizeof(int) * c.nslices, cudaMemcpyDeviceToHost));
  MgHost H;
  const size_t rs = c.kmixed ? sizeof(float) : sizeof(double), budget = smem_budget(m->minb);
  PFEM2_TRY(mg_build(c, A, col, len, tiles, st0, bt0, m->minb == 1 ? 160 : 128, budget / rs, H));
  m->wide = H.r1_col.size() >= 64 * (size_t)std::max(1, H.n[1]);
  m->xsplit = H.xsplit;
  m->s1max = H.s1max;
  m->b2max = H.b2max;
  std::vector<int> bo1(G + 1), bo2(G + 1);
  for (int b = 0; b <= G; ++b) {
    bo1[b] = H.toff[1][bt0[b]];
    bo2[b] = H.toff[2][bt0[b]];
  }
  // ---- shared memory: the vectors, then the static data per category while
  // the budget lasts (maximum over blocks; the kernel stages the same pieces)
  const size_t i4 = 4;
  size_t smem = al16(sizeof(double) * kMgSums * m->items_max) + al16(rs * m->s1max) + al16(rs * m->b2max);
  constexpr int NC = 9;
  size_t cat[NC] = {};
  for (int b = 0; b < G; ++b) {
    const int s0 = bsl[2 * b], s1 = bsl[2 * b + 1], ns = s1 - s0;
    const int n1 = bo1[b + 1] - bo1[b], n2 = bo2[b + 1] - bo2[b];
    const int l0 = H.blk_s1[b], l1 = H.blk_s1[b + 1], nl = l1 - l0;
    const size_t ne = c.h_sl_ptr[s1] - c.h_sl_ptr[s0], np0 = H.p0_ptr[s1] - H.p0_ptr[s0];
    const size_t nm = (size_t)(H.blk_m2[b + 1] - H.blk_m2[b]), nq = H.q2_ptr[bo2[b + 1]] - H.q2_ptr[bo2[b]];
    const size_t nj = H.j1_ptr[l1] - H.j1_ptr[l0], np = H.p1_ptr[l1] - H.p1_ptr[l0];
    const size_t nr = H.r1_ptr[bo1[b + 1]] - H.r1_ptr[bo1[b]];
    const size_t v[NC] = {2 * al16(i4 * (ns + 1)) + 3 * al16(i4 * ns) + al16(i4 * n1) + al16(i4 * (n1 + 1)) +
                              2 * al16(i4 * n2) + al16(i4 * (n2 + 1)) + al16(i4 * nl) + 2 * al16(i4 * (nl + 1)) +
                              al16(rs * 32 * ns) + al16(rs * 7 * 32 * ns),
                          al16(i4 * ne),
                          al16(rs * nm),
                          al16(i4 * nq) + al16(rs * nq),
                          al16(rs * ne),
                          al16(i4 * np0) + al16(rs * np0),
                          al16(i4 * np) + al16(rs * np),
                          al16(i4 * nj) + al16(rs * nj),
                          al16(i4 * nr) + al16(rs * nr)};
    for (int k = 0; k < NC; ++k) cat[k] = std::max(cat[k], v[k]);
  }
  if (smem > budget) {
    set_error("krylov: the pressure multigrid's per-block data exceed shared memory");
    return PFEM2_INVALID_ARG;
  }
  for (m->mask = 0;; ++m->mask) {
    size_t need = smem;
    for (int k = 0; k < NC; ++k)
      if (kMgMask[m->mask] >> k & 1) need += cat[k];
    if (need <= budget) {
      m->smem = need;
      break;
    }
  }
  const void* kern = c.kmixed ? mg_kernel<float>(m->minb, m->mask) : mg_kernel<double>(m->minb, m->mask);
  // one process-wide upper bound, so contexts with different hierarchies coexist
  PFEM2_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget));
  int occ = 0;
  PFEM2_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, mg_threads(m->minb), m->smem));
  if (occ * c.num_sms < G) {
    set_error("krylov: the multigrid solver grid cannot be resident");
    return PFEM2_CUDA_ERROR;
  }
  const long long sz[12] = {c.nv,
                            H.n[1],
                            H.n[2],
                            H.n[3],
                            (long long)H.r1_col.size(),
                            (long long)H.q2_col.size(),
                            0,
                            (long long)H.p0_col.size(),
                            (long long)H.j1_col.size(),
                            (long long)H.p1_col.size(),
                            (long long)H.m2.size(),
                            0};
  for (int k = 0; k < 12; ++k) m->sizes[k] = sz[k];
  PFEM2_TRY(ws_upload(w, &m->blk_sys, bsys));
  PFEM2_TRY(ws_upload(w, &m->blk_sys_off, bsys_off));
  PFEM2_TRY(ws_upload(w, &m->blk_sl, bsl));
  PFEM2_TRY(ws_upload(w, &m->blk_slot, bslot));
  PFEM2_TRY(ws_upload(w, &m->sys_slot0, slot0));
  PFEM2_TRY(ws_upload(w, &m->blk_o1, bo1));
  PFEM2_TRY(ws_upload(w, &m->blk_o2, bo2));
  PFEM2_TRY(ws_upload(w, &m->slk, slk));
  PFEM2_TRY(ws_upload(w, &m->lk1, H.lk[1]));
  PFEM2_TRY(ws_upload(w, &m->lk2, H.lk[2]));
  PFEM2_TRY(ws_upload(w, &m->r1_ptr, H.r1_ptr));
  PFEM2_TRY(ws_upload(w, &m->r1_col, H.r1_col));
  PFEM2_TRY(ws_upload_r(w, c.kmixed, &m->r1_val, H.r1_val));
  PFEM2_TRY(ws_upload(w, &m->q2_ptr, H.q2_ptr));
  PFEM2_TRY(ws_upload(w, &m->q2_col, H.q2_col));
  PFEM2_TRY(ws_upload_r(w, c.kmixed, &m->q2_val, H.q2_val));
  PFEM2_TRY(ws_upload(w, &m->m2_off, H.m2_off));
  PFEM2_TRY(ws_upload(w, &m->blk_m2, H.blk_m2));
  PFEM2_TRY(ws_upload_r(w, c.kmixed, &m->m2, H.m2));
  PFEM2_TRY(ws_upload(w, &m->p0_ptr, H.p0_ptr));
  PFEM2_TRY(ws_upload(w, &m->p0_len, H.p0_len));
  PFEM2_TRY(ws_upload(w, &m->p0_col, H.p0_col));
  PFEM2_TRY(ws_upload_r(w, c.kmixed, &m->p0_val, H.p0_val));
  PFEM2_TRY(ws_upload(w, &m->blk_s1, H.blk_s1));
  PFEM2_TRY(ws_upload(w, &m->s1_lk, H.s1_lk));
  PFEM2_TRY(ws_upload(w, &m->j1_ptr, H.j1_ptr));
  PFEM2_TRY(ws_upload(w, &m->j1_col, H.j1_col));
  PFEM2_TRY(ws_upload_r(w, c.kmixed, &m->j1_val, H.j1_val));
  PFEM2_TRY(ws_upload(w, &m->p1_ptr, H.p1_ptr));
  PFEM2_TRY(ws_upload(w, &m->p1_col, H.p1_col));
  PFEM2_TRY(ws_upload_r(w, c.kmixed, &m->p1_val, H.p1_val));
  PFEM2_TRY(ws_upload(w, &m->sys_n2, H.sys_n2));
  PFEM2_TRY(ws_upload(w, &m->sys_off2, H.sys_off2));
  PFEM2_TRY(ws_upload(w, &m->sys_w, H.w0));
  if (!c.moving) PFEM2_TRY(ws_upload_r(w, c.kmixed, &m->d0, H.d0));
  void** vec[] = {&m->z, &m->dq, &m->jr, &m->c1, &m->b1, &m->x1, &m->b2, &m->x2};
  const size_t nv = c.nv, n1 = H.n[1], n2 = H.n[2], nvec[] = {nv, nv, nv, n1, n1, n1, n2, n2};
  for (int k = 0; k < 8; ++k) {
    unsigned char* d;
    PFEM2_TRY(ws_alloc(w, &d, nvec[k] * rs));
    *vec[k] = d;
  }
  PFEM2_TRY(ws_alloc(w, &m->part, 7 * (size_t)m->nslots));
  return PFEM2_OK;
}

namespace {

template <typename R>
pfem2_status mg_solve_impl(Ctx& c) {
  KrylovWs* w = (KrylovWs*)c.kws;
  MgWs* m = w->mg;
  const int ni = (int)c.inst.size();
  MgArgs<R> a{};
  a.nv = c.nv;
  a.nsys = m->nsys;
  a.ninst = ni;
  a.blk_sys = m->blk_sys;
  a.blk_sys_off = m->blk_sys_off;
  a.blk_sl = m->blk_sl;
  a.blk_slot = m->blk_slot;
  a.sys_slot0 = m->sys_slot0;
  a.blk_o1 = m->blk_o1;
  a.blk_o2 = m->blk_o2;
  a.slk = m->slk;
  a.lk1 = m->lk1;
  a.lk2 = m->lk2;
  a.sl_ptr = c.sl_ptr;
  a.sl_len = c.sl_len;
  a.sl_col = c.sl_col;
  a.A64 = c.A64[3];
  a.A = c.kmixed ? (const R*)c.A32[3] : (const R*)c.A64[3];
  a.dinv = !c.moving ? (const R*)m->d0 : c.kmixed ? (const R*)c.dinv32[3] : (const R*)c.dinv64[3];
  a.r1_wide = m->wide;
  a.raw = c.moving;
  a.xsplit = m->xsplit;
  a.r1_ptr = m->r1_ptr; a.r1_col = m->r1_col; a.r1_val = (const R*)m->r1_val;
  a.q2_ptr = m->q2_ptr; a.q2_col = m->q2_col; a.q2_val = (const R*)m->q2_val;
  a.m2 = (const R*)m->m2; a.m2_off = m->m2_off; a.blk_m2 = m->blk_m2;
  a.p0_ptr = m->p0_ptr; a.p0_len = m->p0_len; a.p0_col = m->p0_col; a.p0_val = (const R*)m->p0_val;
  a.blk_s1 = m->blk_s1; a.s1_lk = m->s1_lk;
  a.j1_ptr = m->j1_ptr; a.j1_col = m->j1_col; a.j1_val = (const R*)m->j1_val;
  a.p1_ptr = m->p1_ptr; a.p1_col = m->p1_col; a.p1_val = (const R*)m->p1_val;
  a.sys_n2 = m->sys_n2; a.sys_off2 = m->sys_off2; a.sys_w = m->sys_w;
  a.items_max = m->items_max;
  a.s1max = m->s1max;
  a.b2max = m->b2max;
  a.x = c.F[PFEM2_FIELD_P];
  a.b = c.rhs[0];
  a.g = c.dirval[3];
  a.isd = c.isdir[3];
  a.tol_i = (const double*)c.sys_scalars + ni;
  a.rtol_i = (const double*)c.sys_scalars + 3 * ni;
  a.maxit_i = c.d_sysinfo;
  a.z = (R*)m->z; a.dq = (R*)m->dq; a.jr = (R*)m->jr;
  a.c1 = (R*)m->c1; a.b1 = (R*)m->b1; a.x1 = (R*)m->x1; a.b2 = (R*)m->b2; a.x2 = (R*)m->x2;
  a.p = (R*)w->s; a.q = (R*)w->v; a.r = (R*)w->r; a.e = (R*)w->e;
  a.r64 = w->r64;
  a.part = m->part;
  a.nslots = m->nslots;
  a.scount = w->scount;
  a.active = w->active;
  a.out_it = w->out_it[1];
  a.out_res = w->out_res[1];
  a.out_tol = w->out_tol[1];
  a.out_outer = w->out_outer[1];
  a.eta = c.kmixed ? c.refine_eta : 0.0;
  // at most six phases per iteration, and two more per restart (at most one per iteration)
  a.iter_cap = 10 * krylov_max_iter(c) + 256;
  a.gb.count = c.barrier;
  a.gb.gen = c.barrier + 1;
  a.gb.err = c.d_err;
  a.gb.spin_limit = c.spin_limit;
  PFEM2_TRY(krylov_init_solve(c, a.nsys));
  void* args[] = {&a};
  PFEM2_CUDA(cudaLaunchCooperativeKernel(mg_kernel<R>(m->minb, m->mask), dim3(m->grid), dim3(mg_threads(m->minb)), args,
                                         m->smem, c.stream));
  c.launches++;
  return PFEM2_OK;
}

}  // namespace

pfem2_status mg_solve(Ctx& c) { return c.kmixed ? mg_solve_impl<float>(c) : mg_solve_impl<double>(c); }

}  // namespace pfem2
