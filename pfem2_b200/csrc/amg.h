// amg.h -- smoothed-aggregation multigrid for the pressure Poisson systems:
// the host-side hierarchy (built once at setup from the eliminated FP64
// matrix) in the layout the persistent solver kernel reads.
//
// The reference preconditions its pressure solve with Trilinos ML
// (TrilinosWrappers::PreconditionAMG, TurekBenchmarkCuda/TurekBenchmark.cc:
// 731-797). Here one V(1,1) cycle with damped Jacobi smoothing and
// smoothed-aggregation transfers is applied in its additive form
//   M_l^-1 = J_l + Pt_l M_{l+1}^-1 Pt_l^T,
//   J_l  = 2 w D^-1 - w^2 D^-1 A_l D^-1,  Pt_l = (I - w D^-1 A_l) P_l,
// D the smoother's diagonal (the absolute row sums on level 0 of a fixed mesh),
// which is algebraically the same V-cycle: the pre- and post-smoothing of a
// level are folded into J_l and into the post-smoothed prolongator Pt_l, so
// a level costs one sparse product each way and no extra synchronisation.
// Levels: 0 = the pressure rows; 1, 2 = aggregates of the level below built
// inside each solver tile; 3 = one aggregate per tile, solved exactly with
// a dense inverse.
#pragma once
#include <vector>

#include "ctx.h"

namespace pfem2 {

constexpr int kMgLevels = 4;

struct MgHost {
  int n[kMgLevels] = {0, 0, 0, 0};        // dofs per level over all systems
  std::vector<int> toff[kMgLevels];       // [l][ntiles+1] first level-l dof of each tile (l >= 1)
  std::vector<int> lsys[kMgLevels];       // [l][n_l] system of each level-l dof (l >= 1)
  std::vector<int> lk[3];                 // [1..2][n_l] index of that system among its block's systems
  // Pt_0^T D (applied to D^-1 v; Pt_0^T on a moving mesh), CSR over the
  // level-1 rows with global level-0 columns
  std::vector<int> r1_ptr, r1_col;
  std::vector<double> r1_val;
  // Pt_1^T, CSR over the level-2 rows with global level-1 columns
  std::vector<int> q2_ptr, q2_col;
  std::vector<double> q2_val;
  // M2 = J_2 + Pt_2 E^-1 Pt_2^T, dense rows of the system's n2 columns in
  // level-2 order: where each block's rows start, and each row's offset there
  std::vector<double> m2;
  std::vector<long long> blk_m2;          // [G+1]
  std::vector<int> m2_off;                // [n2]
  // post-smoothed prolongator of level 0 on SELL slices; columns are the
  // indices into the owning block's level-1 list (global with xsplit)
  std::vector<int> p0_ptr, p0_len, p0_col;
  std::vector<double> p0_val;
  // per-block lists of the level-1 dofs a block evaluates (own dofs, then,
  // unless xsplit, the halo its rows prolong from): system among the block's,
  // J_1 rows with global level-1 columns, Pt_1 rows with global level-2 columns
  bool xsplit = false;
  std::vector<int> blk_s1, s1_lk, j1_ptr, j1_col, p1_ptr, p1_col;
  std::vector<double> j1_val, p1_val;
  std::vector<int> sys_n2, sys_off2;      // level-2 size and first level-2 dof per system
  std::vector<double> w0;                 // level-0 smoother weight per system
  std::vector<double> d0;                 // [nv] level-0 smoother diagonal D^-1 (1 / a_ii on a moving mesh)
  int s1max = 0;
  int b2max = 0;                          // level-2 dofs of the local systems of a block
};

// Builds the hierarchy of every pressure system. A, col, len: host copy of
// the eliminated FP64 pressure matrix in the context's SELL layout; tiles,
// st0: the pressure solve's tiles and first tile per system; bt0: first
// tile per block of the persistent grid; coarse_max: level-3 unknowns per
// system at most (groups of tiles share one); b2_max: level-2 unknowns of a
// block's systems at most (PFEM2_INVALID_ARG above).
pfem2_status mg_build(const Ctx& c, const std::vector<double>& A, const std::vector<int>& col,
                      const std::vector<int>& len, const std::vector<Tile>& tiles, const std::vector<int>& st0,
                      const std::vector<int>& bt0, int coarse_max, size_t b2_max, MgHost& out);

// In-place inverse of an SPD matrix (Cholesky, then L^-T L^-1); false if the
// matrix is not SPD, a pivot being pivot_min times its diagonal entry or less.
bool spd_inverse(std::vector<double>& M, int n, double pivot_min);

}  // namespace pfem2
