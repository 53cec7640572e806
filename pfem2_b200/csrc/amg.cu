// amg.cu -- host setup of the smoothed-aggregation multigrid hierarchy of
// the pressure systems (runs once per pfem2_setup; FP64 throughout).
//
// Per system: level 0 is the eliminated pressure matrix (Dirichlet and
// padding rows have no off-diagonal entries and stay out of every
// aggregate). Levels 1 and 2 aggregate the level below with the classic
// three-pass greedy rule (seed + all-free neighbourhood, attach leftovers to
// the best-connected neighbouring aggregate, group the rest), restricted to
// one solver tile so that restriction never leaves the block that owns the
// tile. Level 3 takes one aggregate per tile. P_l is the tentative
// (piecewise-constant) prolongator smoothed once by (I - w D^-1 A_l), the
// coarse operator is the Galerkin product P_l^T A_l P_l, and w = 4 / (3
// rho(D^-1 A_l)) with rho from 30 power iterations (x 1.05).
#include <algorithm>
#include <cmath>
#include <numeric>

#include "amg.h"

namespace pfem2 {

namespace {

// Entries of J_1 and Pt_1 rows that a block may read for its level-1 halo per
// iteration; above, x1 is formed by the owners in a phase of its own. Pressure
// solve with halo rows / with the phase: channels of 8k to 52k cells (1 to 1.5k
// entries) 0.43 / 0.46 and 0.79 / 0.85 ms; pipes of 1.5k cells (7k) 0.56 / 0.49,
// 3k (13k) 0.99 / 0.52, 12k (12k) 1.31 / 0.73, 131k (23k) 4.2 / 3.4 FP64 and
// 2.8 / 1.8 FP32
constexpr size_t kHaloMax = 4096;

struct Csr {
  int n = 0, m = 0;
  std::vector<int> ptr{0}, col;
  std::vector<double> val;
};

Csr transpose(const Csr& A) {
  Csr T;
  T.n = A.m;
  T.m = A.n;
  T.ptr.assign(A.m + 1, 0);
  for (int c : A.col) T.ptr[c + 1]++;
  for (int i = 0; i < A.m; ++i) T.ptr[i + 1] += T.ptr[i];
  T.col.resize(A.col.size());
  T.val.resize(A.col.size());
  std::vector<int> pos(T.ptr.begin(), T.ptr.end() - 1);
  for (int i = 0; i < A.n; ++i)
    for (int e = A.ptr[i]; e < A.ptr[i + 1]; ++e) {
      const int p = pos[A.col[e]]++;
      T.col[p] = i;
      T.val[p] = A.val[e];
    }
  return T;
}

// C = A B, rows with ascending columns, exact zeros dropped
Csr spgemm(const Csr& A, const Csr& B) {
  Csr C;
  C.n = A.n;
  C.m = B.m;
  C.ptr.assign(A.n + 1, 0);
  std::vector<int> mark(B.m, -1), list;
  std::vector<double> acc(B.m, 0.0);
  for (int i = 0; i < A.n; ++i) {
    list.clear();
    for (int e = A.ptr[i]; e < A.ptr[i + 1]; ++e) {
      const int k = A.col[e];
      const double a = A.val[e];
      for (int f = B.ptr[k]; f < B.ptr[k + 1]; ++f) {
        const int j = B.col[f];
        if (mark[j] != i) {
          mark[j] = i;
          acc[j] = 0.0;
          list.push_back(j);
        }
        acc[j] += a * B.val[f];
      }
    }
    std::sort(list.begin(), list.end());
    for (int j : list)
      if (acc[j] != 0.0) {
        C.col.push_back(j);
        C.val.push_back(acc[j]);
      }
    C.ptr[i + 1] = (int)C.col.size();
  }
  return C;
}

// (I - w D^-1 A) P
Csr smooth(const Csr& A, const std::vector<double>& dinv, double w, const Csr& P) {
  const Csr AP = spgemm(A, P);
  Csr R;
  R.n = P.n;
  R.m = P.m;
  R.ptr.assign(P.n + 1, 0);
  for (int i = 0; i < P.n; ++i) {
    int a = P.ptr[i], b = AP.ptr[i];
    const int ae = P.ptr[i + 1], be = AP.ptr[i + 1];
    const double s = w * dinv[i];
    while (a < ae || b < be) {
      int j;
      double v;
      if (b >= be || (a < ae && P.col[a] < AP.col[b])) {
        j = P.col[a];
        v = P.val[a++];
      } else if (a >= ae || AP.col[b] < P.col[a]) {
        j = AP.col[b];
        v = -s * AP.val[b++];
      } else {
        j = P.col[a];
        v = P.val[a++] - s * AP.val[b++];
      }
      if (v != 0.0) {
        R.col.push_back(j);
        R.val.push_back(v);
      }
    }
    R.ptr[i + 1] = (int)R.col.size();
  }
  return R;
}

double rho_dinv_a(const Csr& A, const std::vector<double>& dinv) {
  const int n = A.n;
  std::vector<double> x(n), y(n);
  for (int i = 0; i < n; ++i) x[i] = 1.0 + 0.5 * std::sin(0.7 * i + 0.3);
  double lam = 1.0;
  for (int it = 0; it < 30; ++it) {
    double nx = 0.0, ny = 0.0;
    for (int i = 0; i < n; ++i) {
      double s = 0.0;
      for (int e = A.ptr[i]; e < A.ptr[i + 1]; ++e) s += A.val[e] * x[A.col[e]];
      y[i] = dinv[i] * s;
      nx += x[i] * x[i];
      ny += y[i] * y[i];
    }
    if (!(ny > 0.0)) break;
    lam = std::sqrt(ny / nx);
    const double inv = 1.0 / std::sqrt(ny);
    for (int i = 0; i < n; ++i) x[i] = y[i] * inv;
  }
  return 1.05 * lam;
}

bool isolated(const Csr& A, int i) {
  for (int e = A.ptr[i]; e < A.ptr[i + 1]; ++e)
    if (A.col[e] != i && A.val[e] != 0.0) return false;
  return true;
}

// Three-pass greedy aggregation inside tiles; aggregates renumbered in tile
// order (stable). Rows without off-diagonal entries get -1.
int aggregate(const Csr& A, const std::vector<int>& tile, std::vector<int>& agg) {
  const int n = A.n;
  agg.assign(n, -1);
  auto strong = [&](int i, int e) {
    const int j = A.col[e];
    return j != i && A.val[e] != 0.0 && tile[j] == tile[i];
  };
  std::vector<int> seed_tile;
  int na = 0;
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    bool any = false, free = true;
    for (int e = A.ptr[i]; e < A.ptr[i + 1]; ++e)
      if (strong(i, e)) {
        any = true;
        if (agg[A.col[e]] >= 0) free = false;
      }
    if (!any || !free) continue;
    agg[i] = na;
    for (int e = A.ptr[i]; e < A.ptr[i + 1]; ++e)
      if (strong(i, e)) agg[A.col[e]] = na;
    seed_tile.push_back(tile[i]);
    ++na;
  }
  std::vector<int> join(n, -1);
  std::vector<std::pair<int, int>> cnt;
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    cnt.clear();
    for (int e = A.ptr[i]; e < A.ptr[i + 1]; ++e) {
      if (!strong(i, e) || agg[A.col[e]] < 0) continue;
      const int a = agg[A.col[e]];
      bool found = false;
      for (auto& pc : cnt)
        if (pc.first == a) {
          pc.second++;
          found = true;
        }
      if (!found) cnt.push_back({a, 1});
    }
    int best = -1, bc = 0;
    for (auto& pc : cnt)
      if (pc.second > bc || (pc.second == bc && pc.first < best)) {
        best = pc.first;
        bc = pc.second;
      }
    join[i] = best;
  }
  for (int i = 0; i < n; ++i)
    if (join[i] >= 0) agg[i] = join[i];
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0 || isolated(A, i)) continue;
    agg[i] = na;
    for (int e = A.ptr[i]; e < A.ptr[i + 1]; ++e)
      if (strong(i, e) && agg[A.col[e]] < 0) agg[A.col[e]] = na;
    seed_tile.push_back(tile[i]);
    ++na;
  }
  std::vector<int> order(na), newid(na);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return seed_tile[a] < seed_tile[b]; });
  for (int k = 0; k < na; ++k) newid[order[k]] = k;
  for (int i = 0; i < n; ++i)
    if (agg[i] >= 0) agg[i] = newid[agg[i]];
  return na;
}

// one aggregate per group of `per` consecutive tiles, counted from tile t0
// (rows with off-diagonal entries only)
int tile_aggregate(const Csr& A, const std::vector<int>& tile, int t0, int per, std::vector<int>& agg) {
  agg.assign(A.n, -1);
  int na = 0, last = -1;
  for (int i = 0; i < A.n; ++i) {
    if (isolated(A, i)) continue;
    const int g = (tile[i] - t0) / per;
    if (g != last) {
      last = g;
      ++na;
    }
    agg[i] = na - 1;
  }
  return na;
}

// aggregates of aggregates: the graph of the tentative (piecewise-constant)
// coarse operator aggregated again inside the tiles, those without neighbours
// (parts of the mesh by themselves) kept, numbered in tile order; the new count
int merge_aggregates(const Csr& A, const std::vector<int>& tile, int na, std::vector<int>& agg) {
  Csr P;
  P.n = A.n;
  P.m = na;
  P.ptr.assign(A.n + 1, 0);
  std::vector<int> ctile(na, -1), cagg;
  for (int i = 0; i < A.n; ++i) {
    if (agg[i] >= 0) {
      P.col.push_back(agg[i]);
      P.val.push_back(1.0);
      ctile[agg[i]] = tile[i];
    }
    P.ptr[i + 1] = (int)P.col.size();
  }
  const Csr Ac = spgemm(transpose(P), spgemm(A, P));
  int nc = aggregate(Ac, ctile, cagg);
  std::vector<int> order(na), newid(na, -1);
  for (int k = 0; k < na; ++k)
    if (cagg[k] < 0) cagg[k] = nc++;
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return ctile[a] != ctile[b] ? ctile[a] < ctile[b] : cagg[a] < cagg[b];
  });
  int next = 0;
  for (int k : order)
    if (newid[cagg[k]] < 0) newid[cagg[k]] = next++;
  for (int i = 0; i < A.n; ++i)
    if (agg[i] >= 0) agg[i] = newid[cagg[agg[i]]];
  return nc;
}

struct Level {
  Csr A, J, P, Pt2;
  std::vector<double> dinv;
  std::vector<int> tile;
  double w = 0.0;
};

}  // namespace

bool spd_inverse(std::vector<double>& M, int n, double pivot_min) {
  std::vector<double> L((size_t)n * n, 0.0);
  for (int j = 0; j < n; ++j) {
    double d = M[(size_t)j * n + j];
    for (int k = 0; k < j; ++k) d -= L[(size_t)j * n + k] * L[(size_t)j * n + k];
    if (!(d > pivot_min * M[(size_t)j * n + j])) return false;
    d = std::sqrt(d);
    L[(size_t)j * n + j] = d;
    for (int i = j + 1; i < n; ++i) {
      double s = M[(size_t)i * n + j];
      for (int k = 0; k < j; ++k) s -= L[(size_t)i * n + k] * L[(size_t)j * n + k];
      L[(size_t)i * n + j] = s / d;
    }
  }
  std::vector<double> Li((size_t)n * n, 0.0);
  for (int j = 0; j < n; ++j) {
    Li[(size_t)j * n + j] = 1.0 / L[(size_t)j * n + j];
    for (int i = j + 1; i < n; ++i) {
      double s = 0.0;
      for (int k = j; k < i; ++k) s -= L[(size_t)i * n + k] * Li[(size_t)k * n + j];
      Li[(size_t)i * n + j] = s / L[(size_t)i * n + i];
    }
  }
  for (int i = 0; i < n; ++i)
    for (int j = 0; j <= i; ++j) {
      double s = 0.0;
      for (int k = i; k < n; ++k) s += Li[(size_t)k * n + i] * Li[(size_t)k * n + j];
      M[(size_t)i * n + j] = s;
      M[(size_t)j * n + i] = s;
    }
  return true;
}

pfem2_status mg_build(const Ctx& c, const std::vector<double>& A, const std::vector<int>& col,
                      const std::vector<int>& len, const std::vector<Tile>& tiles, const std::vector<int>& st0,
                      const std::vector<int>& bt0, int coarse_max, size_t b2_max, MgHost& H) {
  const int ni = (int)c.inst.size(), T = (int)tiles.size(), G = (int)bt0.size() - 1;
  // M2 is dense: level 2 is coarsened further where a system would have more
  // dofs than this. The line bounds memory (151 MB of FP32 rows per system, 4 GB
  // over a batch), not time: every iteration reads M2, and large 2D channels
  // solve faster with fewer dofs in spite of more iterations (144k cells: 2,609
  // dofs 2.8 ms FP64 and 2.6 FP32, 608 dofs 1.3 and 1.6; 262k cells: 4,160 dofs
  // 7.6 and 10.5 ms, 1,196 dofs 4.4 and 3.9). 3D pipes of up to 0.5M cells have
  // 1,700 at most
  const int n2_max = std::max(512, std::min(6144, (int)std::sqrt(1.0e9 / ni)));
  const std::vector<int>& sp = c.h_sl_ptr;
  std::vector<std::vector<Level>> sysL(ni);
  std::vector<std::vector<double>> Einv(ni);
  for (int s = 0; s < ni; ++s) {
    const int v0 = c.inst[s].v_off, n0 = c.inst[s].nv_pad;
    std::vector<Level>& L = sysL[s];
    L.resize(kMgLevels);
    // level 0 from the SELL layout
    Csr& A0 = L[0].A;
    A0.n = A0.m = n0;
    A0.ptr.assign(n0 + 1, 0);
    L[0].tile.assign(n0, -1);
    for (int t = st0[s]; t < st0[s + 1]; ++t)
      for (int sl = tiles[t].s0; sl < tiles[t].s1; ++sl)
        for (int l = 0; l < kSlice; ++l) L[0].tile[sl * kSlice + l - v0] = t;
    for (int i = 0; i < n0; ++i) {
      const int row = v0 + i, sl = row / kSlice, lane = row % kSlice;
      for (int j = 0; j < len[sl]; ++j) {
        const int e = sp[sl] + j * kSlice + lane;
        if ((j > 0 && col[e] == row) || A[e] == 0.0) continue;
        A0.col.push_back(col[e] - v0);
        A0.val.push_back(A[e]);
      }
      A0.ptr[i + 1] = (int)A0.col.size();
    }
    for (int l = 0; l < kMgLevels; ++l) {
      Level& V = L[l];
      const int n = V.A.n;
      if (n == 0) {
        set_error("amg: a pressure system has an empty coarse level");
        return PFEM2_MESH_ERROR;
      }
      V.dinv.assign(n, 0.0);
      for (int i = 0; i < n; ++i) {
        double d = 0.0;
        for (int e = V.A.ptr[i]; e < V.A.ptr[i + 1]; ++e)
          if (V.A.col[e] == i) d = V.A.val[e];
        if (!(d > 0.0)) {
          set_error("amg: a diagonal entry of the pressure matrix is not positive");
          return PFEM2_MESH_ERROR;
        }
        V.dinv[i] = 1.0 / d;
      }
      if (l == kMgLevels - 1) {
        std::vector<double> E((size_t)n * n, 0.0);
        for (int i = 0; i < n; ++i)
          for (int e = V.A.ptr[i]; e < V.A.ptr[i + 1]; ++e) E[(size_t)i * n + V.A.col[e]] = V.A.val[e];
        // symmetrise the Galerkin product's rounding
        for (int i = 0; i < n; ++i)
          for (int j = 0; j < i; ++j) {
            const double m = 0.5 * (E[(size_t)i * n + j] + E[(size_t)j * n + i]);
            E[(size_t)i * n + j] = E[(size_t)j * n + i] = m;
          }
        // a moving mesh has the Jacobi CG to fall back on where the operator is
        // singular up to rounding (no Dirichlet pressure: the last pivot is 6e-13
        // to 1e-10 of its diagonal, of either sign, on channels of 400 to 250k
        // cells; with an outflow pressure the smallest is 0.5)
        if (!spd_inverse(E, n, c.moving ? 1e-7 : 0.0)) {
          set_error("amg: the coarsest pressure operator is not SPD");
          return PFEM2_MESH_ERROR;
        }
        Einv[s] = std::move(E);
        break;
      }
      const double rho = rho_dinv_a(V.A, V.dinv);
      std::vector<int> agg;
      // the coarsest level: groups of tiles, at most coarse_max unknowns per system
      const int ntl = st0[s + 1] - st0[s], per = (ntl + coarse_max - 1) / coarse_max;
      int na = l < kMgLevels - 2 ? aggregate(V.A, V.tile, agg) : tile_aggregate(V.A, V.tile, st0[s], per, agg);
      while (l == 1 && na > n2_max) {
        const int nc = merge_aggregates(V.A, V.tile, na, agg);
        if (nc == na) break;
        na = nc;
      }
      if (na == 0) {
        set_error("amg: aggregation produced no coarse unknowns");
        return PFEM2_MESH_ERROR;
      }
      Csr Pt;
      Pt.n = n;
      Pt.m = na;
      Pt.ptr.assign(n + 1, 0);
      std::vector<int> ctile(na, -1);
      for (int i = 0; i < n; ++i) {
        if (agg[i] >= 0) {
          Pt.col.push_back(agg[i]);
          Pt.val.push_back(1.0);
          ctile[agg[i]] = V.tile[i];
        }
        Pt.ptr[i + 1] = (int)Pt.col.size();
      }
      V.P = smooth(V.A, V.dinv, 4.0 / (3.0 * rho), Pt);
      // smoother. Level 0 of a fixed mesh: 1 / sum_j |a_ij| in place of 1 / a_ii,
      // so that lambda_max <= 1 holds row by row (cells of a distorted part do
      // not damp the rest of the mesh) and w = 1.85 keeps J positive; otherwise
      // 1.6 / rho, on a moving mesh at most 0.49 (J stays positive there for any
      // 2D Q1 mesh). Iterations against 4 / (3 rho): channel with disk, 52k cells,
      // 37 -> 32 (solve 0.77 -> 0.67 ms, FP64), 13k 30 -> 25, 131k-cell pipe
      // 46 -> 42, 16 channels 44 -> 37; 1.8 / rho took 17 instead of 14 on a
      // uniform channel. The coarse levels' weights and an exact level 1 change
      // none of these by more than one. (1.6 / rho stays below 1.7 / lambda_max on
      // the coarse levels of graded, stretched, sheared and randomly distorted
      // channels.) Contexts that round P or V to FP32 for the right-hand sides keep
      // 4 / (3 rho) (34k-cell channel 0.66 ms per solve, 0.60 with the row sums).
      // That is for the same results, not for better ones: the rounding turns
      // differences far below the solver's tolerance into last-bit flips and 1e-6
      // in the loads, whose error against FP64 is 5e-5 with either weight.
      if (c.amixed || c.prmixed) {
        V.w = 4.0 / (3.0 * rho);
        if (l == 0 && c.moving) V.w = std::min(V.w, 0.49);
      } else if (l == 0 && !c.moving) {
        for (int i = 0; i < n; ++i) {
          double sum = 0.0;
          for (int e = V.A.ptr[i]; e < V.A.ptr[i + 1]; ++e) sum += std::fabs(V.A.val[e]);
          V.dinv[i] = 1.0 / sum;
        }
        V.w = 1.85;
      } else {
        V.w = 1.6 / rho;
        if (l == 0) V.w = std::min(V.w, 0.49);
      }
      // J = 2 w D^-1 - w^2 D^-1 A D^-1
      V.J = V.A;
      for (int i = 0; i < n; ++i)
        for (int e = V.J.ptr[i]; e < V.J.ptr[i + 1]; ++e) {
          const int j = V.J.col[e];
          V.J.val[e] = -V.w * V.w * V.dinv[i] * V.A.val[e] * V.dinv[j] + (i == j ? 2.0 * V.w * V.dinv[i] : 0.0);
        }
      V.Pt2 = smooth(V.A, V.dinv, V.w, V.P);
      L[l + 1].A = spgemm(transpose(V.P), spgemm(V.A, V.P));
      L[l + 1].tile = ctile;
    }
    H.w0.push_back(L[0].w);
    H.d0.insert(H.d0.end(), L[0].dinv.begin(), L[0].dinv.end());
  }
  // ---- global numbering: systems in order, dofs tile-ordered inside
  std::vector<std::vector<int>> goff(kMgLevels, std::vector<int>(ni + 1, 0));
  for (int l = 1; l < kMgLevels; ++l) {
    for (int s = 0; s < ni; ++s) goff[l][s + 1] = goff[l][s] + sysL[s][l].A.n;
    H.n[l] = goff[l][ni];
    H.toff[l].assign(T + 1, 0);
    H.lsys[l].resize(H.n[l]);
    for (int s = 0; s < ni; ++s) {
      const std::vector<int>& tl = sysL[s][l].tile;
      for (int a = 0; a < (int)tl.size(); ++a) {
        H.toff[l][tl[a] + 1]++;
        H.lsys[l][goff[l][s] + a] = s;
      }
    }
    for (int t = 0; t < T; ++t) H.toff[l][t + 1] += H.toff[l][t];
  }
  H.n[0] = c.nv;
  std::vector<int> sys_of_tile(T);
  for (int s = 0; s < ni; ++s)
    for (int t = st0[s]; t < st0[s + 1]; ++t) sys_of_tile[t] = s;
  // what a block holds of level 2, before the dense matrices of that size are made
  for (int b = 0; b < G; ++b)
    if (bt0[b + 1] > bt0[b]) {
      const int s0 = sys_of_tile[bt0[b]], s1 = sys_of_tile[bt0[b + 1] - 1];
      H.b2max = std::max(H.b2max, goff[2][s1 + 1] - goff[2][s0]);
    }
  if ((size_t)H.b2max > b2_max) {
    set_error("krylov: the pressure multigrid's per-block data exceed shared memory");
    return PFEM2_INVALID_ARG;
  }
  // ---- restrictions
  auto append_rows = [](const Csr& M, int coff, std::vector<int>& ptr, std::vector<int>& cl, std::vector<double>& vl) {
    if (ptr.empty()) ptr.push_back(0);
    for (int i = 0; i < M.n; ++i) {
      for (int e = M.ptr[i]; e < M.ptr[i + 1]; ++e) {
        cl.push_back(M.col[e] + coff);
        vl.push_back(M.val[e]);
      }
      ptr.push_back((int)cl.size());
    }
  };
  for (int s = 0; s < ni; ++s) {
    std::vector<Level>& L = sysL[s];
    Csr R = transpose(L[0].Pt2);
    if (!c.moving)
      for (size_t e = 0; e < R.col.size(); ++e) R.val[e] /= L[0].dinv[R.col[e]];
    append_rows(R, c.inst[s].v_off, H.r1_ptr, H.r1_col, H.r1_val);
    append_rows(transpose(L[1].Pt2), goff[1][s], H.q2_ptr, H.q2_col, H.q2_val);
    const int n2 = L[2].A.n, n3 = L[3].A.n;
    H.sys_n2.push_back(n2);
    H.sys_off2.push_back(goff[2][s]);
    // M2 = J_2 + (Pt_2 E^-1) Pt_2^T
    const Csr& P = L[2].Pt2;
    const size_t m0 = H.m2.size();
    H.m2.resize(m0 + (size_t)n2 * n2, 0.0);
    std::vector<double> t(n3);
    for (int i = 0; i < n2; ++i) {
      double* row = H.m2.data() + m0 + (size_t)i * n2;
      std::fill(t.begin(), t.end(), 0.0);
      for (int e = P.ptr[i]; e < P.ptr[i + 1]; ++e) {
        const double v = P.val[e];
        const double* E = Einv[s].data() + (size_t)P.col[e] * n3;
        for (int d = 0; d < n3; ++d) t[d] += v * E[d];
      }
      for (int j = 0; j < n2; ++j) {
        double v = 0.0;
        for (int e = P.ptr[j]; e < P.ptr[j + 1]; ++e) v += t[P.col[e]] * P.val[e];
        row[j] = v;
      }
      for (int e = L[2].J.ptr[i]; e < L[2].J.ptr[i + 1]; ++e) row[L[2].J.col[e]] += L[2].J.val[e];
    }
  }
  // ---- per-block lists
  std::vector<int> loc1(H.n[1], -1);
  // the level-1 halo each block's rows prolong from, and the entries of its
  // J_1 and Pt_1 rows
  std::vector<std::vector<int>> halo(G);
  size_t nhalo = 0;
  for (int b = 0; b < G; ++b) {
    const int t_lo = bt0[b], t_hi = bt0[b + 1];
    std::vector<int>& h = halo[b];
    for (int t = t_lo; t < t_hi; ++t) {
      const int s = sys_of_tile[t], v0 = c.inst[s].v_off;
      const Csr& P = sysL[s][0].Pt2;
      for (int e = P.ptr[tiles[t].s0 * kSlice - v0]; e < P.ptr[tiles[t].s1 * kSlice - v0]; ++e) {
        const int g = goff[1][s] + P.col[e];
        if ((g < H.toff[1][t_lo] || g >= H.toff[1][t_hi]) && loc1[g] != b) {
          loc1[g] = b;
          h.push_back(g);
        }
      }
    }
    std::sort(h.begin(), h.end());
    for (int g : h) {
      const int s = H.lsys[1][g], r = g - goff[1][s];
      const Level& V = sysL[s][1];
      nhalo += V.J.ptr[r + 1] - V.J.ptr[r] + V.Pt2.ptr[r + 1] - V.Pt2.ptr[r];
    }
  }
  std::fill(loc1.begin(), loc1.end(), -1);
  H.xsplit = nhalo > (size_t)G * kHaloMax;
  H.blk_s1.assign(1, 0);
  H.j1_ptr.assign(1, 0);
  H.p1_ptr.assign(1, 0);
  H.blk_m2.assign(1, 0);
  H.m2_off.assign(H.n[2], 0);
  H.p0_ptr.assign(c.nslices + 1, 0);
  H.p0_len.assign(c.nslices, 0);
  std::vector<std::vector<int>> p0c(c.nslices);
  std::vector<std::vector<double>> p0v(c.nslices);
  for (int l = 1; l <= 2; ++l) H.lk[l].assign(H.n[l], 0);
  for (int b = 0; b < G; ++b) {
    const int t_lo = bt0[b], t_hi = bt0[b + 1];
    // systems of a block are consecutive; lists store the index among them
    const int sys_first = t_hi > t_lo ? sys_of_tile[t_lo] : 0;
    for (int l = 1; l <= 2; ++l)
      for (int g = H.toff[l][t_lo]; g < H.toff[l][t_hi]; ++g) H.lk[l][g] = H.lsys[l][g] - sys_first;
    long long mo = 0;
    for (int g = H.toff[2][t_lo]; g < H.toff[2][t_hi]; ++g) {
      H.m2_off[g] = (int)mo;
      mo += sysL[H.lsys[2][g]][2].A.n;
    }
    H.blk_m2.push_back(H.blk_m2.back() + mo);
    // own level-1 dofs, then the halo the level-0 prolongation reads
    std::vector<int> S1;
    for (int g = H.toff[1][t_lo]; g < H.toff[1][t_hi]; ++g) S1.push_back(g);
    if (!H.xsplit) S1.insert(S1.end(), halo[b].begin(), halo[b].end());
    for (int k = 0; k < (int)S1.size(); ++k) loc1[S1[k]] = k;
    for (int g : S1) {
      const int s = H.lsys[1][g], r = g - goff[1][s];
      const Level& V = sysL[s][1];
      H.s1_lk.push_back(s - sys_first);
      for (int e = V.J.ptr[r]; e < V.J.ptr[r + 1]; ++e) {
        H.j1_col.push_back(goff[1][s] + V.J.col[e]);
        H.j1_val.push_back(V.J.val[e]);
      }
      H.j1_ptr.push_back((int)H.j1_col.size());
      for (int e = V.Pt2.ptr[r]; e < V.Pt2.ptr[r + 1]; ++e) {
        H.p1_col.push_back(goff[2][s] + V.Pt2.col[e]);
        H.p1_val.push_back(V.Pt2.val[e]);
      }
      H.p1_ptr.push_back((int)H.p1_col.size());
    }
    H.blk_s1.push_back((int)H.s1_lk.size());
    H.s1max = std::max(H.s1max, (int)S1.size());
    // level-0 prolongation rows of the block's slices
    for (int t = t_lo; t < t_hi; ++t) {
      const int s = sys_of_tile[t], v0 = c.inst[s].v_off;
      const Csr& P = sysL[s][0].Pt2;
      for (int sl = tiles[t].s0; sl < tiles[t].s1; ++sl) {
        int mx = 0;
        for (int l = 0; l < kSlice; ++l) {
          const int i = sl * kSlice + l - v0;
          mx = std::max(mx, P.ptr[i + 1] - P.ptr[i]);
        }
        H.p0_len[sl] = mx;
        p0c[sl].assign((size_t)mx * kSlice, 0);
        p0v[sl].assign((size_t)mx * kSlice, 0.0);
        for (int l = 0; l < kSlice; ++l) {
          const int i = sl * kSlice + l - v0;
          for (int e = P.ptr[i]; e < P.ptr[i + 1]; ++e) {
            const int j = e - P.ptr[i];
            const int g = goff[1][s] + P.col[e];
            p0c[sl][(size_t)j * kSlice + l] = H.xsplit ? g : loc1[g];
            p0v[sl][(size_t)j * kSlice + l] = P.val[e];
          }
        }
      }
    }
    for (int g : S1) loc1[g] = -1;
  }
  for (int sl = 0; sl < c.nslices; ++sl) {
    H.p0_ptr[sl + 1] = H.p0_ptr[sl] + H.p0_len[sl] * kSlice;
    H.p0_col.insert(H.p0_col.end(), p0c[sl].begin(), p0c[sl].end());
    H.p0_val.insert(H.p0_val.end(), p0v[sl].begin(), p0v[sl].end());
  }
  return PFEM2_OK;
}

}  // namespace pfem2
