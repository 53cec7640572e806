// ale.cu -- the moving mesh of the reference's cylinderDyM case on the GPU:
// the pseudo-solid elasticity solve for the mesh displacement
// (problem_of_elasticity + solveU, cylinderDyM/cylinderDyM.cc:926-976,
// 886-903), the reinterpolation of the nodal fields at the displaced
// vertices (reinterpolate_fields, cylinderDyM/pfem2particle.cpp:1144-1235),
// the grid transformation (transform_grid, :1237-1261) with the rebuilt
// per-cell records, and the particles' relocation in the moved mesh
// (sort_particles_into_subdomains_and_cells, then check_empty_cells).
//
// The elasticity system couples the dim displacement components. It is one
// scalar system of dim x nv rows, components one after the other, on slices
// of its own: slice c nslices + s holds rows c nv + 32 s ..., with the entries
// of the scalar pattern's slice s once per column component. Assembly is
// node-centric like the flow matrices (a thread owns a vertex' rows and sums
// its cells in ascending order: deterministic, no atomics), Dirichlet rows and
// columns are eliminated symmetrically, and the flow's Jacobi CG kernel solves
// it (krylov.cu, FP64, one reduction per iteration, one thread-block cluster
// for small meshes): 8.2 us per
// iteration on a mesh of 8k cells against 11.6 with two reductions and a grid
// barrier after each.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "fe.cuh"

namespace pfem2 {

__device__ __forceinline__ int ale_entry(const int* __restrict__ sl_ptr, int row, int j) {
  return sl_ptr[row >> 5] + j * 32 + (row & 31);
}

// entry e of vertex row `row` in the scalar pattern, row component a, column
// component b (nell entries in the scalar pattern)
template <int DIM>
__device__ __forceinline__ size_t el_entry(const int* __restrict__ sl_ptr, const int* __restrict__ sl_len, int nell,
                                           int row, int e, int a, int b) {
  const int s = row >> 5, p = sl_ptr[s];
  return (size_t)DIM * ((size_t)a * nell + p) + (size_t)b * sl_len[s] * 32 + (e - p);
}

// K[(a, ci), (b, cj)] += sum over the cells around vertex a and their
// QGauss(2) points of (lambda d_ci N_a d_cj N_b + mu d_cj N_a d_ci N_b
// + delta_ci,cj mu grad N_a . grad N_b) JxW
template <int DIM>
__global__ void __launch_bounds__(128) k_elastic_assemble(int nv, int nell, const int* __restrict__ v2c_ptr,
                                                          const int* __restrict__ v2c_cell,
                                                          const unsigned char* __restrict__ v2c_loc,
                                                          const int* __restrict__ inc_slot, const int* __restrict__ sl_ptr,
                                                          const int* __restrict__ sl_len, const double* __restrict__ X,
                                                          const int* __restrict__ cv, double lambda, double mu,
                                                          double* __restrict__ K) {
  constexpr int NV = Dims<DIM>::NV;
  for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < nv; row += gridDim.x * blockDim.x) {
    for (int k = v2c_ptr[row]; k < v2c_ptr[row + 1]; ++k) {
      const int c = v2c_cell[k], la = v2c_loc[k];
      LocalCell<DIM, double> L;
      double x0[DIM];
      load_local_cell<DIM, double>(X, cv, c, L, x0);
      for (int iq = 0; iq < NV; ++iq) {
        double xi[DIM];
        cell_qp_xi<DIM, double>(iq, xi);
        QP<DIM, double> q;
        eval_qp<DIM, double>(L, xi, cell_qp_w<DIM>(), -1, q);
        for (int lb = 0; lb < NV; ++lb) {
          const int e = inc_slot[(size_t)k * NV + lb];
          double gg = 0.0;
#pragma unroll
          for (int d = 0; d < DIM; ++d) gg += q.G[la][d] * q.G[lb][d];
#pragma unroll
          for (int ci = 0; ci < DIM; ++ci)
#pragma unroll
            for (int cj = 0; cj < DIM; ++cj) {
              double v = lambda * q.G[la][ci] * q.G[lb][cj] + mu * q.G[la][cj] * q.G[lb][ci];
              if (ci == cj) v += mu * gg;
              K[el_entry<DIM>(sl_ptr, sl_len, nell, row, e, ci, cj)] += v * q.JxW;
            }
        }
      }
    }
  }
}

// symmetric elimination of the constrained vertices (fix[v]: all
// components, values g[d * nv + v]): a constrained row keeps its diagonal
// blocks' diagonal (1 where it is 0: padding rows) and gets rhs = K_aa g_a;
// a free row moves its constrained columns to the right-hand side
template <int DIM>
__global__ void k_elastic_eliminate(int nv, int nell, const int* __restrict__ sl_ptr, const int* __restrict__ sl_len,
                                    const int* __restrict__ sl_col, double* __restrict__ K,
                                    const unsigned char* __restrict__ fix, const double* __restrict__ g,
                                    double* __restrict__ rhs, double* __restrict__ dinv) {
  for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < nv; row += gridDim.x * blockDim.x) {
    const int len = sl_len[row >> 5];
    const int e0 = ale_entry(sl_ptr, row, 0);
    const auto at = [&](int e, int a, int b) -> double& { return K[el_entry<DIM>(sl_ptr, sl_len, nell, row, e, a, b)]; };
    if (fix[row]) {
      for (int j = 0; j < len; ++j) {
        const int e = ale_entry(sl_ptr, row, j);
        const bool diag = sl_col[e] == row && j == 0;
#pragma unroll
        for (int a = 0; a < DIM; ++a)
#pragma unroll
          for (int b = 0; b < DIM; ++b)
            if (!(diag && a == b)) at(e, a, b) = 0.0;
      }
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        double& d = at(e0, a, a);
        if (d == 0.0) d = 1.0;
        rhs[(size_t)a * nv + row] = d * g[(size_t)a * nv + row];
        dinv[(size_t)a * nv + row] = 1.0 / d;
      }
    } else {
      double s[DIM];
#pragma unroll
      for (int a = 0; a < DIM; ++a) s[a] = 0.0;
      for (int j = 1; j < len; ++j) {
        const int e = ale_entry(sl_ptr, row, j);
        const int col = sl_col[e];
        if (col == row || !fix[col]) continue;
#pragma unroll
        for (int a = 0; a < DIM; ++a)
#pragma unroll
          for (int b = 0; b < DIM; ++b) {
            s[a] -= at(e, a, b) * g[(size_t)b * nv + col];
            at(e, a, b) = 0.0;
          }
      }
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        rhs[(size_t)a * nv + row] = s[a];
        dinv[(size_t)a * nv + row] = 1.0 / at(e0, a, a);
      }
    }
  }
}

// reinterpolate_fields: interior vertices take Vx, Vy(, Vz), P at their
// displaced position from the lowest-index cell around them that contains
// it (inside with tolerance 1e-5), then the others in ascending order;
// boundary vertices and vertices found nowhere keep their values
template <int DIM>
__global__ void k_reinterpolate(int nv, const double* __restrict__ X, const int* __restrict__ cv,
                                const int* __restrict__ v2c_ptr, const int* __restrict__ v2c_cell,
                                const unsigned char* __restrict__ bnd, const double* __restrict__ U0,
                                const double* __restrict__ U1, const double* __restrict__ U2,
                                const double* __restrict__ F0, const double* __restrict__ F1,
                                const double* __restrict__ F2, const double* __restrict__ F3,
                                double* __restrict__ out) {
  constexpr int NV = Dims<DIM>::NV;
  const double* U[3] = {U0, U1, U2};
  const double* F[4] = {F0, F1, F2, F3};
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
    double val[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) val[k] = F[k] ? F[k][v] : 0.0;
    if (!bnd[v]) {
      for (int k = v2c_ptr[v]; k < v2c_ptr[v + 1]; ++k) {
        const int c = v2c_cell[k];
        LocalCell<DIM, double> L;
        double x0[DIM], xl[DIM], xi[DIM];
        load_local_cell<DIM, double>(X, cv, c, L, x0);
#pragma unroll
        for (int d = 0; d < DIM; ++d) xl[d] = (X[(size_t)v * DIM + d] + U[d][v]) - x0[d];
        if (!local_inverse<DIM, double>(L, xl, xi)) continue;
        bool in = true;
#pragma unroll
        for (int d = 0; d < DIM; ++d) in = in && xi[d] >= -1e-5 && xi[d] <= 1.0 + 1e-5;
        if (!in) continue;
        double N[NV];
        shape_values<DIM, double>(xi, N);
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          if (!F[f]) continue;
          double s = 0.0;
#pragma unroll
          for (int b = 0; b < NV; ++b) s += N[b] * F[f][cv[(size_t)c * NV + b]];
          val[f] = s;
        }
        break;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) out[(size_t)k * nv + v] = val[k];
  }
}

template <int DIM>
__global__ void k_transform(int nv, double* __restrict__ X, const double* __restrict__ U0,
                            const double* __restrict__ U1, const double* __restrict__ U2) {
  const double* U[3] = {U0, U1, U2};
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x)
#pragma unroll
    for (int d = 0; d < DIM; ++d) X[(size_t)v * DIM + d] += U[d][v];
}

// unit direction vertex -> cell centre of every incidence (FP64 and the
// particle kernels' type)
template <int DIM>
__global__ void k_v2c_dir(int nv, const double* __restrict__ X, const int* __restrict__ cv,
                          const int* __restrict__ v2c_ptr, const int* __restrict__ v2c_cell, double* __restrict__ dir,
                          float* __restrict__ dirf) {
  constexpr int NV = Dims<DIM>::NV;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x)
    for (int k = v2c_ptr[v]; k < v2c_ptr[v + 1]; ++k) {
      const int c = v2c_cell[k];
      double ctr[DIM], nn = 0.0;
#pragma unroll
      for (int a = 0; a < DIM; ++a) ctr[a] = 0.0;
      for (int b = 0; b < NV; ++b)
#pragma unroll
        for (int a = 0; a < DIM; ++a) ctr[a] += X[(size_t)cv[(size_t)c * NV + b] * DIM + a];
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        ctr[a] = ctr[a] / NV - X[(size_t)v * DIM + a];
        nn += ctr[a] * ctr[a];
      }
      nn = sqrt(nn);
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        dir[(size_t)k * DIM + a] = ctr[a] / nn;
        if (dirf) dirf[(size_t)k * DIM + a] = (float)(ctr[a] / nn);
      }
    }
}

// the tables and vectors that ale_alloc makes
static void ale_free_tables(Ctx& c) {
  void** p[] = {(void**)&c.ale_K,   (void**)&c.ale_fix, (void**)&c.ale_g,   (void**)&c.ale_rhs,
                (void**)&c.ale_dinv, (void**)&c.ale_x,  (void**)&c.ale_new, (void**)&c.ale_flag,
                (void**)&c.ale_slp, (void**)&c.ale_sll, (void**)&c.ale_slc};
  for (void** q : p) {
    if (*q) cudaFree(*q);
    *q = nullptr;
  }
}

static pfem2_status ale_alloc_tables(Ctx& c) {
  const size_t nv = c.nv, dim = c.dim;
  auto al = [&](void** p, size_t bytes) -> pfem2_status {
    *p = nullptr;
    PFEM2_CUDA(cudaMalloc(p, bytes));
    PFEM2_CUDA(cudaMemset(*p, 0, bytes));
    return PFEM2_OK;
  };
  PFEM2_TRY(al((void**)&c.ale_K, sizeof(double) * dim * dim * c.nell));
  PFEM2_TRY(al((void**)&c.ale_fix, dim * nv));
  PFEM2_TRY(al((void**)&c.ale_g, sizeof(double) * dim * nv));
  PFEM2_TRY(al((void**)&c.ale_rhs, sizeof(double) * dim * nv));
  PFEM2_TRY(al((void**)&c.ale_dinv, sizeof(double) * dim * nv));
  PFEM2_TRY(al((void**)&c.ale_x, sizeof(double) * dim * nv));
  PFEM2_TRY(al((void**)&c.ale_new, sizeof(double) * 4 * nv));
  PFEM2_TRY(al((void**)&c.ale_flag, sizeof(int)));
  // the system's own slices (see the head of this file)
  std::vector<int> len(c.nslices), col(c.nell), slp(1, 0), sll, slc((size_t)dim * dim * c.nell);
  PFEM2_CUDA(cudaMemcpy(len.data(), c.sl_len, sizeof(int) * c.nslices, cudaMemcpyDeviceToHost));
  PFEM2_CUDA(cudaMemcpy(col.data(), c.sl_col, sizeof(int) * c.nell, cudaMemcpyDeviceToHost));
  for (size_t a = 0; a < dim; ++a)
    for (int s = 0; s < c.nslices; ++s) {
      const int n = len[s] * kSlice, p = c.h_sl_ptr[s];
      for (size_t b = 0; b < dim; ++b)
        for (int e = 0; e < n; ++e) slc[slp.back() + b * n + e] = (int)(b * nv) + col[p + e];
      sll.push_back((int)dim * len[s]);
      slp.push_back(slp.back() + (int)dim * n);
    }
  PFEM2_TRY(al((void**)&c.ale_slp, sizeof(int) * slp.size()));
  PFEM2_TRY(al((void**)&c.ale_sll, sizeof(int) * sll.size()));
  PFEM2_TRY(al((void**)&c.ale_slc, sizeof(int) * slc.size()));
  PFEM2_CUDA(cudaMemcpy(c.ale_slp, slp.data(), sizeof(int) * slp.size(), cudaMemcpyHostToDevice));
  PFEM2_CUDA(cudaMemcpy(c.ale_sll, sll.data(), sizeof(int) * sll.size(), cudaMemcpyHostToDevice));
  PFEM2_CUDA(cudaMemcpy(c.ale_slc, slc.data(), sizeof(int) * slc.size(), cudaMemcpyHostToDevice));
  PFEM2_TRY(krylov_elastic_setup(c, slp));
  PFEM2_CUDA(cudaDeviceSynchronize());  // (these copies are on the default stream)
  return PFEM2_OK;
}

// on the first use; a call that fails half-way leaves nothing behind
static pfem2_status ale_alloc(Ctx& c) {
  if (c.ale_ready) return PFEM2_OK;
  const pfem2_status st = ale_alloc_tables(c);
  c.ale_ready = st == PFEM2_OK;
  if (!c.ale_ready) ale_free_tables(c);
  return st;
}

// boundary vertices (on any boundary face) of the mesh, once at setup
pfem2_status ale_setup(Ctx& c) {
  const int NV = 1 << c.dim, NF = 2 * c.dim;
  std::vector<unsigned char> bnd(c.nv, 0);
  for (const HostInst& in : c.inst)
    for (int ce = 0; ce < in.nc; ++ce)
      for (int f = 0; f < NF; ++f) {
        if (in.fb[(size_t)ce * NF + f] < 0) continue;
        for (int v = 0; v < NV; ++v)
          if (((v >> (f / 2)) & 1) == f % 2) bnd[in.v_off + in.cells[(size_t)ce * NV + v]] = 1;
      }
  PFEM2_CUDA(cudaMalloc((void**)&c.ale_bnd, c.nv));
  PFEM2_CUDA(cudaMemcpy(c.ale_bnd, bnd.data(), c.nv, cudaMemcpyHostToDevice));
  return PFEM2_OK;
}

void ale_free(Ctx& c) {
  ale_free_tables(c);
  if (c.ale_bnd) cudaFree(c.ale_bnd);
  if (c.ale_xphys) cudaFree(c.ale_xphys);
}

pfem2_status ale_elasticity(Ctx& c, const pfem2_elasticity& e, const double* body_disp, int* iters, double* res) {
  PFEM2_TRY(ale_alloc(c));
  const int dim = c.dim, NV = 1 << dim, NF = 2 * dim;
  const size_t nv = c.nv;
  // constrained vertices: fixed boundaries (zero) and the body; padding rows
  std::vector<unsigned char> fix(dim * nv, 0);  // (the same per component)
  std::vector<double> g(dim * nv, 0.0);
  for (const HostInst& in : c.inst) {
    for (int k = in.nv; k < in.nv_pad; ++k) fix[in.v_off + k] = 1;
    for (int ce = 0; ce < in.nc; ++ce)
      for (int f = 0; f < NF; ++f) {
        const int b = in.fb[(size_t)ce * NF + f];
        if (b < 0) continue;
        const bool isfix = b < 32 && ((e.fixed_mask >> b) & 1u), isbody = b == e.body_id;
        if (!isfix && !isbody) continue;
        for (int v = 0; v < NV; ++v)
          if (((v >> (f / 2)) & 1) == f % 2) {
            const int gv = in.v_off + in.cells[(size_t)ce * NV + v];
            fix[gv] = 1;
            for (int d = 0; d < dim; ++d) g[(size_t)d * nv + gv] = isbody ? body_disp[d] : 0.0;
          }
      }
  }
  for (int d = 1; d < dim; ++d) std::copy(fix.begin(), fix.begin() + nv, fix.begin() + (size_t)d * nv);
  PFEM2_CUDA(cudaMemcpyAsync(c.ale_fix, fix.data(), dim * nv, cudaMemcpyHostToDevice, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(c.ale_g, g.data(), sizeof(double) * dim * nv, cudaMemcpyHostToDevice, c.stream));
  PFEM2_CUDA(cudaMemsetAsync(c.ale_K, 0, sizeof(double) * dim * dim * c.nell, c.stream));
  PFEM2_CUDA(cudaMemsetAsync(c.ale_x, 0, sizeof(double) * dim * nv, c.stream));  // x0 = g on the constrained rows, else 0
  const int grid = grid_for(c, c.nv, 128, 8), g2 = grid_for(c, c.nv, 256, 8);
  if (dim == 2) {
    k_elastic_assemble<2><<<grid, 128, 0, c.stream>>>(c.nv, c.nell, c.v2c_ptr, c.v2c_cell, c.v2c_loc, c.inc_slot,
                                                      c.sl_ptr, c.sl_len, c.X, c.cv, e.lambda, e.mu, c.ale_K);
    k_elastic_eliminate<2><<<g2, 256, 0, c.stream>>>(c.nv, c.nell, c.sl_ptr, c.sl_len, c.sl_col, c.ale_K, c.ale_fix,
                                                     c.ale_g, c.ale_rhs, c.ale_dinv);
  } else {
    k_elastic_assemble<3><<<grid, 128, 0, c.stream>>>(c.nv, c.nell, c.v2c_ptr, c.v2c_cell, c.v2c_loc, c.inc_slot,
                                                      c.sl_ptr, c.sl_len, c.X, c.cv, e.lambda, e.mu, c.ale_K);
    k_elastic_eliminate<3><<<g2, 256, 0, c.stream>>>(c.nv, c.nell, c.sl_ptr, c.sl_len, c.sl_col, c.ale_K, c.ale_fix,
                                                     c.ale_g, c.ale_rhs, c.ale_dinv);
  }
  c.launches += 2;
  const ElasticSystem E{c.ale_slp, c.ale_sll, c.ale_slc, c.ale_K, c.ale_dinv, c.ale_rhs, c.ale_g, c.ale_fix, c.ale_x};
  PFEM2_TRY(krylov_elastic_solve(c, E, e.tol, e.rtol, e.max_iter > 0 ? e.max_iter : 10000));
  // the displacement into the fields
  for (int d = 0; d < dim; ++d)
    PFEM2_CUDA(cudaMemcpyAsync(c.F[PFEM2_FIELD_DISP_X + d], c.ale_x + (size_t)d * nv, sizeof(double) * nv,
                               cudaMemcpyDeviceToDevice, c.stream));
  int it = 0, err = 0;
  double rr = 0.0, tol = 0.0;
  PFEM2_CUDA(cudaMemcpyAsync(&err, c.d_err, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  PFEM2_TRY(krylov_elastic_read(c, &it, &rr, &tol));
  if (iters) *iters = it;
  if (res) *res = rr;
  if (err) {
    set_error("mesh elasticity: a wait of the solver timed out");
    c.failed = true;
    return PFEM2_TIMEOUT;
  }
  if (!(rr <= tol)) {
    set_error("mesh elasticity: the CG did not converge within max_iter");
    return PFEM2_NOT_CONVERGED;
  }
  return PFEM2_OK;
}

pfem2_status ale_move_mesh(Ctx& c) {
  PFEM2_TRY(ale_alloc(c));
  const int dim = c.dim;
  const size_t nv = c.nv;
  const double* U[3] = {c.F[PFEM2_FIELD_DISP_X], c.F[PFEM2_FIELD_DISP_Y], dim == 3 ? c.F[PFEM2_FIELD_DISP_Z] : nullptr};
  // 1. the particles' physical positions in the old mesh
  if (c.seeded) {
    if (c.ale_xphys_cap < (size_t)c.pcap) {
      if (c.ale_xphys) cudaFree(c.ale_xphys);
      PFEM2_CUDA(cudaMalloc((void**)&c.ale_xphys, sizeof(double) * dim * (size_t)c.pcap));
      c.ale_xphys_cap = c.pcap;
    }
    PFEM2_TRY(launch_particle_positions(c, c.ale_xphys));
  }
  // 2. the fields at the displaced vertices (old mesh)
  const int grid = grid_for(c, c.nv, 128, 8);
  const double* Fv[4] = {c.F[PFEM2_FIELD_VX], c.F[PFEM2_FIELD_VY], dim == 3 ? c.F[PFEM2_FIELD_VZ] : nullptr,
                         c.F[PFEM2_FIELD_P]};
  if (dim == 2)
    k_reinterpolate<2><<<grid, 128, 0, c.stream>>>(c.nv, c.X, c.cv, c.v2c_ptr, c.v2c_cell, c.ale_bnd, U[0], U[1], U[2],
                                                   Fv[0], Fv[1], Fv[2], Fv[3], c.ale_new);
  else
    k_reinterpolate<3><<<grid, 128, 0, c.stream>>>(c.nv, c.X, c.cv, c.v2c_ptr, c.v2c_cell, c.ale_bnd, U[0], U[1], U[2],
                                                   Fv[0], Fv[1], Fv[2], Fv[3], c.ale_new);
  c.launches++;
  for (int k = 0; k < 4; ++k)
    if (Fv[k])
      PFEM2_CUDA(cudaMemcpyAsync((void*)Fv[k], c.ale_new + (size_t)k * nv, sizeof(double) * nv,
                                 cudaMemcpyDeviceToDevice, c.stream));
  // the particle kernels' mirrors of V and V - V_old follow (the re-seeding
  // of check_empty_cells below interpolates V)
  PFEM2_TRY(launch_sync_real_fields(c));
  // 3. move the vertices; the per-cell records and directions follow
  if (dim == 2) k_transform<2><<<grid, 128, 0, c.stream>>>(c.nv, c.X, U[0], U[1], U[2]);
  else k_transform<3><<<grid, 128, 0, c.stream>>>(c.nv, c.X, U[0], U[1], U[2]);
  if (dim == 2)
    k_v2c_dir<2><<<grid, 128, 0, c.stream>>>(c.nv, c.X, c.cv, c.v2c_ptr, c.v2c_cell, c.v2c_dir,
                                             c.pmixed ? (float*)c.v2c_dir_r : nullptr);
  else
    k_v2c_dir<3><<<grid, 128, 0, c.stream>>>(c.nv, c.X, c.cv, c.v2c_ptr, c.v2c_cell, c.v2c_dir,
                                             c.pmixed ? (float*)c.v2c_dir_r : nullptr);
  c.launches += 2;
  PFEM2_CUDA(cudaMemsetAsync(c.ale_flag, 0, sizeof(int), c.stream));
  PFEM2_TRY(launch_cell_geo(c, c.ale_flag));
  // 4. the particles in the moved mesh, then check_empty_cells
  if (c.seeded) PFEM2_TRY(launch_relocate(c, c.ale_xphys));
  int flag = 0;
  PFEM2_CUDA(cudaMemcpyAsync(&flag, c.ale_flag, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  PFEM2_CUDA(cudaStreamSynchronize(c.stream));
  PFEM2_CUDA(cudaGetLastError());
  if (flag) {
    set_error("move_mesh: a cell turned inside out (non-positive Jacobian)");
    return PFEM2_MESH_ERROR;
  }
  return PFEM2_OK;
}

}  // namespace pfem2
