// particles.cu -- particle kernels of the PFEM2 step (sm_100a).
//
// Layout: particles are SoA and sorted by cell (cell_start offsets), with
// reference coordinates xi[d][cap] and carried velocity u[d][cap] in the
// arithmetic type R (float for the mixed path, double for the plain path).
//
// Kernels and the reference routines they replace:
//   k_seed          seed_particles / seed_particles_into_cell
//                   (TurekBenchmark/pfem2particle.cpp:701-721,774-790)
//   k_correct       correct_particles_velocities (:792-811)
//   k_advect_stay,  move_particles sub-steps (:813-848) + point location
//   k_advect_leave, (k_advect_one: the same in one kernel)
//                   sort_particles_into_subdomains_and_cells (:276-507),
//                   find_closest_vertex_of_cell (:142-166),
//                   compare_particle_association (:268-274)
//   k_rebin_*       the re-sort by cell plus check_cell_for_empty_parts
//                   (:723-772), with the projection partials fused in
//   k_project_*     distribute_particle_velocities_to_grid (:858-918)
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>

#include "common.cuh"
#include "ctx.h"

namespace pfem2 {

constexpr int kRebinWarps = 8;
constexpr int kMaxBuckets = 256;
// Resident blocks per SM that the re-sort kernels' registers are capped for.
// Both wait for dependent loads, so resident warps pay until the spilled
// registers' traffic (every store reaches the L2) outweighs them. Re-sort of
// the 1M-cell FP32 mesh with 6 / 5 blocks (gather / write) 1.04 ms; 6 / 6:
// 1.66, 4 / 4: 1.15, 8 / 5: 1.06; 201k-cell FP64 mesh with 6 / 4 0.240 ms,
// 4 / 4: 0.262, 3 / 4: 0.301; 131k-cell pipe, FP32 particles, 4 / 3 0.367 ms,
// 3 / 3: 0.435, 4 / 4: 0.53; 10k-cell pipe, FP64, 3 / 2 0.038 ms, 4 / 3: 0.053.
template <int DIM, typename R>
struct RebinMinBlocks {
  static constexpr int gather = sizeof(R) == 4 ? (DIM == 2 ? 6 : 4) : (DIM == 2 ? 6 : 3);
  static constexpr int write = sizeof(R) == 4 ? (DIM == 2 ? 5 : 3) : (DIM == 2 ? 4 : 2);
};

// ------------------------------------------------------------------ seed
template <int DIM, typename R>
__global__ void k_seed(int c0, int c1, int q0, int q1, int q2, int pbase, uint64_t seed, double jitter,
                       const double* __restrict__ X, const int* __restrict__ cv, const double* __restrict__ V0,
                       const double* __restrict__ V1, const double* __restrict__ V2, int* __restrict__ cell,
                       R* __restrict__ xi, R* __restrict__ u, size_t cap, int* __restrict__ cell_start) {
  constexpr int NV = Dims<DIM>::NV;
  const int Q = q0 * q1 * q2;
  const double h[3] = {1.0 / q0, 1.0 / q1, 1.0 / q2};
  const double* V[3] = {V0, V1, V2};
  for (int c = c0 + blockIdx.x * blockDim.x + threadIdx.x; c < c1; c += gridDim.x * blockDim.x) {
    const size_t pc = (size_t)pbase + (size_t)(c - c0) * Q;
    cell_start[c] = (int)pc;
    for (int t = 0; t < Q; ++t) {
      int idx[3] = {t / (q1 * q2), (t / q2) % q1, t % q2};
      uint64_t ord = (uint64_t)(c - c0) * Q + t;
      double x[3];
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        x[d] = (idx[d] + 1.0 / 2) * h[d];
        if (jitter != 0.0) x[d] += jitter * (2.0 * uniform01(seed, ord, d) - 1.0);
      }
      double N[NV];
      shape_values<DIM, double>(x, N);
      double uu[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        int g = __ldg(cv + (size_t)c * NV + v);
#pragma unroll
        for (int d = 0; d < DIM; ++d) uu[d] = uu[d] + N[v] * V[d][g];
      }
      size_t p = pc + t;
      cell[p] = c;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        xi[d * cap + p] = R(x[d]);
        u[d * cap + p] = R(uu[d]);
      }
    }
  }
}

template <int DIM, typename R>
static pfem2_status seed_impl(Ctx& c, uint64_t seed, double jitter) {
  int b = c.cur;
  size_t total = 0;
  for (auto& in : c.inst) total += (size_t)in.nc * in.q[0] * in.q[1] * (DIM == 3 ? in.q[2] : 1);
  if (total > (size_t)c.pcap) {
    set_error("seed: particle capacity exceeded");
    return PFEM2_PARTICLE_OVERFLOW;
  }
  size_t pbase = 0;
  for (auto& in : c.inst) {
    int q2 = DIM == 3 ? (int)in.q[2] : 1;
    int grid = grid_for(c, in.nc, 128, 16);
    k_seed<DIM, R><<<grid, 128, 0, c.stream>>>(in.c_off, in.c_off + in.nc, in.q[0], in.q[1], q2, (int)pbase, seed,
                                               jitter, c.X, c.cv, c.F[PFEM2_FIELD_VX], c.F[PFEM2_FIELD_VY],
                                               c.F[PFEM2_FIELD_VZ], c.pcell[b], (R*)c.pxi[b], (R*)c.pu[b],
                                               (size_t)c.pcap, c.cell_start[b]);
    c.launches++;
    pbase += (size_t)in.nc * in.q[0] * in.q[1] * q2;
  }
  int tot = (int)total;
  PFEM2_CUDA(cudaMemcpyAsync(c.cell_start[b] + c.nc, &tot, sizeof(int), cudaMemcpyHostToDevice, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(c.d_np + b, &tot, sizeof(int), cudaMemcpyHostToDevice, c.stream));
  PFEM2_CUDA(cudaStreamSynchronize(c.stream));
  PFEM2_CUDA(cudaGetLastError());
  return PFEM2_OK;
}

pfem2_status launch_seed(Ctx& c, int instance, const uint32_t q[3], uint64_t seed, double jitter) {
  (void)instance;
  if (c.dim == 2) return c.pmixed ? seed_impl<2, float>(c, seed, jitter) : seed_impl<2, double>(c, seed, jitter);
  return c.pmixed ? seed_impl<3, float>(c, seed, jitter) : seed_impl<3, double>(c, seed, jitter);
}

// -------------------------------------------------------- real mirrors
template <int DIM, typename R>
__global__ void k_sync_real(int nv, const double* __restrict__ V0, const double* __restrict__ V1,
                            const double* __restrict__ V2, const double* __restrict__ O0,
                            const double* __restrict__ O1, const double* __restrict__ O2, R* __restrict__ Vr,
                            R* __restrict__ dVr) {
  const double* V[3] = {V0, V1, V2};
  const double* O[3] = {O0, O1, O2};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      double v = V[d][i];
      Vr[(size_t)d * nv + i] = R(v);
      dVr[(size_t)d * nv + i] = R(v - O[d][i]);
    }
  }
}

template <int DIM, typename R>
static pfem2_status sync_real_impl(Ctx& c) {
  k_sync_real<DIM, R><<<grid_for(c, c.nv, 256), 256, 0, c.stream>>>(
      c.nv, c.F[PFEM2_FIELD_VX], c.F[PFEM2_FIELD_VY], c.F[PFEM2_FIELD_VZ], c.F[PFEM2_FIELD_OLD_VX],
      c.F[PFEM2_FIELD_OLD_VY], c.F[PFEM2_FIELD_OLD_VZ], (R*)c.Vr, (R*)c.dVr);
  c.launches++;
  return PFEM2_OK;
}

pfem2_status launch_sync_real_fields(Ctx& c) {
  if (c.dim == 2) return c.pmixed ? sync_real_impl<2, float>(c) : sync_real_impl<2, double>(c);
  return c.pmixed ? sync_real_impl<3, float>(c) : sync_real_impl<3, double>(c);
}

// --------------------------------------------------------------- correct
template <int DIM, typename R>
__global__ void __launch_bounds__(256) k_correct(const int* __restrict__ cell, const R* __restrict__ xi,
                                                 R* __restrict__ u, size_t cap, const int* __restrict__ d_np,
                                                 const int* __restrict__ cv, const R* __restrict__ dV, int nv) {
  constexpr int NV = Dims<DIM>::NV;
  const int n = min(*d_np, (int)cap);
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int c = cell[p];
    R x[DIM], up[DIM], N[NV];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      x[d] = xi[d * cap + p];
      up[d] = u[d * cap + p];
    }
    shape_values<DIM, R>(x, N);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      int g = __ldg(cv + (size_t)c * NV + v);
#pragma unroll
      for (int d = 0; d < DIM; ++d) up[d] = up[d] + N[v] * __ldg(dV + (size_t)d * nv + g);
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) u[d * cap + p] = up[d];
  }
}

template <int DIM, typename R>
static pfem2_status correct_impl(Ctx& c) {
  int b = c.cur;
  k_correct<DIM, R><<<grid_for(c, c.pcap, 256, 8), 256, 0, c.stream>>>(
      c.pcell[b], (const R*)c.pxi[b], (R*)c.pu[b], (size_t)c.pcap, c.d_np + b, c.cv, (const R*)c.dVr, c.nv);
  c.launches++;
  return PFEM2_OK;
}

pfem2_status launch_correct(Ctx& c) {
  if (c.dim == 2) return c.pmixed ? correct_impl<2, float>(c) : correct_impl<2, double>(c);
  return c.pmixed ? correct_impl<3, float>(c) : correct_impl<3, double>(c);
}

// ---------------------------------------------------------------- advect
// One thread per particle; all PARTICLES_MOVEMENT_STEPS sub-steps run in
// registers (the nodal field is fixed during move_particles). After each
// sub-step the particle is located like the reference does: current cell
// first, then the patch of the "closest" vertex in alignment order; a
// particle found nowhere is deleted (newcell = -1).
// resident 256-thread blocks per SM the one-kernel advection is compiled for:
// it is latency-bound, so the FP32 2D variant trades its few extra
// registers for four blocks (32 warps) per SM, and the FP64 3D variant
// (240 registers uncapped, one block) runs two at 128 registers in spite of
// its spills (2.72 -> 2.40 ms on the 442k-cell pipe; three: 4.0 ms); the
// FP64 2D variant measured slower with three than with two
template <int DIM, typename R>
struct AdvectMinBlocks {
  static constexpr int value = DIM == 2 ? (sizeof(R) == 4 ? 4 : 2) : 2;
};


// Resident blocks per SM of the two-kernel form (stay: 256 threads, leave: 128),
// measured as advection per step. Stay, without the point location's registers:
// 1M-cell FP32 mesh 1.04 ms with 6 (5: 1.07, 7: more spills, 1.39); 131k-cell
// pipe, FP64, 0.86 ms with 2 (3: 1.13, 1: 1.04). Leave: 16 channels, FP64, 0.57 ms
// with 6 (4: 0.67, 8: 0.68); 1M cells FP32 1.04 with 8 (7: 1.22, 10: 1.34);
// 10k-cell pipe, FP64, 0.128 with 3 (4: 0.134).
template <int DIM, typename R>
struct StayMinBlocks {
  static constexpr int value = sizeof(R) == 4 ? (DIM == 2 ? 6 : 3) : (DIM == 2 ? 4 : 2);
};
template <int DIM, typename R>
struct LeaveMinBlocks {
  static constexpr int value = sizeof(R) == 4 ? (DIM == 2 ? 8 : 4) : (DIM == 2 ? 6 : 3);
};

constexpr int kAdvLeft = -2;  // advect_steps<.., false>: the particle left its cell

// patches of at most this many cells are searched without the sort's
// local-memory arrays
constexpr int kSmallPatch = 8;

// The reference's search for a point xn (cell-local frame of cell c, whose
// record is G / L / x0) that left cell c (sort_particles_into_subdomains_and_
// cells, TurekBenchmark/pfem2particle.cpp:276-507): the vertex of c best
// aligned with the direction uf from the old position xo
// (find_closest_vertex_of_cell, :142-166), then that vertex's cells ordered
// by the alignment of their centre directions with vertex -> point
// (compare_particle_association, :268-274), the first that contains the
// point. On success c, G, L, x0 and the reference coordinates x are those of
// the new cell; false when no cell of the patch contains the point.
template <int DIM, typename R>
__device__ __forceinline__ bool locate_from(int& c, CellGeo<DIM, R>& G, LocalCell<DIM, R>& L, double* x0,
                                            const R* xo, const R* xn, const R* uf, R* x, const int* gvx,
                                            const CellGeo<DIM, R>* __restrict__ geo,
                                            const int* __restrict__ v2c_ptr, const int* __restrict__ v2c_cell,
                                            const R* __restrict__ v2c_dir) {
  constexpr int NV = Dims<DIM>::NV;
  R x2[DIM];
  {
    // closest vertex of the old cell seen along the velocity
    R un = R(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) un += uf[d] * uf[d];
    un = sqrt(un);
    R best = R(0);
    int bv = 0;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      R t[DIM], tn = R(0), dot = R(0);
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        t[d] = L.D[v][d] - xo[d];
        tn += t[d] * t[d];
      }
      tn = sqrt(tn);
#pragma unroll
      for (int d = 0; d < DIM; ++d) dot += (uf[d] / un) * (t[d] / tn);
      if (v == 0) best = dot;
      else if (dot > best) { best = dot; bv = v; }
    }
    const int gv = gvx[bv];
    R vp[DIM], vpn = R(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      vp[d] = xn[d] - L.D[bv][d];
      vpn += vp[d] * vp[d];
    }
    vpn = sqrt(vpn);
#pragma unroll
    for (int d = 0; d < DIM; ++d) vp[d] /= vpn;
    const int k0 = __ldg(v2c_ptr + gv);
    int nk = __ldg(v2c_ptr + gv + 1) - k0;
    if (nk > kMaxPatch) nk = kMaxPatch;
    bool found = false;
    // the point in patch cell i (i in v2c order): on success the new cell
    auto try_cell = [&](int i) {
      const int cc = __ldg(v2c_cell + k0 + i);
      const CellGeo<DIM, R> Gc = geo[cc];
      LocalCell<DIM, R> Lc;
      double xc[DIM];
      geo_to_local<DIM, R>(Gc, Lc, xc);
      R t[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) t[d] = xn[d] + R(x0[d] - xc[d]);
      if (geo_inverse<DIM, R>(Gc, Lc, t, x2) && inside_unit<DIM, R>(x2)) {
        found = true;
        c = cc;
        G = Gc;
        L = Lc;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          x0[d] = xc[d];
          x[d] = x2[d];
        }
      }
    };
    auto align = [&](int i) {
      R sdot = R(0);
#pragma unroll
      for (int d = 0; d < DIM; ++d) sdot += __ldg(v2c_dir + (size_t)(k0 + i) * DIM + d) * vp[d];
      return sdot;
    };
    if (nk <= kSmallPatch) {
      // small patches: the cells are tried in order by repeated selection of
      // the best aligned remaining one (the lowest index among equal
      // alignments), which is the order of the stable sort below without
      // its local-memory arrays; the alignments are recomputed per round
      // from cached loads, and usually the first cell tried holds the point
      unsigned left = (1u << nk) - 1u;
      while (left && !found) {
        int bi = -1;
        R bk = R(0);
        for (int i = 0; i < nk; ++i) {
          if (!((left >> i) & 1u)) continue;
          const R k = align(i);
          if (bi < 0 || k > bk) {
            bi = i;
            bk = k;
          }
        }
        left &= ~(1u << bi);
        try_cell(bi);
      }
      return found;
    }
    R key[kMaxPatch];
    int perm[kMaxPatch];
    for (int i = 0; i < nk; ++i) {
      const R sdot = align(i);
      key[i] = sdot;
      // stable insertion by descending alignment (std::sort is an
      // insertion sort, hence stable, for patches of <= 16 cells)
      int j = i - 1;
      while (j >= 0 && sdot > key[perm[j]]) {
        perm[j + 1] = perm[j];
        --j;
      }
      perm[j + 1] = i;
    }
    for (int i = 0; i < nk && !found; ++i) try_cell(perm[i]);
    return found;
  }
}

// Sub-steps s0 .. S-1 of the S forward-Euler sub-steps of one particle with
// the Q1-interpolated mesh velocity (move_particles,
// TurekBenchmark/pfem2particle.cpp:813-856), starting in cell c0 at
// reference coordinates x (updated). After a sub-step
// the point is first tried in the current cell; if it left, FULL runs the
// reference's search (sort_particles_into_subdomains_and_cells: the vertex
// of the old cell best aligned with the velocity, then that vertex's cells
// ordered by alignment with the directions to their centres, :276-507) and
// returns the new cell, or -1 when no cell of the patch contains the point
// (the particle is deleted); without FULL it returns kAdvLeft at the first
// sub-step that leaves the cell, with x still at the start of that
// sub-step and its index in s_left. Otherwise it returns the cell.
template <int DIM, typename R, bool FULL>
__device__ __forceinline__ int advect_steps(int c0, R* x, R dts, int s0, int& s_left, int S,
                                            const CellGeo<DIM, R>* __restrict__ geo,
                                            const int* __restrict__ cv, const R* __restrict__ Vr, int nv,
                                            const int* __restrict__ v2c_ptr, const int* __restrict__ v2c_cell,
                                            const R* __restrict__ v2c_dir) {
  constexpr int NV = Dims<DIM>::NV;
  int c = c0;
  // vertex ids and velocities of the current cell, reloaded only when the
  // particle changes cell
  int gvx[NV];
  R vv[NV][DIM], N[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) gvx[v] = __ldg(cv + (size_t)c * NV + v);
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int d = 0; d < DIM; ++d) vv[v][d] = __ldg(Vr + (size_t)d * nv + gvx[v]);
  CellGeo<DIM, R> G = geo[c];
  LocalCell<DIM, R> L;
  double x0[DIM];
  geo_to_local<DIM, R>(G, L, x0);
  for (int s = s0; s < S; ++s) {
    shape_values<DIM, R>(x, N);
    R uf[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) uf[d] = R(0);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) uf[d] = uf[d] + N[v] * vv[v][d];
    }
    R xo[DIM], xn[DIM], x2[DIM];
    local_map<DIM, R>(L, x, xo);
#pragma unroll
    for (int d = 0; d < DIM; ++d) xn[d] = xo[d] + uf[d] * dts;
    if (geo_inverse<DIM, R>(G, L, xn, x2) && inside_unit<DIM, R>(x2)) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) x[d] = x2[d];
      continue;
    }
    if (!FULL) {
      s_left = s;
      return kAdvLeft;
    }
    if (!locate_from<DIM, R>(c, G, L, x0, xo, xn, uf, x, gvx, geo, v2c_ptr, v2c_cell, v2c_dir)) return -1;
#pragma unroll
    for (int v = 0; v < NV; ++v) gvx[v] = __ldg(cv + (size_t)c * NV + v);
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int d = 0; d < DIM; ++d) vv[v][d] = __ldg(Vr + (size_t)d * nv + gvx[v]);
  }
  return c;
}

// deletion count and far movers of one advected particle (c: its new cell,
// -1 when deleted)
__device__ __forceinline__ void advect_record(int p, int c0, int c, const int* __restrict__ ring_ptr,
                                              const int* __restrict__ ring_cell,
                                              unsigned long long* __restrict__ far_keys, int far_cap,
                                              int* __restrict__ counters, const Movers mv) {
  if (c < 0) {
    atomicAdd(counters + CNT_DELETED, 1);
  } else if (c != c0) {
    // a particle that stays in the 1-ring of its old cell goes to the mover
    // list of its new cell; one that left it to the far list, and its place
    // in the mover list, drawn before the ring is searched, stays empty
    const int k = atomicAdd(mv.cnt + c, 1);
    bool near = false;
    for (int rr = __ldg(ring_ptr + c0); rr < __ldg(ring_ptr + c0 + 1); ++rr)
      if (__ldg(ring_cell + rr) == c) {
        near = true;
        break;
      }
    if (k < mv.cap) mv.list[(size_t)c * mv.cap + k] = near ? p : INT_MAX;
    if (!near) {
      int slot = atomicAdd(counters + CNT_FAR, 1);
      if (slot < far_cap) far_keys[slot] = ((unsigned long long)(unsigned)c << 32) | (unsigned)p;
      else atomicExch(counters + CNT_FAR_OVERFLOW, 1);
    }
  }
}

// Advection in one kernel (small 2D sets, see advect_split): correction, every
// sub-step with the full point location in line. Same arithmetic as the
// two-kernel form.
template <int DIM, typename R, bool FUSE>
__global__ void __launch_bounds__(256, AdvectMinBlocks<DIM, R>::value) k_advect_one(
    const int* __restrict__ cell, R* __restrict__ xi, R* __restrict__ u, int* __restrict__ newcell, size_t cap,
    const int* __restrict__ d_np, const CellGeo<DIM, R>* __restrict__ geo, const int* __restrict__ cv,
    const R* __restrict__ Vr, const R* __restrict__ dVr, int nv, int S, const DevInst* __restrict__ inst,
    const int* __restrict__ cell_inst, const int* __restrict__ v2c_ptr, const int* __restrict__ v2c_cell,
    const R* __restrict__ v2c_dir, const int* __restrict__ ring_ptr, const int* __restrict__ ring_cell,
    unsigned long long* __restrict__ far_keys, int far_cap, int* __restrict__ counters, const Movers mv) {
  constexpr int NV = Dims<DIM>::NV;
  const int n = min(*d_np, (int)cap);
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int c0 = cell[p];
    R x[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) x[d] = xi[d * cap + p];
    if (FUSE) {
      R N[NV], up[DIM];
      shape_values<DIM, R>(x, N);
#pragma unroll
      for (int d = 0; d < DIM; ++d) up[d] = u[d * cap + p];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int g = __ldg(cv + (size_t)c0 * NV + v);
#pragma unroll
        for (int d = 0; d < DIM; ++d) up[d] = up[d] + N[v] * __ldg(dVr + (size_t)d * nv + g);
      }
#pragma unroll
      for (int d = 0; d < DIM; ++d) u[d * cap + p] = up[d];
    }
    const R dts = R(inst[__ldg(cell_inst + c0)].dt_sub);
    int s_left = 0;
    int c = advect_steps<DIM, R, true>(c0, x, dts, 0, s_left, S, geo, cv, Vr, nv, v2c_ptr, v2c_cell, v2c_dir);
    if (c < 0) c = -1;
    advect_record(p, c0, c, ring_ptr, ring_cell, far_keys, far_cap, counters, mv);
    newcell[p] = c;
#pragma unroll
    for (int d = 0; d < DIM; ++d) xi[d * cap + p] = x[d];
  }
}

// Advection in two kernels. k_advect_stay: a block walks the 32-particle slices
// of a contiguous chunk; every particle is corrected (FUSE) and takes the lean
// sub-steps while it stays in its cell; one that leaves goes to the chunk's part
// of the queue, with its reference coordinates at the start of the sub-step it
// left in xi and that sub-step's index in newcell. k_advect_leave: a warp takes
// units of up to 32 leavers of one chunk and resumes them with the full point
// location, so that the divergent patch search runs on full warps.
//
// Both are bound by dependent loads, the FP64 3D form by the FP64 pipe. In one
// kernel (a queue per warp, resumed in place) the point location's registers
// held every warp to its occupancy: 131k-cell pipe, 3.5M FP64 particles, 1.28
// ms against 0.86 now; 16 channels, 8.7M, FP64, 0.70 against 0.57; 52k cells,
// 1.7M, FP64, 0.164 against 0.149; 13k cells, FP64, 0.074 against 0.058; 1M
// cells, 28M, FP32, 1.10 against 1.04. Units keep a chunk's leavers together:
// one queue over all chunks lost the cell data's L1 hits (1M cells 1.19 ms, 16
// channels 0.64), a block per chunk waited for the fastest region (16 channels
// 0.78). The arithmetic is that of k_advect_one (bitwise equal results).
constexpr int kAdvThreads = 256, kLeaveThreads = 128;

template <int DIM, typename R, bool FUSE>
__global__ void __launch_bounds__(kAdvThreads, StayMinBlocks<DIM, R>::value) k_advect_stay(
    const int* __restrict__ cell, R* __restrict__ xi, R* __restrict__ u, int* __restrict__ newcell, size_t cap,
    const int* __restrict__ d_np, const CellGeo<DIM, R>* __restrict__ geo, const int* __restrict__ cv,
    const R* __restrict__ Vr, const R* __restrict__ dVr, int nv, int S, const DevInst* __restrict__ inst,
    const int* __restrict__ cell_inst, int* __restrict__ queue, int2* __restrict__ units, int* __restrict__ n_units) {
  constexpr int NV = Dims<DIM>::NV;
  __shared__ int s_n, s_at;
  const int n = min(*d_np, (int)cap);
  const int chunk = (n + gridDim.x - 1) / gridDim.x;
  const int lo = (int)min((long long)n, (long long)blockIdx.x * chunk), hi = min(n, lo + chunk);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  for (int base = lo + warp * 32; base < hi; base += kAdvThreads) {
    const int p = base + lane;
    bool leave = false;
    if (p < hi) {
      const int c0 = cell[p];
      R x[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) x[d] = xi[d * cap + p];
      if (FUSE) {
        R N[NV], up[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) up[d] = u[d * cap + p];
        shape_values<DIM, R>(x, N);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const int g = __ldg(cv + (size_t)c0 * NV + v);
#pragma unroll
          for (int d = 0; d < DIM; ++d) up[d] = up[d] + N[v] * __ldg(dVr + (size_t)d * nv + g);
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d) u[d * cap + p] = up[d];
      }
      const R dts = R(inst[__ldg(cell_inst + c0)].dt_sub);
      int s_left = 0;
      const int c = advect_steps<DIM, R, false>(c0, x, dts, 0, s_left, S, geo, cv, Vr, nv, nullptr, nullptr, nullptr);
      leave = c == kAdvLeft;
      newcell[p] = leave ? s_left : c;
#pragma unroll
      for (int d = 0; d < DIM; ++d) xi[d * cap + p] = x[d];
    }
    const unsigned m = __ballot_sync(PFEM2_FULL_MASK, leave);
    if (m) {
      int k = 0;
      if (lane == 0) k = atomicAdd(&s_n, __popc(m));
      k = __shfl_sync(PFEM2_FULL_MASK, k, 0);
      if (leave) queue[lo + k + __popc(m & lanemask_lt())] = p;
    }
  }
  __syncthreads();
  const int left = s_n, nu = (left + 31) / 32;
  if (threadIdx.x == 0) s_at = atomicAdd(n_units, nu);
  __syncthreads();
  for (int j = threadIdx.x; j < nu; j += kAdvThreads) units[s_at + j] = make_int2(lo + 32 * j, min(32, left - 32 * j));
}

template <int DIM, typename R>
__global__ void __launch_bounds__(kLeaveThreads, LeaveMinBlocks<DIM, R>::value) k_advect_leave(
    const int* __restrict__ cell, R* __restrict__ xi, int* __restrict__ newcell, size_t cap,
    const CellGeo<DIM, R>* __restrict__ geo, const int* __restrict__ cv,
    const R* __restrict__ Vr, int nv, int S, const DevInst* __restrict__ inst, const int* __restrict__ cell_inst,
    const int* __restrict__ v2c_ptr, const int* __restrict__ v2c_cell, const R* __restrict__ v2c_dir,
    const int* __restrict__ ring_ptr, const int* __restrict__ ring_cell, unsigned long long* __restrict__ far_keys,
    int far_cap, int* __restrict__ counters, const Movers mv, const int* __restrict__ queue,
    const int2* __restrict__ units, const int* __restrict__ n_units) {
  const int nu = *n_units, lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * kLeaveThreads + threadIdx.x) >> 5; i < nu; i += gridDim.x * (kLeaveThreads / 32)) {
    const int2 unit = units[i];
    if (lane >= unit.y) continue;
    const int p = queue[unit.x + lane], c0 = cell[p];
    R x[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) x[d] = xi[d * cap + p];
    const R dts = R(inst[__ldg(cell_inst + c0)].dt_sub);
    int s_left = 0;
    int c = advect_steps<DIM, R, true>(c0, x, dts, newcell[p], s_left, S, geo, cv, Vr, nv, v2c_ptr, v2c_cell, v2c_dir);
    if (c < 0) c = -1;
    advect_record(p, c0, c, ring_ptr, ring_cell, far_keys, far_cap, counters, mv);
    newcell[p] = c;
#pragma unroll
    for (int d = 0; d < DIM; ++d) xi[d * cap + p] = x[d];
  }
}

__global__ void k_far_sort(unsigned long long* keys, const int* __restrict__ counters, int cap);

// ------------------------------------------------------------ moving mesh
// physical position of every particle (FP64) from its cell record, before
// the mesh moves
template <int DIM, typename R>
__global__ void k_particle_positions(const int* __restrict__ cell, const R* __restrict__ xi, size_t cap,
                                     const int* __restrict__ d_np, const CellGeo<DIM, R>* __restrict__ geo,
                                     double* __restrict__ out) {
  const int n = min(*d_np, (int)cap);
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const CellGeo<DIM, R> G = geo[cell[p]];
    LocalCell<DIM, R> L;
    double x0[DIM];
    geo_to_local<DIM, R>(G, L, x0);
    R x[DIM], xl[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) x[d] = xi[d * cap + p];
    local_map<DIM, R>(L, x, xl);
#pragma unroll
    for (int d = 0; d < DIM; ++d) out[d * cap + p] = x0[d] + (double)xl[d];
  }
}

// sort_particles_into_subdomains_and_cells after transform_grid: every
// particle keeps its physical position xphys and is located in the moved
// mesh: its cell first, else the reference's vertex-patch search from its
// cell along the direction it moved relative to the mesh (from where its
// old reference coordinates now map to); the new cell (-1: deleted) goes
// to newcell with the moves recorded for the re-sort like the advection's
template <int DIM, typename R>
__global__ void __launch_bounds__(256) k_relocate(
    const int* __restrict__ cell, R* __restrict__ xi, int* __restrict__ newcell, size_t cap,
    const int* __restrict__ d_np, const CellGeo<DIM, R>* __restrict__ geo, const int* __restrict__ cv,
    const int* __restrict__ v2c_ptr, const int* __restrict__ v2c_cell, const R* __restrict__ v2c_dir,
    const double* __restrict__ xphys, const int* __restrict__ ring_ptr, const int* __restrict__ ring_cell,
    unsigned long long* __restrict__ far_keys, int far_cap, int* __restrict__ counters,
    const Movers mv) {
  constexpr int NV = Dims<DIM>::NV;
  const int n = min(*d_np, (int)cap);
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int c0 = cell[p];
    int c = c0;
    CellGeo<DIM, R> G = geo[c0];
    LocalCell<DIM, R> L;
    double x0[DIM];
    geo_to_local<DIM, R>(G, L, x0);
    R x[DIM], xo[DIM], xn[DIM], uf[DIM], x2[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) x[d] = xi[d * cap + p];
    local_map<DIM, R>(L, x, xo);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      xn[d] = R(xphys[d * cap + p] - x0[d]);
      uf[d] = xn[d] - xo[d];
    }
    if (geo_inverse<DIM, R>(G, L, xn, x2) && inside_unit<DIM, R>(x2)) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) x[d] = x2[d];
    } else {
      int gvx[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) gvx[v] = __ldg(cv + (size_t)c0 * NV + v);
      if (!locate_from<DIM, R>(c, G, L, x0, xo, xn, uf, x, gvx, geo, v2c_ptr, v2c_cell, v2c_dir)) c = -1;
    }
    advect_record(p, c0, c, ring_ptr, ring_cell, far_keys, far_cap, counters, mv);
    newcell[p] = c;
    if (c >= 0)
#pragma unroll
      for (int d = 0; d < DIM; ++d) xi[d * cap + p] = x[d];
  }
}

// per-cell records of the particle kernels rebuilt from the vertices on the
// device (the same arithmetic as at setup); *flag = 1 if a cell has a
// non-positive Jacobian at its centre
template <int DIM, typename R>
__global__ void k_cell_geo(int nc, const double* __restrict__ X, const int* __restrict__ cv,
                           CellGeo<DIM, R>* __restrict__ geo, int* __restrict__ flag) {
  constexpr int NV = Dims<DIM>::NV;
  for (int ce = blockIdx.x * blockDim.x + threadIdx.x; ce < nc; ce += gridDim.x * blockDim.x) {
    CellGeo<DIM, R> g;
    double D[NV][DIM];
    const int g0 = cv[(size_t)ce * NV];
#pragma unroll
    for (int a = 0; a < DIM; ++a) g.x0[a] = X[(size_t)g0 * DIM + a];
    double scale = 0.0;
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        D[v][a] = X[(size_t)cv[(size_t)ce * NV + v] * DIM + a] - g.x0[a];
        scale = fmax(scale, fabs(D[v][a]));
        if (v > 0) g.D[v - 1][a] = (R)D[v][a];
      }
    double J[DIM * DIM];
#pragma unroll
    for (int k = 0; k < DIM * DIM; ++k) J[k] = 0.0;
    const double w0 = DIM == 2 ? 0.5 : 0.25;
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int b = 0; b < DIM; ++b) {
        const double w = ((v >> b) & 1) ? w0 : -w0;
#pragma unroll
        for (int a = 0; a < DIM; ++a) J[a * DIM + b] += D[v][a] * w;
      }
    double Ji[DIM * DIM];
    const double det = det_inv<DIM, double>(J, Ji);
    if (!(det > 0.0)) atomicExch(flag, 1);
#pragma unroll
    for (int k = 0; k < DIM * DIM; ++k) g.Ji[k] = (R)Ji[k];
    bool aff = true;
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        double s = 0.0;
#pragma unroll
        for (int b = 0; b < DIM; ++b)
          if ((v >> b) & 1) s += D[1 << b][a];
        if (fabs(D[v][a] - s) > 1e-13 * scale) aff = false;
      }
    g.affine = aff ? 1 : 0;
    geo[ce] = g;
  }
}

template <int DIM, typename R>
static pfem2_status positions_impl(Ctx& c, double* out) {
  const int b = c.cur;
  k_particle_positions<DIM, R><<<grid_for(c, c.pcap, 256, 8), 256, 0, c.stream>>>(
      c.pcell[b], (const R*)c.pxi[b], (size_t)c.pcap, c.d_np + b, (const CellGeo<DIM, R>*)c.cell_geo, out);
  c.launches++;
  return PFEM2_OK;
}

pfem2_status launch_particle_positions(Ctx& c, double* out) {
  if (c.dim == 2) return c.pmixed ? positions_impl<2, float>(c, out) : positions_impl<2, double>(c, out);
  return c.pmixed ? positions_impl<3, float>(c, out) : positions_impl<3, double>(c, out);
}

template <int DIM, typename R>
static pfem2_status relocate_impl(Ctx& c, const double* xphys) {
  const int b = c.cur;
  PFEM2_CUDA(cudaMemsetAsync(c.d_counters, 0, sizeof(int) * CNT_N_STATS, c.stream));
  PFEM2_CUDA(cudaMemsetAsync(c.movers.cnt, 0, sizeof(int) * c.nc, c.stream));
  k_relocate<DIM, R><<<grid_for(c, c.pcap, 256, 8), 256, 0, c.stream>>>(
      c.pcell[b], (R*)c.pxi[b], c.newcell, (size_t)c.pcap, c.d_np + b, (const CellGeo<DIM, R>*)c.cell_geo, c.cv,
      c.v2c_ptr, c.v2c_cell, (const R*)c.v2c_dir_r, xphys, c.ring_ptr, c.ring_cell, c.far_keys, c.far_cap,
      c.d_counters, c.movers);
  k_far_sort<<<1, 1024, sizeof(unsigned long long) * c.far_cap, c.stream>>>(c.far_keys, c.d_counters, c.far_cap);
  c.launches += 2;
  return PFEM2_OK;
}

pfem2_status launch_relocate(Ctx& c, const double* xphys) {
  const pfem2_status s = c.dim == 2 ? (c.pmixed ? relocate_impl<2, float>(c, xphys) : relocate_impl<2, double>(c, xphys))
                                    : (c.pmixed ? relocate_impl<3, float>(c, xphys) : relocate_impl<3, double>(c, xphys));
  if (s != PFEM2_OK) return s;
  // the re-sort into the moved cells with check_empty_cells
  return launch_rebin(c, true, false, true);
}

pfem2_status launch_cell_geo(Ctx& c, int* flag) {
  const int grid = grid_for(c, c.nc, 128, 8);
  if (c.dim == 2) {
    if (c.pmixed) k_cell_geo<2, float><<<grid, 128, 0, c.stream>>>(c.nc, c.X, c.cv, (CellGeo<2, float>*)c.cell_geo, flag);
    else k_cell_geo<2, double><<<grid, 128, 0, c.stream>>>(c.nc, c.X, c.cv, (CellGeo<2, double>*)c.cell_geo, flag);
  } else {
    if (c.pmixed) k_cell_geo<3, float><<<grid, 128, 0, c.stream>>>(c.nc, c.X, c.cv, (CellGeo<3, float>*)c.cell_geo, flag);
    else k_cell_geo<3, double><<<grid, 128, 0, c.stream>>>(c.nc, c.X, c.cv, (CellGeo<3, double>*)c.cell_geo, flag);
  }
  c.launches++;
  PFEM2_CUDA(cudaGetLastError());
  return PFEM2_OK;
}

// single-CTA bitonic sort of the (cell, particle) keys of the far movers
__global__ void k_far_sort(unsigned long long* keys, const int* __restrict__ counters, int cap) {
  extern __shared__ unsigned long long sk[];
  int n = counters[CNT_FAR];
  if (n > cap) n = cap;
  if (n <= 1) return;
  int m = 1;
  while (m < n) m <<= 1;
  for (int i = threadIdx.x; i < m; i += blockDim.x) sk[i] = i < n ? keys[i] : ~0ull;
  __syncthreads();
  for (int k = 2; k <= m; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < m; i += blockDim.x) {
        int l = i ^ j;
        if (l > i) {
          bool up = (i & k) == 0;
          unsigned long long a = sk[i], b = sk[l];
          if ((a > b) == up) { sk[i] = b; sk[l] = a; }
        }
      }
      __syncthreads();
    }
  for (int i = threadIdx.x; i < n; i += blockDim.x) keys[i] = sk[i];
}

// the far-mover sort's shared memory beyond the 48 KB default
pfem2_status far_sort_setup(Ctx& c) {
  PFEM2_CUDA(cudaFuncSetAttribute((const void*)k_far_sort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(unsigned long long) * c.far_cap)));
  return PFEM2_OK;
}

// One kernel or two. In 2D the second kernel's launch and its own chain of
// point locations pay from about 130k particles on. Move (advection and
// re-sort), FP64, one / two kernels, at a third and at four fifths of a cell
// per step: 28k particles 0.038 / 0.042 and 0.050 / 0.063 ms, 83k 0.050 / 0.049
// and 0.050 / 0.058, 171k 0.065 / 0.060 and 0.065 / 0.073, 398k 0.099 / 0.089
// and 0.156 / 0.168, 1.0M 0.206 / 0.157 and 0.215 / 0.229. In 3D the one kernel's
// registers leave it half the warps: 0.7k particles, FP64, 0.129
// / 0.107 ms, 46k 0.190 / 0.141, 0.6M 0.905 / 0.538.
constexpr size_t kSplitMin2D = 131072;

bool advect_split(const Ctx& c) {
  if (c.tune.advect_split) return c.tune.advect_split == 2;
  if (c.adv_split_min >= 0) return (long long)c.pcap >= c.adv_split_min;
  return c.dim == 3 || c.n_seeded >= kSplitMin2D;
}

template <int DIM, typename R>
static pfem2_status advect_impl(Ctx& c, bool fuse) {
  int b = c.cur;
  int S = c.cfg.movement_steps;
  if (!advect_split(c)) {
    const int grid = grid_for(c, c.pcap, 256, c.tune.advect_blocks_per_sm);
    if (fuse)
      k_advect_one<DIM, R, true><<<grid, 256, 0, c.stream>>>(
          c.pcell[b], (R*)c.pxi[b], (R*)c.pu[b], c.newcell, (size_t)c.pcap, c.d_np + b,
          (const CellGeo<DIM, R>*)c.cell_geo, c.cv, (const R*)c.Vr, (const R*)c.dVr, c.nv, S, c.d_inst, c.cell_inst,
          c.v2c_ptr, c.v2c_cell, (const R*)c.v2c_dir_r, c.ring_ptr, c.ring_cell, c.far_keys, c.far_cap, c.d_counters,
          c.movers);
    else
      k_advect_one<DIM, R, false><<<grid, 256, 0, c.stream>>>(
          c.pcell[b], (R*)c.pxi[b], (R*)c.pu[b], c.newcell, (size_t)c.pcap, c.d_np + b,
          (const CellGeo<DIM, R>*)c.cell_geo, c.cv, (const R*)c.Vr, (const R*)c.dVr, c.nv, S, c.d_inst, c.cell_inst,
          c.v2c_ptr, c.v2c_cell, (const R*)c.v2c_dir_r, c.ring_ptr, c.ring_cell, c.far_keys, c.far_cap, c.d_counters,
          c.movers);
    c.launches++;
  } else {
    // every resident block walks one contiguous chunk
    const int grid = grid_for(c, c.pcap, kAdvThreads, c.tune.advect_blocks_per_sm);
    int* const queue = c.rebin_list + (size_t)c.nc * kListStride;  // the re-sort's overflow part, free until then
    int* const n_units = c.movers.cnt + c.nc;
    int2* const units = (int2*)c.pu[1 - b];  // filled by the re-sort later
    const auto stay = fuse ? k_advect_stay<DIM, R, true> : k_advect_stay<DIM, R, false>;
    stay<<<grid, kAdvThreads, 0, c.stream>>>(
        c.pcell[b], (R*)c.pxi[b], (R*)c.pu[b], c.newcell, (size_t)c.pcap, c.d_np + b,
        (const CellGeo<DIM, R>*)c.cell_geo, c.cv, (const R*)c.Vr, (const R*)c.dVr, c.nv, S, c.d_inst, c.cell_inst,
        queue, units, n_units);
    k_advect_leave<DIM, R><<<grid, kLeaveThreads, 0, c.stream>>>(
        c.pcell[b], (R*)c.pxi[b], c.newcell, (size_t)c.pcap, (const CellGeo<DIM, R>*)c.cell_geo, c.cv, (const R*)c.Vr, c.nv, S, c.d_inst, c.cell_inst, c.v2c_ptr, c.v2c_cell, (const R*)c.v2c_dir_r, c.ring_ptr,
        c.ring_cell, c.far_keys, c.far_cap, c.d_counters, c.movers, queue, units, n_units);
    c.launches++;
    c.launches++;
  }
  k_far_sort<<<1, 1024, sizeof(unsigned long long) * c.far_cap, c.stream>>>(c.far_keys, c.d_counters, c.far_cap);
  c.launches++;
  return PFEM2_OK;
}

pfem2_status launch_advect(Ctx& c, bool fuse) {
  PFEM2_CUDA(cudaMemsetAsync(c.d_counters, 0, sizeof(int) * CNT_N_STATS, c.stream));
  PFEM2_CUDA(cudaMemsetAsync(c.movers.cnt, 0, sizeof(int) * (c.nc + 1), c.stream));
  if (c.dim == 2) return c.pmixed ? advect_impl<2, float>(c, fuse) : advect_impl<2, double>(c, fuse);
  return c.pmixed ? advect_impl<3, float>(c, fuse) : advect_impl<3, double>(c, fuse);
}

// ----------------------------------------------------------------- rebin
// One warp per target cell. The incoming particles of cell c are its stayers,
// the movers that advection listed for it and particles from beyond its 1-ring
// in the sorted far list, in ascending old index, so the result is a stable
// sort by cell of the old storage order.
// With CHECK the per-sub-cell counts are walked in that order: a particle
// whose bucket already holds MAX_PARTICLES_PER_CELL_PART is removed, and
// every empty sub-cell receives one particle at its centre, appended in
// (i,j,k) order with the interpolated nodal velocity.
template <int DIM, typename R>
struct ProjAcc {
  R a[Dims<DIM>::NV][DIM + 1];
};

template <int DIM, typename R>
__device__ __forceinline__ void proj_add(ProjAcc<DIM, R>& acc, const R* x, const R* uu) {
  R N[Dims<DIM>::NV];
  shape_values<DIM, R>(x, N);
#pragma unroll
  for (int v = 0; v < Dims<DIM>::NV; ++v) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) acc.a[v][d] += N[v] * uu[d];
    acc.a[v][DIM] += N[v];
  }
}

template <int DIM, typename R>
__device__ __forceinline__ void proj_store(ProjAcc<DIM, R>& acc, R* __restrict__ partial, int c, int lane) {
  constexpr int K = Dims<DIM>::NV * (DIM + 1);
  constexpr int N = K <= 16 ? 16 : 32;
  static_assert(K <= N, "projection partials exceed a warp");
  R v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = i < K ? acc.a[i / (DIM + 1)][i % (DIM + 1)] : R(0);
  const R tot = warp_sum_many<N, R>(v, lane);
  const int idx = warp_sum_many_index<N>(lane);
  // every value is held by 32 / N lanes; the first of them stores it
  if ((lane & (32 / N - 1)) == 0 && idx < K) partial[(size_t)c * K + idx] = tot;
}

// sub-cell index of check_cell_for_empty_parts: unsigned(xi / h) with
// h = 1.0 / q, which is q for xi == 1 (a bucket of its own, as in the
// reference); clamped to [0, q]. xi * q has the same integer part unless it
// lies within rounding of an integer, and only there the quotient is formed.
// For FP32 coordinates xi * q is exact in FP64, so that happens only when
// it is an integer; for FP64 coordinates a relative 1e-12 decides.
template <typename R>
__device__ __forceinline__ int sub_bucket_fp64(R xr, const double& h, int q) {
  const double xi = (double)xr;
  double t = xi * (double)q;
  if (sizeof(R) == 4) {
    if (t == rint(t)) t = xi / h;
  } else if (fabs(t - rint(t)) <= 1e-12 * fmax(1.0, fabs(t))) {
    t = xi / h;
  }
  if (!(t >= 0.0)) t = 0.0;
  if (t > (double)q) t = (double)q;
  return (int)(unsigned)t;
}

template <typename R>
__device__ __forceinline__ int sub_bucket(R xr, const double& h, int q) {
  return sub_bucket_fp64<R>(xr, h, q);
}

// FP32 coordinates: for 0 < xi < 1, xi = m 2^-s with the 24-bit significand
// m and s = 150 - (biased exponent) >= 24, so xi q = (m q) 2^-s exactly in
// 64-bit integers (q < 2^16): its integer part is the bucket unless xi q
// is itself an integer, where the quotient xi / h decides (the FP64 form,
// as for 0, 1 and anything outside (0, 1)). Same results as the FP64 form,
// with integer instructions only.
template <>
__device__ __forceinline__ int sub_bucket<float>(float xr, const double& h, int q) {
  const unsigned b = __float_as_uint(xr);
  if (b - 1u < 0x3f7fffffu) {  // 0 < xi < 1 (positive, below the bits of 1.0f)
    const int e = (int)(b >> 23);
    if (e == 0) return 0;  // subnormal: 0 < xi q < 1
    const int sh = 150 - e;
    if (sh < 64) {
      const unsigned long long prod = (unsigned long long)((b & 0x7fffffu) | 0x800000u) * (unsigned)q;
      if (prod & ((1ull << sh) - 1ull)) return (int)(prod >> sh);
    } else {
      return 0;  // xi < 2^-40: 0 < xi q < 1
    }
  }
  return sub_bucket_fp64<float>(xr, h, q);
}

// t / q for t, q < 2^16 with qm = ceil(2^32 / q)
__device__ __forceinline__ int div_small(int t, unsigned long long qm) {
  return (int)(((unsigned long long)(unsigned)t * qm) >> 32);
}

// (i, j, k) of sub-cell t in (i, j, k) order with extents (q0, q1, q2)
__device__ __forceinline__ void sub_cell_ijk(int t, int q1, int q2, const unsigned long long* qm, int id[3]) {
  const int u = div_small(t, qm[2]);  // t / q2
  id[2] = t - u * q2;
  id[0] = div_small(u, qm[1]);        // t / (q1 q2)
  id[1] = u - id[0] * q1;
}

__device__ __forceinline__ int far_lower_bound(const unsigned long long* keys, int n, unsigned long long k) {
  int lo = 0, hi = n;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (keys[mid] < k) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// The re-sort runs as three kernels. k_rebin_gather: a warp per target cell
// gathers and checks its incoming particles and stores their list and count.
// k_rebin_scan: exclusive sums of the counts. k_rebin_write: a warp per cell
// copies its particles to their new place with the projection partials. No
// warp waits for another, except in the scan (0.013 ms for 1M cells). As one
// kernel, where a block of eight cells looked back over the blocks before it
// for its offset, the ticket, the look-back and the block barriers cost more
// than the lists' way through memory. All are bound by dependent loads and by
// issue (gather 560, write 340 warp instructions a cell of 28 FP32 particles,
// 50% and 42% of the issue slots), not by bytes. 1M cells, 28M particles, FP32:
// 1.73 -> 1.04 ms (1.51 with the mover lists alone); 201k cells, 3M particles,
// FP64: 0.365 -> 0.240 ms; 52k cells, 1.7M, FP32: 0.147 -> 0.117 ms; 131k-cell
// pipe, 3.5M, FP32: 0.575 -> 0.370 ms.

// Incoming particles of cell c in ascending old index, written to list by the
// calling warp: the stayers are a run of the cell's old segment, the movers
// come unordered from the cell's mover list and are ranked by comparing each
// with all (scratch: kMaxBuckets ints, 16-byte aligned); movers from cells
// before c precede the stayers, the others follow. Returns their number (the
// entries beyond list_cap are dropped). A cell with more movers than its list
// holds scans the old segments of its whole 1-ring.
__device__ __forceinline__ int gather_incoming(int c, const int* __restrict__ old_start,
                                               const int* __restrict__ newcell, int cap,
                                               const int* __restrict__ ring_ptr, const int* __restrict__ ring_cell,
                                               const Movers& mv, int* list, int* scratch, int list_cap) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  const int nm = mv.cnt[c], sb = min(old_start[c], cap), se = min(old_start[c + 1], cap);
  int m0 = lane < nm ? mv.list[(size_t)c * mv.cap + lane] : INT_MAX;
  int v = sb + lane < se ? newcell[sb + lane] : -1;
  int n = 0;
  const auto append = [&](int p, bool in) {
    const unsigned m = __ballot_sync(PFEM2_FULL_MASK, in);
    const int pos = n + __popc(m & lt);
    if (in && pos < list_cap) list[pos] = p;
    n += __popc(m);
  };
  if (nm > mv.cap) {
    for (int r = __ldg(ring_ptr + c); r < __ldg(ring_ptr + c + 1); ++r) {
      const int s = __ldg(ring_cell + r);
      const int e = min(old_start[s + 1], cap);
      for (int base = min(old_start[s], cap); base < e; base += 32)
        append(base + lane, base + lane < e && newcell[base + lane] == c);
    }
    return n;
  }
  int n_mv = __popc(__ballot_sync(PFEM2_FULL_MASK, m0 != INT_MAX));
  if (nm > 0) scratch[lane] = m0;
  n = __popc(__ballot_sync(PFEM2_FULL_MASK, m0 < sb));
  for (int i = 32; i < nm; i += 32) {
    const int m = i + lane < nm ? mv.list[(size_t)c * mv.cap + i + lane] : INT_MAX;
    scratch[i + lane] = m;
    n += __popc(__ballot_sync(PFEM2_FULL_MASK, m < sb));
    n_mv += __popc(__ballot_sync(PFEM2_FULL_MASK, m != INT_MAX));
  }
  const int n_lo = n;
  append(sb + lane, v == c);
  for (int base = sb + 32; base < se; base += 32) {
    v = base + lane < se ? newcell[base + lane] : -1;
    append(base + lane, v == c);
  }
  __syncwarp();
  const int n_stay = n - n_lo;
  for (int i = lane; i < nm; i += 32) {
    const int m = i < 32 ? m0 : scratch[i];
    int rank = 0;
    for (int k = 0; k < nm; k += 4) {
      const int4 q = *reinterpret_cast<const int4*>(scratch + k);
      rank += (q.x < m) + (q.y < m) + (q.z < m) + (q.w < m);
    }
    const int pos = rank < n_lo ? rank : rank + n_stay;
    if (m != INT_MAX && pos < list_cap) list[pos] = m;
  }
  __syncwarp();
  return n_mv + n_stay;
}

template <int DIM, typename R, bool CHECK>
__global__ void __launch_bounds__(kRebinWarps * 32, RebinMinBlocks<DIM, R>::gather) k_rebin_gather(
    const int* __restrict__ old_start, const int* __restrict__ newcell, const R* __restrict__ oxi, size_t cap, int nc,
    const int* __restrict__ ring_ptr, const int* __restrict__ ring_cell, const Movers mv, const unsigned long long* __restrict__ far_keys, int far_cap,
    const DevInst* __restrict__ inst, const int* __restrict__ cell_inst, int list_cap, int* __restrict__ counters,
    int* __restrict__ cnt, int* __restrict__ glist, int* __restrict__ glist_pos, int* __restrict__ novf) {
  extern __shared__ int smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* bcnt = smem + warp * kMaxBuckets;
  int* list = smem + kRebinWarps * kMaxBuckets + warp * list_cap;
  const unsigned lt = lanemask_lt();
  int nfar = counters[CNT_FAR];
  if (nfar > far_cap) nfar = far_cap;
  for (int c = blockIdx.x * kRebinWarps + warp; c < nc; c += gridDim.x * kRebinWarps) {
    int n_in = gather_incoming(c, old_start, newcell, (int)cap, ring_ptr, ring_cell, mv, list, bcnt, list_cap);
    if (nfar > 0) {
      const int lo = far_lower_bound(far_keys, nfar, (unsigned long long)(unsigned)c << 32);
      const int hi = far_lower_bound(far_keys, nfar, (unsigned long long)(unsigned)(c + 1) << 32);
      __syncwarp();
      if (hi > lo && lane == 0) {
        int m = n_in < list_cap ? n_in : list_cap;
        for (int k = lo; k < hi; ++k) {
          const int p = (int)(far_keys[k] & 0xffffffffu);
          if (p < 0 || p >= (int)cap) continue;
          int j = m - 1;
          while (j >= 0 && list[j] > p) {
            if (j + 1 < list_cap) list[j + 1] = list[j];
            --j;
          }
          if (j + 1 < list_cap) list[j + 1] = p;
          if (m < list_cap) ++m;
        }
      }
      n_in += hi - lo;
      __syncwarp();
    }
    if (n_in > list_cap) {
      if (lane == 0) atomicExch(counters + CNT_LIST_OVERFLOW, 1);
      n_in = list_cap;
    }
    int n_keep = n_in, n_new = 0;
    if (CHECK) {
      const DevInst& I = inst[__ldg(cell_inst + c)];
      const int q0 = I.q[0], q1 = I.q[1], q2 = DIM == 3 ? I.q[2] : 1;
      const int nb1 = q1 + 1, nb2 = q2 + 1;
      // one chunk of 32 particles needs no counts in shared memory, and up to
      // 32 sub-cells fit a mask of the occupied ones
      const int Q = q0 * q1 * q2;
      const bool masked = Q <= 32, counts = n_in > 32 || !masked;
      unsigned occupied = 0;
      if (counts) {
        const int nb = (q0 + 1) * nb1 * nb2;
        for (int k = lane; k < nb; k += 32) bcnt[k] = 0;
        __syncwarp();
      }
      n_keep = 0;
      for (int base = 0; base < n_in; base += 32) {
        const int i = base + lane;
        const bool active = i < n_in;
        const int p = active ? list[i] : -1;
        int bi = -1;
        unsigned bit = 0;
        if (active) {
          const int b0 = sub_bucket<R>(oxi[p], I.h[0], q0);
          const int b1 = sub_bucket<R>(oxi[cap + p], I.h[1], q1);
          const int b2 = DIM == 3 ? sub_bucket<R>(oxi[2 * cap + p], I.h[2], q2) : 0;
          bi = (b0 * nb1 + b1) * nb2 + b2;
          if (masked && b0 < q0 && b1 < q1 && b2 < q2) bit = 1u << ((b0 * q1 + b1) * q2 + b2);
        }
        occupied |= __reduce_or_sync(PFEM2_FULL_MASK, bit);
        const unsigned peers = __match_any_sync(PFEM2_FULL_MASK, bi);
        int prev = 0;
        if (counts) {
          if (active) prev = bcnt[bi];
          __syncwarp();
          if (active && (peers & lt) == 0) bcnt[bi] = prev + __popc(peers);
        }
        const bool keep = active && prev + __popc(peers & lt) + 1 <= I.max_per_part;
        const unsigned km = __ballot_sync(PFEM2_FULL_MASK, keep);
        const int kpos = n_keep + __popc(km & lt);
        __syncwarp();
        if (keep && kpos != i) list[kpos] = p;  // kpos <= i: no particle is overwritten before it is read
        n_keep += __popc(km);
        __syncwarp();
      }
      // empty sub-cells -> new particles, (i,j,k) order
      for (int base = 0; base < Q; base += 32) {
        const int t = base + lane;
        bool e = false;
        if (masked) {
          e = t < Q && !((occupied >> lane) & 1u);
        } else if (t < Q) {
          int ijk[3];
          sub_cell_ijk(t, q1, q2, I.qm, ijk);
          e = bcnt[(ijk[0] * nb1 + ijk[1]) * nb2 + ijk[2]] == 0;
        }
        const unsigned em = __ballot_sync(PFEM2_FULL_MASK, e);
        const int pos = n_keep + n_new + __popc(em & lt);
        if (e && pos < list_cap) list[pos] = -1 - t;
        n_new += __popc(em);
      }
      if (n_keep + n_new > list_cap) {
        if (lane == 0) atomicExch(counters + CNT_LIST_OVERFLOW, 1);
        n_new = list_cap - n_keep;
      }
      if (lane == 0) {
        if (n_in - n_keep) atomicAdd(counters + CNT_REMOVED, n_in - n_keep);
        if (n_new) atomicAdd(counters + CNT_RESEEDED, n_new);
      }
    }
    __syncwarp();
    // the list and its length; the overflow part holds cap entries, enough
    // for every list that fits the particle storage
    const int n = n_keep + n_new;
    int pos = -1;
    int* dst = glist + (size_t)c * kListStride;
    if (n > kListStride) {
      if (lane == 0) pos = atomicAdd(novf, n);
      pos = __shfl_sync(PFEM2_FULL_MASK, pos, 0);
      if (pos < 0 || (size_t)pos + n > cap) pos = -1;
      dst = glist + (size_t)nc * kListStride + pos;
    }
    if (n <= kListStride || pos >= 0)
      for (int i = lane; i < n; i += 32) dst[i] = list[i];
    if (lane == 0) {
      cnt[c] = n;
      if (n > kListStride) glist_pos[c] = pos;
    }
    __syncwarp();
  }
}

// status words of the scan's tiles: bits 62-63 = 1 (tile aggregate known) or 2
// (inclusive prefix known), the low bits the value
constexpr unsigned long long kTileAgg = 1ull << 62, kTilePre = 2ull << 62, kTileVal = (1ull << 62) - 1;
constexpr int kScanThreads = 256, kScanItems = kScanTile / kScanThreads;

// new_start[c] = sum of the counts before cell c, new_start[nc] and *np_out =
// their sum: one pass over tiles in ticket order (a block waits only on tiles
// taken by blocks already running) with decoupled look-back; waits bounded, a
// timeout is flagged in CNT_SCAN_TIMEOUT
__global__ void __launch_bounds__(kScanThreads) k_rebin_scan(int nc, const int* __restrict__ cnt,
                                                             int* __restrict__ new_start, int* __restrict__ np_out,
                                                             int* __restrict__ counters,
                                                             unsigned long long* __restrict__ tiles,
                                                             unsigned spin_limit) {
  __shared__ int s_tile, s_base, s_w[kScanThreads / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned long long* status = tiles + 1;
  if (threadIdx.x == 0) s_tile = (int)atomicAdd(tiles, 1ull);
  __syncthreads();
  const int t = s_tile, c0 = t * kScanTile + threadIdx.x * kScanItems;
  int v[kScanItems], sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = c0 + k < nc ? cnt[c0 + k] : 0;
    sum += v[k];
  }
  int inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(PFEM2_FULL_MASK, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) s_w[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    unsigned long long agg = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) agg += (unsigned)s_w[w];
    unsigned long long excl = 0;
    if (t == 0) {
      if (lane == 0) atomicExch(status, kTilePre | agg);
    } else {
      if (lane == 0) atomicExch(status + t, kTileAgg | agg);
      // look back over windows of 32 predecessors (lane k reads tile j - k):
      // the window ends at the nearest tile with a published prefix; the
      // tiles before it must have published their aggregates
      int j = t - 1;
      unsigned spins = 0;
      for (;;) {
        if (spins++ >= spin_limit) {
          if (lane == 0) atomicExch(counters + CNT_SCAN_TIMEOUT, 1);
          break;
        }
        const int k = j - lane;
        const unsigned long long wd =
            k >= 0 ? *(volatile const unsigned long long*)(status + k) : kTilePre;  // before tile 0: prefix 0
        const unsigned pre = __ballot_sync(PFEM2_FULL_MASK, (wd >> 62) == 2);
        const unsigned wait = __ballot_sync(PFEM2_FULL_MASK, (wd >> 62) == 0);
        const int lp = pre ? __ffs(pre) - 1 : 31;
        const unsigned upto = lp == 31 ? PFEM2_FULL_MASK : (2u << lp) - 1u;
        if (wait & upto) {
          __nanosleep(32);
          continue;
        }
        excl += warp_sum((unsigned long long)(lane <= lp ? (wd & kTileVal) : 0ull));
        if (pre) break;
        j -= 32;
      }
      if (lane == 0) atomicExch(status + t, kTilePre | ((excl + agg) & kTileVal));
    }
    if (lane == 0) s_base = (int)excl;
  }
  __syncthreads();
  int out = s_base + inc - sum;
  for (int w = 0; w < warp; ++w) out += s_w[w];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (c0 + k < nc) new_start[c0 + k] = out;
    out += v[k];
    if (c0 + k == nc - 1) {
      new_start[nc] = out;
      *np_out = out;
    }
  }
}

template <int DIM, typename R, bool PROJ>
__global__ void __launch_bounds__(kRebinWarps * 32, RebinMinBlocks<DIM, R>::write) k_rebin_write(
    const R* __restrict__ oxi, const R* __restrict__ ou, size_t cap, int* __restrict__ ncell, R* __restrict__ nxi,
    R* __restrict__ nu, const int* __restrict__ new_start, int nc, const DevInst* __restrict__ inst,
    const int* __restrict__ cell_inst, const int* __restrict__ cv, const R* __restrict__ Vr, int nv,
    R* __restrict__ partial, const int* __restrict__ cnt, const int* __restrict__ glist,
    const int* __restrict__ glist_pos) {
  constexpr int NV = Dims<DIM>::NV;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the next cell's count, place and list are loaded while a cell is worked on
  // (the list's entries from the count on are not used)
  const int step = gridDim.x * kRebinWarps;
  int n_next = 0, out_next = 0, code_next = 0;
  const auto fetch = [&](int c) {
    if (c < nc) {
      n_next = cnt[c];
      out_next = new_start[c];
      code_next = glist[(size_t)c * kListStride + lane];
    }
  };
  fetch(blockIdx.x * kRebinWarps + warp);
  for (int c = blockIdx.x * kRebinWarps + warp; c < nc; c += step) {
    const int n = n_next, out = out_next;
    int code = code_next;
    fetch(c + step);
    const int* list = glist + (size_t)c * kListStride;
    bool stored = true;
    if (n > kListStride) {
      const int pos = glist_pos[c];
      stored = pos >= 0;  // else more particles than their storage holds (reported): any particle will do
      list = glist + (size_t)nc * kListStride + max(pos, 0);
      code = stored ? list[lane] : -1;
    }
    ProjAcc<DIM, R> acc;
    if (PROJ) {
#pragma unroll
      for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int k = 0; k <= DIM; ++k) acc.a[v][k] = R(0);
    }
    for (int j = lane; j < n; j += 32) {
      if (j >= 32) code = stored ? list[j] : -1;
      R x[DIM], uu[DIM];
      if (code >= 0) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          x[d] = oxi[d * cap + code];
          uu[d] = ou[d * cap + code];
        }
      } else {
        const DevInst& I = inst[__ldg(cell_inst + c)];
        const int t = -1 - code;
        int id[3];
        sub_cell_ijk(t, I.q[1], DIM == 3 ? I.q[2] : 1, I.qm, id);
#pragma unroll
        for (int d = 0; d < DIM; ++d) x[d] = R((id[d] + 1.0 / 2) * I.h[d]);
        R N[NV];
        shape_values<DIM, R>(x, N);
#pragma unroll
        for (int d = 0; d < DIM; ++d) uu[d] = R(0);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const int g = __ldg(cv + (size_t)c * NV + v);
#pragma unroll
          for (int d = 0; d < DIM; ++d) uu[d] = uu[d] + N[v] * Vr[(size_t)d * nv + g];
        }
      }
      const size_t o = (size_t)out + j;
      if (o < cap) {
        ncell[o] = c;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
          nxi[d * cap + o] = x[d];
          nu[d * cap + o] = uu[d];
        }
      }
      if (PROJ) proj_add<DIM, R>(acc, x, uu);
    }
    if (PROJ) proj_store<DIM, R>(acc, partial, c, lane);
  }
}

template <int DIM, typename R, bool CHECK, bool PROJ>
static pfem2_status rebin_launch(Ctx& c, const int* newcell) {
  const int o = c.cur, nb = 1 - c.cur;
  const size_t smem = (size_t)kRebinWarps * (c.list_cap + kMaxBuckets) * sizeof(int);
  const int ntiles = (c.nc + kScanTile - 1) / kScanTile;
  // resident blocks only: a cell per warp at a time, the cells in turn
  const int ggrid = grid_for(c, (long long)c.nc * 32, kRebinWarps * 32,
                             std::min(c.tune.rebin_blocks_per_sm, RebinMinBlocks<DIM, R>::gather));
  const int wgrid = grid_for(c, (long long)c.nc * 32, kRebinWarps * 32,
                             std::min(c.tune.rebin_blocks_per_sm, RebinMinBlocks<DIM, R>::write));
  PFEM2_CUDA(cudaFuncSetAttribute((const void*)k_rebin_gather<DIM, R, CHECK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
  // ticket and status words of the scan, then the overflow part's fill count
  PFEM2_CUDA(cudaMemsetAsync(c.rebin_tiles, 0, sizeof(unsigned long long) * ((size_t)ntiles + 2), c.stream));
  int* novf = (int*)(c.rebin_tiles + ntiles + 1);
  k_rebin_gather<DIM, R, CHECK><<<ggrid, kRebinWarps * 32, smem, c.stream>>>(
      c.cell_start[o], newcell, (const R*)c.pxi[o], (size_t)c.pcap, c.nc, c.ring_ptr, c.ring_cell, c.movers,
      c.far_keys, c.far_cap, c.d_inst, c.cell_inst, c.list_cap, c.d_counters, c.rebin_cnt, c.rebin_list,
      c.rebin_pos, novf);
  k_rebin_scan<<<ntiles, kScanThreads, 0, c.stream>>>(c.nc, c.rebin_cnt, c.cell_start[nb], c.d_np + nb, c.d_counters,
                                                      c.rebin_tiles, c.spin_limit >> 2);
  k_rebin_write<DIM, R, PROJ><<<wgrid, kRebinWarps * 32, 0, c.stream>>>(
      (const R*)c.pxi[o], (const R*)c.pu[o], (size_t)c.pcap, c.pcell[nb], (R*)c.pxi[nb], (R*)c.pu[nb],
      c.cell_start[nb], c.nc, c.d_inst, c.cell_inst, c.cv, (const R*)c.Vr, c.nv, (R*)c.partial, c.rebin_cnt,
      c.rebin_list, c.rebin_pos);
  c.launches += 3;
  c.cur = nb;
  return PFEM2_OK;
}

template <int DIM, typename R>
static pfem2_status rebin_impl(Ctx& c, bool check, bool proj, bool from_advect) {
  const int* nc_arr = from_advect ? c.newcell : c.pcell[c.cur];
  if (check) return proj ? rebin_launch<DIM, R, true, true>(c, nc_arr) : rebin_launch<DIM, R, true, false>(c, nc_arr);
  return proj ? rebin_launch<DIM, R, false, true>(c, nc_arr) : rebin_launch<DIM, R, false, false>(c, nc_arr);
}

pfem2_status launch_rebin(Ctx& c, bool check, bool proj, bool from_advect) {
  if (!from_advect) {
    // no movers: make sure their lists are empty
    PFEM2_CUDA(cudaMemsetAsync(c.d_counters + CNT_FAR, 0, sizeof(int), c.stream));
    PFEM2_CUDA(cudaMemsetAsync(c.movers.cnt, 0, sizeof(int) * c.nc, c.stream));
  }
  if (c.dim == 2) return c.pmixed ? rebin_impl<2, float>(c, check, proj, from_advect) : rebin_impl<2, double>(c, check, proj, from_advect);
  return c.pmixed ? rebin_impl<3, float>(c, check, proj, from_advect) : rebin_impl<3, double>(c, check, proj, from_advect);
}

// --------------------------------------------------------------- project
template <int DIM, typename R>
__global__ void __launch_bounds__(256) k_project_cells(const int* __restrict__ cell_start, const R* __restrict__ xi,
                                                       const R* __restrict__ u, size_t cap, int nc,
                                                       R* __restrict__ partial) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (int c = blockIdx.x * wpb + warp; c < nc; c += gridDim.x * wpb) {
    const int b = min(cell_start[c], (int)cap), n = min(cell_start[c + 1], (int)cap) - b;
    ProjAcc<DIM, R> acc;
#pragma unroll
    for (int v = 0; v < Dims<DIM>::NV; ++v)
#pragma unroll
      for (int k = 0; k <= DIM; ++k) acc.a[v][k] = R(0);
    for (int j = lane; j < n; j += 32) {
      R x[DIM], uu[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        x[d] = xi[d * cap + b + j];
        uu[d] = u[d * cap + b + j];
      }
      proj_add<DIM, R>(acc, x, uu);
    }
    proj_store<DIM, R>(acc, partial, c, lane);
  }
}

// node gather: u_n = sum_k N u / sum_k N over the cells around node n, in
// ascending cell order (deterministic, no float atomics)
template <int DIM, typename R>
__global__ void __launch_bounds__(256) k_project_nodes(int nv, const int* __restrict__ v2c_ptr,
                                                       const int* __restrict__ v2c_cell,
                                                       const unsigned char* __restrict__ v2c_loc,
                                                       const R* __restrict__ partial,
                                                       const unsigned char* __restrict__ zero_flag,
                                                       double* __restrict__ V0, double* __restrict__ V1,
                                                       double* __restrict__ V2, double* __restrict__ W,
                                                       R* __restrict__ Vr, int* __restrict__ counters,
                                                       double* __restrict__ wall_dv) {
  constexpr int K = Dims<DIM>::NV * (DIM + 1);
  double* V[3] = {V0, V1, V2};
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
    R s[DIM + 1];
#pragma unroll
    for (int k = 0; k <= DIM; ++k) s[k] = R(0);
    const int k1 = v2c_ptr[v + 1];
    for (int k = v2c_ptr[v]; k < k1; ++k) {
      const R* pp = partial + (size_t)v2c_cell[k] * K + v2c_loc[k] * (DIM + 1);
#pragma unroll
      for (int q = 0; q <= DIM; ++q) s[q] += pp[q];
    }
    const R w = s[DIM];
    const bool z = zero_flag[v] != 0;
    if (w == R(0) && k1 > v2c_ptr[v]) atomicAdd(counters + CNT_ZERO_WEIGHT, 1);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      R val = (w != R(0)) ? s[d] / w : R(0);
      if (z) {
        if (wall_dv) wall_dv[(size_t)d * nv + v] = (double)val;  // for the wall push-back
        val = R(0);
      }
      V[d][v] = (double)val;
      Vr[(size_t)d * nv + v] = val;
    }
    W[v] = (double)w;
  }
}

// Wall push-back after the projection (nacaAirfoil/pfem2particle.cpp:
// 919-952): a warp per cell touching a zero-flag vertex; every particle of
// the cell loses N_v(xi_p) times the projected velocity of each such vertex v
// whose velocity has a component above 1e-5 in magnitude (vertices in
// ascending local order, FP64 products).
template <int DIM, typename R>
__global__ void __launch_bounds__(256) k_wall_pushback(int ncells, const int* __restrict__ cells,
                                                       const int* __restrict__ cell_start, const int* __restrict__ cv,
                                                       const unsigned char* __restrict__ zero_flag,
                                                       const double* __restrict__ dv, int nv,
                                                       const R* __restrict__ xi, R* __restrict__ u, size_t cap) {
  constexpr int NV = Dims<DIM>::NV;
  const int lane = threadIdx.x & 31;
  for (int wc = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5); wc < ncells;
       wc += (int)((gridDim.x * (size_t)blockDim.x) >> 5)) {
    const int c = cells[wc];
    double d[NV][DIM];
    bool on[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int g = __ldg(cv + (size_t)c * NV + v);
      on[v] = false;
#pragma unroll
      for (int a = 0; a < DIM; ++a) d[v][a] = 0.0;
      if (zero_flag[g]) {
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
          d[v][a] = dv[(size_t)a * nv + g];
          on[v] |= fabs(d[v][a]) > 1e-5;
        }
      }
    }
    const int p1 = cell_start[c + 1];
    for (int p = cell_start[c] + lane; p < p1; p += 32) {
      double x[DIM], N[NV];
#pragma unroll
      for (int a = 0; a < DIM; ++a) x[a] = (double)xi[(size_t)a * cap + p];
      shape_values<DIM, double>(x, N);
      double uu[DIM];
#pragma unroll
      for (int a = 0; a < DIM; ++a) uu[a] = (double)u[(size_t)a * cap + p];
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (on[v])
#pragma unroll
          for (int a = 0; a < DIM; ++a) uu[a] -= N[v] * d[v][a];
#pragma unroll
      for (int a = 0; a < DIM; ++a) u[(size_t)a * cap + p] = R(uu[a]);
    }
  }
}

template <int DIM, typename R>
static pfem2_status project_impl(Ctx& c, bool partials_ready) {
  const int b = c.cur;
  if (!partials_ready) {
    k_project_cells<DIM, R><<<grid_for(c, (long long)c.nc * 32, 256, 8), 256, 0, c.stream>>>(
        c.cell_start[b], (const R*)c.pxi[b], (const R*)c.pu[b], (size_t)c.pcap, c.nc, (R*)c.partial);
    c.launches++;
  }
  k_project_nodes<DIM, R><<<grid_for(c, c.nv, 256, 8), 256, 0, c.stream>>>(
      c.nv, c.v2c_ptr, c.v2c_cell, c.v2c_loc, (const R*)c.partial, c.zero_flag, c.F[PFEM2_FIELD_VX],
      c.F[PFEM2_FIELD_VY], c.dim == 3 ? c.F[PFEM2_FIELD_VZ] : c.F[PFEM2_FIELD_VZ], c.F[PFEM2_FIELD_NODE_WEIGHT],
      (R*)c.Vr, c.d_counters, c.wall_dv);
  c.launches++;
  if (c.n_wall_cells > 0) {
    k_wall_pushback<DIM, R><<<grid_for(c, (long long)c.n_wall_cells * 32, 256, 8), 256, 0, c.stream>>>(
        c.n_wall_cells, c.wall_cells, c.cell_start[b], c.cv, c.zero_flag, c.wall_dv, c.nv, (const R*)c.pxi[b],
        (R*)c.pu[b], (size_t)c.pcap);
    c.launches++;
  }
  return PFEM2_OK;
}

pfem2_status launch_project(Ctx& c, bool partials_ready) {
  if (c.dim == 2) return c.pmixed ? project_impl<2, float>(c, partials_ready) : project_impl<2, double>(c, partials_ready);
  return c.pmixed ? project_impl<3, float>(c, partials_ready) : project_impl<3, double>(c, partials_ready);
}

// -------------------------------------------------- particle state access
template <int DIM, typename R>
__global__ void k_pack_out(const int* __restrict__ cell, const R* __restrict__ xi, const R* __restrict__ u,
                           size_t cap, int p0, int n, int c_off, int* __restrict__ ocell, double* __restrict__ oxi,
                           double* __restrict__ ou) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const size_t p = (size_t)p0 + j;
    ocell[j] = cell[p] - c_off;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      oxi[(size_t)j * DIM + d] = (double)xi[d * cap + p];
      ou[(size_t)j * DIM + d] = (double)u[d * cap + p];
    }
  }
}

template <int DIM, typename R>
static pfem2_status read_impl(Ctx& c, int instance, int* cell, double* xi, double* u, int* n_out) {
  const int b = c.cur;
  const HostInst& in = c.inst[instance];
  int se[2];
  PFEM2_CUDA(cudaMemcpyAsync(&se[0], c.cell_start[b] + in.c_off, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(&se[1], c.cell_start[b] + in.c_off + in.nc, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  PFEM2_CUDA(cudaStreamSynchronize(c.stream));
  const int n = se[1] - se[0];
  *n_out = n;
  if (!cell) return PFEM2_OK;
  if (n == 0) return PFEM2_OK;
  // packed in the buffers that the next re-sort fills, as many at a time as
  // their coordinates hold in FP64 (allocating three buffers per call took 0.8
  // of 1.1 ms for 53k particles)
  const int per = std::max(1, (int)((size_t)c.pcap * sizeof(R) / sizeof(double)));
  int* dc = c.pcell[1 - b];
  double *dx = (double*)c.pxi[1 - b], *du = (double*)c.pu[1 - b];
  for (int i = 0; i < n; i += per) {
    const int m = std::min(per, n - i);
    k_pack_out<DIM, R><<<grid_for(c, m, 256), 256, 0, c.stream>>>(c.pcell[b], (const R*)c.pxi[b], (const R*)c.pu[b],
                                                                 (size_t)c.pcap, se[0] + i, m, in.c_off, dc, dx, du);
    c.launches++;
    PFEM2_CUDA(cudaMemcpyAsync(cell + i, dc, sizeof(int) * m, cudaMemcpyDeviceToHost, c.stream));
    PFEM2_CUDA(cudaMemcpyAsync(xi + (size_t)i * DIM, dx, sizeof(double) * m * DIM, cudaMemcpyDeviceToHost, c.stream));
    PFEM2_CUDA(cudaMemcpyAsync(u + (size_t)i * DIM, du, sizeof(double) * m * DIM, cudaMemcpyDeviceToHost, c.stream));
  }
  PFEM2_CUDA(cudaStreamSynchronize(c.stream));
  return PFEM2_OK;
}

pfem2_status read_particles(Ctx& c, int instance, int* cell, double* xi, double* u, int* n) {
  if (c.dim == 2) return c.pmixed ? read_impl<2, float>(c, instance, cell, xi, u, n) : read_impl<2, double>(c, instance, cell, xi, u, n);
  return c.pmixed ? read_impl<3, float>(c, instance, cell, xi, u, n) : read_impl<3, double>(c, instance, cell, xi, u, n);
}

// unsorted particles in, stable sort by cell through the rebin machinery:
// the particles are first placed one per "virtual old segment" (all in the
// segment of their own cell, in input order) and then rebinned without check.
template <int DIM, typename R>
__global__ void k_unpack_in(int n, const int* __restrict__ pos, const int* __restrict__ icell,
                            const double* __restrict__ ixi, const double* __restrict__ iu, int* __restrict__ cell,
                            R* __restrict__ xi, R* __restrict__ u, size_t cap) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const size_t p = pos[j];
    cell[p] = icell[j];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      xi[d * cap + p] = R(ixi[(size_t)j * DIM + d]);
      u[d * cap + p] = R(iu[(size_t)j * DIM + d]);
    }
  }
}

// refused before anything of the context changes
pfem2_status check_set_particles(const Ctx& c, const int* counts, const int* cell, const double* xi, const double* u) {
  size_t k = 0;
  for (size_t i = 0; i < c.inst.size(); ++i)
    for (int j = 0; j < counts[i]; ++j, ++k) {
      if (cell[k] < 0 || cell[k] >= c.inst[i].nc) {
        set_error("set_particles: cell out of range");
        return PFEM2_INVALID_ARG;
      }
      for (int d = 0; d < c.dim; ++d)
        if (!std::isfinite(xi[k * c.dim + d]) || !std::isfinite(u[k * c.dim + d])) {
          set_error("set_particles: a coordinate or velocity is not finite");
          return PFEM2_INVALID_ARG;
        }
    }
  return PFEM2_OK;
}

template <int DIM, typename R>
static pfem2_status set_impl(Ctx& c, const int* counts, const int* cell, const double* xi, const double* u) {
  // host-side stable placement by cell (a state-loading utility, not the step)
  size_t n = 0;
  for (size_t i = 0; i < c.inst.size(); ++i) n += counts[i];
  if (n > (size_t)c.pcap) {
    set_error("set_particles: capacity exceeded");
    return PFEM2_PARTICLE_OVERFLOW;
  }
  std::vector<int> gcell(n), cnt(c.nc + 1, 0), pos(n);
  size_t k = 0;
  for (size_t i = 0; i < c.inst.size(); ++i)
    for (int j = 0; j < counts[i]; ++j, ++k) {
      gcell[k] = cell[k] + c.inst[i].c_off;
      cnt[gcell[k] + 1]++;
    }
  for (int i = 0; i < c.nc; ++i) cnt[i + 1] += cnt[i];
  std::vector<int> start(cnt.begin(), cnt.end());
  for (size_t j = 0; j < n; ++j) pos[j] = cnt[gcell[j]]++;
  const int b = c.cur;
  int *dpos, *dcell;
  double *dxi, *du;
  size_t nn = n ? n : 1;
  PFEM2_CUDA(cudaMalloc(&dpos, sizeof(int) * nn));
  PFEM2_CUDA(cudaMalloc(&dcell, sizeof(int) * nn));
  PFEM2_CUDA(cudaMalloc(&dxi, sizeof(double) * nn * DIM));
  PFEM2_CUDA(cudaMalloc(&du, sizeof(double) * nn * DIM));
  // (on the context's stream, which does not wait for the default stream's
  // copies: those may still be in flight when the call returns)
  PFEM2_CUDA(cudaMemcpyAsync(dpos, pos.data(), sizeof(int) * n, cudaMemcpyHostToDevice, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(dcell, gcell.data(), sizeof(int) * n, cudaMemcpyHostToDevice, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(dxi, xi, sizeof(double) * n * DIM, cudaMemcpyHostToDevice, c.stream));
  PFEM2_CUDA(cudaMemcpyAsync(du, u, sizeof(double) * n * DIM, cudaMemcpyHostToDevice, c.stream));
  if (n) {
    k_unpack_in<DIM, R><<<grid_for(c, n, 256), 256, 0, c.stream>>>((int)n, dpos, dcell, dxi, du, c.pcell[b],
                                                                 (R*)c.pxi[b], (R*)c.pu[b], (size_t)c.pcap);
    c.launches++;
  }
  PFEM2_CUDA(cudaMemcpyAsync(c.cell_start[b], start.data(), sizeof(int) * (c.nc + 1), cudaMemcpyHostToDevice, c.stream));
  int nint = (int)n;
  PFEM2_CUDA(cudaMemcpyAsync(c.d_np + b, &nint, sizeof(int), cudaMemcpyHostToDevice, c.stream));
  PFEM2_CUDA(cudaStreamSynchronize(c.stream));
  cudaFree(dpos); cudaFree(dcell); cudaFree(dxi); cudaFree(du);
  PFEM2_CUDA(cudaGetLastError());
  return PFEM2_OK;
}

pfem2_status launch_set_particles(Ctx& c, const int* counts, const int* cell, const double* xi, const double* u) {
  if (c.dim == 2) return c.pmixed ? set_impl<2, float>(c, counts, cell, xi, u) : set_impl<2, double>(c, counts, cell, xi, u);
  return c.pmixed ? set_impl<3, float>(c, counts, cell, xi, u) : set_impl<3, double>(c, counts, cell, xi, u);
}

}  // namespace pfem2
