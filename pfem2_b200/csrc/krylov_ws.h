// krylov_ws.h -- the Krylov workspace and the device helpers shared by the
// Jacobi solver kernel (krylov.cu) and the multigrid CG kernel (mgcg.cu).
#pragma once
#include <string>
#include <vector>

#include "common.cuh"
#include "ctx.h"

namespace pfem2 {

constexpr int kMaxLocalSys = 16;  // systems a block of the multigrid's grid may own parts of

__device__ __forceinline__ float fma_r(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_r(double a, double b, double c) { return fma(a, b, c); }

template <int GL, typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
  for (int o = GL / 2; o > 0; o >>= 1) v += __shfl_xor_sync(PFEM2_FULL_MASK, v, o);
  return v;
}

// acc + sum over the entries of a SELL row of val(ei) * x(col), in entry
// order, with the loads of CH entries issued before their products are
// accumulated (one memory round trip per CH entries instead of one per entry)
template <typename T, int CH = 8, typename Cols, typename Val, typename X>
__device__ __forceinline__ T sell_dot(T acc, Cols cols, int base, int len, int lane, Val val, X x) {
  for (int j0 = 0; j0 < len; j0 += CH) {
    T av[CH], xv[CH];
#pragma unroll
    for (int u = 0; u < CH; ++u) {
      const int j = j0 + u;
      if (j < len) {
        const int ei = base + j * 32 + lane;
        av[u] = val(ei);
        xv[u] = x(cols[ei]);
      } else {
        av[u] = T(0);
        xv[u] = T(0);
      }
    }
#pragma unroll
    for (int u = 0; u < CH; ++u) acc = fma_r(av[u], xv[u], acc);
  }
  return acc;
}

// acc + sum over CSR entries [k0, k1) of val(k) * x(col(k)), the lanes of a
// group of GL taking every GL-th entry, loads issued CH entries at a time
template <int GL, int CH, typename T, typename Cols, typename Val, typename X>
__device__ __forceinline__ T csr_dot(T acc, int k0, int k1, int sub, Cols cols, Val val, X x) {
  for (int kb = k0 + sub; kb < k1; kb += CH * GL) {
    T av[CH], xv[CH];
#pragma unroll
    for (int u = 0; u < CH; ++u) {
      const int k = kb + u * GL;
      if (k < k1) {
        av[u] = val[k];
        xv[u] = x(cols[k]);
      } else {
        av[u] = T(0);
        xv[u] = T(0);
      }
    }
#pragma unroll
    for (int u = 0; u < CH; ++u) acc = fma_r(av[u], xv[u], acc);
  }
  return acc;
}

__device__ __forceinline__ size_t al16_dev(size_t b) { return (b + 15) & ~(size_t)15; }

// copies src[0, n) into shared memory at `cur` (16-byte aligned pieces); the
// caller syncs before reading it
template <typename T>
__device__ __forceinline__ const T* stage_copy(unsigned char*& cur, const T* src, int n) {
  T* dst = reinterpret_cast<T*>(cur);
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
  cur += al16_dev((size_t)n * sizeof(T));
  return dst;
}

// Waits (acquire) until system counter *cnt has reached target (release adds
// of the blocks that own parts of the system); false after spin_limit polls
// or when another block has flagged an error.
__device__ __forceinline__ bool wait_count(const unsigned* cnt, unsigned target, const GridBarrier& gb) {
  unsigned spins = 0;
  while ((int)(ld_acquire_u32(cnt) - target) < 0) {
    if (++spins > gb.spin_limit || *(volatile int*)gb.err != 0) return false;
    __nanosleep(20);
  }
  return true;
}

// ------------------------------------------------------------------ host
struct MgWs;  // mgcg.cu

// partition of a Jacobi solve over its grid
struct JacobiPlan {
  int *blk_inst = nullptr, *blk_inst_off = nullptr, *blk_slot = nullptr, *blk_sl = nullptr, *sys_slot0 = nullptr,
      *slk = nullptr;
  int grid = 0, nslots = 0, items_max = 0, sys_max = 0, minb = 2, split = 1;
  int ts = 0;                                      // no cluster: least slices of a block
  int sm = 0;                                      // cluster: what a block keeps in shared memory
  bool cluster = false, bicg = false;
  size_t st_meta = 0, st_entries = 0;              // per block: static index bytes, SELL entries
  double* item_part = nullptr;                     // the items' partial sums, where they do not fit shared memory
};

struct KrylovWs {
  JacobiPlan plan[2];                              // [0] pressure (without multigrid), [1] velocity components
  JacobiPlan elastic;                              // mesh elasticity
  double *el_pk = nullptr, *el_e = nullptr, *el_r = nullptr, *el_v = nullptr, *el_s = nullptr, *el_t = nullptr,
         *el_r64 = nullptr, *el_part = nullptr, *el_res = nullptr;
  int* el_int = nullptr;
  bool mass_share = false;                         // the components' mass matrices are equal
  void *pk = nullptr, *rh = nullptr, *s = nullptr, *t = nullptr, *v = nullptr;
  MgWs* mg = nullptr;
  void *e = nullptr, *r = nullptr;
  double* r64 = nullptr;
  double* part = nullptr;
  unsigned* scount = nullptr;
  int* active = nullptr;
  int* out_it[3] = {};
  double* out_res[3] = {};
  double* out_tol[3] = {};
  int* out_outer[3] = {};
  std::vector<void*> allocs;            // every device allocation of the workspace
};

template <typename T>
inline pfem2_status ws_alloc(KrylovWs* w, T** p, size_t n) {
  *p = nullptr;
  if (n == 0) n = 1;
  PFEM2_CUDA(cudaMalloc((void**)p, sizeof(T) * n));
  w->allocs.push_back(*p);
  PFEM2_CUDA(cudaMemset(*p, 0, sizeof(T) * n));
  return PFEM2_OK;
}

template <typename T>
inline pfem2_status ws_upload(KrylovWs* w, T** p, const std::vector<T>& v) {
  PFEM2_TRY(ws_alloc(w, p, v.size()));
  if (!v.empty()) PFEM2_CUDA(cudaMemcpy(*p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice));
  return PFEM2_OK;
}

// FP64 host values as the inner type R (float for the mixed path)
inline pfem2_status ws_upload_r(KrylovWs* w, bool mixed, void** p, const std::vector<double>& v) {
  if (mixed) {
    std::vector<float> f(v.begin(), v.end());
    float* d;
    PFEM2_TRY(ws_upload(w, &d, f));
    *p = d;
  } else {
    double* d;
    PFEM2_TRY(ws_upload(w, &d, v));
    *p = d;
  }
  return PFEM2_OK;
}

inline size_t al16(size_t b) { return (b + 15) & ~(size_t)15; }

// shared-memory budget of a solver block (dynamic part) with MINB resident blocks per SM
constexpr size_t smem_budget(int minb) { return minb == 1 ? 200 * 1024 : 108 * 1024; }

// krylov.cu: resets a solve's shared state (counters, barrier, error word)
pfem2_status krylov_init_solve(Ctx& c, int nsys);
int krylov_max_iter(const Ctx& c);

// mgcg.cu: the multigrid CG of the pressure systems
pfem2_status mg_setup(Ctx& c);
pfem2_status mg_solve(Ctx& c);
void mg_free(KrylovWs* w);
void mg_sizes(const KrylovWs* w, long long* out12);
void mg_forms(const KrylovWs* w, int* out6);

}  // namespace pfem2
