// blas.cuh -- qkxTM BLAS on device fields (reference lib/blas_qkxTM.cpp:4-56,
// Vector::norm2 lib/lattice_util.cpp:464-477), plus the fused CG updates.
//
// Reductions are deterministic: a fixed grid writes one partial per block and
// a one-block finalize sums the partials in a fixed order, so repeated runs
// give bit-identical scalars.  Scalars that drive the solvers (alpha, beta,
// r2) live in device memory so an iteration needs no host round trip.
#pragma once
#include "qkx_common.cuh"

namespace qkx {

constexpr int BLAS_NT = 256;

// Solver scalars for up to QKX_MAX_RHS right-hand sides.
constexpr int MAX_RHS = 64;
struct CgScalars {
  double r2[MAX_RHS];
  double r2_old[MAX_RHS];
  double pAp[MAX_RHS];
  double alpha[MAX_RHS];
  double beta[MAX_RHS];
  double stop[MAX_RHS];   // FP64 true residual^2 at which the RHS has converged ((0.9 tol)^2 |b|^2)
  int active[MAX_RHS];   // 1 while the RHS still iterates
  int iters[MAX_RHS];
  double aux[MAX_RHS];   // per-RHS results of the batched FP64 residual steps
  double aux2[MAX_RHS];
  int restart[MAX_RHS];  // 1: restart the search direction from the residual (p = r)
};

template <int NT>
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double red[NT / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double w = 0.0;
  if (threadIdx.x < 32) {
    w = threadIdx.x < NT / 32 ? red[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  }
  __syncthreads();
  return w;  // valid in thread 0
}

// Re <x, y> over n complex numbers (partials per block)
static __global__ void __launch_bounds__(BLAS_NT) k_redot(const double2* x, const double2* y, size_t n,
                                                   double* part) {
  pdl_start();
  double acc = 0.0;
  for (size_t i = (size_t)blockIdx.x * BLAS_NT + threadIdx.x; i < n; i += (size_t)gridDim.x * BLAS_NT) {
    double2 a = x[i], b = y[i];
    acc += a.x * b.x + a.y * b.y;
  }
  double s = block_sum<BLAS_NT>(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// what a sum of partials is for
enum { FIN_STORE = 0, FIN_PAP = 1, FIN_R2 = 2, FIN_R2_INIT = 3 };

// Sum part[0..n) in a fixed order: FIN_STORE *dst = sum; FIN_R2_INIT r2 = sum
static __global__ void __launch_bounds__(1024) k_finalize(const double* part, int n, double* dst, int mode,
                                                   CgScalars* sc, int rhs) {
  pdl_start();
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += 1024) acc += part[i];
  double s = block_sum<1024>(acc);
  if (threadIdx.x == 0) {
    if (mode == FIN_STORE) *dst = s;
    else sc->r2[rhs] = s;
  }
}

// ---- the FP64 CG iteration (solvers.cpp:40-70) in five kernels: the two hops, the two sums and the update.
// active[0] says whether the next iteration runs, restart[0] whether the current one does: iterations
// the host has queued past the stopping one do nothing, so it need not wait for r2 between them.

// start of the loop: the first iteration runs while r2 is above the stop
static __global__ void k_cg_begin(CgScalars* sc, double stop) {
  sc->stop[0] = stop;
  sc->active[0] = sc->r2[0] > stop ? 1 : 0;
  sc->restart[0] = 0;
}

// FIN_PAP: <p, M^+M p> = |M p|^2 from the first hop, alpha; FIN_R2: |r|^2 from the second, beta, the
// stopping rule, and r2 to page-locked host memory
static __global__ void __launch_bounds__(1024) k_cg_finalize(const double* part, int n, int mode,
                                                      CgScalars* sc, double* r2_host) {
  pdl_start();
  if (mode == FIN_PAP) {
    if (!sc->active[0]) {
      __syncthreads();
      if (threadIdx.x == 0) sc->restart[0] = 0;
      return;
    }
  } else if (!sc->restart[0]) {
    return;
  }
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += 1024) acc += part[i];
  const double s = block_sum<1024>(acc);
  if (threadIdx.x != 0) return;
  if (mode == FIN_PAP) {
    sc->restart[0] = 1;
    sc->pAp[0] = s;
    sc->alpha[0] = sc->r2[0] / s;
  } else {
    sc->r2_old[0] = sc->r2[0];
    sc->r2[0] = s;
    sc->beta[0] = s / sc->r2_old[0];
    sc->active[0] = s > sc->stop[0] ? 1 : 0;
    *r2_host = s;
  }
}

// x = x + alpha p, p = r + beta p in one pass (X_eq_X_p_aY and X_eq_aX_p_Y, lib/blas_qkxTM.cpp:31, 45)
static __global__ void __launch_bounds__(BLAS_NT) k_cg_update(const CgScalars* sc, const double2* r, double2* x,
                                                       double2* p, size_t n) {
  pdl_start();
  if (!sc->restart[0]) return;
  const double a = sc->alpha[0], b = sc->beta[0];
  for (size_t i = (size_t)blockIdx.x * BLAS_NT + threadIdx.x; i < n; i += (size_t)gridDim.x * BLAS_NT) {
    const double2 pv = p[i], xv = x[i], rv = r[i];
    x[i] = make_double2(xv.x + a * pv.x, xv.y + a * pv.y);
    p[i] = make_double2(b * pv.x + rv.x, b * pv.y + rv.y);
  }
}

// y = y + a x with a host scalar
static __global__ void __launch_bounds__(BLAS_NT) k_axpy_h(double a, const double2* x, double2* y, size_t n) {
  pdl_start();
  for (size_t i = (size_t)blockIdx.x * BLAS_NT + threadIdx.x; i < n; i += (size_t)gridDim.x * BLAS_NT) {
    double2 xv = x[i], yv = y[i];
    y[i] = make_double2(yv.x + a * xv.x, yv.y + a * xv.y);
  }
}

// y = a y + x with a host scalar
static __global__ void __launch_bounds__(BLAS_NT) k_xpay_h(const double2* x, double a, double2* y, size_t n) {
  pdl_start();
  for (size_t i = (size_t)blockIdx.x * BLAS_NT + threadIdx.x; i < n; i += (size_t)gridDim.x * BLAS_NT) {
    double2 xv = x[i], yv = y[i];
    y[i] = make_double2(a * yv.x + xv.x, a * yv.y + xv.y);
  }
}

// z = x - y, with partial sums of |z|^2 (true-residual helper)
static __global__ void __launch_bounds__(BLAS_NT) k_sub_norm(const double2* __restrict__ x, const double2* __restrict__ y,
                                                      double2* __restrict__ z, size_t n, double* __restrict__ part) {
  double acc = 0.0;
  for (size_t i = (size_t)blockIdx.x * BLAS_NT + threadIdx.x; i < n; i += (size_t)gridDim.x * BLAS_NT) {
    double2 a = x[i], b = y[i];
    double2 d = make_double2(a.x - b.x, a.y - b.y);
    z[i] = d;
    acc += d.x * d.x + d.y * d.y;
  }
  double s = block_sum<BLAS_NT>(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

}  // namespace qkx
