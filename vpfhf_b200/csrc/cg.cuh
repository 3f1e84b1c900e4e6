// cg.cuh -- preconditioned CG with device-resident scalars (no host round trip per
// iteration) and deterministic reductions.
//
// Semantics of PETSc's KSPCG with KSP_NORM_PRECONDITIONED and the default
// convergence test (KSPConvergedDefault): x0 = 0, z = D^-1 r, converged when
// ||z|| <= max(rtol ||z0||, atol), diverged on ||z|| >= dtol ||z0||, NaN, or a
// non-positive p.Ap.  Vectors are T (double, or float for the inner solve of the
// mixed-precision path); every dot product and step length is FP64.
#pragma once

#include "common.cuh"

namespace vfgpu {

// Reason codes (PETSc KSPConvergedReason numbering where one exists).
enum { CG_RUNNING = 0, CG_CONVERGED_RTOL = 2, CG_CONVERGED_ATOL = 3, CG_DIVERGED_ITS = -3,
       CG_DIVERGED_DTOL = -4, CG_DIVERGED_INDEFINITE = -8, CG_DIVERGED_NAN = -9 };

struct CGState {
  // by iteration parity: the iteration reads [par] and leaves [par ^ 1], so that no block reads
  // what another one writes
  double rz[2];
  int itn[2];
  double pw, zz, alpha, beta, rnorm0, ttol, dtol;
  double xalpha;  // step of the current iteration (0 if it made none); see cg_iteration
  int its, maxit, done, reason;
  int yield;      // the device loop also ends at this iteration count (the host's time check)
};

// Fixed reduction grids (at most 4 blocks per SM of a B200): the block partials are summed in
// a fixed order, so every reduction is deterministic.
constexpr int RED_THREADS = 256, RED_BLOCKS = 592;

// The vectors are whole device allocations (16-byte aligned: the kernels use 16-byte
// loads and stores).
template <typename T> struct CGVecs {
  T* x;              // solution
  T* r;              // residual
  T* p;              // search direction
  T* w;              // A p
  const T* dinv;     // Jacobi: 1 / diag
  const T* b;        // right-hand side
  const uint8_t* mask;  // nonzero => dof removed from the system (or null)
  int64_t n;
  const double* dotp;   // the operator's block partials of p.w (written by the apply)
  int ndot;
};

#ifdef __CUDACC__
// Fixed-order sum of K values per thread over a block of RED_THREADS (shuffle trees, then the
// warps in order), in every thread.
template <int K>
__device__ __forceinline__ void block_total(double (&v)[K]) {
  __shared__ double red[K][RED_THREADS / 32];
#pragma unroll
  for (int q = 0; q < K; q++)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  __syncthreads();  // a previous call's totals have been read
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int q = 0; q < K; q++) red[q][threadIdx.x >> 5] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < K; q++) {
    v[q] = red[q][0];
#pragma unroll
    for (int w = 1; w < RED_THREADS / 32; w++) v[q] += red[q][w];
  }
}

// Fixed-order sum of n blocks' partials by one block, in every thread (identical in every
// block that calls it).  L1 is bypassed: an earlier kernel of the same graph wrote them.
template <int K>
__device__ __forceinline__ void final_sum(const double* __restrict__ partial, int n, double (&out)[K]) {
#pragma unroll
  for (int q = 0; q < K; q++) out[q] = 0.;
  for (int b = threadIdx.x; b < n; b += RED_THREADS)
#pragma unroll
    for (int q = 0; q < K; q++) out[q] += __ldcg(partial + b * K + q);
  block_total<K>(out);
}
#endif

// Blocks of a CG vector kernel over n values in 16-byte packets: two packets per thread on
// small systems (fewer partials to sum), one wave of 4 blocks per SM on large ones.
inline int cg_blocks(int64_t n, int bytes) {
  const int64_t per = 2 * RED_THREADS * (16 / bytes);
  const int64_t b = (n + per - 1) / per;
  return (int)(b < 1 ? 1 : b > RED_BLOCKS ? RED_BLOCKS : b);
}

// Host-side driver pieces (solver.cu).  One iteration is: the operator apply
// w = A p, which also writes the block partials of p.w to v.dotp (the tile
// engine's A.dot), then cg_iteration: the update kernel moves r only (r -= alpha w,
// z = D^-1 r, block partials of (r,z), (z,z)), and the direction kernel sums those,
// tests for convergence and does x += alpha p together with p = z + beta p, in one pass
// over p.  The iteration that stops the solve does not move x and p, so cg_finish_x adds
// its step to x after the loop.  par: the parity of the iteration (0 for the first).
template <typename T>
cudaError_t cg_init(const CGVecs<T>& v, CGState* st, double* partial, double rtol, double atol,
                    double dtol, int maxit, cudaStream_t s);
template <typename T>
cudaError_t cg_iteration(const CGVecs<T>& v, CGState* st, double* partial, int par,
                         cudaStream_t s);
template <typename T>
cudaError_t cg_finish_x(const CGVecs<T>& v, const CGState* st, cudaStream_t s);
// The PCG around a multigrid preconditioner (FP64 vectors; z = M^-1 r in TZ = double or
// float, the V-cycle's own vector).  One iteration is: the V-cycle without its first and last
// smoothing steps on the fine level; mgcg_direction (the last step z += zdinv (r - t) / theta
// with the block partials of r.z; then beta, x += alpha p of the iteration before and
// p = z + beta p); the operator apply w = A p with the partials of p.w; mgcg_update
// (r -= alpha w, the V-cycle's FP32 copy of r and its first step z = zdinv r / theta, block
// partials of (D^-1 r).(D^-1 r), the Jacobi solve's stopping test); and the end of the iteration from those partials, which also sets
// the while node's condition (mgcg_end in cg_loop.cu; loop null: no condition).  So the test
// comes before the next V-cycle, and no vector is passed over for a dot alone.  cg_finish_x
// adds the last step to x.
template <typename TZ> struct MgcgVecs {
  double *x, *r, *p, *w;
  const double *dinv, *b;
  TZ* z;
  float* r32;  // the V-cycle's right-hand side (FP32), or null: it reads r
  int64_t n;
  const double* dotp;
  int ndot;
  const TZ *t, *zdinv;  // fine level: K z, the smoother's inverse diagonal and coefficients
  const double* zcoef;  // (zcoef[1] = 1 / theta)
};
template <typename TZ>
cudaError_t mgcg_init(const MgcgVecs<TZ>& v, CGState* st, double* partial, double rtol, double atol, double dtol,
                      int maxit, cudaStream_t s);
template <typename TZ>
cudaError_t mgcg_direction(const MgcgVecs<TZ>& v, CGState* st, double* partial, cudaStream_t s);
template <typename TZ>
cudaError_t mgcg_update(const MgcgVecs<TZ>& v, CGState* st, double* partial, cudaStream_t s);
cudaError_t mgcg_end(CGState* st, const double* partial, int64_t n, const cudaGraphConditionalHandle* loop,
                     cudaStream_t s);

// Device loop (cg_loop.cu): sets the condition of the while node `loop` from the state after
// its body's iterations; and st->yield, the iteration count from which the loop returns.
cudaError_t cg_set_condition(const CGState* st, cudaGraphConditionalHandle loop, cudaStream_t s);
cudaError_t cg_set_yield(CGState* st, int yield, cudaStream_t s);

}  // namespace vfgpu
