// solver.cu -- reductions, PCG kernels and the vector kernels of the U/V solves.
#include <algorithm>
#include <climits>
#include <cmath>

#include "cg.cuh"
#include "solver.h"

namespace vfgpu {

namespace {

// Block-level fixed-order sum of K values per thread into partial[blockIdx*K + q].
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K], double* __restrict__ partial) {
  block_total<K>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < K; q++) partial[blockIdx.x * K + q] = v[q];
}

#define GRID_LOOP(i, n)                                                                  \
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n);              \
       i += (int64_t)gridDim.x * blockDim.x)

// 16-byte packets for the bandwidth-bound CG kernels: W values of T per load/store.
// The CG vectors are whole cudaMalloc allocations (256-byte aligned); the n % W tail
// is done with scalar accesses by the first threads of the grid.
template <typename T> struct Pack {
  static constexpr int W = 16 / sizeof(T);
  T e[W];
};
template <typename T>
__device__ __forceinline__ Pack<T> ld16(const T* __restrict__ a, int64_t c) {
  Pack<T> p;
  if constexpr (sizeof(T) == 8) {
    const double2 q = reinterpret_cast<const double2*>(a)[c];
    p.e[0] = q.x;
    p.e[1] = q.y;
  } else {
    const float4 q = reinterpret_cast<const float4*>(a)[c];
    p.e[0] = q.x;
    p.e[1] = q.y;
    p.e[2] = q.z;
    p.e[3] = q.w;
  }
  return p;
}
// The same with evict-first caching: for a vector that is not read again before others push
// it out of L2.
template <typename T>
__device__ __forceinline__ Pack<T> ld16s(const T* __restrict__ a, int64_t c) {
  Pack<T> p;
  if constexpr (sizeof(T) == 8) {
    const double2 q = __ldcs(reinterpret_cast<const double2*>(a) + c);
    p.e[0] = q.x;
    p.e[1] = q.y;
  } else {
    const float4 q = __ldcs(reinterpret_cast<const float4*>(a) + c);
    p.e[0] = q.x;
    p.e[1] = q.y;
    p.e[2] = q.z;
    p.e[3] = q.w;
  }
  return p;
}
template <typename T>
__device__ __forceinline__ void st16(T* __restrict__ a, int64_t c, const Pack<T>& p) {
  if constexpr (sizeof(T) == 8) {
    reinterpret_cast<double2*>(a)[c] = make_double2(p.e[0], p.e[1]);
  } else {
    reinterpret_cast<float4*>(a)[c] = make_float4(p.e[0], p.e[1], p.e[2], p.e[3]);
  }
}
// Visits the n values as 16-byte packets (fp(packet index)), then the tail of
// n % W values one by one (ft(element index)).
template <typename T, class FP, class FT>
__device__ __forceinline__ void pack_loop(int64_t n, FP fp, FT ft) {
  constexpr int W = Pack<T>::W;
  const int64_t np = n / W;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t st = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = t0; c < np; c += st) fp(c);
  for (int64_t i = np * W + t0; i < n; i += st) ft(i);
}
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) cg_init_kernel(CGVecs<T> v, double* partial) {
  double acc[2] = {0., 0.};
  GRID_LOOP(i, v.n) {
    const bool m = v.mask && v.mask[i];
    const T r = m ? T(0) : v.b[i];
    const T z = r * v.dinv[i];
    v.x[i] = T(0);
    v.r[i] = r;
    v.p[i] = z;
    acc[0] += (double)z * (double)r;
    acc[1] += (double)z * (double)z;
  }
  block_sum<2>(acc, partial);
}

__global__ void cg_init_final(CGState* st, const double* partial, double rtol, double atol,
                              double dtol, int maxit) {
  double s[2];
  final_sum<2>(partial, RED_BLOCKS, s);
  if (threadIdx.x == 0) {
    st->rz[0] = st->rz[1] = s[0];
    st->itn[0] = st->itn[1] = 0;
    st->zz = s[1];
    st->rnorm0 = sqrt(s[1]);
    st->ttol = fmax(rtol * st->rnorm0, atol);
    st->dtol = dtol;
    st->its = 0;
    st->xalpha = 0.;
    st->maxit = maxit;
    st->yield = INT_MAX;
    st->done = 0;
    st->reason = CG_RUNNING;
    if (!(st->rnorm0 == st->rnorm0)) {
      st->done = 1;
      st->reason = CG_DIVERGED_NAN;
    } else if (st->rnorm0 <= st->ttol) {
      st->done = 1;
      st->reason = st->rnorm0 <= atol ? CG_CONVERGED_ATOL : CG_CONVERGED_RTOL;
    } else if (s[0] == 0.) {
      st->done = 1;
      st->reason = CG_CONVERGED_ATOL;
    }
  }
}

// r -= alpha w and the block partials of (r, z), (z, z) with z = D^-1 r, after w = A p: every
// block sums the operator's p.w partials (written by the apply's kernels) to the same
// alpha = (r,z)/(p,w).  The block's first packets are on their way while it does: the sum is a
// memory latency and a block reduction that would otherwise come before any of the kernel's
// traffic.  w is not read again: evict-first, so that r and dinv stay in L2 for the
// direction kernel (41.0 -> 37.2 us at 129^3 FP64 beside 43.1 -> 44.3 us there).
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) cg_update_kernel(CGVecs<T> v, CGState* st,
                                                                double* partial, int par) {
  // block 0 may set done while other blocks start: the whole block takes one view of it
  if (__syncthreads_or(st->done)) return;
  constexpr int W = Pack<T>::W;
  const int64_t np = v.n / W, t0 = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * RED_THREADS;
  Pack<T> r, w, d;
  if (t0 < np) {
    r = ld16(v.r, t0);
    w = ld16s(v.w, t0);
    d = ld16(v.dinv, t0);
  }
  double pws[1];
  final_sum<1>(v.dotp, v.ndot, pws);
  const double pw = pws[0];
  if (!(pw > 0.)) {  // same value in every block: all of them stop here
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->pw = pw;
      st->xalpha = 0.;  // no step of this iteration reaches x
      st->its = st->itn[par];
      st->done = 1;
      st->reason = (pw == pw) ? CG_DIVERGED_INDEFINITE : CG_DIVERGED_NAN;
    }
    return;
  }
  const double alpha = st->rz[par] / pw;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->pw = pw;
    st->alpha = alpha;
    st->xalpha = alpha;  // x += alpha p: in cg_p_kernel, or in cg_finish_x if the solve stops here
  }
  const T a = (T)alpha;
  double acc[2] = {0., 0.};
  for (int64_t c = t0; c < np;) {
#pragma unroll
    for (int k = 0; k < W; k++) {
      r.e[k] = r.e[k] - a * w.e[k];
      const T z = r.e[k] * d.e[k];
      acc[0] += (double)z * (double)r.e[k];
      acc[1] += (double)z * (double)z;
    }
    st16(v.r, c, r);
    c += step;
    if (c < np) {
      r = ld16(v.r, c);
      w = ld16s(v.w, c);
      d = ld16(v.dinv, c);
    }
  }
  for (int64_t i = np * W + t0; i < v.n; i += step) {
    const T ri = v.r[i] - a * v.w[i];
    const T z = ri * v.dinv[i];
    v.r[i] = ri;
    acc[0] += (double)z * (double)ri;
    acc[1] += (double)z * (double)z;
  }
  block_sum<2>(acc, partial);
}

// End of a CG iteration: every block sums the update kernel's partials to the same (r, z),
// (z, z) and takes the same decision -- convergence tests of KSPConvergedDefault on the
// preconditioned norm, or beta -- of which block 0 keeps the record; then x += alpha p and
// p = z + beta p in one pass, back from the end of the vectors: the update kernel's forward
// pass left the tail of r and dinv in L2.  As there, the first packets are on their way while
// the block sums.  (Ending the iteration in the update kernel's last block instead costs a
// fence, an atomic and that block's serial reduction.)
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) cg_p_kernel(CGVecs<T> v, CGState* st, const double* partial,
                                                           int nblk, int par) {
  // done is set from an earlier iteration, or by block 0 of this launch (which then takes the
  // same decision as this block would): the whole block takes one view of it
  if (__syncthreads_or(st->done)) return;
  constexpr int W = Pack<T>::W;
  const int64_t np = v.n / W, t0 = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * RED_THREADS;
  Pack<T> p, x, r, d;
  int64_t c = np - 1 - t0;
  auto load = [&]() {
    p = ld16(v.p, c);
    r = ld16(v.r, c);
    d = ld16(v.dinv, c);
    x = ld16(v.x, c);
  };
  if (c >= 0) load();
  double s[2];
  final_sum<2>(partial, nblk, s);
  const double rz = s[0], zz = s[1], dp = sqrt(zz), rz0 = st->rz[par];
  const int its = st->itn[par] + 1;
  int reason = CG_RUNNING;
  double beta = 0.;
  if (!(dp == dp)) {
    reason = CG_DIVERGED_NAN;
  } else if (dp <= st->ttol) {
    reason = CG_CONVERGED_RTOL;
  } else if (dp >= st->dtol * st->rnorm0) {
    reason = CG_DIVERGED_DTOL;
  } else if (its >= st->maxit) {
    reason = CG_DIVERGED_ITS;
  } else {
    beta = rz / rz0;
    if (rz == 0.) reason = CG_CONVERGED_ATOL;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->its = its;
    st->itn[par ^ 1] = its;
    st->zz = zz;
    st->beta = beta;
    st->rz[par ^ 1] = rz;
    if (reason) {
      st->reason = reason;
      st->done = 1;
    }
  }
  if (reason) return;
  const T a = (T)st->alpha, b = (T)beta;
  while (c >= 0) {
#pragma unroll
    for (int k = 0; k < W; k++) {
      x.e[k] = x.e[k] + a * p.e[k];
      p.e[k] = r.e[k] * d.e[k] + b * p.e[k];
    }
    st16(v.x, c, x);
    st16(v.p, c, p);
    c -= step;
    if (c >= 0) load();
  }
  for (int64_t i = np * W + t0; i < v.n; i += step) {
    v.x[i] = v.x[i] + a * v.p[i];
    v.p[i] = v.r[i] * v.dinv[i] + b * v.p[i];
  }
}

// ---- PCG around the multigrid V-cycle (cg.cuh)
// The V-cycle's first smoothing step from z = 0 (the product rounded).
__device__ __forceinline__ double presmooth(double dinv, double r, double inv_theta) {
  return __dmul_rn(dinv * r, inv_theta);
}
__device__ __forceinline__ float presmooth(float dinv, double r, float inv_theta) {
  return __fmul_rn(dinv * (float)r, inv_theta);
}
// Its last one, z + dinv (r - t) / theta.
__device__ __forceinline__ double postsmooth(double z, double dinv, double r, double t, double inv_theta) {
  return z + __dmul_rn(dinv * (r - t), inv_theta);
}
__device__ __forceinline__ float postsmooth(float z, float dinv, double r, float t, float inv_theta) {
  return z + __fmul_rn(dinv * ((float)r - t), inv_theta);
}

template <typename TZ>
__global__ void __launch_bounds__(RED_THREADS) mgcg_init_kernel(MgcgVecs<TZ> v, double* partial) {
  const TZ th = TZ(v.zcoef[1]);
  double acc[1] = {0.};
  GRID_LOOP(i, v.n) {
    const double r = v.b[i], z = r * v.dinv[i];
    v.x[i] = 0.;
    v.r[i] = r;
    if (v.r32) v.r32[i] = (float)r;
    v.z[i] = presmooth(v.zdinv[i], r, th);
    acc[0] += z * z;
  }
  block_sum<1>(acc, partial);
}

__global__ void __launch_bounds__(RED_THREADS) mgcg_init_final(CGState* st, const double* partial, int nblk,
                                                               double rtol, double atol, double dtol, int maxit) {
  double s[1];
  final_sum<1>(partial, nblk, s);
  if (threadIdx.x) return;
  st->rnorm0 = sqrt(s[0]);
  st->zz = s[0];
  st->ttol = fmax(rtol * st->rnorm0, atol);
  st->dtol = dtol;
  st->its = 0;
  st->xalpha = 0.;
  st->maxit = maxit;
  st->yield = INT_MAX;
  st->done = 0;
  st->reason = CG_RUNNING;
  if (!(st->rnorm0 == st->rnorm0)) {
    st->done = 1;
    st->reason = CG_DIVERGED_NAN;
  } else if (st->rnorm0 <= st->ttol) {
    st->done = 1;
    st->reason = st->rnorm0 <= atol ? CG_CONVERGED_ATOL : CG_CONVERGED_RTOL;
  }
}

template <typename TZ> struct Two {
  TZ x, y;
};
__device__ __forceinline__ Two<double> ld2(const double* a, int64_t c) {
  const double2 q = reinterpret_cast<const double2*>(a)[c];
  return {q.x, q.y};
}
__device__ __forceinline__ Two<float> ld2(const float* a, int64_t c) {
  const float2 q = reinterpret_cast<const float2*>(a)[c];
  return {q.x, q.y};
}
__device__ __forceinline__ void st2(double* a, int64_t c, double x, double y) {
  reinterpret_cast<double2*>(a)[c] = make_double2(x, y);
}
__device__ __forceinline__ void st2(float* a, int64_t c, float x, float y) {
  reinterpret_cast<float2*>(a)[c] = make_float2(x, y);
}

template <typename TZ>
__global__ void __launch_bounds__(RED_THREADS) mgcg_smooth_rz_kernel(MgcgVecs<TZ> v, const CGState* st,
                                                                     double* partial) {
  if (__syncthreads_or(st->done)) return;
  const TZ th = TZ(v.zcoef[1]);
  double acc[1] = {0.};
  const int64_t np = v.n / 2, t0 = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * RED_THREADS;
  for (int64_t c = t0; c < np; c += step) {
    const Two<double> r = ld2(v.r, c);
    const Two<TZ> z = ld2(v.z, c), t = ld2(v.t, c), d = ld2(v.zdinv, c);
    const TZ zx = postsmooth(z.x, d.x, r.x, t.x, th), zy = postsmooth(z.y, d.y, r.y, t.y, th);
    st2(v.z, c, zx, zy);
    acc[0] += r.x * (double)zx;
    acc[0] += r.y * (double)zy;
  }
  for (int64_t i = 2 * np + t0; i < v.n; i += step) {
    const TZ z = postsmooth(v.z[i], v.zdinv[i], v.r[i], v.t[i], th);
    v.z[i] = z;
    acc[0] += v.r[i] * (double)z;
  }
  block_sum<1>(acc, partial);
}

// x += alpha p (the iteration before) and p = z + beta p; the first iteration has neither.  The
// parity of the finished iterations, which only the end of an iteration moves, picks the
// (r, z) that every block reads and the one that block 0 leaves.
template <typename TZ>
__global__ void __launch_bounds__(RED_THREADS) mgcg_p_kernel(MgcgVecs<TZ> v, CGState* st, const double* partial,
                                                             int nblk) {
  if (__syncthreads_or(st->done)) return;
  const int64_t np = v.n / 2, t0 = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * RED_THREADS;
  const int its = st->its, par = its & 1;
  Two<double> p{0., 0.}, x = p;
  Two<TZ> z{TZ(0), TZ(0)};
  auto load = [&](int64_t c) {
    z = ld2(v.z, c);
    if (its) {
      p = ld2(v.p, c);
      x = ld2(v.x, c);
    }
  };
  if (t0 < np) load(t0);
  double s[1];
  final_sum<1>(partial, nblk, s);
  const double rz = s[0];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->rz[par ^ 1] = rz;
    if (!(rz > 0.)) {
      st->reason = rz == 0. ? CG_CONVERGED_ATOL : CG_DIVERGED_INDEFINITE;
      st->done = 1;
    }
  }
  if (!(rz > 0.)) return;
  const double b = its ? rz / st->rz[par] : 0., a = st->xalpha;
  for (int64_t c = t0; c < np;) {
    double qx = z.x, qy = z.y;
    if (its) {
      st2(v.x, c, x.x + a * p.x, x.y + a * p.y);
      qx += b * p.x;
      qy += b * p.y;
    }
    st2(v.p, c, qx, qy);
    c += step;
    if (c < np) load(c);
  }
  for (int64_t i = 2 * np + t0; i < v.n; i += step) {
    const double zi = v.z[i];
    if (its) v.x[i] += a * v.p[i];
    v.p[i] = its ? zi + b * v.p[i] : zi;
  }
}

template <typename TZ>
__global__ void __launch_bounds__(RED_THREADS) mgcg_update_kernel(MgcgVecs<TZ> v, CGState* st, double* partial) {
  if (__syncthreads_or(st->done)) return;
  const int64_t np = v.n / 2, t0 = (int64_t)blockIdx.x * RED_THREADS + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * RED_THREADS;
  Two<double> r{0., 0.}, w = r, d = r;
  Two<TZ> zd{TZ(0), TZ(0)};
  const TZ th = TZ(v.zcoef[1]);
  auto load = [&](int64_t c) {
    r = ld2(v.r, c);
    w = ld2(v.w, c);
    d = ld2(v.dinv, c);
    zd = ld2(v.zdinv, c);
  };
  if (t0 < np) load(t0);
  double pws[1];
  final_sum<1>(v.dotp, v.ndot, pws);
  const double pw = pws[0];
  if (!(pw > 0.)) {  // same value in every block; x and r stay as they are
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->pw = pw;
      st->xalpha = 0.;
      st->done = 1;
      st->reason = (pw == pw) ? CG_DIVERGED_INDEFINITE : CG_DIVERGED_NAN;
    }
    return;
  }
  const double alpha = st->rz[(st->its & 1) ^ 1] / pw;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->pw = pw;
    st->alpha = alpha;
    st->xalpha = alpha;
  }
  double acc[1] = {0.};
  for (int64_t c = t0; c < np;) {
    r.x += -alpha * w.x;
    r.y += -alpha * w.y;
    const double zx = r.x * d.x, zy = r.y * d.y;
    acc[0] += zx * zx;
    acc[0] += zy * zy;
    st2(v.r, c, r.x, r.y);
    if (v.r32) st2(v.r32, c, (float)r.x, (float)r.y);
    st2(v.z, c, presmooth(zd.x, r.x, th), presmooth(zd.y, r.y, th));
    c += step;
    if (c < np) load(c);
  }
  for (int64_t i = 2 * np + t0; i < v.n; i += step) {
    const double ri = v.r[i] - alpha * v.w[i], zi = ri * v.dinv[i];
    v.r[i] = ri;
    if (v.r32) v.r32[i] = (float)ri;
    v.z[i] = presmooth(v.zdinv[i], ri, th);
    acc[0] += zi * zi;
  }
  block_sum<1>(acc, partial);
}

// The step of the iteration that stopped the solve (its cg_p_kernel did not run):
// x += xalpha p; nothing after an indefinite p.w (xalpha = 0) or while the solve is
// still going (a watchdog stop between iterations: every step has reached x).
template <typename T>
__global__ void cg_finish_x_kernel(CGVecs<T> v, const CGState* st) {
  if (!st->done) return;
  const double alpha = st->xalpha;
  if (alpha == 0.) return;
  const T a = (T)alpha;
  pack_loop<T>(
      v.n,
      [&](int64_t c) {
        Pack<T> x = ld16(v.x, c);
        const Pack<T> p = ld16(v.p, c);
#pragma unroll
        for (int k = 0; k < Pack<T>::W; k++) x.e[k] = x.e[k] + a * p.e[k];
        st16(v.x, c, x);
      },
      [&](int64_t i) { v.x[i] = v.x[i] + a * v.p[i]; });
}

// ---- generic vector kernels ----
template <int K> struct PtrPack {
  const double* p[K];
};

template <int K>
__global__ void __launch_bounds__(RED_THREADS) dots_kernel(PtrPack<K> a, PtrPack<K> b, int64_t n,
                                                           double* partial) {
  double acc[K];
#pragma unroll
  for (int q = 0; q < K; q++) acc[q] = 0.;
  GRID_LOOP(i, n) {
#pragma unroll
    for (int q = 0; q < K; q++) acc[q] += a.p[q][i] * b.p[q][i];
  }
  block_sum<K>(acc, partial);
}

template <int K>
__global__ void dots_final(const double* partial, double* out) {
  double s[K];
  final_sum<K>(partial, RED_BLOCKS, s);
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < K; q++) out[q] = s[q];
}

__global__ void __launch_bounds__(RED_THREADS) absmax_diff_kernel(const double* a, const double* b,
                                                                  int64_t n, double* partial) {
  __shared__ double red[RED_THREADS];
  double m = 0.;
  GRID_LOOP(i, n) m = fmax(m, fabs(a[i] - b[i]));
  red[threadIdx.x] = m;
  __syncthreads();
  for (int st = RED_THREADS / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + st]);
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

__global__ void absmax_final(const double* partial, double* out) {
  if (threadIdx.x == 0) {
    double m = 0.;
    for (int b = 0; b < RED_BLOCKS; b++) m = fmax(m, partial[b]);
    out[0] = m;
  }
}

// F = y - f on free dofs, F = u - ubc on Dirichlet dofs (ResidualApplyDirichletBC).
__global__ void u_residual_kernel(const double* y, const double* f, const double* u,
                                  const uint8_t* kind, const double* bcu, double* F, int64_t n3) {
  GRID_LOOP(i, n3) {
    const int k = kind ? kind[i] : 0;
    if (k == 0)
      F[i] = y[i] - f[i];
    else
      F[i] = u[i] - (k == 1 ? 0. : k == 2 ? 1. : bcu[i]);
  }
}

// U := Dirichlet value on Dirichlet dofs (VecApplyDirichletBC).
__global__ void apply_bc_kernel(double* u, const uint8_t* kind, const double* bcu, int64_t n) {
  GRID_LOOP(i, n) {
    const int k = kind[i];
    if (k) u[i] = k == 1 ? 0. : k == 2 ? 1. : (bcu ? bcu[i] : u[i]);
  }
}

__global__ void axpy_kernel(double* y, double a, const double* x, int64_t n) {
  GRID_LOOP(i, n) y[i] += a * x[i];
}
__global__ void axpby_kernel(double* z, const double* x, double a, const double* y, int64_t n) {
  GRID_LOOP(i, n) z[i] = x[i] + a * y[i];
}
__global__ void inv_kernel(const double* d, double* dinv, float* dinv32, int64_t n) {
  GRID_LOOP(i, n) {
    const double r = 1. / d[i];
    dinv[i] = r;
    if (dinv32) dinv32[i] = (float)r;
  }
}
__global__ void to_f32_kernel(const double* x, float* y, int64_t n) {
  GRID_LOOP(i, n) y[i] = (float)x[i];
}
__global__ void add_f32_kernel(double* y, const float* x, int64_t n) {
  GRID_LOOP(i, n) y[i] += (double)x[i];
}

// ---- V (phase field) ----
// F_V = y - b; AT2 irreversibility rows 0 (VF_IrrevApplyEQVec); BC rows v - bc.
__global__ void v_residual_kernel(const double* y, const double* b, const double* v,
                                  const double* virrev, const uint8_t* kind, double irrevtol,
                                  int at2, double* F, int64_t n) {
  GRID_LOOP(i, n) {
    double f = y[i] - b[i];
    if (at2 && virrev[i] <= irrevtol) f = 0.;
    const int k = kind ? kind[i] : 0;
    if (k) f = v[i] - (k == 1 ? 0. : k == 2 ? 1. : v[i]);
    F[i] = f;
  }
}

// VI norm (SNESVIComputeInactiveSetFnorm) partial sums.
__global__ void __launch_bounds__(RED_THREADS) vi_norm_kernel(const double* F, const double* x,
                                                              const double* lb, const double* ub,
                                                              int64_t n, double* partial) {
  double acc[1] = {0.};
  GRID_LOOP(i, n) {
    const double f = F[i];
    if ((x[i] > lb[i] + 1.e-8 || f <= 0.) && (x[i] < ub[i] - 1.e-8 || f >= 0.)) acc[0] += f * f;
  }
  block_sum<1>(acc, partial);
}

// Active set of SNESVINEWTONRSLS (x at a bound with F pushing outward) plus the
// dofs removed from the reduced system (Dirichlet rows, AT2 irreversibility).
__global__ void v_mask_kernel(const double* F, const double* x, const double* lb, const double* ub,
                              const double* virrev, const uint8_t* kind, double irrevtol, int at2,
                              uint8_t* mask, int64_t n) {
  GRID_LOOP(i, n) {
    const double f = F[i];
    const bool inactive = (x[i] > lb[i] + 1.e-8 || f < 0.) && (x[i] < ub[i] - 1.e-8 || f > 0.);
    const bool fixed = (kind && kind[i]) || (at2 && virrev[i] <= irrevtol);
    mask[i] = (!inactive || fixed) ? 1 : 0;
  }
}

// Newton step on the removed dofs: Dirichlet rows are identity (Y = F), active
// and irreversible dofs do not move.
__global__ void v_fix_step_kernel(double* Y, const double* F, const uint8_t* mask,
                                  const uint8_t* kind, int64_t n) {
  GRID_LOOP(i, n) {
    if (mask[i]) Y[i] = (kind && kind[i]) ? F[i] : 0.;
  }
}

// W = clamp(v - lambda Y, lb, ub) (SNESVIProjectOntoBounds), and partial |W - v|^2.
__global__ void __launch_bounds__(RED_THREADS) v_project_kernel(const double* v, const double* Y,
                                                                double lambda, const double* lb,
                                                                const double* ub, double* W,
                                                                int64_t n, double* partial) {
  double acc[1] = {0.};
  GRID_LOOP(i, n) {
    const double w = fmin(fmax(v[i] - lambda * Y[i], lb[i]), ub[i]);
    W[i] = w;
    acc[0] += (w - v[i]) * (w - v[i]);
  }
  block_sum<1>(acc, partial);
}

__global__ void v_bounds_kernel(const double* virrev, int at1, double* lb, double* ub, double* v,
                                int64_t n) {
  GRID_LOOP(i, n) {
    const double l = 0., u = at1 ? virrev[i] : 1.;
    lb[i] = l;
    ub[i] = u;
    v[i] = fmin(fmax(v[i], l), u);
  }
}

inline int vgrid(int64_t n) { return (int)std::min<int64_t>((n + 255) / 256, 148 * 16); }

}  // namespace

// ------------------------------------------------------------------ host wrappers
template <typename T>
cudaError_t cg_init(const CGVecs<T>& v, CGState* st, double* partial, double rtol, double atol,
                    double dtol, int maxit, cudaStream_t s) {
  cg_init_kernel<T><<<RED_BLOCKS, RED_THREADS, 0, s>>>(v, partial);
  cg_init_final<<<1, RED_THREADS, 0, s>>>(st, partial, rtol, atol, dtol, maxit);
  return cudaGetLastError();
}

template <typename T> static bool aligned16(const CGVecs<T>& v) {
  const void* ps[] = {v.x, v.r, v.p, v.w, v.dinv};
  for (const void* p : ps)
    if (reinterpret_cast<uintptr_t>(p) % 16) return false;
  return true;
}

template <typename T>
cudaError_t cg_iteration(const CGVecs<T>& v, CGState* st, double* partial, int par, cudaStream_t s) {
  if (!aligned16(v)) return cudaErrorMisalignedAddress;  // caught on the host, nothing launched
  if (!v.dotp || v.ndot <= 0) return cudaErrorInvalidValue;
  const int nb = cg_blocks(v.n, (int)sizeof(T));
  cg_update_kernel<T><<<nb, RED_THREADS, 0, s>>>(v, st, partial, par);
  cg_p_kernel<T><<<nb, RED_THREADS, 0, s>>>(v, st, partial, nb, par);
  return cudaGetLastError();
}

template <typename T>
cudaError_t cg_finish_x(const CGVecs<T>& v, const CGState* st, cudaStream_t s) {
  if (reinterpret_cast<uintptr_t>(v.x) % 16 || reinterpret_cast<uintptr_t>(v.p) % 16) return cudaErrorMisalignedAddress;
  cg_finish_x_kernel<T><<<RED_BLOCKS, RED_THREADS, 0, s>>>(v, st);
  return cudaGetLastError();
}

template cudaError_t cg_init<double>(const CGVecs<double>&, CGState*, double*, double, double,
                                     double, int, cudaStream_t);
template cudaError_t cg_init<float>(const CGVecs<float>&, CGState*, double*, double, double,
                                    double, int, cudaStream_t);
// r.z partials in partial[0, RED_BLOCKS), those of the stopping test in the next RED_BLOCKS
template <typename TZ>
cudaError_t mgcg_init(const MgcgVecs<TZ>& v, CGState* st, double* partial, double rtol, double atol, double dtol,
                      int maxit, cudaStream_t s) {
  for (const void* q : {(const void*)v.x, (const void*)v.r, (const void*)v.p, (const void*)v.w, (const void*)v.dinv,
                        (const void*)v.z, (const void*)v.r32, (const void*)v.t, (const void*)v.zdinv})
    if (reinterpret_cast<uintptr_t>(q) % 16) return cudaErrorMisalignedAddress;
  if (!v.dotp || v.ndot <= 0) return cudaErrorInvalidValue;
  mgcg_init_kernel<TZ><<<RED_BLOCKS, RED_THREADS, 0, s>>>(v, partial);
  mgcg_init_final<<<1, RED_THREADS, 0, s>>>(st, partial, RED_BLOCKS, rtol, atol, dtol, maxit);
  return cudaGetLastError();
}
template <typename TZ>
cudaError_t mgcg_direction(const MgcgVecs<TZ>& v, CGState* st, double* partial, cudaStream_t s) {
  const int nb = cg_blocks(v.n, 8);
  mgcg_smooth_rz_kernel<TZ><<<nb, RED_THREADS, 0, s>>>(v, st, partial);
  mgcg_p_kernel<TZ><<<nb, RED_THREADS, 0, s>>>(v, st, partial, nb);
  return cudaGetLastError();
}
template <typename TZ>
cudaError_t mgcg_update(const MgcgVecs<TZ>& v, CGState* st, double* partial, cudaStream_t s) {
  mgcg_update_kernel<TZ><<<cg_blocks(v.n, 8), RED_THREADS, 0, s>>>(v, st, partial + RED_BLOCKS);
  return cudaGetLastError();
}
template cudaError_t mgcg_init<double>(const MgcgVecs<double>&, CGState*, double*, double, double, double, int,
                                       cudaStream_t);
template cudaError_t mgcg_init<float>(const MgcgVecs<float>&, CGState*, double*, double, double, double, int,
                                      cudaStream_t);
template cudaError_t mgcg_direction<double>(const MgcgVecs<double>&, CGState*, double*, cudaStream_t);
template cudaError_t mgcg_direction<float>(const MgcgVecs<float>&, CGState*, double*, cudaStream_t);
template cudaError_t mgcg_update<double>(const MgcgVecs<double>&, CGState*, double*, cudaStream_t);
template cudaError_t mgcg_update<float>(const MgcgVecs<float>&, CGState*, double*, cudaStream_t);

template cudaError_t cg_iteration<double>(const CGVecs<double>&, CGState*, double*, int, cudaStream_t);
template cudaError_t cg_iteration<float>(const CGVecs<float>&, CGState*, double*, int, cudaStream_t);
template cudaError_t cg_finish_x<double>(const CGVecs<double>&, const CGState*, cudaStream_t);
template cudaError_t cg_finish_x<float>(const CGVecs<float>&, const CGState*, cudaStream_t);

template <int K>
static void launch_dots(const double* const* a, const double* const* b, int64_t n, double* partial,
                        double* out, cudaStream_t s) {
  PtrPack<K> pa, pb;
  for (int q = 0; q < K; q++) {
    pa.p[q] = a[q];
    pb.p[q] = b[q];
  }
  dots_kernel<K><<<RED_BLOCKS, RED_THREADS, 0, s>>>(pa, pb, n, partial);
  dots_final<K><<<1, RED_THREADS, 0, s>>>(partial, out);
}

cudaError_t dev_dots(const double* const* a, const double* const* b, int k, int64_t n,
                     double* partial, double* out, cudaStream_t s) {
  // a, b: host arrays of k device pointers; out[q] = a[q] . b[q] (device memory)
  switch (k) {
    case 1: launch_dots<1>(a, b, n, partial, out, s); break;
    case 2: launch_dots<2>(a, b, n, partial, out, s); break;
    case 3: launch_dots<3>(a, b, n, partial, out, s); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

namespace {
__global__ void __launch_bounds__(RED_THREADS) znorm_kernel(const double* r, const double* dinv,
                                                            int64_t n, double* partial) {
  double acc[1] = {0.};
  GRID_LOOP(i, n) {
    const double z = r[i] * dinv[i];
    acc[0] += z * z;
  }
  block_sum<1>(acc, partial);
}
}  // namespace

cudaError_t dev_znorm2(const double* r, const double* dinv, int64_t n, double* partial,
                       double* out, cudaStream_t s) {
  znorm_kernel<<<RED_BLOCKS, RED_THREADS, 0, s>>>(r, dinv, n, partial);
  dots_final<1><<<1, RED_THREADS, 0, s>>>(partial, out);
  return cudaGetLastError();
}

cudaError_t dev_absmax_diff(const double* a, const double* b, int64_t n, double* partial,
                            double* out, cudaStream_t s) {
  absmax_diff_kernel<<<RED_BLOCKS, RED_THREADS, 0, s>>>(a, b, n, partial);
  absmax_final<<<1, 32, 0, s>>>(partial, out);
  return cudaGetLastError();
}

cudaError_t dev_u_residual(const double* y, const double* f, const double* u, const uint8_t* kind,
                           const double* bcu, double* F, int64_t n3, cudaStream_t s) {
  u_residual_kernel<<<vgrid(n3), 256, 0, s>>>(y, f, u, kind, bcu, F, n3);
  return cudaGetLastError();
}
cudaError_t dev_apply_bc(double* u, const uint8_t* kind, const double* bcu, int64_t n,
                         cudaStream_t s) {
  apply_bc_kernel<<<vgrid(n), 256, 0, s>>>(u, kind, bcu, n);
  return cudaGetLastError();
}
cudaError_t dev_axpy(double* y, double a, const double* x, int64_t n, cudaStream_t s) {
  axpy_kernel<<<vgrid(n), 256, 0, s>>>(y, a, x, n);
  return cudaGetLastError();
}
cudaError_t dev_axpby(double* z, const double* x, double a, const double* y, int64_t n,
                      cudaStream_t s) {
  axpby_kernel<<<vgrid(n), 256, 0, s>>>(z, x, a, y, n);
  return cudaGetLastError();
}
cudaError_t dev_inv(const double* d, double* dinv, float* dinv32, int64_t n, cudaStream_t s) {
  inv_kernel<<<vgrid(n), 256, 0, s>>>(d, dinv, dinv32, n);
  return cudaGetLastError();
}
cudaError_t dev_to_f32(const double* x, float* y, int64_t n, cudaStream_t s) {
  to_f32_kernel<<<vgrid(n), 256, 0, s>>>(x, y, n);
  return cudaGetLastError();
}
cudaError_t dev_add_f32(double* y, const float* x, int64_t n, cudaStream_t s) {
  add_f32_kernel<<<vgrid(n), 256, 0, s>>>(y, x, n);
  return cudaGetLastError();
}
cudaError_t dev_v_residual(const double* y, const double* b, const double* v, const double* virrev,
                           const uint8_t* kind, double irrevtol, int at2, double* F, int64_t n,
                           cudaStream_t s) {
  v_residual_kernel<<<vgrid(n), 256, 0, s>>>(y, b, v, virrev, kind, irrevtol, at2, F, n);
  return cudaGetLastError();
}
cudaError_t dev_vi_norm2(const double* F, const double* x, const double* lb, const double* ub,
                         int64_t n, double* partial, double* out, cudaStream_t s) {
  vi_norm_kernel<<<RED_BLOCKS, RED_THREADS, 0, s>>>(F, x, lb, ub, n, partial);
  dots_final<1><<<1, RED_THREADS, 0, s>>>(partial, out);
  return cudaGetLastError();
}
cudaError_t dev_v_mask(const double* F, const double* x, const double* lb, const double* ub,
                       const double* virrev, const uint8_t* kind, double irrevtol, int at2,
                       uint8_t* mask, int64_t n, cudaStream_t s) {
  v_mask_kernel<<<vgrid(n), 256, 0, s>>>(F, x, lb, ub, virrev, kind, irrevtol, at2, mask, n);
  return cudaGetLastError();
}
cudaError_t dev_v_fix_step(double* Y, const double* F, const uint8_t* mask, const uint8_t* kind,
                           int64_t n, cudaStream_t s) {
  v_fix_step_kernel<<<vgrid(n), 256, 0, s>>>(Y, F, mask, kind, n);
  return cudaGetLastError();
}
cudaError_t dev_v_project(const double* v, const double* Y, double lambda, const double* lb,
                          const double* ub, double* W, int64_t n, double* partial, double* out,
                          cudaStream_t s) {
  v_project_kernel<<<RED_BLOCKS, RED_THREADS, 0, s>>>(v, Y, lambda, lb, ub, W, n, partial);
  dots_final<1><<<1, RED_THREADS, 0, s>>>(partial, out);
  return cudaGetLastError();
}
cudaError_t dev_v_bounds(const double* virrev, int at1, double* lb, double* ub, double* v,
                         int64_t n, cudaStream_t s) {
  v_bounds_kernel<<<vgrid(n), 256, 0, s>>>(virrev, at1, lb, ub, v, n);
  return cudaGetLastError();
}

}  // namespace vfgpu
