// common.cuh -- shared helpers for the vfgpu kernels (sm_100a).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace vfgpu {

// 1-D 3-point Gauss rule on the reference interval t in [-1/2, 1/2]
// (VFCartFE.c:100-107: nodes (1 -+ sqrt(3/5))/2 on [0,1], weights 5/18, 8/18, 5/18).
#define VF_TAU 0.38729833462074168852   /* sqrt(3/5)/2 */
#define VF_W0 0.27777777777777777778    /* 5/18 */
#define VF_W1 0.44444444444444444444    /* 8/18 */

// Element-layer material table (per-layer VFMatProp, VFCommon.h:69-80).
#define VF_MAXLAYER 16
struct LayerTable {
  double lambda[VF_MAXLAYER];   // Lame lambda (VFCommon.c:584)
  double mu[VF_MAXLAYER];       // Lame mu     (VFCommon.c:585)
  double lamfac[VF_MAXLAYER];   // lambda / E  (for per-cell E)
  double mufac[VF_MAXLAYER];    // mu / E
  double alpha[VF_MAXLAYER];    // thermal expansion
  double beta[VF_MAXLAYER];     // Biot coefficient
  double Gc[VF_MAXLAYER];
};

// Coefficients of the U operator's separable stencil (u_stencil.cuh) at spacing (h0, h1, h2)
// for the axes (0, 1, 2), rounded once: of 6 P, 36 Q and 36 R from sums over 6 m and 36 m m.
struct StencilCoefs {
  double xx, xy, yx, yy, xd, q, qz, rx, ry;
  double g;               // R's multiple on the lowest plane
  double em, el, fl, fm;  // a face across axis 1, its missing half: of P_0, P_1; of R_1, R_2
};
inline StencilCoefs stencil_coefs(double lambda, double mu_, double d0, double d1, double d2) {
  const long double lam = lambda, mu = mu_, h0 = d0, h1 = d1, h2 = d2, l2 = lam + 2 * mu, lm = lam + mu;
  const long double a0 = h1 * h2 / h0, a1 = h0 * h2 / h1, a2 = h0 * h1 / h2;
  StencilCoefs c;
  c.xx = (double)(-l2 * a0);
  c.xy = (double)(-mu * a1);
  c.yx = (double)(-mu * a0);
  c.yy = (double)(-l2 * a1);
  c.xd = (double)(-1.5L * lm * h2);
  c.q = (double)(-mu * a2);
  c.qz = (double)(-l2 * a2);
  c.rx = (double)(-1.5L * lm * h1);
  c.ry = (double)(-1.5L * lm * h0);
  c.g = (double)((mu - lam) / lm);
  c.em = (double)(3 * mu * h2);
  c.el = (double)(3 * lam * h2);
  c.fl = (double)(3 * lam * h0);
  c.fm = (double)(3 * mu * h0);
  return c;
}

// Per-problem parameters the operator kernels read through a device pointer, so
// that captured CUDA graphs stay valid when a ctx is re-used for another problem
// (set-up calls rewrite this block instead of the kernels' by-value arguments).
struct DevParams {
  LayerTable L;
  double eta;                  // eta (VFProp.eta)
  StencilCoefs st[2];          // layer 0: axes x, y, z, and y, x, z (the U stencil)
};

template <typename T> struct Vec3 { T x, y, z; };

__host__ __device__ inline int64_t node_index(int i, int j, int k, int nx, int ny) {
  return ((int64_t)k * ny + j) * nx + i;
}

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Deterministic sum of one double per thread over a block (any 1-3D shape with a
// multiple of 32 threads): warp shuffle trees, then warp 0 sums the warp totals in
// order.  `scratch` is shared memory for >= 32 doubles; every thread must call
// (it contains a barrier); the result is valid in thread 0.
__device__ __forceinline__ double block_sum_dbl(double v, double* scratch) {
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nw = (blockDim.x * blockDim.y * blockDim.z) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((tid & 31) == 0) scratch[tid >> 5] = v;
  __syncthreads();
  double s = 0.;
  if (tid == 0)
    for (int w = 0; w < nw; w++) s += scratch[w];
  return s;
}

}  // namespace vfgpu
