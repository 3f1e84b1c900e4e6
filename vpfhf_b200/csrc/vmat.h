// vmat.h -- the assembled damage operator K_V (VF_BilinearFormVAT1/AT23D_local +
// VF_BilinearFormVCoupling3D_local, VFMech.c:2040-2115) as a symmetric 27-point stencil:
// per node its own entry and the 13 couplings to the neighbours ahead of it in (z, y, x)
// order, one array per coupling, a[d * vmat_stride(N) + node]; couplings that leave the
// grid are 0; and the row sums, which are the sums of the mass part alone (the stiffness
// part's are 0): the apply takes its differences with them.  120 bytes per node in FP64,
// against 216 for the element form's 27 Gauss-point coefficients per cell.
#pragma once

#include "common.cuh"

namespace vfgpu {

constexpr int kVCouplings = 14;
constexpr int kVRowSum = kVCouplings, kVArrays = kVCouplings + 1;
// (dx, dy, dz) of each coupling
__host__ __device__ constexpr int kVForward[kVCouplings][3] = {
    {0, 0, 0},  {1, 0, 0}, {-1, 1, 0}, {0, 1, 0}, {1, 1, 0},  {-1, -1, 1}, {0, -1, 1},
    {1, -1, 1}, {-1, 0, 1}, {0, 0, 1},  {1, 0, 1}, {-1, 1, 1}, {0, 1, 1},   {1, 1, 1}};
__host__ __device__ inline int64_t vmat_stride(int64_t n) { return (n + 31) & ~int64_t(31); }

template <typename T> struct VMatArgs {
  const T* __restrict__ a;           // kVArrays arrays: couplings, row sums
  const T* __restrict__ x;           // N input; must be 0 on masked dofs (the reduced-space CG
                                     // keeps its directions 0 there), which makes the masked
                                     // columns drop out
  T* __restrict__ y;                 // N output
  const uint8_t* __restrict__ mask;  // N: nonzero => dof removed (y = 0); or null
  const int* __restrict__ skip;      // if non-null and *skip != 0 the launch does nothing
  double* __restrict__ dot;          // if non-null: vmat_blocks() partials of x.y
  int nx, ny, nz;
};
// Blocks of one launch (and x.y partials it writes).
int vmat_blocks(int64_t n);
// y = K_V x with the masked rows 0; T = double or float.
template <typename T> cudaError_t launch_vmat_apply(const VMatArgs<T>& A, cudaStream_t s);

}  // namespace vfgpu
