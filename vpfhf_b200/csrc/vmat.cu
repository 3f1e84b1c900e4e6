// vmat.cu -- y = K_V x with the assembled couplings (vmat.h).
#include <algorithm>

#include "vmat.h"

namespace vfgpu {

namespace {

constexpr int VM_THREADS = 256;
// 4 blocks of 256 threads on each of 148 SMs: one wave
constexpr int VM_BLOCKS = 592;

// One thread per node, nodes in memory order, one wave of blocks that sweeps the planes
// together, so that the 13 couplings a node shares with the nodes behind it (the planes just
// read) come from L1 and L2 and HBM sees each coupling once.  A masked node costs its mask
// byte: where the bounds are active (most of the grid in an AT1 problem) whole warps leave
// at once.  On the faces of the box (FACE) the neighbours that do not exist are left out by
// their coordinates, not by their zero couplings: in memory order the node one past a row's end
// is the next row's first, and 0 times a value that is not finite there would reach this row.
// A row is sum_j a_j x_j = (sum_j a_j) r + sum_j a_j (x_j - r) for any r: with r a mean of the node
// (1/4) and its 6 face neighbours (1/8 each) no full-size products cancel, neither where the
// stiffness part dominates and x is smooth nor where the mass part does.  Normwise error of
// one FP32 apply, element form / plain products / this form, in 1e-8 (x random, smooth): no mass
// part 6.1 / 11.5 / 5.1, 338 / 788 / 8.7; mass 30 times the stiffness 6.8 / 13.0 / 5.1, 5.6 / 10.8
// / 3.2; FP64 alike.  (With r = x of the node and one sum 7.7 and 19 for x random.)
// Measured at 129^3 inside the AT1 penny crack's StepV (few nodes free): 7.9 us a launch in
// FP64 and 4.4 us in FP32, where the element form with its staged coefficients took 63.5 + 4.5
// (seams) and 33.7 + 2.8 us (averages over a solve's launches, finished ones included); with
// every node free 102 us in FP64 (element form 96 + 8.7; the plain products 96).  A warp takes one form
// of the row: with a branch per node nearly every warp of a 65^3 grid ran both (AT2 multigrid AM step 65^3
// 21.5 -> 21.1 ms).
template <typename T, bool FACE>
__device__ __forceinline__ T vmat_row(const VMatArgs<T>& A, int64_t n, int i, int j, int k, int64_t st) {
  const int64_t row = A.nx, pl = (int64_t)A.nx * A.ny;
  // whether the neighbour one step along -, 0, + of an axis exists
  const bool ex[3] = {i > 0, true, i < A.nx - 1}, ey[3] = {j > 0, true, j < A.ny - 1},
             ez[3] = {k > 0, true, k < A.nz - 1};
  const T x0 = A.x[n];
  T m = T(0);  // 8 times the reference value
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const int64_t o = q == 0 ? 1 : q == 1 ? row : pl;
    const bool hi = q == 0 ? ex[2] : q == 1 ? ey[2] : ez[2], lo = q == 0 ? ex[0] : q == 1 ? ey[0] : ez[0];
    m += (!FACE || hi ? A.x[n + o] : x0) + (!FACE || lo ? A.x[n - o] : x0);
  }
  const T ref = T(0.125) * fma(T(2), x0, m);
  T s[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
  for (int d = 1; d < kVCouplings; d++) {
    const int dx = kVForward[d][0], dy = kVForward[d][1], dz = kVForward[d][2];
    const int64_t o = dx + dy * row + dz * pl;
    T &f = s[d & 1], &b = s[2 + (d & 1)];
    if (!FACE || (ex[1 + dx] && ey[1 + dy] && ez[1 + dz])) f = fma(A.a[d * st + n], A.x[n + o] - ref, f);
    if (!FACE || (ex[1 - dx] && ey[1 - dy] && ez[1 - dz])) b = fma(A.a[d * st + n - o], A.x[n - o] - ref, b);
  }
  return fma(A.a[kVRowSum * st + n], ref, fma(A.a[n], x0 - ref, (s[0] + s[1]) + (s[2] + s[3])));
}

template <typename T, bool DOT>
__global__ void __launch_bounds__(VM_THREADS, 4) vmat_apply_kernel(const __grid_constant__ VMatArgs<T> A) {
  __shared__ double red[32];
  if (A.skip && *A.skip) return;  // converged solve
  const int64_t N = (int64_t)A.nx * A.ny * A.nz, st = vmat_stride(N);
  const unsigned nx = A.nx, ny = A.ny;
  double acc = 0.;
  for (int64_t n = (int64_t)blockIdx.x * VM_THREADS + threadIdx.x; n < N; n += (int64_t)gridDim.x * VM_THREADS) {
    T y = T(0);
    if (!(A.mask && A.mask[n])) {
      // (N < 2^32: 14 couplings of 2^32 nodes do not fit a device)
      const unsigned m = (unsigned)n, rows = m / nx;
      const int i = (int)(m - rows * nx), k = (int)(rows / ny), j = (int)(rows - (unsigned)k * ny);
      const bool face = i == 0 || i == A.nx - 1 || j == 0 || j == A.ny - 1 || k == 0 || k == A.nz - 1;
      // one form for the whole warp (the same bits where no neighbour is missing)
      y = __any_sync(__activemask(), face) ? vmat_row<T, true>(A, n, i, j, k, st) : vmat_row<T, false>(A, n, i, j, k, st);
      if constexpr (DOT) acc += (double)A.x[n] * (double)y;
    }
    A.y[n] = y;
  }
  if constexpr (DOT) {
    const double s = block_sum_dbl(acc, red);
    if (threadIdx.x == 0) A.dot[blockIdx.x] = s;
  }
}

}  // namespace

int vmat_blocks(int64_t n) { return (int)std::min<int64_t>(VM_BLOCKS, (n + VM_THREADS - 1) / VM_THREADS); }

template <typename T> cudaError_t launch_vmat_apply(const VMatArgs<T>& A, cudaStream_t s) {
  const int b = vmat_blocks((int64_t)A.nx * A.ny * A.nz);
  if (A.dot) vmat_apply_kernel<T, true><<<b, VM_THREADS, 0, s>>>(A);
  else vmat_apply_kernel<T, false><<<b, VM_THREADS, 0, s>>>(A);
  return cudaGetLastError();
}
template cudaError_t launch_vmat_apply<double>(const VMatArgs<double>&, cudaStream_t);
template cudaError_t launch_vmat_apply<float>(const VMatArgs<float>&, cudaStream_t);

}  // namespace vfgpu
