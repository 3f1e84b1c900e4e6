// u_twophase.cuh -- the U operator on small grids: every element by itself, then every node.
//
// The tile engine marches tiles of 32 x 8 elements up the planes: on a small grid a block has
// one to three planes, recomputes the element layer below them and runs its layers one after
// the other at 8 warps per SM, so the apply is a chain of element latencies whatever the size.
// Here one thread computes one element and leaves its 24 nodal values in scratch (one array
// per value, so that loads and stores are coalesced), and a second launch sums the up to 8
// values of each node component in the tile engine's order: inside a tile the elements left
// and right, then the rows, then the layers; on a seam of the tiles each tile's share that way,
// then the shares.  So an apply has the same bits on either path, and the entry points that
// take tiles where a ctx takes two phases (the fixed-scratch apply, launches without
// scratch) agree with it bit for bit.  The price is 48 values per element through L2, which is
// why large grids keep the tiles.
#pragma once

#include "ops.cuh"

namespace vfgpu {

constexpr int TP_THREADS = 128, TP_NODE_THREADS = 256, TP_NODE_BLOCKS = 592;

__host__ __device__ inline int64_t twophase_stride(int nx, int ny, int nz) {
  return ((int64_t)(nx - 1) * (ny - 1) * (nz - 1) + 31) & ~int64_t(31);
}
// Values of scratch one apply of the grid takes.
inline size_t twophase_values(int nx, int ny, int nz) { return (size_t)24 * twophase_stride(nx, ny, nz); }
inline int twophase_node_blocks(int nx, int ny, int nz) {
  return (int)std::min<int64_t>(TP_NODE_BLOCKS, ((int64_t)nx * ny * nz + TP_NODE_THREADS - 1) / TP_NODE_THREADS);
}

template <class Op>
__global__ void __launch_bounds__(TP_THREADS, sizeof(typename Op::T) == 8 ? 2 : 4)
    u_element_kernel(const __grid_constant__ typename Op::Args A, const LayerTable L) {
  using T = typename Op::T;
  if (A.skip && *A.skip) return;
  const int nex = A.nx - 1, ney = A.ny - 1, nez = A.nz - 1;
  const int cell = blockIdx.x * TP_THREADS + threadIdx.x;
  if (cell >= nex * ney * nez) return;
  const int ez = cell / (nex * ney), r = cell - ez * (nex * ney), ey = r / nex, ex = r - ey * nex;
  T in[8][4], out[8][3];
#pragma unroll
  for (int a = 0; a < 8; a++) {
    const int64_t n = node_index(ex + (a & 1), ey + ((a >> 1) & 1), ez + (a >> 2), A.nx, A.ny);
#pragma unroll
    for (int c = 0; c < 3; c++) in[a][c] = A.x[3 * n + c];
    in[a][3] = A.v[n];
  }
  Op::element(A, L, ex, ey, ez, in, out);
  const int64_t st = twophase_stride(A.nx, A.ny, A.nz);
#pragma unroll
  for (int a = 0; a < 8; a++)
#pragma unroll
    for (int c = 0; c < 3; c++) A.scr[(a * 3 + c) * st + cell] = out[a][c];
}

template <class Op, int TY, bool DOT>
__global__ void __launch_bounds__(TP_NODE_THREADS)
    u_node_sum_kernel(const __grid_constant__ typename Op::Args A) {
  using T = typename Op::T;
  __shared__ double red[32];
  if (A.skip && *A.skip) return;
  const int nx = A.nx, ny = A.ny, nz = A.nz, nex = nx - 1, ney = ny - 1, nez = nz - 1;
  const int64_t st = twophase_stride(nx, ny, nz);
  const int N = nx * ny * nz;
  double dacc = 0.;
  for (int n = blockIdx.x * TP_NODE_THREADS + threadIdx.x; n < N; n += gridDim.x * TP_NODE_THREADS) {
    const int k = n / (nx * ny), r = n - k * (nx * ny), j = r / nx, i = r - j * nx;
    const unsigned fl = Op::node_flags(A, n);
    T e[8][3];  // the value of the node in the element of which it is corner a
#pragma unroll
    for (int a = 0; a < 8; a++) {
      const int ex = i - (a & 1), ey = j - ((a >> 1) & 1), ez = k - (a >> 2);
      const bool in = ex >= 0 && ex < nex && ey >= 0 && ey < ney && ez >= 0 && ez < nez;
      const int64_t q = in ? ((int64_t)ez * ney + ey) * nex + ex : 0;
#pragma unroll
      for (int c = 0; c < 3; c++) e[a][c] = in ? A.scr[(a * 3 + c) * st + q] : T(0);
    }
    // e[a]: corners 0..3 of the layer above, 4..7 of the one below; odd a: the element to the left,
    // a & 2: the row before
    T val[3], xin[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {  // layer below and above
      val[c] = ((e[7][c] + e[6][c]) + (e[5][c] + e[4][c])) + ((e[3][c] + e[2][c]) + (e[1][c] + e[0][c]));
      xin[c] = (DOT || ((fl >> c) & 1u)) ? A.x[3 * (int64_t)n + c] : T(0);
    }
    // tile seams (seam_range in tile_engine.cuh)
    const bool sx = i % 32 == 0 && i > 0 && i < nx - 1, sy = j % TY == 0 && j > 0 && j < ny - 1;
    if (sx || sy) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        // the four columns of elements, both layers of each
        if (sx && sy)
          val[c] = (((e[7][c] + e[3][c]) + (e[6][c] + e[2][c])) + (e[5][c] + e[1][c])) + (e[4][c] + e[0][c]);
        else if (sx)  // left and right tile
          val[c] = ((e[7][c] + e[5][c]) + (e[3][c] + e[1][c])) + ((e[6][c] + e[4][c]) + (e[2][c] + e[0][c]));
        else  // tiles of the rows before and after
          val[c] = ((e[7][c] + e[6][c]) + (e[3][c] + e[2][c])) + ((e[5][c] + e[4][c]) + (e[1][c] + e[0][c]));
      }
    }
    dacc += Op::template finish_node_in<DOT>(A, n, val, fl, xin);
  }
  if constexpr (DOT) {
    const double s = block_sum_dbl(dacc, red);
    if (threadIdx.x == 0) A.dot[blockIdx.x] = s;
  }
}

// Both launches; with A.dot, twophase_node_blocks partials of x.y.  TY: element rows of the
// operator's tiles.
template <class Op, int TY>
cudaError_t launch_u_twophase(const typename Op::Args& A, const LayerTable& L, cudaStream_t s) {
  const int ncell = (A.nx - 1) * (A.ny - 1) * (A.nz - 1), nb = twophase_node_blocks(A.nx, A.ny, A.nz);
  u_element_kernel<Op><<<(ncell + TP_THREADS - 1) / TP_THREADS, TP_THREADS, 0, s>>>(A, L);
  if (A.dot) u_node_sum_kernel<Op, TY, true><<<nb, TP_NODE_THREADS, 0, s>>>(A);
  else u_node_sum_kernel<Op, TY, false><<<nb, TP_NODE_THREADS, 0, s>>>(A);
  return cudaGetLastError();
}

}  // namespace vfgpu
