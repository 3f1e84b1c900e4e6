// apply.cu -- instantiations of the tile engine for the U operator.
#include <atomic>
#include <mutex>
#include <type_traits>

#include "kernels.h"
#include "mbar.cuh"
#include "ops.cuh"
#include "u_stencil.cuh"
#include "u_twophase.cuh"

namespace vfgpu {

// FP64 U operator tiles: 32 x U64_TY elements (1 CTA per SM: ~250 registers per thread).
// 12 rows (12 warps per SM at 168 registers, with 288 bytes of spills) measured slower
// on B200: 0.280 against 0.253 ms at 129^3, 0.814 against 0.733 ms at 193^3.
#ifndef VFGPU_U64_TY
#define VFGPU_U64_TY 8
#endif
constexpr int U_TY = 8, U64_TY = VFGPU_U64_TY;
// Blocks per SM of the FP64 U operator: 1 (~250 registers, two corner-contribution
// buffers) or, as a build option, 2 (128 registers: the row closed form of the
// non-constant elements spills; one buffer and a second barrier per layer).
#ifndef VFGPU_U64_MINB
#define VFGPU_U64_MINB 1
#endif
constexpr int U64_MINB = VFGPU_U64_MINB;
// The fixed-weight U kernel of a split launch (UOpConst: fewer registers, and the x-summed
// corner buffers leave room for both stages) takes more blocks per SM than the general
// one: 2 (FP64) and 3 (FP32) measured 0.117 / 0.089 ms at 129^3 on the penny field against
// 0.134 / 0.091 ms with the general kernel's 1 and 2.
#ifndef VFGPU_U64C_MINB
#define VFGPU_U64C_MINB 2
#endif
#ifndef VFGPU_U32C_MINB
#define VFGPU_U32C_MINB 3
#endif
// The FP32 fixed-weight wave on packed two-lane FP32 (UOpF2Const: two element rows per
// thread, 4 warps per block; the same bits as the scalar UOpConst<float>) or scalar.
// Measured at 129^3 on the penny field, whole FP32 apply: packed at 4 blocks per SM
// (118-126 registers) 0.0855 ms, at 3 0.0905, at 5 (spilling) 0.0879, at 2 0.0981;
// scalar at 3 blocks per SM 0.0900 ms.
#ifndef VFGPU_U32C_PACKED
#define VFGPU_U32C_PACKED 1
#endif
#ifndef VFGPU_U32C2_MINB
#define VFGPU_U32C2_MINB 4
#endif
constexpr bool kU32CPacked = VFGPU_U32C_PACKED != 0;
constexpr int U64C_MINB = VFGPU_U64C_MINB,
              U32C_MINB = kU32CPacked ? VFGPU_U32C2_MINB : VFGPU_U32C_MINB;
using U32COp = std::conditional_t<kU32CPacked, UOpF2Const<false>, UOpConst<float>>;
using U32COpC = std::conditional_t<kU32CPacked, UOpF2Const<true>, UOpConst<float, true>>;
// FP32 U operator: scalar UOp<float> (2 CTAs of 8 warps per SM) by default.  The
// packed two-lane variant (UOpF2: two elements per thread, half the arithmetic
// instructions) is kept as a build option; it needs 242 registers, so one CTA of
// 8 warps per SM, and measured slower on B200: 0.185 ms against 0.161 ms at 129^3,
// 0.353 ms against 0.298 ms at 161^3 (16 element rows; 0.189 / 0.339 ms with 8).
#ifndef VFGPU_U32_PACKED
#define VFGPU_U32_PACKED 0
#endif
#ifndef VFGPU_U32_PACKED_TY
#define VFGPU_U32_PACKED_TY 16
#endif
constexpr bool kU32Packed = VFGPU_U32_PACKED != 0;
constexpr int U32_TY = kU32Packed ? VFGPU_U32_PACKED_TY : U_TY;
#ifndef VFGPU_U32_MINB
#define VFGPU_U32_MINB 2
#endif
constexpr int U32_MINB = kU32Packed ? (VFGPU_U32_PACKED_TY == 16 ? 1 : 2) : VFGPU_U32_MINB;
using U32Op = std::conditional_t<kU32Packed, UOpF2, UOp<float>>;
using U32OpC = std::conditional_t<kU32Packed, UOpF2, UOp<float, true>>;

template <typename T, int MINB> cudaError_t set_stencil_attributes();

// Blocks per SM of the stencil kernel.
#ifndef VFGPU_ST64_MINB
#define VFGPU_ST64_MINB 2
#endif
#ifndef VFGPU_ST32_MINB
#define VFGPU_ST32_MINB 3
#endif
constexpr int ST64_MINB = VFGPU_ST64_MINB, ST32_MINB = VFGPU_ST32_MINB;
// Smallest grids, in (tile, plane) units, whose homogeneous nodes take the stencil.  Per apply, two
// cracks, tiles split by phase field against stencil, us: FP64 75^3 (2250 units) 46.2 / 46.5,
// 81^3 (2430) 52.4 / 48.3, 70 x 70 x 128 (3456) 65.3 / 59.3, 97^3 (3492) 61.2 / 50.4, 129^3 (8256)
// 108 / 63; FP32 113^3 (6328) 65.7 / 61.8, 129^3 76 / 55 (below 6000 the FP32 tiles run one wave).
#ifndef VFGPU_ST64_MIN_UNITS
#define VFGPU_ST64_MIN_UNITS 2000
#endif
#ifndef VFGPU_ST32_MIN_UNITS
#define VFGPU_ST32_MIN_UNITS 6000
#endif

// Cubic cells take the U element with every 1/h folded into the row weight.
template <typename T> bool cubic(const UApplyArgs<T>& A) { return A.ihx == A.ihy && A.ihy == A.ihz; }

cudaError_t apply_kernel_attributes() {
  static std::mutex m;  // contexts may be created from several threads
  std::lock_guard<std::mutex> lk(m);
  cudaError_t e = set_tile_attributes<UOp<double>, U64_TY, U64_MINB>();
  if (e == cudaSuccess) e = set_tile_attributes<UOp<double, true>, U64_TY, U64_MINB>();
  if (e == cudaSuccess) e = set_tile_attributes<UOpConst<double>, U64_TY, U64C_MINB>();
  if (e == cudaSuccess) e = set_tile_attributes<UOpConst<double, true>, U64_TY, U64C_MINB>();
  if constexpr (!kU32Packed) {
    if (e == cudaSuccess) e = set_tile_attributes<U32COp, U32_TY, U32C_MINB>();
    if (e == cudaSuccess) e = set_tile_attributes<U32COpC, U32_TY, U32C_MINB>();
  }
  if (e == cudaSuccess) e = set_tile_attributes<U32Op, U32_TY, U32_MINB>();
  if (e == cudaSuccess) e = set_tile_attributes<U32OpC, U32_TY, U32_MINB>();
  if (e == cudaSuccess) e = set_tile_attributes<UOpNC<double>, U64_TY, 1>();
  if (e == cudaSuccess) e = set_tile_attributes<UOpNC<float>, U_TY, 2>();
  if (e == cudaSuccess) e = set_tile_attributes<UOpMarked<double>, U64_TY, U64_MINB>();
  if (e == cudaSuccess) e = set_tile_attributes<UOpMarked<double, true>, U64_TY, U64_MINB>();
  if constexpr (!kU32Packed) {
    if (e == cudaSuccess) e = set_tile_attributes<UOpMarked<float>, U32_TY, U32_MINB>();
    if (e == cudaSuccess) e = set_tile_attributes<UOpMarked<float, true>, U32_TY, U32_MINB>();
  }
  if (e == cudaSuccess) e = set_stencil_attributes<double, ST64_MINB>();
  if (e == cudaSuccess) e = set_stencil_attributes<float, ST32_MINB>();
  return e;
}

// One CTA waits on an mbarrier whose phase completes (complete = 1: the arrival is
// made) or never does (complete = 0: 16 transaction bytes are expected and no copy is
// issued); *err is set when the bounded wait gives up.
__global__ void wait_selftest_kernel(unsigned* err, long long limit, int complete) {
  __shared__ uint64_t bar;
  const uint32_t b = smem_u32(&bar);
  if (threadIdx.x == 0) {
    mbar_init(b, 1);
    mbar_fence_init();
    if (complete) mbar_arrive(b);
    else mbar_expect_tx(b, 16);
  }
  __syncthreads();
  if (!mbar_wait(b, 0, limit)) atomicOr(err, 1u);
}

cudaError_t wait_selftest(long long cycles, int complete, int* timed_out) {
  unsigned* d = nullptr;
  unsigned h = 0;
  cudaError_t e = cudaMalloc(&d, sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(unsigned));
  if (e == cudaSuccess) {
    wait_selftest_kernel<<<1, 64>>>(d, cycles, complete);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(unsigned), cudaMemcpyDeviceToHost);
  cudaFree(d);
  *timed_out = h ? 1 : 0;
  return e;
}

// ------------------------------------------------------------------ unit lists
// cls[(by ntx + bx) (nz - 1) + k] = 1 when every element of tile (bx, by) (32 x TY
// elements) in element layer k has 8 equal nodal v (elements beyond the grid count as
// equal).  One block per tile and run of kClsLayers layers: each thread loads its
// element column's 2 x 2 node quads of the run's kClsLayers + 1 planes at once, then
// votes per layer.
constexpr int kClsLayers = 8;
template <int TY>
__global__ void __launch_bounds__(32 * TY) u_classify_kernel(const double* __restrict__ v,
                                                              uint8_t* __restrict__ cls, int nx,
                                                              int ny, int nez) {
  __shared__ int all[kClsLayers];
  const int tid = threadIdx.y * 32 + threadIdx.x;
  if (tid < kClsLayers) all[tid] = 1;
  const int ex = blockIdx.x * 32 + threadIdx.x, ey = blockIdx.y * TY + threadIdx.y;
  const int k0 = blockIdx.z * kClsLayers;
  const bool in = ex < nx - 1 && ey < ny - 1;
  const int64_t pl = (int64_t)nx * ny;
  const double* w = v + (in ? (int64_t)k0 * pl + (int64_t)ey * nx + ex : 0);
  double q[kClsLayers + 1][4];
#pragma unroll
  for (int i = 0; i <= kClsLayers; i++) {
    const bool ld = in && k0 + i <= nez;
    q[i][0] = ld ? w[i * pl] : 0.;
    q[i][1] = ld ? w[i * pl + 1] : 0.;
    q[i][2] = ld ? w[i * pl + nx] : 0.;
    q[i][3] = ld ? w[i * pl + nx + 1] : 0.;
  }
  __syncthreads();  // all[] initialised
#pragma unroll
  for (int i = 0; i < kClsLayers; i++) {
    const double a = q[i][0];
    const bool c = !in || (q[i][1] == a && q[i][2] == a && q[i][3] == a && q[i + 1][0] == a &&
                           q[i + 1][1] == a && q[i + 1][2] == a && q[i + 1][3] == a);
    if (!__all_sync(0xffffffffu, c) && threadIdx.x == 0) all[i] = 0;
  }
  __syncthreads();
  if (tid < kClsLayers && k0 + tid < nez)
    cls[(int64_t)(blockIdx.y * gridDim.x + blockIdx.x) * nez + k0 + tid] = all[tid] ? 1 : 0;
}

// Exclusive prefix sum of a[0, n) in shared memory over the whole block (blockDim.x a
// multiple of 32, at most 1024); returns the total.  wsum: 32 ints of shared scratch.
__device__ int block_scan_excl(int* a, int n, int* wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int b0 = min((int)threadIdx.x * per, n), b1 = min(b0 + per, n);
  int sum = 0;
  for (int i = b0; i < b1; i++) sum += a[i];
  int x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = lane < nw ? wsum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    wsum[lane] = w;
  }
  __syncthreads();
  int run = x - sum + (warp ? wsum[warp - 1] : 0);
  const int total = wsum[nw - 1];
  for (int i = b0; i < b1; i++) {
    const int t = a[i];
    a[i] = run;
    run += t;
  }
  __syncthreads();  // wsum is reused by the next scan
  return total;
}

// Unit type of node plane z of a tile column: from its layer flags f[0, nz - 1), 0 when the
// element layers below and above are constant (or absent), else 1; or (PLANES) its own
// flag f[z], 1 when the unit holds a node the stencil does not write.
template <bool PLANES>
__device__ __forceinline__ int unit_type(const uint8_t* f, int z, int nez) {
  if (PLANES) return f[z];
  const bool below = z == 0 || f[z - 1], above = z == nez || f[z];
  return below && above ? 0 : 1;
}

// One block of 1024 threads builds both unit lists of a plan from its layer flags:
// per tile column (one thread each) the runs of equal unit type up its nz planes,
// counted, offset by prefix sums over the columns in tile order, written; then, per
// list l and block b of its wave of ncta_l blocks, the run holding the list's unit
// U b / ncta_l (binary search on the runs' unit offsets).
template <bool PLANES>
__global__ void __launch_bounds__(1024) unit_lists_kernel(const uint8_t* __restrict__ cls, int nz,
                                                          int ncol, int ncta0, int ncta1, int4* __restrict__ runs0,
                                                          int4* __restrict__ runs1, int* __restrict__ start0,
                                                          int* __restrict__ start1, int* __restrict__ total) {
  extern __shared__ int sh[];  // [4][ncol] counts, then 32 ints of scan scratch
  int* cnt = sh;
  int* wsum = sh + 4 * ncol;
  const int nez = nz - 1;
  for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
    const uint8_t* f = cls + (int64_t)c * (PLANES ? nz : nez);
    int nr[2] = {0, 0}, nu[2] = {0, 0}, prev = -1;
    for (int z = 0; z < nz; z++) {
      const int t = unit_type<PLANES>(f, z, nez);
      nu[t]++;
      if (t != prev) nr[t]++;
      prev = t;
    }
    cnt[c] = nr[0];
    cnt[ncol + c] = nr[1];
    cnt[2 * ncol + c] = nu[0];
    cnt[3 * ncol + c] = nu[1];
  }
  __syncthreads();
  int tot[4];
#pragma unroll
  for (int a = 0; a < 4; a++) tot[a] = block_scan_excl(cnt + a * ncol, ncol, wsum);
  int4* runs[2] = {runs0, runs1};
  for (int c = threadIdx.x; c < ncol; c += blockDim.x) {
    const uint8_t* f = cls + (int64_t)c * (PLANES ? nz : nez);
    int r[2] = {cnt[c], cnt[ncol + c]}, u[2] = {cnt[2 * ncol + c], cnt[3 * ncol + c]};
    int z0 = 0, t0 = unit_type<PLANES>(f, 0, nez);
    for (int z = 1; z <= nz; z++) {
      const int t = z < nz ? unit_type<PLANES>(f, z, nez) : -1;
      if (t != t0) {
        runs[t0][r[t0]++] = make_int4(c, z0, z, u[t0]);
        u[t0] += z - z0;
        z0 = z;
        t0 = t;
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ncta0 + ncta1; i += blockDim.x) {
    const int l = i < ncta0 ? 0 : 1, b = l ? i - ncta0 : i, ncta = l ? ncta1 : ncta0, nrun = tot[l];
    const int64_t ub = (int64_t)tot[2 + l] * b / ncta;
    int lo = 0, hi = nrun - 1;
    while (lo < hi) {  // the last run whose first unit is <= ub
      const int mid = (lo + hi + 1) / 2;
      if (runs[l][mid].w <= ub) lo = mid; else hi = mid - 1;
    }
    (l ? start1 : start0)[b] = nrun > 0 ? lo : 0;
  }
  if (threadIdx.x == 0) {
    total[0] = tot[2];
    total[1] = tot[3];
  }
}

constexpr int kMaxListCols = 2048;  // tile columns the one-block list builder takes
// Grids below this many (tile, plane) units keep the plain split: there the general
// wave's latency (about one segment) and the list build cost more than the fixed-weight
// kernel saves.  Measured on the penny field, split against plain, us per apply FP64 /
// FP32: 41^3 35.8 / 29.7 against 25.7 / 23.6; 65^3 44.1 / 35.9 against 44.0 / 29.5;
// 81^3 54.3 / 46.0 against 60.4 / 42.1; 97^3 64.5 / 56.3 against 72.7 / 52.2; 113^3
// 93.3 / 72.8 against 109.6 / 74.8; 161^3 189.4 / 140.3 against 247.0 / 154.7.
#ifndef VFGPU_U64_LISTS_MIN_UNITS
#define VFGPU_U64_LISTS_MIN_UNITS 2000
#endif
#ifndef VFGPU_U32_LISTS_MIN_UNITS
#define VFGPU_U32_LISTS_MIN_UNITS 6000
#endif

bool unit_lists_pay(const TilePlan& p, int nz, int prec_bytes) {
  const int64_t min_units = prec_bytes == 8 ? VFGPU_U64_LISTS_MIN_UNITS : VFGPU_U32_LISTS_MIN_UNITS;
  return (int64_t)p.ntx * p.nty * nz >= min_units;
}

size_t unit_lists_bytes(const TilePlan& p, int nz) {
  const int64_t ncol = (int64_t)p.ntx * p.nty;
  if (nz < 2 || ncol > kMaxListCols) return 0;
  auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
  return up(ncol * nz) + 2 * up(ncol * nz * sizeof(int4)) + up(p.ncta0 * sizeof(int)) +
         up(p.ncta * sizeof(int)) + up(2 * sizeof(int));
}

UnitLists unit_lists_carve(void* base, const TilePlan& p, int nz) {
  UnitLists L;
  if (!base || !unit_lists_bytes(p, nz)) return L;
  const size_t ncol = (size_t)p.ntx * p.nty;
  auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
  char* q = static_cast<char*>(base);
  L.cls = reinterpret_cast<uint8_t*>(q);
  q += up(ncol * nz);
  for (int l = 0; l < 2; l++) {
    L.runs[l] = reinterpret_cast<int4*>(q);
    q += up(ncol * nz * sizeof(int4));
  }
  for (int l = 0; l < 2; l++) {
    L.start[l] = reinterpret_cast<int*>(q);
    q += up((l ? p.ncta : p.ncta0) * sizeof(int));
  }
  L.total = reinterpret_cast<int*>(q);
  return L;
}

template <int TY>
static cudaError_t classify(const double* v, uint8_t* cls, int nx, int ny, int nz, const TilePlan& p,
                            cudaStream_t s) {
  const int runs = (nz - 1 + kClsLayers - 1) / kClsLayers;
  if (runs > 65535 || p.nty > 65535) return cudaErrorInvalidValue;
  u_classify_kernel<TY><<<dim3(p.ntx, p.nty, runs), dim3(32, TY), 0, s>>>(v, cls, nx, ny, nz - 1);
  return cudaGetLastError();
}

cudaError_t build_unit_lists(const double* v, int nx, int ny, int nz, const TilePlan& p,
                             const UnitLists& L, cudaStream_t s) {
  if (!L.cls) return cudaSuccess;
  cudaError_t e;
  switch (p.ty) {
    case 4: e = classify<4>(v, L.cls, nx, ny, nz, p, s); break;
    case 8: e = classify<8>(v, L.cls, nx, ny, nz, p, s); break;
    case 16: e = classify<16>(v, L.cls, nx, ny, nz, p, s); break;
    default: return cudaErrorInvalidValue;
  }
  if (e != cudaSuccess) return e;
  const int ncol = p.ntx * p.nty;
  unit_lists_kernel<false><<<1, 1024, (4 * ncol + 32) * sizeof(int), s>>>(
      L.cls, nz, ncol, p.ncta0, p.ncta, L.runs[0], L.runs[1], L.start[0], L.start[1], L.total);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ node flags
// node[n] = the Dirichlet bits, kNodeOne where v = 1, kNodeElement where one of the up to 26
// neighbours has another v.
__global__ void __launch_bounds__(256) u_node_kernel(const double* __restrict__ v, const uint8_t* __restrict__ bc,
                                                     uint8_t* __restrict__ node, int nx, int ny, int nz) {
  const int64_t plane = (int64_t)nx * ny, N = plane * nz;
  const int64_t n = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (n >= N) return;
  const int k = (int)(n / plane), r = (int)(n - k * plane), j = r / nx, i = r - j * nx;
  const double a = v[n];
  bool same = true;
#pragma unroll
  for (int c = -1; c < 2; c++)
#pragma unroll
    for (int b = -1; b < 2; b++)
#pragma unroll
      for (int d = -1; d < 2; d++)
        same &= v[node_index(min(max(i + d, 0), nx - 1), min(max(j + b, 0), ny - 1), min(max(k + c, 0), nz - 1), nx,
                             ny)] == a;
  node[n] = (uint8_t)(bc[n] | (a == 1. ? kNodeOne : 0u) | (same ? 0u : kNodeElement));
}

// type[col nz + z] = 1 when the 33 x (TY + 1) nodes of tile col in plane z hold one of the
// element operator's.
template <int TY>
__global__ void __launch_bounds__(32 * TY) u_unit_type_kernel(const uint8_t* __restrict__ node,
                                                               uint8_t* __restrict__ type, int nx, int ny, int nz) {
  const int tid = threadIdx.y * 32 + threadIdx.x, k0 = blockIdx.z * kClsLayers;
  for (int k = k0; k < min(k0 + kClsLayers, nz); k++) {
    bool any = false;
    for (int s = tid; s < 33 * (TY + 1); s += 32 * TY) {
      const int X = blockIdx.x * 32 + s % 33, Y = blockIdx.y * TY + s / 33;
      if (X < nx && Y < ny) any = any || (node[node_index(X, Y, k, nx, ny)] & kNodeElement);
    }
    const int t = __syncthreads_or(any);
    if (tid == 0) type[(int64_t)(blockIdx.y * gridDim.x + blockIdx.x) * nz + k] = t ? 1 : 0;
  }
}

// A homogeneous node that only listed units hold goes to the element operator too (those
// units run in any case): the stencil keeps the nodes of at least one unlisted unit.
__global__ void __launch_bounds__(256) u_node_demote_kernel(const uint8_t* __restrict__ type,
                                                            uint8_t* __restrict__ node, int nx, int ny, int nz,
                                                            int ty, int ntx, int nty) {
  const int64_t plane = (int64_t)nx * ny, n = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (n >= plane * nz) return;
  const unsigned f = node[n];
  if (f & kNodeElement) return;
  const int k = (int)(n / plane), r = (int)(n - k * plane), j = r / nx, i = r - j * nx;
  // the tiles whose boxes hold the node: the one it starts and, on a seam, the one before
  const int bx1 = min(i / 32, ntx - 1), by1 = min(j / ty, nty - 1);
  const int bx0 = i % 32 == 0 && i > 0 ? i / 32 - 1 : bx1, by0 = j % ty == 0 && j > 0 ? j / ty - 1 : by1;
  bool all = true;
  for (int by = by0; by <= by1; by++)
    for (int bx = bx0; bx <= bx1; bx++) all = all && type[(int64_t)(by * ntx + bx) * nz + k];
  if (all) node[n] = (uint8_t)(f | kNodeElement);
}

// range[b]: the planes [x, y) of stencil block b's chunk that hold nodes of the stencil.
__global__ void __launch_bounds__(256) u_srange_kernel(const uint8_t* __restrict__ node, int2* __restrict__ range,
                                                       int nx, int ny, int nz, StencilPlan p) {
  const int b = blockIdx.x, bx = b % p.ntx, by = (b / p.ntx) % p.nty, bz = b / (p.ntx * p.nty);
  const int ka = bz * p.zc, kb = min(ka + p.zc, nz);
  int lo = kb, hi = ka;
  for (int k = ka; k < kb; k++) {
    bool hit = false;
    for (int s = threadIdx.x; s < ST_X * ST_Y; s += 256) {
      const int i = 1 + bx * ST_X + s % ST_X, j = 1 + by * ST_Y + s / ST_X;
      if (i < nx - 1 && j < ny - 1) hit = hit || !(node[node_index(i, j, k, nx, ny)] & kNodeElement);
    }
    if (__syncthreads_or(hit)) {
      lo = min(lo, k);
      hi = k + 1;
    }
  }
  if (threadIdx.x == 0) range[b] = make_int2(lo, hi);
}

cudaError_t build_node_flags(const double* v, const uint8_t* bc, int nx, int ny, int nz, uint8_t* node,
                             cudaStream_t s) {
  const int64_t N = (int64_t)nx * ny * nz;
  u_node_kernel<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(v, bc, node, nx, ny, nz);
  return cudaGetLastError();
}

cudaError_t build_stencil_lists(uint8_t* node, int2* range, int nx, int ny, int nz, const TilePlan& p,
                                const UnitLists& L, cudaStream_t s) {
  const int runs = (nz + kClsLayers - 1) / kClsLayers, ncol = p.ntx * p.nty;
  const int64_t N = (int64_t)nx * ny * nz;
  const dim3 grid(p.ntx, p.nty, runs);
  switch (p.ty) {
    case 4: u_unit_type_kernel<4><<<grid, dim3(32, 4), 0, s>>>(node, L.cls, nx, ny, nz); break;
    case 8: u_unit_type_kernel<8><<<grid, dim3(32, 8), 0, s>>>(node, L.cls, nx, ny, nz); break;
    case 16: u_unit_type_kernel<16><<<grid, dim3(32, 16), 0, s>>>(node, L.cls, nx, ny, nz); break;
    default: return cudaErrorInvalidValue;
  }
  u_node_demote_kernel<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(L.cls, node, nx, ny, nz, p.ty, p.ntx, p.nty);
  u_srange_kernel<<<p.st.blocks(), 256, 0, s>>>(node, range, nx, ny, nz, p.st);
  unit_lists_kernel<true><<<1, 1024, (4 * ncol + 32) * sizeof(int), s>>>(
      L.cls, nz, ncol, p.ncta0, p.ncta, L.runs[0], L.runs[1], L.start[0], L.start[1], L.total);
  return cudaGetLastError();
}

// Largest grids, in cells, whose applies run in two phases.  Per apply, two cracks, tiles (with
// the stencil where it is taken) against two phases, us AT1 / AT2: FP64 17^3 16.4 / 14.4 and
// 9.3 / 9.3 (of which about 8 are the call), 41^3 22.6 / 21.6 and 14.4 / 14.7, 65^3 36.9 / 34.9
// and 28.7 / 34.2, 81^3 48.3 / 71.7 and 59.3 / 69.7, 97^3 50.4 / 93.2 and 95.7 / 112.8; FP32 41^3
// 18.5 / 20.5 and 11.3 / 11.3, 65^3 24.6 / 27.9 and 18.5 / 23.8, 81^3 42.0 / 48.5 and 28.7 / 39.0,
// 97^3 52.3 / 65.0 and 53.6 / 70.9; 97 x 61 x 83 (tiles that fit) - / 31.6 and - / 33.2.
#ifndef VFGPU_TWOPHASE64_CELLS
#define VFGPU_TWOPHASE64_CELLS 300000
#endif
#ifndef VFGPU_TWOPHASE32_CELLS
#define VFGPU_TWOPHASE32_CELLS 400000
#endif
bool twophase_pays(int nx, int ny, int nz, int prec_bytes) {
  const int64_t most = prec_bytes == 8 ? VFGPU_TWOPHASE64_CELLS : VFGPU_TWOPHASE32_CELLS;
  return (int64_t)(nx - 1) * (ny - 1) * (nz - 1) <= most;
}

size_t twophase_scratch(int nx, int ny, int nz) { return twophase_values(nx, ny, nz); }
int twophase_dots(int nx, int ny, int nz) { return twophase_node_blocks(nx, ny, nz); }

bool stencil_pays(const TilePlan& p, int nx, int ny, int nz, int prec_bytes) {
  if (U64_TY != U32_TY || (prec_bytes == 4 && kU32Packed)) return false;  // the plans share the node flags
  const int64_t ncol = (int64_t)p.ntx * p.nty;
  if (std::min(nx, std::min(ny, nz)) < 8 || ncol > kMaxListCols || ceil_div(nz, kClsLayers) > 65535) return false;
  return ncol * nz >= (prec_bytes == 8 ? VFGPU_ST64_MIN_UNITS : VFGPU_ST32_MIN_UNITS);
}

TilePlan u_plan(int nx, int ny, int nz, int prec_bytes, int num_sms) {
  TilePlan p = tile_plan(nx, ny, nz, prec_bytes == 8 ? U64_TY : U32_TY, 3,
                         prec_bytes == 8 ? U64_MINB : U32_MINB, num_sms);
  const TilePlan q = tile_plan(nx, ny, nz, p.ty, 3, prec_bytes == 8 ? U64C_MINB : U32C_MINB, num_sms);
  p.ncta0 = q.ncta;
  p.st = stencil_plan(nx, ny, nz, num_sms * (prec_bytes == 8 ? ST64_MINB : ST32_MINB));
  return p;
}

template <typename T, int MINB> cudaError_t set_stencil_attributes() {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  constexpr int smem = (int)stencil_smem<T>();
  e = cudaFuncSetAttribute(u_stencil_kernel<T, MINB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(u_stencil_kernel<T, MINB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

// Homogeneous nodes by the stencil, then the others by the element operator over unit list
// 1, then the faces with the element operator's seams.  With A.dot the x.y partials go to
// A.dot[0, blocks) (stencil), then ncta (elements), then nface + seam_blocks.
template <class OpG, int TY, int MINB, int STB>
static cudaError_t launch_u_stencil(typename OpG::Args A, const TilePlan& p, const LayerTable& L, cudaStream_t s) {
  using T = typename OpG::T;
  A.ntx = p.ntx;
  A.nty = p.nty;
  cudaError_t e = set_stencil_attributes<T, STB>();
  if (e == cudaSuccess) e = set_tile_attributes<OpG, TY, MINB>();
  if (e != cudaSuccess) return e;
  constexpr size_t smem = stencil_smem<T>(), smemG = tile_smem_bytes<OpG, TY, MINB>();
  const int nb = p.st.blocks(), oblocks = p.st.nface + seam_blocks(p, A.nx, A.ny, A.nz);
  const dim3 block(32, TY);
  typename OpG::Args AG = A;
  if (AG.dot) AG.dot += nb;
  if (A.dot) {
    u_stencil_kernel<T, STB, true><<<nb, ST_THREADS, smem, s>>>(A, p.st);
    tile_apply_kernel<OpG, TY, MINB, true><<<p.ncta, block, smemG, s>>>(AG, L);
    u_outer_kernel<OpG, true><<<oblocks, 256, 0, s>>>(AG, TY, p.ncta, p.st.nface);
  } else {
    u_stencil_kernel<T, STB, false><<<nb, ST_THREADS, smem, s>>>(A, p.st);
    tile_apply_kernel<OpG, TY, MINB, false><<<p.ncta, block, smemG, s>>>(AG, L);
    u_outer_kernel<OpG, false><<<oblocks, 256, 0, s>>>(AG, TY, p.ncta, p.st.nface);
  }
  return cudaGetLastError();
}

template <>
cudaError_t launch_u_apply<double>(const UApplyArgs<double>& A, const TilePlan& p,
                                   const LayerTable& L, cudaStream_t s) {
  if (A.scr) {
    if (A.cflag) return launch_u_twophase<UOpNC<double>, U64_TY>(A, L, s);
    if (cubic(A)) return launch_u_twophase<UOp<double, true>, U64_TY>(A, L, s);
    return launch_u_twophase<UOp<double>, U64_TY>(A, L, s);
  }
  if (A.cflag) return launch_tile_apply<UOpNC<double>, U64_TY, 1>(A, p, L, s);
  if (A.node) {
    if (cubic(A)) return launch_u_stencil<UOpMarked<double, true>, U64_TY, U64_MINB, ST64_MINB>(A, p, L, s);
    return launch_u_stencil<UOpMarked<double>, U64_TY, U64_MINB, ST64_MINB>(A, p, L, s);
  }
  if (A.ur[0] && A.ur[1]) {
    if (cubic(A))
      return launch_tile_apply_split<UOpConst<double, true>, UOp<double, true>, U64_TY, U64C_MINB, U64_MINB>(
          A, p, L, s);
    return launch_tile_apply_split<UOpConst<double>, UOp<double>, U64_TY, U64C_MINB, U64_MINB>(A, p, L, s);
  }
  if (cubic(A)) return launch_tile_apply<UOp<double, true>, U64_TY, U64_MINB>(A, p, L, s);
  return launch_tile_apply<UOp<double>, U64_TY, U64_MINB>(A, p, L, s);
}
template <>
cudaError_t launch_u_apply<float>(const UApplyArgs<float>& A, const TilePlan& p,
                                  const LayerTable& L, cudaStream_t s) {
  if (A.scr) {
    if (A.cflag) return launch_u_twophase<UOpNC<float>, U_TY>(A, L, s);
    if (cubic(A)) return launch_u_twophase<UOp<float, true>, U32_TY>(A, L, s);
    return launch_u_twophase<UOp<float>, U32_TY>(A, L, s);
  }
  // NOCOMPRESSION needs the scalar layout: its plan is the FP32 plan only with the
  // scalar tile (the packed build option keeps the plain operator packed)
  if (A.cflag) return launch_tile_apply<UOpNC<float>, U_TY, 2>(A, p, L, s);
  if constexpr (!kU32Packed) {
    if (A.node) {
      if (cubic(A)) return launch_u_stencil<UOpMarked<float, true>, U32_TY, U32_MINB, ST32_MINB>(A, p, L, s);
      return launch_u_stencil<UOpMarked<float>, U32_TY, U32_MINB, ST32_MINB>(A, p, L, s);
    }
    if (A.ur[0] && A.ur[1]) {
      if (cubic(A))
        return launch_tile_apply_split<U32COpC, U32OpC, U32_TY, U32C_MINB, U32_MINB>(A, p, L, s);
      return launch_tile_apply_split<U32COp, U32Op, U32_TY, U32C_MINB, U32_MINB>(A, p, L, s);
    }
  }
  if (cubic(A)) return launch_tile_apply<U32OpC, U32_TY, U32_MINB>(A, p, L, s);
  return launch_tile_apply<U32Op, U32_TY, U32_MINB>(A, p, L, s);
}
}  // namespace vfgpu

extern "C" int vfgpu_wait_selftest(long long cycles, int complete, int* timed_out) {
  if (!timed_out || cycles < 0 || cycles > 4000000000ll) return -1;
  return vfgpu::wait_selftest(cycles, complete ? 1 : 0, timed_out) == cudaSuccess ? 0 : -2;
}
