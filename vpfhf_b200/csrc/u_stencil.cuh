// u_stencil.cuh -- the U operator at nodes inside a homogeneous patch, as a separable
// node-centred stencil.
//
// A node is homogeneous when every element around it has the same 8 nodal v and the grid
// one material.  There K(v) is S = v^2 + eta times a sum of tensor products of the 1-D
// operators of linear elements -- mass M, stiffness K, and the first derivative C with its
// transpose T -- so with d2 f = (f- - f) + (f+ - f), m f = f + d2 f / 6, d f = f+ - f- along
// an axis (interior nodes: M = h m, K = -d2 / h, C = -T = d / 2) the rows of a node are
//   y_c = S [ m_z P_c + d2_z Q_c + d_z R_c ]
//   P_x = -(lam + 2 mu) (hy hz / hx) m_y d2_x u_x - mu (hx hz / hy) d2_y m_x u_x
//         - (lam + mu) (hz / 4) d_x d_y u_y,    Q_x = -mu (hx hy / hz) m_x m_y u_x,
//   R_x = -(lam + mu) (hy / 4) d_x m_y u_z      (y alike),
//   P_z = -mu ((hy hz / hx) m_y d2_x u_z + (hx hz / hy) d2_y m_x u_z),
//   Q_z = -(lam + 2 mu) (hx hy / hz) m_x m_y u_z,
//   R_z = -(lam + mu) ((hy / 4) d_x m_y u_x + (hx / 4) m_x d_y u_y):
// what the element sums give there (the 3-point Gauss rule is exact for these degrees), in
// about 95 operations per node against 234 per element plus the exchange and summation of
// its 24 nodal values.  Every difference is taken before it is averaged, as in the
// element's modal form.
//
// Columns inside the box in x and y: a block owns 32 x 16 of them and marches up a chunk of
// planes, 4 rows of one column per thread.  Planes of 34 x 18 nodes stream through a 5-slot
// shared-memory ring by asynchronous copies three planes ahead, one barrier per plane; a
// thread makes the x-passes of the 6 rows its 4 outputs need (13.5 shared reads per node) and
// keeps per row what planes k - 1 and k give to node k, so nothing is exchanged between
// threads and no seam is summed.  127 = 4 x 32 - 1 = 8 x 16 - 1: the inside of the 2^k + 1 grids
// fills the tiles.  On the lowest and highest plane M is h (f / 2 + (f' - f) / 6), K is
// (f - f') / h, C = (f' - f) / 2 and T = -C -+ f: the node keeps P / 3 - Q and a multiple of R.
// x and y faces (their edges aside): runs of 4 nodes up a column, 30 columns per warp, with the
// one-sided operators across the face; an x face is a y face with x and y exchanged.  The
// box's 12 edges: 9 lanes per node from the 27 neighbours and the 1-D coefficients.  Both
// run beside the element operator's seams in the apply's last launch: a march up whole face
// columns inside the main launch is a serial chain of memory latencies (57 us at 161^3).
// Nodes that are not homogeneous are left to the element operator (UApplyArgs::node).
#pragma once

#include "ops.cuh"

namespace vfgpu {

constexpr int ST_ROW = 3 * (ST_X + 2), ST_PLANE = ST_ROW * (ST_Y + 2), ST_RING = 5;
template <typename T> constexpr size_t stencil_smem() { return sizeof(T) * ST_RING * ST_PLANE; }

// 1-D operators of node i of n at spacing h: coefficients at i - 1, i, i + 1.
template <typename T> struct Axis1D {
  T M[3], K[3], C[3], D[3];  // D: the transpose of C
  __device__ __forceinline__ Axis1D(int i, int n, T h) {
    const T l = T(i > 0), r = T(i < n - 1), ih = T(1) / h;
    M[0] = l * h * T(1.0 / 6.0);
    M[1] = (l + r) * h * T(1.0 / 3.0);
    M[2] = r * h * T(1.0 / 6.0);
    K[0] = -l * ih;
    K[1] = (l + r) * ih;
    K[2] = -r * ih;
    C[0] = T(-0.5) * l;
    C[1] = T(0.5) * (l - r);
    C[2] = T(0.5) * r;
    D[0] = -C[0];
    D[1] = C[1];
    D[2] = -C[2];
  }
};

// The share of node (i, j, k)'s rows (without S) that the three neighbours i - 1 .. i + 1 of
// row j + b - 1, plane k + c - 1 give, for any node of the box (used on its edges).
template <typename T>
__device__ __forceinline__ void stencil_edge_row(const UApplyArgs<T>& A, int i, int j, int k, int b, int c, T lam,
                                                 T mu, T hx, T hy, T hz, T (&y)[3]) {
  const Axis1D<T> X(i, A.nx, hx), Y(j, A.ny, hy), Z(k, A.nz, hz);
  const T l2 = lam + T(2) * mu;
  const int kk = min(max(k + c - 1, 0), A.nz - 1), jj = min(max(j + b - 1, 0), A.ny - 1);  // beyond: weight 0
  T M[3], K[3], C[3], D[3];
#pragma unroll
  for (int q = 0; q < 3; q++) M[q] = K[q] = C[q] = D[q] = T(0);
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const T* u = A.x + 3 * node_index(min(max(i + a - 1, 0), A.nx - 1), jj, kk, A.nx, A.ny);
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const T v = __ldg(u + q);
      M[q] = fma(X.M[a], v, M[q]);
      K[q] = fma(X.K[a], v, K[q]);
      C[q] = fma(X.C[a], v, C[q]);
      D[q] = fma(X.D[a], v, D[q]);
    }
  }
  auto at = [](const T (&f)[3], int q) { return q == 0 ? f[0] : q == 1 ? f[1] : f[2]; };
  const T My = at(Y.M, b), Ky = at(Y.K, b), Cy = at(Y.C, b), Dy = at(Y.D, b);
  const T Mz = at(Z.M, c), Kz = at(Z.K, c), Cz = at(Z.C, c), Dz = at(Z.D, c);
  y[0] = Mz * (l2 * (K[0] * My) + mu * (M[0] * Ky) + lam * (D[1] * Cy) + mu * (C[1] * Dy)) +
         Kz * (mu * (M[0] * My)) + My * (lam * (D[2] * Cz) + mu * (C[2] * Dz));
  y[1] = Mz * (mu * (K[1] * My) + l2 * (M[1] * Ky) + lam * (C[0] * Dy) + mu * (D[0] * Cy)) +
         Kz * (mu * (M[1] * My)) + M[2] * (lam * (Dy * Cz) + mu * (Cy * Dz));
  y[2] = Mz * (mu * (K[2] * My + M[2] * Ky)) + Kz * (l2 * (M[2] * My)) +
         My * (lam * (C[0] * Dz) + mu * (D[0] * Cz)) + M[1] * (lam * (Cy * Dz) + mu * (Dy * Cz));
}

// StencilCoefs in the kernel's type (rounded once each).
template <typename T> struct StencilCoef {
  T xx, xy, yx, yy, xd, q, qz, rx, ry, g;
  __device__ __forceinline__ explicit StencilCoef(const StencilCoefs& c)
      : xx(T(c.xx)), xy(T(c.xy)), yx(T(c.yx)), yy(T(c.yy)), xd(T(c.xd)), q(T(c.q)), qz(T(c.qz)), rx(T(c.rx)),
        ry(T(c.ry)), g(T(c.g)) {}
};

// Takes in plane k's P, Q, R of a row: fin = node k - 1, then acc = what planes k - 1 and k give
// to node k, up = what plane k gives to node k + 1.
template <typename T>
__device__ __forceinline__ void stencil_march(const T (&P)[3], const T (&Q)[3], const T (&R)[3], T (&acc)[3],
                                              T (&up)[3], T (&fin)[3]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const T t = fma(P[c], T(1.0 / 6.0), Q[c]);
    fin[c] = acc[c] + (t + R[c]);
    acc[c] = fma(T(2.0 / 3.0), P[c], fma(T(-2), Q[c], up[c]));
    up[c] = t - R[c];
  }
}
// acc on the lowest (g) or highest (-g) plane, from the rows' P, Q, R and what the plane below
// gave (0 on the lowest).
template <typename T>
__device__ __forceinline__ void stencil_end(const T (&P)[3], const T (&Q)[3], const T (&R)[3], T g,
                                            const T (&below)[3], T (&acc)[3]) {
#pragma unroll
  for (int c = 0; c < 3; c++) acc[c] = below[c] + fma(c < 2 ? g : -g, R[c], fma(P[c], T(1.0 / 3.0), -Q[c]));
}

// Writes a finished node from its rows (without S), flags and x; with DOT returns its x.y.
// S1 = 1 + eta.
template <typename T, bool DOT>
__device__ __forceinline__ double stencil_put(const UApplyArgs<T>& A, T S1, T eta, int64_t n, unsigned f,
                                              const T (&r)[3], const T* xin) {
  T S = S1;
  if (!(f & kNodeOne)) {
    const T v = A.v[n];
    S = fma(v, v, eta);
  }
  T y[3];
#pragma unroll
  for (int c = 0; c < 3; c++) y[c] = S * r[c];
  if (f & 7u)
#pragma unroll
    for (int c = 0; c < 3; c++)
      if ((f >> c) & 1u) y[c] = xin[c];
  T* yo = A.y + 3 * n;
  double d = 0.;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    yo[c] = y[c];
    if constexpr (DOT) d += (double)xin[c] * (double)y[c];
  }
  return d;
}

template <typename T, int MINB, bool DOT>
__global__ void __launch_bounds__(ST_THREADS, MINB)
    u_stencil_kernel(const __grid_constant__ UApplyArgs<T> A, const StencilPlan p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);
  __shared__ double red[32];
  if (A.skip && *A.skip) return;  // converged solve
  const int tid = threadIdx.x, lane = tid & 31, wy = tid >> 5;
  const int nx = A.nx, ny = A.ny, nz = A.nz;
  const int b = blockIdx.x;
  const int2 zr = A.srange[b];  // the chunk's planes that hold nodes of the stencil
  if (zr.x >= zr.y) {           // none: uniform exit
    if (DOT && tid == 0) A.dot[blockIdx.x] = 0.;
    return;
  }
  const T eta = T(A.P->eta);
  const int64_t plane = (int64_t)nx * ny;
  const T sixth = T(1.0 / 6.0), S1 = T(1) + eta;
  double dacc = 0.;
  auto put = [&](int64_t n, unsigned f, const T (&r)[3], const T* xin) { dacc += stencil_put<T, DOT>(A, S1, eta, n, f, r, xin); };
  const int bx = b % p.ntx, by = (b / p.ntx) % p.nty;
  const int X0 = bx * ST_X, Y0 = by * ST_Y;  // the halo corner: first inner column X0 + 1
  const int ka = zr.x, kb = zr.y;                       // planes [ka, kb) are written,
  const int kf = max(ka - 1, 0), kl = min(kb, nz - 1);  // [kf, kl] read
  // a warp copies rows wy, wy + ST_W, ... of a plane, 102 values each (columns and rows
  // beyond the box repeat its last one: they feed no node that is written)
  constexpr int NR = (ST_Y + 2 + ST_W - 1) / ST_W;
  int off[4], rof[NR];
#pragma unroll
  for (int q = 0; q < 4; q++) off[q] = min(lane + 32 * q, 3 * (nx - X0) - 1);
#pragma unroll
  for (int q = 0; q < NR; q++) rof[q] = 3 * (min(Y0 + wy + q * ST_W, ny - 1) * nx + X0);
  const T* src = A.x + 3 * plane * kf;  // the next plane to fetch, into slot fs
  int fs = 0, left = kl - kf + 1;
  auto fetch = [&]() {
    if (left > 0) {
      T* dst = ring + fs * ST_PLANE + wy * ST_ROW + lane;
#pragma unroll
      for (int r = 0; r < NR; r++) {
        if (r == NR - 1 && wy + r * ST_W >= ST_Y + 2) break;
        const T* a = src + rof[r];
#pragma unroll
        for (int q = 0; q < 3; q++) cp_async_val(dst + r * ST_W * ST_ROW + 32 * q, a + off[q], true);
        if (lane < ST_ROW - 96) cp_async_val(dst + r * ST_W * ST_ROW + 96, a + off[3], true);
      }
    }
    left--;
    src += 3 * plane;
    fs = fs == ST_RING - 1 ? 0 : fs + 1;
    cp_async_commit();  // also when empty: the waits count groups
  };
  const StencilCoef<T> C(A.P->st[0]);
  const int i = X0 + 1 + lane, j0 = Y0 + 1 + wy * ST_RY;
  // rows of this thread whose nodes lie inside the x and y faces
  const int rows = i < nx - 1 ? min(max(ny - 1 - j0, 0), ST_RY) : 0;
  int64_t nk = (int64_t)j0 * nx + i + kf * plane;  // node of row 0 in plane k
  T acc[ST_RY][3], up[ST_RY][3];
#pragma unroll
  for (int r = 0; r < ST_RY; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) acc[r][c] = up[r][c] = T(0);
  unsigned fl[ST_RY];
#pragma unroll
  for (int r = 0; r < ST_RY; r++) fl[r] = kNodeElement;
  // writes row r of the plane whose row 0 is node n and whose ring slot starts at xr
  auto finish = [&](int r, int64_t n, const T (&fin)[3], const T* xr) {
    if (fl[r] & kNodeElement) return;
    T xin[3];
#pragma unroll
    for (int c = 0; c < 3; c++) xin[c] = T(0);
    if (DOT || (fl[r] & 7u))
#pragma unroll
      for (int c = 0; c < 3; c++) xin[c] = xr[(r + 1) * ST_ROW + 3 + c];
    put(n + r * nx, fl[r], fin, xin);
  };
  fetch();
  fetch();
  fetch();
  const T* const mine = ring + wy * ST_RY * ST_ROW + 3 * lane;  // this thread's corner of slot 0
  const T *s = mine, *sp = mine;  // of plane k and of plane k - 1
  int slot = 0;
#pragma unroll 1
  for (int k = kf; k <= kl; k++) {
    asm volatile("cp.async.wait_group 2;\n" ::: "memory");
    __syncthreads();  // plane k is everyone's; the slot of plane k - 2 is no longer read
    fetch();
    // this plane's flags, for the finish one plane on
    unsigned nf[ST_RY];
    const int live = k >= ka && k < kb ? rows : 0;
#pragma unroll
    for (int r = 0; r < ST_RY; r++) {
      nf[r] = kNodeElement;
      if (r < live) nf[r] = A.node[nk + r * nx];
    }
    const bool end = k == 0 || k == nz - 1;
    T d2[3][3], m[3][3], d[3][3];  // [row mod 3][component]: x-passes
#pragma unroll
    for (int q = 0; q < ST_RY + 2; q++) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const T lo = s[q * ST_ROW + c], u = s[q * ST_ROW + 3 + c], hi = s[q * ST_ROW + 6 + c];
        const T e = (lo - u) + (hi - u);
        d2[q % 3][c] = e;
        m[q % 3][c] = fma(e, sixth, u);
        d[q % 3][c] = hi - lo;
      }
      if (q < 2) continue;
      const int r = q - 2, lo = (q - 2) % 3, mid = (q - 1) % 3, hi = q % 3;
      auto D2 = [&](const T (&f)[3][3], int c) { return (f[lo][c] - f[mid][c]) + (f[hi][c] - f[mid][c]); };
      auto Mm = [&](const T (&f)[3][3], int c, T dd) { return fma(dd, sixth, f[mid][c]); };
      auto Dd = [&](const T (&f)[3][3], int c) { return f[hi][c] - f[lo][c]; };
      T P[3], Q[3], R[3], fin[3];
      {
        const T y2 = D2(m, 0);
        P[0] = fma(C.xd, Dd(d, 1), fma(C.xy, y2, C.xx * Mm(d2, 0, D2(d2, 0))));
        Q[0] = C.q * Mm(m, 0, y2);
      }
      {
        const T y2 = D2(m, 1);
        P[1] = fma(C.xd, Dd(d, 0), fma(C.yy, y2, C.yx * Mm(d2, 1, D2(d2, 1))));
        Q[1] = C.q * Mm(m, 1, y2);
      }
      {
        const T y2 = D2(m, 2);
        P[2] = fma(C.xy, y2, C.yx * Mm(d2, 2, D2(d2, 2)));
        Q[2] = C.qz * Mm(m, 2, y2);
      }
      R[0] = C.rx * Mm(d, 2, D2(d, 2));
      R[1] = C.ry * Dd(m, 2);
      R[2] = fma(C.ry, Dd(m, 1), C.rx * Mm(d, 0, D2(d, 0)));
      T below[3];
#pragma unroll
      for (int c = 0; c < 3; c++) below[c] = up[r][c];
      stencil_march<T>(P, Q, R, acc[r], up[r], fin);
      if (end) {
        asm volatile("");  // a branch, not selects: it is taken on two planes
        stencil_end<T>(P, Q, R, k == 0 ? C.g : -C.g, below, acc[r]);
      }
      finish(r, nk - plane, fin, sp);
    }
#pragma unroll
    for (int r = 0; r < ST_RY; r++) fl[r] = nf[r];
    nk += plane;
    sp = s;
    slot = slot == ST_RING - 1 ? 0 : slot + 1;
    s = mine + slot * ST_PLANE;
  }
  if (kb == nz)  // the highest plane takes nothing from above
#pragma unroll
    for (int r = 0; r < ST_RY; r++) finish(r, nk - plane, acc[r], sp);
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if constexpr (DOT) {
    const double s = block_sum_dbl(dacc, red);
    if (tid == 0) A.dot[blockIdx.x] = s;
  }
}

// A face across axis n with tangential axis t: node strides along t and inward, components of
// t and n, sg with d_n f = sg (inner - face), and the terms of the missing half (of P, of R).
template <typename T> struct FaceAxes {
  int st, sn, ct, cn;
  T sg, em, el, fl, fm;
};
// P, Q, R of the face node with index n in its plane; the lanes of a warp hold consecutive nodes
// along t, so that the x-passes along t take their neighbours from the lanes beside (6 loads
// instead of 18: on an x face every lane's load is a cache line of its own).  Components t, n, z.
template <typename T>
__device__ __forceinline__ void stencil_face_plane(const T* __restrict__ x, int64_t n, const FaceAxes<T>& F,
                                                   const StencilCoef<T>& C, T (&P)[3], T (&Q)[3], T (&R)[3]) {
  const T sixth = T(1.0 / 6.0);
  T e2[2][3], m[2][3], d[2][3];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const T* u = x + 3 * (n + r * (int64_t)F.sn);
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const T mi = __ldg(u + (q == 0 ? F.ct : q == 1 ? F.cn : 2));
      const T lo = __shfl_up_sync(0xffffffffu, mi, 1), hi = __shfl_down_sync(0xffffffffu, mi, 1);
      const T e = (lo - mi) + (hi - mi);
      e2[r][q] = e;
      m[r][q] = fma(e, sixth, mi);
      d[r][q] = hi - lo;
    }
  }
  // across the face: mass f / 3 + f' / 6, second difference f' - f, d = sg (f' - f)
  auto Mn = [&](const T (&f)[2][3], int q) { return fma(f[1][q], sixth, f[0][q] * T(1.0 / 3.0)); };
  auto Dn = [&](const T (&f)[2][3], int q) { return f[1][q] - f[0][q]; };
  P[0] = fma(F.em, d[0][1], fma(C.xd * F.sg, Dn(d, 1), fma(C.xy, Dn(m, 0), C.xx * Mn(e2, 0))));
  P[1] = fma(F.el, d[0][0], fma(C.xd * F.sg, Dn(d, 0), fma(C.yy, Dn(m, 1), C.yx * Mn(e2, 1))));
  P[2] = fma(C.xy, Dn(m, 2), C.yx * Mn(e2, 2));
  Q[0] = C.q * Mn(m, 0);
  Q[1] = C.q * Mn(m, 1);
  Q[2] = C.qz * Mn(m, 2);
  R[0] = C.rx * Mn(d, 2);
  R[1] = fma(F.fl, m[0][2], C.ry * F.sg * Dn(m, 2));
  R[2] = fma(F.fm, m[0][1], fma(C.ry * F.sg, Dn(m, 1), C.rx * Mn(d, 0)));
}

// The x and y faces and the edges, by threads first, first + step, ... (whole warps); returns
// this thread's share of x.y.
template <typename T, bool DOT>
__device__ __forceinline__ double stencil_outer(const UApplyArgs<T>& A, int64_t first, int64_t step) {
  double dacc = 0.;
  const int nx = A.nx, ny = A.ny, nz = A.nz, ncx = nx - 2, ncy = ny - 2;
  const int64_t plane = (int64_t)nx * ny;
  const T eta = T(A.P->eta), S1 = T(1) + eta;
  const int lane = (int)(first & 31);
  // faces: groups of 30 columns (lanes 1 .. 30; 0 and 31 hold their neighbours), y and x faces in
  // turn, then runs of planes
  const int ngy = ceil_div(ncx, 30), ngx = ceil_div(ncy, 30), ng = face_groups(nx, ny), nmin = 2 * min(ngy, ngx);
  const int nw = face_warps(nx, ny, nz);
  for (int w = (int)(first >> 5); w < nw; w += (int)(step >> 5)) {
    const int g = w % ng, k0 = 1 + (w / ng) * ST_FACE_Z;
    const bool yf = g < 2 * nmin ? !(g & 1) : ngy > ngx;
    const int h = g < 2 * nmin ? g >> 1 : g - nmin;  // group among the faces of this axis
    const bool high = h & 1;
    const int nt = yf ? ncx : ncy, pos = (h >> 1) * 30 + lane;
    const bool mine = lane >= 1 && lane <= 30 && pos <= nt;
    const int at = min(pos, nt + 1);
    const int64_t n0 = k0 * plane + (yf ? (int64_t)(high ? ny - 1 : 0) * nx + at
                                        : (int64_t)at * nx + (high ? nx - 1 : 0));
    const int cnt = min(ST_FACE_Z, nz - 1 - k0);
    unsigned f[ST_FACE_Z];
    bool any = false;
#pragma unroll
    for (int c = 0; c < ST_FACE_Z; c++) {
      f[c] = kNodeElement;
      if (mine && c < cnt) f[c] = A.node[n0 + c * plane];
      any = any || !(f[c] & kNodeElement);
    }
    if (!__any_sync(0xffffffffu, any)) continue;
    const StencilCoefs& cc = A.P->st[yf ? 0 : 1];
    const StencilCoef<T> C(cc);
    FaceAxes<T> F;
    F.st = yf ? 1 : nx;
    F.sn = (yf ? nx : 1) * (high ? -1 : 1);
    F.ct = yf ? 0 : 1;
    F.cn = 1 - F.ct;
    F.sg = high ? T(-1) : T(1);
    F.em = -F.sg * T(cc.em);
    F.el = -F.sg * T(cc.el);
    F.fl = -F.sg * T(cc.fl);
    F.fm = -F.sg * T(cc.fm);
    T acc[3] = {T(0), T(0), T(0)}, up[3] = {T(0), T(0), T(0)}, out[ST_FACE_Z + 1][3];
    // every plane is evaluated (those beyond the run again its last one), so that the loads
    // of one plane do not wait for the others
#pragma unroll
    for (int c = -1; c <= ST_FACE_Z; c++) {
      T P[3], Q[3], R[3], fin[3];
      stencil_face_plane<T>(A.x, n0 + min(c, cnt) * plane, F, C, P, Q, R);
      stencil_march<T>(P, Q, R, acc, up, fin);
#pragma unroll
      for (int q = 0; q < 3; q++) out[c > 0 ? c - 1 : ST_FACE_Z][q] = fin[q];
    }
#pragma unroll
    for (int c = 0; c < ST_FACE_Z; c++)
      if (!(f[c] & kNodeElement)) {
        const T r3[3] = {yf ? out[c][0] : out[c][1], yf ? out[c][1] : out[c][0], out[c][2]};
        dacc += stencil_put<T, DOT>(A, S1, eta, n0 + c * plane, f[c], r3, A.x + 3 * (n0 + c * plane));
      }
  }
  // edges: 9 lanes per node, one per row of neighbours, three nodes per warp; summed in a fixed
  // order (one thread per node is a chain of 1500 dependent operations)
  const int nedge = edge_nodes(nx, ny, nz), g = lane / 9, rc = lane - 9 * g;
  for (int64_t w = first >> 5; w * 3 < nedge; w += step >> 5) {
    int q = (int)(3 * w) + g, i = 0, j = 0, k = 0;
    const bool on = g < 3 && q < nedge;
    if (q < 4 * ncx) {  // 4 (nx - 2) along x, 4 (ny - 2) along y, 4 nz along z with the corners
      i = 1 + (q >> 2);
      j = (q & 1) ? ny - 1 : 0;
      k = (q & 2) ? nz - 1 : 0;
    } else if ((q -= 4 * ncx) < 4 * ncy) {
      j = 1 + (q >> 2);
      i = (q & 1) ? nx - 1 : 0;
      k = (q & 2) ? nz - 1 : 0;
    } else {
      q -= 4 * ncy;
      k = q >> 2;
      i = (q & 1) ? nx - 1 : 0;
      j = (q & 2) ? ny - 1 : 0;
    }
    const int64_t n = on ? node_index(i, j, k, nx, ny) : 0;
    const unsigned f = on ? A.node[n] : kNodeElement;
    T r[3] = {T(0), T(0), T(0)};
    if (!(f & kNodeElement))
      stencil_edge_row<T>(A, i, j, k, rc % 3, rc / 3, T(A.P->L.lambda[0]), T(A.P->L.mu[0]), T(A.hx), T(A.hy),
                          T(A.hz), r);
    T sum[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      sum[c] = r[c];
#pragma unroll
      for (int s = 1; s < 9; s++) sum[c] += __shfl_sync(0xffffffffu, r[c], min(9 * g + s, 31));
    }
    if (rc == 0 && !(f & kNodeElement)) dacc += stencil_put<T, DOT>(A, S1, eta, n, f, sum, A.x + 3 * n);
  }
  return dacc;
}

// UOp for the nodes that the stencil (u_stencil.cuh) leaves to the elements: unit list 1
// of a plan built from the node flags.
template <typename T_, bool CUBIC = false> struct UOpMarked : UOp<T_, CUBIC> {
  using T = T_;
  using Args = UApplyArgs<T>;
  __device__ __forceinline__ static unsigned node_flags(const Args& A, int64_t n) { return A.node[n]; }
  __device__ __forceinline__ static bool skip_node(unsigned flags) { return !(flags & kNodeElement); }
  template <bool DOT>
  __device__ __forceinline__ static double finish_node(const Args& A, int64_t n, const T (&val)[3]) {
    const unsigned b = node_flags(A, n);
    T xin[3];
#pragma unroll
    for (int c = 0; c < 3; c++) xin[c] = (DOT || ((b >> c) & 1u)) ? A.x[3 * n + c] : T(0);
    return UOp<T_, CUBIC>::template finish_node_in<DOT>(A, n, val, b, xin);
  }
};

// The apply's last launch: blocks [0, nface) the stencil's faces and edges, the rest the element
// operator's seams; x.y partials to A.dot[dot_base + block].
template <class Op, bool DOT>
__global__ void __launch_bounds__(256, sizeof(typename Op::T) == 8 ? 2 : 3) u_outer_kernel(const __grid_constant__ typename Op::Args A, int TY,
                                                         int dot_base, int nface) {
  __shared__ double red[32];
  if (A.skip && *A.skip) return;
  double dacc;
  if ((int)blockIdx.x < nface)
    dacc = stencil_outer<typename Op::T, DOT>(A, (int64_t)blockIdx.x * 256 + threadIdx.x, (int64_t)nface * 256);
  else
    dacc = seam_range<Op, DOT>(A, TY, (int64_t)(blockIdx.x - nface) * 256 + threadIdx.x,
                               (int64_t)(gridDim.x - nface) * 256);
  if constexpr (DOT) {
    const double s = block_sum_dbl(dacc, red);
    if (threadIdx.x == 0) A.dot[dot_base + blockIdx.x] = s;
  }
}

}  // namespace vfgpu
