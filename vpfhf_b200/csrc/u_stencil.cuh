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
// about 115 operations per node against 234 per element plus the exchange and summation of
// its 24 nodal values.
//
// Rounding.  K(v) maps a constant to 0, so every sum is of values less the node's own: e = d2_x u and the
// second difference u2 across y (differences of neighbours) give 6 d2_y m_x u = 6 u2 + d2_y e and
// G = 36 (m_x m_y u - u) = 6 e + 6 d2_y m_x u; from plane to plane the own value moves by du, of
// which G takes 36.  Averages of full-size values would cancel for smooth u.  In FP64 the own value is
// taken without its low bits, which G gets back, so that du is exact (its rounding would be the
// largest of all for random u).  The 36 is left to S, which is held in two parts: one factor for all
// rows, whose rounding does not average out; then the coefficients are the rows' own.  P +- R are formed
// before the larger q G.  Passes in the vectors' type, rows in FP64 in both types: in FP32 alone the rows'
// chain of sums rounds random u more than the element sums do (7.4e-8).  Normwise error of one apply,
// element form / averages of u in the vectors' type / this form, x random and smooth (about a wave per box):
// FP32 129^3 5.5 / 6.6 / 5.1 and 1690 / 3320 / 20 in 1e-8; FP64 86 x 87 x 88 cubic cells 2.0 / 2.9 / 1.3
// and 160 / 293 / 8.4 in 1e-16, cells of 47 x 36 x 25 1.33 / 1.39 / 1.32.  Time of an apply in a loop
// (two cracks), same order: FP32 129^3 76 / 44 / 55 us, 161^3 136 / 68 / 93, 257 x 257 x 129 279 / 115 /
// 168; FP64 129^3 108 / 55 / 63, 97^3 60 / 47 / 51.  With FP32's passes in FP64 too (2.5e-8, the
// rounding of the result alone) 57.5, 97 and 176 us.
//
// Columns inside the box in x and y: a block owns 32 x 16 of them and marches up a chunk of
// planes, 4 rows of one column per thread.  Planes of 34 x 18 nodes stream through a 5-slot
// shared-memory ring by asynchronous copies three planes ahead, one barrier per plane; a
// thread makes the x-passes of the 6 rows its 4 outputs need (16.5 shared reads per node) and
// keeps per row what planes k - 1 and k give to node k, so nothing is exchanged between
// threads and no seam is summed.  127 = 4 x 32 - 1 = 8 x 16 - 1: the inside of the 2^k + 1 grids
// fills the tiles.  On the lowest and highest plane M is h (f / 2 + (f' - f) / 6), K is
// (f - f') / h, C = (f' - f) / 2 and T = -C -+ f: the node keeps 2 P - Q and a multiple of R.
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
using StencilReal = double;  // the arithmetic of the rows (the passes are in the vectors' type)

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
// row j + b - 1, plane k + c - 1 give, as values less the node's own, for any node of the box
// (used on its edges).
template <typename T, typename W>
__device__ __forceinline__ void stencil_edge_row(const UApplyArgs<T>& A, int i, int j, int k, int b, int c, W lam,
                                                 W mu, W hx, W hy, W hz, W (&y)[3]) {
  const Axis1D<W> X(i, A.nx, hx), Y(j, A.ny, hy), Z(k, A.nz, hz);
  const W l2 = lam + W(2) * mu;
  const int kk = min(max(k + c - 1, 0), A.nz - 1), jj = min(max(j + b - 1, 0), A.ny - 1);  // beyond: weight 0
  const T* own = A.x + 3 * node_index(i, j, k, A.nx, A.ny);
  W M[3], K[3], C[3], D[3];
#pragma unroll
  for (int q = 0; q < 3; q++) M[q] = K[q] = C[q] = D[q] = W(0);
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const T* u = A.x + 3 * node_index(min(max(i + a - 1, 0), A.nx - 1), jj, kk, A.nx, A.ny);
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const W v = W(__ldg(u + q)) - W(__ldg(own + q));
      M[q] = fma(X.M[a], v, M[q]);
      K[q] = fma(X.K[a], v, K[q]);
      C[q] = fma(X.C[a], v, C[q]);
      D[q] = fma(X.D[a], v, D[q]);
    }
  }
  auto at = [](const W (&f)[3], int q) { return q == 0 ? f[0] : q == 1 ? f[1] : f[2]; };
  const W My = at(Y.M, b), Ky = at(Y.K, b), Cy = at(Y.C, b), Dy = at(Y.D, b);
  const W Mz = at(Z.M, c), Kz = at(Z.K, c), Cz = at(Z.C, c), Dz = at(Z.D, c);
  y[0] = Mz * (l2 * (K[0] * My) + mu * (M[0] * Ky) + lam * (D[1] * Cy) + mu * (C[1] * Dy)) +
         Kz * (mu * (M[0] * My)) + My * (lam * (D[2] * Cz) + mu * (C[2] * Dz));
  y[1] = Mz * (mu * (K[1] * My) + l2 * (M[1] * Ky) + lam * (C[0] * Dy) + mu * (D[0] * Cy)) +
         Kz * (mu * (M[1] * My)) + M[2] * (lam * (Dy * Cz) + mu * (Cy * Dz));
  y[2] = Mz * (mu * (K[2] * My + M[2] * Ky)) + Kz * (l2 * (M[2] * My)) +
         My * (lam * (C[0] * Dz) + mu * (D[0] * Cz)) + M[1] * (lam * (Cy * Dz) + mu * (Dy * Cz));
}

// u without its low 32 bits (FP64): the difference of two of them near one another is exact.  FP32 as it is.
__device__ __forceinline__ double stencil_high(double u) { return __hiloint2double(__double2hiint(u), 0); }
__device__ __forceinline__ float stencil_high(float u) { return u; }

// Takes in plane k of a row: fin = its share of node k - 1, whose rest acc holds; then acc = what planes
// k - 1 and k give to node k, up = what plane k gives to node k + 1.  P is 6 times, q G and R 36 times
// the rows' P, Q, R; G and R of the values less the plane's own reference, which changes by du from plane k - 1
// (M: G's multiple of a constant; on a FACE R changes by f dr).
template <int M, bool FACE, typename W>
__device__ __forceinline__ void stencil_march(W P, W q, W G, W R, W du, W f, W dr, W& acc, W& up, W& rest, W& fin) {
  rest = acc;
  fin = fma(q, fma(W(M), du, G), P + (FACE ? fma(f, dr, R) : R));
  acc = fma(W(4), P, fma(W(-2) * q, fma(W(M / 2), du, G), FACE ? fma(f, dr, up) : up));
  up = fma(q, G, P - R);
}

// v^2 + eta, or its 36th, as a rounded value and the rest: one factor for every row of a homogeneous
// patch, so its rounding would not average out.
struct StencilScale {
  double hi, lo;
  __device__ __forceinline__ StencilScale(double v, double eta, bool over36) {
    const double s = fma(v, v, eta), b = s - eta, r = fma(v, v, -b) + (eta - (s - b));
    hi = s;
    lo = r;
    if (over36) {
      const double c = 1.0 / 36.0, q = s * c;
      hi = fma(fma(-36., q, s), c, q);
      lo = (fma(-36., hi, s) + r) * c;
    }
  }
};

// Writes a node from the two parts of its rows (without S; 36 times them where OVER36), flags and x; with
// DOT returns its x.y.  S1: the scale at v = 1.
template <typename T, bool DOT, bool OVER36, typename W>
__device__ __forceinline__ double stencil_put(const UApplyArgs<T>& A, const StencilScale& S1, double eta, int64_t n, unsigned f,
                                              const W (&r)[3], const W (&r2)[3], const T* xin) {
  StencilScale S = S1;
  if (!(f & kNodeOne)) S = StencilScale(A.v[n], eta, OVER36);
  T y[3];
#pragma unroll
  for (int c = 0; c < 3; c++)
    y[c] = T(fma(S.hi, r[c], sizeof(T) == 8 ? fma(S.lo, r[c] + r2[c], S.hi * r2[c]) : S.hi * r2[c]));
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
  using W = StencilReal;
  const double eta = A.P->eta;
  const StencilScale S1(1., eta, true);
  const int64_t plane = (int64_t)nx * ny;
  double dacc = 0.;
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
  const StencilCoefs C = A.P->st[0];
  const T rx = T(C.rx), ry = T(C.ry);
  const int i = X0 + 1 + lane, j0 = Y0 + 1 + wy * ST_RY;
  // rows of this thread whose nodes lie inside the x and y faces
  const int rows = i < nx - 1 ? min(max(ny - 1 - j0, 0), ST_RY) : 0;
  int64_t nk = (int64_t)j0 * nx + i + kf * plane;  // node of row 0 in plane k
  W acc[ST_RY][3], up[ST_RY][3];
#pragma unroll
  for (int r = 0; r < ST_RY; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) acc[r][c] = up[r][c] = W(0);
  unsigned fl[ST_RY];
#pragma unroll
  for (int r = 0; r < ST_RY; r++) fl[r] = kNodeElement;
  // writes row r of the plane whose row 0 is node n and whose ring slot starts at xr
  auto finish = [&](int r, int64_t n, const W (&rest)[3], const W (&fin)[3], const T* xr) {
    if (fl[r] & kNodeElement) return;
    T xin[3];
#pragma unroll
    for (int c = 0; c < 3; c++) xin[c] = T(0);
    if (DOT || (fl[r] & 7u))
#pragma unroll
      for (int c = 0; c < 3; c++) xin[c] = xr[(r + 1) * ST_ROW + 3 + c];
    dacc += stencil_put<T, DOT, true>(A, S1, eta, n + r * nx, fl[r], rest, fin, xin);
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
    T u[3][3], e[3][3], d[3][3];  // [row mod 3][component]: x-passes
#pragma unroll
    for (int q = 0; q < ST_RY + 2; q++) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const T lo = s[q * ST_ROW + c], at = s[q * ST_ROW + 3 + c], hi = s[q * ST_ROW + 6 + c];
        u[q % 3][c] = at;
        e[q % 3][c] = (lo - at) + (hi - at);
        d[q % 3][c] = hi - lo;
      }
      if (q < 2) continue;
      const int r = q - 2, lo = (q - 2) % 3, mid = (q - 1) % 3, hi = q % 3;
      auto M6 = [&](const T (&f)[3][3], int c) { return fma(T(4), f[mid][c], f[lo][c] + f[hi][c]); };  // 6 m_y f
      auto Dd = [&](const T (&f)[3][3], int c) { return f[hi][c] - f[lo][c]; };
      auto Dm = [&](int c) { return fma(T(6), Dd(u, c), Dd(e, c)); };  // 6 d_y m_x u
      T G[3], du[3];
      W P[3], R[3], rest[3], fin[3];
      {
        T y2[3], me[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const T u2 = (u[lo][c] - u[mid][c]) + (u[hi][c] - u[mid][c]), es = e[lo][c] + e[hi][c];
          y2[c] = fma(T(6), u2, fma(T(-2), e[mid][c], es));  // 6 d2_y m_x u
          me[c] = fma(T(4), e[mid][c], es);                  // 6 m_y d2_x u
          const T own = stencil_high(u[mid][c]);
          du[c] = own - stencil_high(sp[(r + 1) * ST_ROW + 3 + c]);  // 0 at the first plane
          G[c] = fma(T(6), u2, sizeof(T) == 8 ? fma(T(36), u[mid][c] - own, me[c]) : me[c]);
        }
        P[0] = fma(C.xd, W(Dd(d, 1)), fma(C.xy, W(y2[0]), C.xx * W(me[0])));
        P[1] = fma(C.xd, W(Dd(d, 0)), fma(C.yy, W(y2[1]), C.yx * W(me[1])));
        P[2] = fma(C.xy, W(y2[2]), C.yx * W(me[2]));
      }
      R[0] = W(rx * M6(d, 2));
      R[1] = W(ry * Dm(2));
      R[2] = W(fma(ry, Dm(1), rx * M6(d, 0)));
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const W qc = c < 2 ? C.q : C.qz, below = up[r][c];
        stencil_march<36, false, W>(P[c], qc, G[c], R[c], du[c], W(0), W(0), acc[r][c], up[r][c], rest[c], fin[c]);
        if (end) {
          asm volatile("");  // a branch, not selects: it is taken on two planes
          const W g = (k == 0) == (c < 2) ? C.g : -C.g;
          acc[r][c] = fma(-qc, fma(W(36), W(du[c]), W(G[c])), fma(W(2), P[c], fma(g, R[c], below)));
        }
      }
      finish(r, nk - plane, rest, fin, sp);
    }
#pragma unroll
    for (int r = 0; r < ST_RY; r++) fl[r] = nf[r];
    nk += plane;
    sp = s;
    slot = slot == ST_RING - 1 ? 0 : slot + 1;
    s = mine + slot * ST_PLANE;
  }
  if (kb == nz) {  // the highest plane takes nothing from above
    const W none[3] = {W(0), W(0), W(0)};
#pragma unroll
    for (int r = 0; r < ST_RY; r++) finish(r, nk - plane, acc[r], none, sp);
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  if constexpr (DOT) {
    const double s = block_sum_dbl(dacc, red);
    if (tid == 0) A.dot[blockIdx.x] = s;
  }
}

// A face across axis n with tangential axis t: node strides along t and inward, components of
// t and n, sg with d_n f = sg (inner - face), and the terms of the missing half (of P, of R).
template <typename W> struct FaceAxes {
  int st, sn, ct, cn;
  W sg, em, el, fl, fm;
};
// P, G, R of the face node with index n in its plane, and its references; the lanes of a warp hold
// consecutive nodes along t, so that the x-passes along t take their neighbours from the lanes
// beside (6 loads instead of 18: on an x face every lane's load is a cache line of its own).
// Components t, n, z.
template <typename T, typename W>
__device__ __forceinline__ void stencil_face_plane(const T* __restrict__ x, int64_t n, const FaceAxes<W>& F,
                                                   const StencilCoefs& C, W (&P)[3], W (&G)[3], W (&R)[3],
                                                   W (&u0)[3]) {
  W e[2][3], d[2][3], u[2][3];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const T* a = x + 3 * (n + r * (int64_t)F.sn);
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const T mi = __ldg(a + (q == 0 ? F.ct : q == 1 ? F.cn : 2));
      const W lo = __shfl_up_sync(0xffffffffu, mi, 1), hi = __shfl_down_sync(0xffffffffu, mi, 1);
      u[r][q] = mi;
      e[r][q] = (lo - u[r][q]) + (hi - u[r][q]);
      d[r][q] = hi - lo;
    }
  }
  // across the face: mass f / 3 + f' / 6, second difference f' - f, d = sg (f' - f)
  auto M6 = [&](const W (&f)[2][3], int q) { return fma(W(2), f[0][q], f[1][q]); };
  auto Dn = [&](const W (&f)[2][3], int q) { return f[1][q] - f[0][q]; };
  W dm[3], m0[3];  // 6 (m_t u' - m_t u) and 6 (m_t u - u0)
#pragma unroll
  for (int q = 0; q < 3; q++) {
    dm[q] = fma(W(6), Dn(u, q), Dn(e, q));
    u0[q] = stencil_high(u[0][q]);
    m0[q] = fma(W(6), u[0][q] - u0[q], e[0][q]);
    G[q] = fma(W(3), m0[q], dm[q]);
  }
  P[0] = fma(F.em, d[0][1], fma(C.xd * F.sg, Dn(d, 1), fma(C.xy, dm[0], C.xx * M6(e, 0))));
  P[1] = fma(F.el, d[0][0], fma(C.xd * F.sg, Dn(d, 0), fma(C.yy, dm[1], C.yx * M6(e, 1))));
  P[2] = fma(C.xy, dm[2], C.yx * M6(e, 2));
  R[0] = C.rx * M6(d, 2);
  R[1] = fma(F.fl, m0[2], C.ry * F.sg * dm[2]);
  R[2] = fma(F.fm, m0[1], fma(C.ry * F.sg, dm[1], C.rx * M6(d, 0)));
}

// The x and y faces and the edges, by threads first, first + step, ... (whole warps); returns
// this thread's share of x.y.
template <typename T, bool DOT>
__device__ __forceinline__ double stencil_outer(const UApplyArgs<T>& A, int64_t first, int64_t step) {
  double dacc = 0.;
  const int nx = A.nx, ny = A.ny, nz = A.nz, ncx = nx - 2, ncy = ny - 2;
  const int64_t plane = (int64_t)nx * ny;
  using W = StencilReal;
  const double eta = A.P->eta;
  const StencilScale S1(1., eta, true);
  const W none[3] = {W(0), W(0), W(0)};
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
    const StencilCoefs& C = A.P->st[yf ? 0 : 1];
    FaceAxes<W> F;
    F.st = yf ? 1 : nx;
    F.sn = (yf ? nx : 1) * (high ? -1 : 1);
    F.ct = yf ? 0 : 1;
    F.cn = 1 - F.ct;
    F.sg = high ? W(-1) : W(1);
    F.em = -F.sg * C.em;
    F.el = -F.sg * C.el;
    F.fl = -F.sg * C.fl;
    F.fm = -F.sg * C.fm;
    const W cR[3] = {W(0), W(6) * F.fl, W(6) * F.fm};
    W acc[3] = {W(0), W(0), W(0)}, up[3] = {W(0), W(0), W(0)}, last[3];
    // every plane is evaluated (those beyond the run again its last one), so that the loads
    // of one plane do not wait for the others
#pragma unroll
    for (int c = -1; c <= ST_FACE_Z; c++) {
      W P[3], G[3], R[3], u[3], du[3], rest[3], fin[3];
      stencil_face_plane<T>(A.x, n0 + min(c, cnt) * plane, F, C, P, G, R, u);
#pragma unroll
      for (int q = 0; q < 3; q++) {
        du[q] = c >= 0 ? u[q] - last[q] : W(0);
        last[q] = u[q];
      }
#pragma unroll
      for (int q = 0; q < 3; q++)
        stencil_march<18, true, W>(P[q], q < 2 ? C.q : C.qz, G[q], R[q], du[q], cR[q], du[q == 1 ? 2 : 1], acc[q],
                                   up[q], rest[q], fin[q]);
      if (c > 0 && !(f[c - 1] & kNodeElement)) {
        const W a[3] = {yf ? rest[0] : rest[1], yf ? rest[1] : rest[0], rest[2]};
        const W b[3] = {yf ? fin[0] : fin[1], yf ? fin[1] : fin[0], fin[2]};
        const int64_t n = n0 + (c - 1) * plane;
        dacc += stencil_put<T, DOT, true>(A, S1, eta, n, f[c - 1], a, b, A.x + 3 * n);
      }
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
    W r[3] = {W(0), W(0), W(0)};
    if (!(f & kNodeElement))
      stencil_edge_row<T, W>(A, i, j, k, rc % 3, rc / 3, A.P->L.lambda[0], A.P->L.mu[0], A.hx, A.hy, A.hz, r);
    W sum[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      sum[c] = r[c];
#pragma unroll
      for (int s = 1; s < 9; s++) sum[c] += __shfl_sync(0xffffffffu, r[c], min(9 * g + s, 31));
    }
    if (rc == 0 && !(f & kNodeElement)) dacc += stencil_put<T, DOT, false>(A, StencilScale(1., eta, false), eta, n, f, sum, none, A.x + 3 * n);
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
__global__ void __launch_bounds__(256, 2) u_outer_kernel(const __grid_constant__ typename Op::Args A, int TY, int dot_base,
                                                         int nface) {
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
