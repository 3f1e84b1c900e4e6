// ops.cuh -- element operators plugged into the tile engine.
//
//   UOp: y = K(v) x, the degraded elasticity operator of VF_BilinearFormU3D_local
//        (VFMech.c:227-290) with Dirichlet rows identity (VFCartFE.c:1147-1296).
#pragma once

#include "f2.cuh"
#include "tile_engine.cuh"
#include "u_apply.cuh"

namespace vfgpu {

// CUBIC: hx = hy = hz, every 1/h factor folds into the row weight (u_element).
template <typename T_, bool CUBIC = false> struct UOp {
  using T = T_;
  using Args = UApplyArgs<T>;
  static constexpr int NC = 3, NIN = 4, EPT = 1;
  static constexpr int LIST = 1;  // the unit list this operator takes in a split launch
  __device__ __forceinline__ static void node_src(const Args& A, int64_t n, const T* (&src)[NIN]) {
    src[0] = A.x + 3 * n;
    src[1] = A.x + 3 * n + 1;
    src[2] = A.x + 3 * n + 2;
    src[3] = A.v + n;
  }
  // The cell's Lame coefficients (material layer table, or per-cell modulus).
  __device__ __forceinline__ static void lame(const Args& A, const LayerTable& L, int ex, int ey,
                                              int ez, T& lam, T& mu) {
    const int layer = A.elayer ? A.elayer[ez] : 0;
    const LayerTable& LT = A.P ? A.P->L : L;
    if (A.cellE) {
      const T E = T(A.cellE[((int64_t)ez * (A.ny - 1) + ey) * (A.nx - 1) + ex]);
      lam = E * T(LT.lamfac[layer]);
      mu = E * T(LT.mufac[layer]);
    } else {
      lam = T(LT.lambda[layer]);
      mu = T(LT.mu[layer]);
    }
  }
  __device__ __forceinline__ static T eta_of(const Args& A) { return A.P ? T(A.P->eta) : A.eta; }
  __device__ __forceinline__ static void element(const Args& A, const LayerTable& L, int ex,
                                                 int ey, int ez, const T (&in)[8][NIN],
                                                 T (&out)[8][NC]) {
    T xn[8][3], vn[8];
#pragma unroll
    for (int a = 0; a < 8; a++) {
      xn[a][0] = in[a][0];
      xn[a][1] = in[a][1];
      xn[a][2] = in[a][2];
      vn[a] = in[a][3];
    }
    T lam, mu;
    lame(A, L, ex, ey, ez, lam, mu);
    const T eta = eta_of(A);
    // an element whose nodal phase field is constant (the intact bulk, v = 1) takes the
    // fixed-weight form; the rest the row closed form
    const T v0 = vn[0];
    bool cst = true;
#pragma unroll
    for (int a = 1; a < 8; a++) cst = cst && vn[a] == v0;
    if (cst)
      u_element_const<T, CUBIC>(xn, fma(v0, v0, eta), lam, mu, A.ihx, A.ihy, A.ihz, A.vol, out);
    else
      u_element<T, CUBIC>(xn, vn, lam, mu, eta, A.ihx, A.ihy, A.ihz, A.vol, out);
  }
  // The same for an element known to have a constant nodal phase field (the choice
  // element makes for it, without the general form in the code path).
  __device__ __forceinline__ static void element_const(const Args& A, const LayerTable& L, int ex,
                                                       int ey, int ez, const T (&in)[8][NIN],
                                                       T (&out)[8][NC]) {
    T xn[8][3];
#pragma unroll
    for (int a = 0; a < 8; a++) {
      xn[a][0] = in[a][0];
      xn[a][1] = in[a][1];
      xn[a][2] = in[a][2];
    }
    T lam, mu;
    lame(A, L, ex, ey, ez, lam, mu);
    const T v0 = in[0][3];
    u_element_const<T, CUBIC>(xn, fma(v0, v0, eta_of(A)), lam, mu, A.ihx, A.ihy, A.ihz, A.vol, out);
  }
  // The per-node flags finish_node needs (Dirichlet bits), loaded ahead by the tiles.
  __device__ __forceinline__ static unsigned node_flags(const Args& A, int64_t n) {
    return A.bc ? A.bc[n] : 0u;
  }
  __device__ __forceinline__ static bool skip_node(unsigned) { return false; }
  // Writes y of node n (Dirichlet rows: y = x) from the node's flags b and input
  // values xin; with DOT, returns x.y over its dofs (the launch accumulates the CG dot
  // into A.dot).
  template <bool DOT>
  __device__ __forceinline__ static double finish_node_in(const Args& A, int64_t n, const T (&val)[NC],
                                                          unsigned b, const T (&xin)[NC]) {
    double d = 0.;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const T y = ((b >> c) & 1u) ? xin[c] : val[c];
      A.y[3 * n + c] = y;
      if constexpr (DOT) d += (double)xin[c] * (double)y;
    }
    return d;
  }
  // The same with the flags and inputs read from global memory (the seam fix-up).
  template <bool DOT>
  __device__ __forceinline__ static double finish_node(const Args& A, int64_t n, const T (&val)[NC]) {
    const unsigned b = node_flags(A, n);
    T xin[NC];
#pragma unroll
    for (int c = 0; c < 3; c++) xin[c] = (DOT || ((b >> c) & 1u)) ? A.x[3 * n + c] : T(0);
    return finish_node_in<DOT>(A, n, val, b, xin);
  }
};

// UOp for the units of unit list 0, whose elements all have a constant nodal phase
// field: the fixed-weight element alone (the choice UOp::element makes for them, with
// the same arithmetic), compiled without the general element.
template <typename T_, bool CUBIC = false> struct UOpConst : UOp<T_, CUBIC> {
  using Base = UOp<T_, CUBIC>;
  using T = T_;
  using Args = UApplyArgs<T>;
  static constexpr int LIST = 0;
  __device__ __forceinline__ static void element(const Args& A, const LayerTable& L, int ex,
                                                 int ey, int ez, const T (&in)[8][Base::NIN],
                                                 T (&out)[8][Base::NC]) {
    Base::element_const(A, L, ex, ey, ez, in, out);
  }
};

// The NOCOMPRESSION U operator: UOp with the per-point element u_element_nc and the
// per-cell compression bits A.cflag.
template <typename T_> struct UOpNC {
  using T = T_;
  using Args = UApplyArgs<T>;
  static constexpr int NC = 3, NIN = 4, EPT = 1;
  static constexpr int LIST = -1;
  __device__ __forceinline__ static void node_src(const Args& A, int64_t n, const T* (&src)[NIN]) {
    UOp<T>::node_src(A, n, src);
  }
  __device__ __forceinline__ static void element(const Args& A, const LayerTable& L, int ex,
                                                 int ey, int ez, const T (&in)[8][NIN],
                                                 T (&out)[8][NC]) {
    T xn[8][3], vn[8];
#pragma unroll
    for (int a = 0; a < 8; a++) {
      xn[a][0] = in[a][0];
      xn[a][1] = in[a][1];
      xn[a][2] = in[a][2];
      vn[a] = in[a][3];
    }
    const int layer = A.elayer ? A.elayer[ez] : 0;
    const LayerTable& LT = A.P ? A.P->L : L;
    const T eta = A.P ? T(A.P->eta) : A.eta;
    const int64_t cell = ((int64_t)ez * (A.ny - 1) + ey) * (A.nx - 1) + ex;
    T lam, mu;
    if (A.cellE) {
      const T E = T(A.cellE[cell]);
      lam = E * T(LT.lamfac[layer]);
      mu = E * T(LT.mufac[layer]);
    } else {
      lam = T(LT.lambda[layer]);
      mu = T(LT.mu[layer]);
    }
    u_element_nc<T>(xn, vn, lam, mu, eta, A.ihx, A.ihy, A.ihz, A.vol, A.cflag[cell], out);
  }
  __device__ __forceinline__ static unsigned node_flags(const Args& A, int64_t n) {
    return UOp<T>::node_flags(A, n);
  }
  __device__ __forceinline__ static bool skip_node(unsigned) { return false; }
  template <bool DOT>
  __device__ __forceinline__ static double finish_node_in(const Args& A, int64_t n, const T (&val)[NC],
                                                          unsigned b, const T (&xin)[NC]) {
    return UOp<T>::template finish_node_in<DOT>(A, n, val, b, xin);
  }
  template <bool DOT>
  __device__ __forceinline__ static double finish_node(const Args& A, int64_t n, const T (&val)[NC]) {
    return UOp<T>::template finish_node<DOT>(A, n, val);
  }
};

// The FP32 U operator on two y-adjacent elements per thread, one per lane of the
// packed FP32 instructions (f2): the same arithmetic as UOp<float> with half the
// instructions.
struct UOpF2 {
  using T = float;
  using Args = UApplyArgs<float>;
  static constexpr int NC = 3, NIN = 4, EPT = 2;
  static constexpr int LIST = -1;
  __device__ __forceinline__ static void node_src(const Args& A, int64_t n, const T* (&src)[NIN]) {
    UOp<float>::node_src(A, n, src);
  }
  __device__ __forceinline__ static void element_multi(const Args& A, const LayerTable& L, int ex,
                                                       const int (&ey)[2], int ez, const bool (&ok)[2],
                                                       const T (&in)[2][8][NIN], T (&out)[2][8][NC]) {
    f2 xn[8][3], vn[8];
#pragma unroll
    for (int a = 0; a < 8; a++) {
#pragma unroll
      for (int c = 0; c < 3; c++) xn[a][c] = f2(in[0][a][c], in[1][a][c]);
      vn[a] = f2(in[0][a][3], in[1][a][3]);
    }
    const int layer = A.elayer ? A.elayer[ez] : 0;
    const LayerTable& LT = A.P ? A.P->L : L;
    const float eta = A.P ? float(A.P->eta) : A.eta;
    f2 lam, mu;
    if (A.cellE) {
      float E[2];
#pragma unroll
      for (int e = 0; e < 2; e++)
        E[e] = ok[e] ? A.cellE[((int64_t)ez * (A.ny - 1) + ey[e]) * (A.nx - 1) + ex] : 0.f;
      const f2 Ep(E[0], E[1]);
      lam = Ep * f2(float(LT.lamfac[layer]));
      mu = Ep * f2(float(LT.mufac[layer]));
    } else {
      lam = f2(float(LT.lambda[layer]));
      mu = f2(float(LT.mu[layer]));
    }
    f2 y[8][3];
    u_element<f2>(xn, vn, lam, mu, f2(eta), f2(A.ihx), f2(A.ihy), f2(A.ihz), f2(A.vol), y);
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
      for (int c = 0; c < 3; c++) {
        out[0][a][c] = ok[0] ? y[a][c].v.x : 0.f;
        out[1][a][c] = ok[1] ? y[a][c].v.y : 0.f;
      }
  }
  __device__ __forceinline__ static unsigned node_flags(const Args& A, int64_t n) {
    return UOp<float>::node_flags(A, n);
  }
  __device__ __forceinline__ static bool skip_node(unsigned) { return false; }
  template <bool DOT>
  __device__ __forceinline__ static double finish_node_in(const Args& A, int64_t n, const T (&val)[NC],
                                                          unsigned b, const T (&xin)[NC]) {
    return UOp<float>::finish_node_in<DOT>(A, n, val, b, xin);
  }
  template <bool DOT>
  __device__ __forceinline__ static double finish_node(const Args& A, int64_t n, const T (&val)[NC]) {
    return UOp<float>::finish_node<DOT>(A, n, val);
  }
};

// UOpConst<float, CUBIC> on two y-adjacent elements per thread, one per lane of the
// packed FP32 instructions (f2): unit list 0 of the FP32 split.  u_element_const has no
// contractible multiply-add, so each lane gives the scalar kernel's bits.
template <bool CUBIC = false> struct UOpF2Const {
  using T = float;
  using Args = UApplyArgs<float>;
  static constexpr int NC = 3, NIN = 4, EPT = 2;
  static constexpr int LIST = 0;
  __device__ __forceinline__ static void node_src(const Args& A, int64_t n, const T* (&src)[NIN]) {
    UOp<float>::node_src(A, n, src);
  }
  __device__ __forceinline__ static void element_multi(const Args& A, const LayerTable& L, int ex,
                                                       const int (&ey)[2], int ez, const bool (&ok)[2],
                                                       const T (&in)[2][8][NIN], T (&out)[2][8][NC]) {
    f2 xn[8][3];
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
      for (int c = 0; c < 3; c++) xn[a][c] = f2(in[0][a][c], in[1][a][c]);
    const int layer = A.elayer ? A.elayer[ez] : 0;
    const LayerTable& LT = A.P ? A.P->L : L;
    const float eta = A.P ? float(A.P->eta) : A.eta;
    f2 lam, mu;
    if (A.cellE) {
      float E[2];
#pragma unroll
      for (int e = 0; e < 2; e++)
        E[e] = ok[e] ? A.cellE[((int64_t)ez * (A.ny - 1) + ey[e]) * (A.nx - 1) + ex] : 0.f;
      const f2 Ep(E[0], E[1]);
      lam = Ep * f2(float(LT.lamfac[layer]));
      mu = Ep * f2(float(LT.mufac[layer]));
    } else {
      lam = f2(float(LT.lambda[layer]));
      mu = f2(float(LT.mu[layer]));
    }
    const f2 v0(in[0][0][3], in[1][0][3]);
    f2 y[8][3];
    u_element_const<f2, CUBIC>(xn, fma(v0, v0, f2(eta)), lam, mu, f2(A.ihx), f2(A.ihy), f2(A.ihz),
                               f2(A.vol), y);
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
      for (int c = 0; c < 3; c++) {
        out[0][a][c] = ok[0] ? y[a][c].v.x : 0.f;
        out[1][a][c] = ok[1] ? y[a][c].v.y : 0.f;
      }
  }
  __device__ __forceinline__ static unsigned node_flags(const Args& A, int64_t n) {
    return UOp<float>::node_flags(A, n);
  }
  __device__ __forceinline__ static bool skip_node(unsigned) { return false; }
  template <bool DOT>
  __device__ __forceinline__ static double finish_node_in(const Args& A, int64_t n, const T (&val)[NC],
                                                          unsigned b, const T (&xin)[NC]) {
    return UOp<float>::template finish_node_in<DOT>(A, n, val, b, xin);
  }
  template <bool DOT>
  __device__ __forceinline__ static double finish_node(const Args& A, int64_t n, const T (&val)[NC]) {
    return UOp<float>::template finish_node<DOT>(A, n, val);
  }
};

}  // namespace vfgpu
