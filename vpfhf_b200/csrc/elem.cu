// elem.cu -- once-per-solve element kernels, after the reference's element routines.  The plain
// operator's element vectors are summed in one pass (cell_gather_kernel); the NOCOMPRESSION
// forms are written per Gauss point and scattered to nodes in 8 parity colours of elements, so
// that no two threads of a launch touch the same node.  Both are deterministic, without
// atomics.  The element tables travel by value in the kernel parameters (__grid_constant__):
// every thread of a warp reads the same entry, which the constant bank broadcasts.
#include <algorithm>
#include <cmath>

#include "elem.h"
#include "vmat.h"

namespace vfgpu {

void etab_host(double hx, double hy, double hz, ETab* e) {
  // VFCartFEElement1DInit (VFCartFE.c:90-116), tensor product as VFCartFEElement3DInit.
  auto t1 = [](double l, double w[3], double phi[2][3], double dphi[2][3]) {
    w[0] = 5. * l / 18.;
    w[1] = 8. * l / 18.;
    w[2] = 5. * l / 18.;
    phi[0][0] = (1. + sqrt(3. / 5.)) * .5;
    phi[0][1] = .5;
    phi[0][2] = (1. - sqrt(3. / 5.)) * .5;
    phi[1][0] = (1. - sqrt(3. / 5.)) * .5;
    phi[1][1] = .5;
    phi[1][2] = (1. + sqrt(3. / 5.)) * .5;
    for (int g = 0; g < 3; g++) {
      dphi[0][g] = -1. / l;
      dphi[1][g] = 1. / l;
    }
  };
  double wx[3], wy[3], wz[3], px[2][3], py[2][3], pz[2][3], dx[2][3], dy[2][3], dz[2][3];
  t1(hx, wx, px, dx);
  t1(hy, wy, py, dy);
  t1(hz, wz, pz, dz);
  for (int gk = 0, g = 0; gk < 3; gk++)
    for (int gj = 0; gj < 3; gj++)
      for (int gi = 0; gi < 3; gi++, g++) {
        e->w[g] = wz[gk] * wy[gj] * wx[gi];
        for (int k = 0; k < 2; k++)
          for (int j = 0; j < 2; j++)
            for (int i = 0; i < 2; i++) {
              const int a = i + 2 * j + 4 * k;
              e->phi[a][g] = pz[k][gk] * py[j][gj] * px[i][gi];
              e->dphi[a][0][g] = pz[k][gk] * py[j][gj] * dx[i][gi];
              e->dphi[a][1][g] = pz[k][gk] * dy[j][gj] * px[i][gi];
              e->dphi[a][2][g] = dz[k][gk] * py[j][gj] * px[i][gi];
            }
      }
}

namespace {

struct CellMat {
  double lambda, mu, alpha, beta, Gc;
};

__device__ __forceinline__ CellMat cell_mat(const ElemArgs& E, int ei, int ej, int ek) {
  const int l = E.elayer ? E.elayer[ek] : 0;
  CellMat m;
  if (E.cellE) {
    const double Ec = (double)E.cellE[((int64_t)ek * (E.ny - 1) + ej) * (E.nx - 1) + ei];
    m.lambda = Ec * E.L.lamfac[l];
    m.mu = Ec * E.L.mufac[l];
  } else {
    m.lambda = E.L.lambda[l];
    m.mu = E.L.mu[l];
  }
  m.alpha = E.L.alpha[l];
  m.beta = E.L.beta[l];
  m.Gc = E.L.Gc[l];
  return m;
}

__device__ __forceinline__ void cell_nodes(const ElemArgs& E, int ei, int ej, int ek,
                                           int64_t (&n)[8]) {
#pragma unroll
  for (int a = 0; a < 8; a++)
    n[a] = node_index(ei + (a & 1), ej + ((a >> 1) & 1), ek + (a >> 2), E.nx, E.ny);
}

// Element (ei,ej,ek) of colour (cx,cy,cz) for the linear thread index t, or false.
__device__ __forceinline__ bool colour_cell(const ElemArgs& E, int color, int64_t t, int& ei,
                                            int& ej, int& ek) {
  const int cx = color & 1, cy = (color >> 1) & 1, cz = color >> 2;
  const int hx = (E.nx - 1 - cx + 1) / 2, hy = (E.ny - 1 - cy + 1) / 2, hz = (E.nz - 1 - cz + 1) / 2;
  if (t >= (int64_t)hx * hy * hz) return false;
  ei = cx + 2 * (int)(t % hx);
  ej = cy + 2 * (int)((t / hx) % hy);
  ek = cz + 2 * (int)(t / ((int64_t)hx * hy));
  return true;
}

// tr(eps(u)) at Gauss point g from the 8 nodal displacements, in the reference's order
__device__ __forceinline__ double trace_at(const ETab& e, const double (&u8)[8][3], int g) {
  double tr = 0.;
  for (int a = 0; a < 8; a++)
    tr += e.dphi[a][0][g] * u8[a][0] + e.dphi[a][1][g] * u8[a][1] + e.dphi[a][2][g] * u8[a][2];
  return tr;
}

__device__ __forceinline__ void gather_u8(const int64_t (&n)[8], const double* __restrict__ u,
                                          double (&u8)[8][3]) {
  for (int a = 0; a < 8; a++)
    for (int c = 0; c < 3; c++) u8[a][c] = u ? u[3 * n[a] + c] : 0.;
}

// ---- tensor-product forms (the plain operator).  On the uniform grid the 27-point rule
// is the tensor product of the 1-D rule, and every table entry is a product of 1-D
// factors: phi_a(g) = b_k(gz) b_j(gy) b_i(gx), dphi_a,x(g) = b_k(gz) b_j(gy) (-+1/hx),
// w_g = W_gx W_gy W_gz vol, with b_0(g) = (1 + sqrt(3/5))/2, 1/2, (1 - sqrt(3/5))/2 at
// the three points, b_1 the mirror, W = 5/18, 8/18, 5/18 (VFCartFEElement1DInit,
// VFCartFE.c:90-116).  So fields at the points, the integrals against products of
// basis functions and the scatter back to the nodes are each three 1-D passes.
constexpr double kB0 = 0.5 * (1.0 + 0.774596669241483377035853079956);  // (1 + sqrt(3/5))/2
constexpr double kB2 = 0.5 * (1.0 - 0.774596669241483377035853079956);
__device__ __forceinline__ constexpr double bas(int i, int g) {
  return g == 1 ? 0.5 : ((g == 0) == (i == 0) ? kB0 : kB2);
}
__device__ __forceinline__ constexpr double w1(int g) { return g == 1 ? 8.0 / 18.0 : 5.0 / 18.0; }

// Modal form of a trilinear field on the unit cell t in [-1/2, 1/2]^3: f = sum_p m_p t^p
// (p = px + 2 py + 4 pz; m_0 the mean, m_1 the x slope, ...).
__device__ __forceinline__ void modal_of(const double (&f)[8], double (&m)[8]) {
  double a[8], b[8];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    a[2 * p] = 0.5 * (f[2 * p] + f[2 * p + 1]);
    a[2 * p + 1] = f[2 * p + 1] - f[2 * p];
  }
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int al = 0; al < 2; al++) {
      const double lo = a[al + 4 * k], hi = a[al + 2 + 4 * k];
      b[al + 4 * k] = 0.5 * (lo + hi);
      b[al + 2 + 4 * k] = hi - lo;
    }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const double lo = b[q], hi = b[q + 4];
    m[q] = 0.5 * (lo + hi);
    m[q + 4] = hi - lo;
  }
}
// Trilinear field at the 27 points, g = gx + 3 gy + 9 gz.
__device__ __forceinline__ void interp27(const double (&f)[8], double (&o)[27]) {
  double fx[4][3], fy[2][3][3];
#pragma unroll
  for (int jk = 0; jk < 4; jk++)
#pragma unroll
    for (int g = 0; g < 3; g++) fx[jk][g] = bas(0, g) * f[2 * jk] + bas(1, g) * f[2 * jk + 1];
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int gy = 0; gy < 3; gy++)
#pragma unroll
      for (int gx = 0; gx < 3; gx++)
        fy[k][gy][gx] = bas(0, gy) * fx[2 * k][gx] + bas(1, gy) * fx[2 * k + 1][gx];
#pragma unroll
  for (int gz = 0; gz < 3; gz++)
#pragma unroll
    for (int gy = 0; gy < 3; gy++)
#pragma unroll
      for (int gx = 0; gx < 3; gx++)
        o[gx + 3 * gy + 9 * gz] = bas(0, gz) * fy[0][gy][gx] + bas(1, gz) * fy[1][gy][gx];
}

// Products of two trilinear fields against the basis, in closed form (the 3-point rule is exact
// for their degrees).  For axis d the other two, in increasing order, are bits ax1 and ax2 of a
// modal index (modal_of), and a field's 4 transverse coefficients at power 0 or 1 of t_d are
// m[(P ? d's bit : 0) + ...].
__device__ __forceinline__ constexpr int ax1(int d) { return d == 0 ? 2 : 1; }
__device__ __forceinline__ constexpr int ax2(int d) { return d == 2 ? 2 : 4; }
template <int P> __device__ __forceinline__ void transverse(const double (&m)[8], int d, double (&f)[4]) {
#pragma unroll
  for (int q = 0; q < 4; q++) f[q] = m[(P ? 1 << d : 0) + ((q & 1) ? ax1(d) : 0) + ((q & 2) ? ax2(d) : 0)];
}
// X[a][b] (+)= coefficient of t1^a t2^b in the product of two bilinear fields.
template <bool ADD>
__device__ __forceinline__ void bilinear_product(const double (&f)[4], const double (&g)[4], double (&X)[3][3]) {
  const double q[3][3] = {{f[0] * g[0], fma(f[0], g[2], f[2] * g[0]), f[2] * g[2]},
                          {fma(f[0], g[1], f[1] * g[0]),
                           fma(f[0], g[3], f[3] * g[0]) + fma(f[1], g[2], f[2] * g[1]), fma(f[2], g[3], f[3] * g[2])},
                          {f[1] * g[1], fma(f[1], g[3], f[3] * g[1]), f[3] * g[3]}};
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) X[a][b] = ADD ? X[a][b] + q[a][b] : q[a][b];
}
// F[p][q] = integral of sum X[a][b] t1^a t2^b against b_p(t1) b_q(t2), b = 1/2 -+ t.
__device__ __forceinline__ void bilinear_moments(const double (&X)[3][3], double (&F)[2][2]) {
  double C[2][3];
#pragma unroll
  for (int b = 0; b < 3; b++) {
    const double e = .5 * fma(X[2][b], 1. / 12., X[0][b]), o = X[1][b] * (1. / 12.);
    C[0][b] = e - o;
    C[1][b] = e + o;
  }
#pragma unroll
  for (int p = 0; p < 2; p++) {
    const double e = .5 * fma(C[p][2], 1. / 12., C[p][0]), o = C[p][1] * (1. / 12.);
    F[p][0] = e - o;
    F[p][1] = e + o;
  }
}
// F[p][q]: the product of two fields (modal) integrated over axis d and against the basis along
// the other two.
__device__ __forceinline__ void product_face(const double (&f)[8], const double (&g)[8], int d, double (&F)[2][2]) {
  double a[4], b[4], X[3][3];
  transverse<0>(f, d, a);
  transverse<0>(g, d, b);
  bilinear_product<false>(a, b, X);
  transverse<1>(f, d, a);
  transverse<1>(g, d, b);
#pragma unroll
  for (int q = 0; q < 4; q++) b[q] *= 1. / 12.;
  bilinear_product<true>(a, b, X);
  bilinear_moments(X, F);
}

// Integrals of q against the squared or plain basis products that carry no factor
// along axis d: F[d][p][q] = sum_g q_g f_p(g_e1) f_q(g_e2) with (e1, e2) the other two
// axes in increasing order, f = b (SQ = false) or b^2 (SQ = true).
template <bool SQ>
__device__ __forceinline__ void face_moments(const double (&q)[27], double (&F)[3][2][2]) {
  auto f = [](int p, int g) { return SQ ? bas(p, g) * bas(p, g) : bas(p, g); };
  double R[3][3][3];  // R[d][ga][gb]: q summed along axis d, indexed by the other two
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) {
      R[0][a][b] = (q[0 + 3 * a + 9 * b] + q[1 + 3 * a + 9 * b]) + q[2 + 3 * a + 9 * b];  // (gy, gz)
      R[1][a][b] = (q[a + 0 + 9 * b] + q[a + 3 + 9 * b]) + q[a + 6 + 9 * b];              // (gx, gz)
      R[2][a][b] = (q[a + 3 * b] + q[a + 3 * b + 9]) + q[a + 3 * b + 18];                 // (gx, gy)
    }
#pragma unroll
  for (int d = 0; d < 3; d++)
#pragma unroll
    for (int pq = 0; pq < 2; pq++) {
      double t[3];
#pragma unroll
      for (int a = 0; a < 3; a++) t[a] = (f(pq, 0) * R[d][a][0] + f(pq, 1) * R[d][a][1]) + f(pq, 2) * R[d][a][2];
#pragma unroll
      for (int p = 0; p < 2; p++) F[d][p][pq] = (f(p, 0) * t[0] + f(p, 1) * t[1]) + f(p, 2) * t[2];
    }
}

// The U diagonal in tensor form (plain operator): diag of node (i,j,k), component x, is
//   (lambda + 2 mu) Jx[j][k] / hx^2 + mu (Jy[i][k] / hy^2 + Jz[i][j] / hz^2)
// with J_d the integrals of w (v^2 + eta) against the squared basis functions of the
// other two axes (and similarly for y, z).
struct UDiagCell {
  static constexpr int NF = 1, NV = 3, MINB = 2;  // nodal fields, values per corner, blocks per SM
  const double* __restrict__ v;
  const uint8_t* __restrict__ bc;  // Dirichlet bits or null
  double* __restrict__ d;
  __device__ __forceinline__ void load(int64_t n, double (&q)[NF]) const { q[0] = v[n]; }
  __device__ __forceinline__ void put(int64_t n, const double (&y)[NV]) const {
    const unsigned b = bc ? bc[n] : 0u;
#pragma unroll
    for (int c = 0; c < 3; c++) d[3 * n + c] = (b >> c) & 1u ? 1. : y[c];
  }
  __device__ __forceinline__ void cell(const ElemArgs& E, int ei, int ej, int ek, const double (&q)[NF][8],
                                       double (&out)[8][NV]) const {
    double v27[27], s27[27];
    interp27(q[0], v27);
    const double vol = E.hx * E.hy * E.hz;
#pragma unroll
    for (int gz = 0; gz < 3; gz++)
#pragma unroll
      for (int gy = 0; gy < 3; gy++)
#pragma unroll
        for (int gx = 0; gx < 3; gx++) {
          const int g = gx + 3 * gy + 9 * gz;
          s27[g] = (vol * (w1(gx) * w1(gy) * w1(gz))) * fma(v27[g], v27[g], E.eta);
        }
    double J[3][2][2];
    face_moments<true>(s27, J);
    const CellMat m = cell_mat(E, ei, ej, ek);
    const double l2m = m.lambda + 2. * m.mu;
    const double ih2[3] = {1. / (E.hx * E.hx), 1. / (E.hy * E.hy), 1. / (E.hz * E.hz)};
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const double jx = J[0][j][k] * ih2[0], jy = J[1][i][k] * ih2[1], jz = J[2][i][j] * ih2[2];
          const int a = i + 2 * j + 4 * k;
          out[a][0] = fma(l2m, jx, m.mu * (jy + jz));
          out[a][1] = fma(l2m, jy, m.mu * (jx + jz));
          out[a][2] = fma(l2m, jz, m.mu * (jx + jy));
        }
  }
};

// The U load in tensor form (plain operator): the thermo-poro load
// sum_g w dphi_a,c S_g, S = 3 kappa alpha (theta - thetaRef)(v^2 + eta) + beta p v, as
// face moments of w S times -+1/h_c (the beta term in closed form, the thermal one point by point
// and only where theta differs from thetaRef at a node), and the crack-pressure load
// sum_g w p grad_c v phi_a in closed form.  The crack-pressure term of an element with 8 equal
// nodal v (and finite p) is 0 and not evaluated: grad v is exactly 0 there.
struct URhsCell {
  static constexpr int NF = 3, NV = 3, MINB = 1;
  const double *__restrict__ v, *__restrict__ theta, *__restrict__ thetaRef, *__restrict__ p;
  double* __restrict__ f;
  __device__ __forceinline__ void load(int64_t n, double (&q)[NF]) const {
    q[0] = v[n];
    q[1] = theta ? theta[n] - (thetaRef ? thetaRef[n] : 0.) : 0.;
    q[2] = p ? p[n] : 0.;
  }
  __device__ __forceinline__ void put(int64_t n, const double (&y)[NV]) const {
#pragma unroll
    for (int c = 0; c < 3; c++) f[3 * n + c] = y[c];
  }
  __device__ __forceinline__ void cell(const ElemArgs& E, int ei, int ej, int ek, const double (&fld)[NF][8],
                                       double (&rl)[8][NV]) const {
    const double (&v8)[8] = fld[0], (&th8)[8] = fld[1], (&p8)[8] = fld[2];
    const CellMat m = cell_mat(E, ei, ej, ek);
    const double coefalpha = (3. * m.lambda + 2. * m.mu) * m.alpha, beta = m.beta;
    const double vol = E.hx * E.hy * E.hz;
    const double ih[3] = {1. / E.hx, 1. / E.hy, 1. / E.hz};
    double vm[8], pm[8], F[3][2][2];
    modal_of(v8, vm);
    modal_of(p8, pm);
    bool thermal = false;
#pragma unroll
    for (int a = 0; a < 8; a++) thermal = thermal || !(th8[a] == 0.);
    if (thermal) {
      double ve[27], ws[27], te[27];
      interp27(v8, ve);
      interp27(th8, te);
#pragma unroll
      for (int gz = 0; gz < 3; gz++)
#pragma unroll
        for (int gy = 0; gy < 3; gy++)
#pragma unroll
          for (int gx = 0; gx < 3; gx++) {
            const int g = gx + 3 * gy + 9 * gz;
            ws[g] = (vol * (w1(gx) * w1(gy) * w1(gz))) * (coefalpha * te[g] * (ve[g] * ve[g] + E.eta));
          }
      face_moments<false>(ws, F);
    } else {
#pragma unroll
      for (int d = 0; d < 3; d++) F[d][0][0] = F[d][0][1] = F[d][1][0] = F[d][1][1] = 0.;
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
      double G[2][2];
      product_face(pm, vm, d, G);
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int k = 0; k < 2; k++) F[d][j][k] = fma(vol * beta, G[j][k], F[d][j][k]);
    }
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const int a = i + 2 * j + 4 * k;
          rl[a][0] = (i ? ih[0] : -ih[0]) * F[0][j][k];
          rl[a][1] = (j ? ih[1] : -ih[1]) * F[1][i][k];
          rl[a][2] = (k ? ih[2] : -ih[2]) * F[2][i][j];
        }
    bool flat = true;
    double ps = 0.;
#pragma unroll
    for (int a = 0; a < 8; a++) {
      flat = flat && v8[a] == v8[0];
      ps += fabs(p8[a]);
    }
    if (E.hasCrackPressure && !(flat && ps - ps == 0.)) {
      // d_c v has no power of t_c: transverse products with p at powers 0 and 1 of t_c
#pragma unroll
      for (int c = 0; c < 3; c++) {
        double g[4], q[4], X[3][3], F0[2][2], F1[2][2];
        transverse<1>(vm, c, g);
        transverse<0>(pm, c, q);
        bilinear_product<false>(q, g, X);
        bilinear_moments(X, F0);
        transverse<1>(pm, c, q);
        bilinear_product<false>(q, g, X);
        bilinear_moments(X, F1);
        const double w = vol * ih[c];
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
          for (int j = 0; j < 2; j++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
              const int t = c == 0 ? i : (c == 1 ? j : k), p = c == 0 ? j : i, r = c == 2 ? j : k;
              const double m = fma(t ? 1. / 12. : -1. / 12., F1[p][r], .5 * F0[p][r]);
              rl[i + 2 * j + 4 * k][c] = fma(w, m, rl[i + 2 * j + 4 * k][c]);
            }
      }
    }
  }
};

// The U load under NOCOMPRESSION, one colour of elements.
__global__ void u_rhs_kernel(const __grid_constant__ ElemArgs E, int color, const double* __restrict__ v,
                             const double* __restrict__ theta, const double* __restrict__ thetaRef,
                             const double* __restrict__ p, double* __restrict__ f,
                             const double* __restrict__ u0) {
  int ei, ej, ek;
  if (!colour_cell(E, color, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, ei, ej, ek)) return;
  const ETab& e = E.tab;
  int64_t n[8];
  cell_nodes(E, ei, ej, ek, n);
  double v8[8], th8[8], p8[8], rl[24];
#pragma unroll
  for (int a = 0; a < 8; a++) {
    v8[a] = v[n[a]];
    th8[a] = theta ? theta[n[a]] - (thetaRef ? thetaRef[n[a]] : 0.) : 0.;
    p8[a] = p ? p[n[a]] : 0.;
  }
  for (int l = 0; l < 24; l++) rl[l] = 0.;
  const CellMat m = cell_mat(E, ei, ej, ek);
  // VF_GradientUThermoPoro3D_local (VFMech.c:386-447); NOCOMPRESSION
  // (VFMech.c:456-524): undegraded thermal term and p instead of p v where tr < 0
  const double coefalpha = (3. * m.lambda + 2. * m.mu) * m.alpha, beta = m.beta;
  double u8[8][3];
  gather_u8(n, u0, u8);
  for (int g = 0; g < 27; g++) {
    double te = 0., pe = 0., ve = 0.;
    for (int a = 0; a < 8; a++) {
      te += e.phi[a][g] * th8[a];
      pe += e.phi[a][g] * p8[a];
      ve += e.phi[a][g] * v8[a];
    }
    const bool comp = trace_at(e, u8, g) < 0.;
    const double s = comp ? coefalpha * te * (1. + E.eta) + beta * pe
                          : coefalpha * te * (ve * ve + E.eta) + beta * pe * ve;
    for (int a = 0; a < 8; a++)
      for (int c = 0; c < 3; c++) rl[3 * a + c] += e.w[g] * e.dphi[a][c][g] * s;
  }
  // VF_GradientUCrackPressure3D_local (VFMech.c:533-589)
  if (E.hasCrackPressure) {
    for (int g = 0; g < 27; g++) {
      double pe = 0., gv[3] = {0., 0., 0.};
      for (int a = 0; a < 8; a++) {
        pe += e.phi[a][g] * p8[a];
        for (int c = 0; c < 3; c++) gv[c] += e.dphi[a][c][g] * v8[a];
      }
      for (int a = 0; a < 8; a++)
        for (int c = 0; c < 3; c++) rl[3 * a + c] += e.w[g] * pe * gv[c] * e.phi[a][g];
    }
  }
  for (int a = 0; a < 8; a++)
    for (int c = 0; c < 3; c++) f[3 * n[a] + c] += rl[3 * a + c];
}

// The U diagonal under NOCOMPRESSION, one colour of elements.
__global__ void u_diag_kernel(const __grid_constant__ ElemArgs E, int color, const double* __restrict__ v,
                              double* __restrict__ d, const double* __restrict__ u0) {
  int ei, ej, ek;
  if (!colour_cell(E, color, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, ei, ej, ek)) return;
  const ETab& e = E.tab;
  int64_t n[8];
  cell_nodes(E, ei, ej, ek, n);
  double v8[8], dg[24];
#pragma unroll
  for (int a = 0; a < 8; a++) v8[a] = v[n[a]];
  for (int l = 0; l < 24; l++) dg[l] = 0.;
  const CellMat m = cell_mat(E, ei, ej, ek);
  double u8[8][3];
  gather_u8(n, u0, u8);
  const double kappa = m.lambda + 2. * m.mu / 3.;
  for (int g = 0; g < 27; g++) {
    double s = 0.;
    for (int a = 0; a < 8; a++) s += v8[a] * e.phi[a][g];
    const double sv = s * s + E.eta, ws = e.w[g] * sv;
    // spherical coefficient: lambda s, or kappa (1 + eta) - 2 mu s / 3 in compression
    const bool comp = trace_at(e, u8, g) < 0.;
    const double lw = comp ? e.w[g] * (kappa * (1. + E.eta) - 2. * m.mu * sv / 3.) : ws * m.lambda;
    for (int a = 0; a < 8; a++) {
      const double d0 = e.dphi[a][0][g], d1 = e.dphi[a][1][g], d2 = e.dphi[a][2][g];
      const double g2 = d0 * d0 + d1 * d1 + d2 * d2;
      dg[3 * a + 0] += (lw + ws * m.mu) * d0 * d0 + ws * m.mu * g2;
      dg[3 * a + 1] += (lw + ws * m.mu) * d1 * d1 + ws * m.mu * g2;
      dg[3 * a + 2] += (lw + ws * m.mu) * d2 * d2 + ws * m.mu * g2;
    }
  }
  for (int a = 0; a < 8; a++)
    for (int c = 0; c < 3; c++) d[3 * n[a] + c] += dg[3 * a + c];
}

__global__ void nc_flags_kernel(const __grid_constant__ ElemArgs E, const double* __restrict__ u,
                                uint32_t* __restrict__ flags) {
  const int64_t NCELL = (int64_t)(E.nx - 1) * (E.ny - 1) * (E.nz - 1);
  const int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= NCELL) return;
  const int ei = (int)(cell % (E.nx - 1));
  const int ej = (int)((cell / (E.nx - 1)) % (E.ny - 1));
  const int ek = (int)(cell / ((int64_t)(E.nx - 1) * (E.ny - 1)));
  int64_t n[8];
  cell_nodes(E, ei, ej, ek, n);
  double u8[8][3];
  gather_u8(n, u, u8);
  uint32_t bits = 0u;
  for (int g = 0; g < 27; g++)
    if (trace_at(E.tab, u8, g) < 0.) bits |= 1u << g;
  flags[cell] = bits;
}

__global__ void bc_diag_kernel(const uint8_t* __restrict__ bcbits, double* __restrict__ d, int64_t N) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned b = bcbits[i];
    for (int c = 0; c < 3; c++)
      if ((b >> c) & 1u) d[3 * i + c] = 1.;
  }
}

// ---- the assembled V operator (vmat.h): 14 couplings per node.
//
// Along a Gauss row the strain is linear in t = tx, so twice the energy density (the
// coupling coefficient 2 W, ElasticEnergyDensity3D_local, VFMech.c:32-106, plus the AT2 mass
// coefficient, VFMech.c:2040-2058) is c0 + c1 t + c2 t^2 there and its row moments against
// 1, t, t^2 follow from mean t^2 = 1/12, mean t^4 = 1/80 (odd means vanish): the reference's
// 3-point sums.  Products of two 1-D basis functions are 1/4 - t + t^2 (both at the low
// node), 1/4 - t^2 (one each) and 1/4 + t + t^2 (both high), so the cell's element matrix has
// 27 distinct entries, one per product type and axis, built by sum factorisation; the
// stiffness part (Gc / 2 c_w) eps grad . grad is a constant per type.  A corner's row sum R is
// the sum of the mass part over the 8 types it is in (the stiffness part's row sums are 0).  NOCOMPRESSION
// (VFMech.c:115-218, 2125-2153) evaluates the row's three points instead (sign per point).
__device__ __forceinline__ void v_cell_types(const ElemArgs& E, const CellMat& mat,
                                             const double (&m)[3][8], const double (&mth)[8],
                                             double (&M)[27], double (&R)[8]) {
  const double ih[3] = {1. / E.hx, 1. / E.hy, 1. / E.hz};
  const double vol = E.hx * E.hy * E.hz;
  const double mass = E.atnum == 2 ? mat.Gc / E.atcv * .5 / E.epsilon : 0.;
  const double lam = mat.lambda, mu = mat.mu;
  // product of the basis functions of type p (0: low low, 1: low high, 2: high high) at point g
  auto bb = [](int p, int g) { return bas(p == 2 ? 1 : 0, g) * bas(p == 0 ? 0 : 1, g); };
#pragma unroll
  for (int t = 0; t < 27; t++) M[t] = 0.;
#pragma unroll
  for (int gz = 0; gz < 3; gz++) {
    const double tz = gz == 1 ? 0. : (gz == 0 ? -VF_TAU : VF_TAU);
    double cxy[3][3];  // [py][px]
#pragma unroll
    for (int q = 0; q < 9; q++) cxy[q / 3][q % 3] = 0.;
#pragma unroll
    for (int gy = 0; gy < 3; gy++) {
      const double ty = gy == 1 ? 0. : (gy == 0 ? -VF_TAU : VF_TAU);
      double X[3], ay[3], by[3], az[3], bz[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        X[c] = ih[0] * fma(fma(m[c][7], tz, m[c][3]), ty, fma(m[c][5], tz, m[c][1]));
        ay[c] = ih[1] * fma(m[c][6], tz, m[c][2]);
        by[c] = ih[1] * fma(m[c][7], tz, m[c][3]);
        az[c] = ih[2] * fma(m[c][6], ty, m[c][4]);
        bz[c] = ih[2] * fma(m[c][7], ty, m[c][5]);
      }
      const double a0 = mat.alpha * fma(fma(mth[6], tz, mth[2]), ty, fma(mth[4], tz, mth[0]));
      const double a1 = mat.alpha * fma(fma(mth[7], tz, mth[3]), ty, fma(mth[5], tz, mth[1]));
      // twice the shear strains, value and slope along the row
      const double s01 = X[1] + ay[0], s02 = X[2] + az[0], s12 = ay[2] + az[1], r12 = by[2] + bz[1];
      double S0, S1, S2;  // row moments of the coefficient against 1, t, t^2
      if (E.unilateral) {
        S0 = S1 = S2 = 0.;
        const double kappa = lam + 2. * mu / 3.;
#pragma unroll
        for (int gx = 0; gx < 3; gx++) {
          const double t = gx == 1 ? 0. : (gx == 0 ? -VF_TAU : VF_TAU);
          const double exx = X[0], eyy = fma(by[1], t, ay[1]), ezz = fma(bz[2], t, az[2]);
          const double at = fma(a1, t, a0);
          const double g01 = fma(by[0], t, s01), g02 = fma(bz[0], t, s02), g12 = fma(r12, t, s12);
          // W = sigma(eps - e0) : eps, less (kappa/2) tr^2 where tr < 0
          const double tr = exx + eyy + ezz, te = tr - 3. * at;
          const double Wf = .5 * (lam * te * tr + 2. * mu * ((exx - at) * exx + (eyy - at) * eyy + (ezz - at) * ezz)) +
                            .5 * mu * (g01 * g01 + g02 * g02 + g12 * g12);
          const double S = tr < 0. ? 0. : kappa * tr * tr * .5, D = Wf - kappa * tr * tr * .5;
          const double c = w1(gx) * (2. * (S + D) + mass);
          S0 += c;
          S1 = fma(t, c, S1);
          S2 = fma(t * t, c, S2);
        }
      } else {
        const double e0 = X[0] - a0, e1 = ay[1] - a0, e2 = az[2] - a0;
        const double f0 = -a1, f1 = by[1] - a1, f2 = bz[2] - a1;
        const double T0 = (e0 + e1) + e2, T1 = (f0 + f1) + f2;
        const double c0 = fma(lam * T0, T0, fma(2. * mu, fma(e0, e0, fma(e1, e1, e2 * e2)),
                                                mu * fma(s01, s01, fma(s02, s02, s12 * s12)))) + mass;
        const double c1 = 2. * fma(lam * T0, T1, fma(2. * mu, fma(e0, f0, fma(e1, f1, e2 * f2)),
                                                     mu * fma(s01, by[0], fma(s02, bz[0], s12 * r12))));
        const double c2 = fma(lam * T1, T1, fma(2. * mu, fma(f0, f0, fma(f1, f1, f2 * f2)),
                                                mu * fma(by[0], by[0], fma(bz[0], bz[0], r12 * r12))));
        S0 = fma(c2, 1. / 12., c0);
        S1 = c1 * (1. / 12.);
        S2 = fma(c2, 1. / 80., c0 * (1. / 12.));
      }
      const double q = fma(S0, .25, S2);
      const double px[3] = {q - S1, fma(S0, .25, -S2), q + S1};
#pragma unroll
      for (int py = 0; py < 3; py++)
#pragma unroll
        for (int x = 0; x < 3; x++) cxy[py][x] = fma(w1(gy) * bb(py, gy), px[x], cxy[py][x]);
    }
#pragma unroll
    for (int pz = 0; pz < 3; pz++)
#pragma unroll
      for (int py = 0; py < 3; py++)
#pragma unroll
        for (int x = 0; x < 3; x++)
          M[x + 3 * py + 9 * pz] = fma(w1(gz) * bb(pz, gz), cxy[py][x], M[x + 3 * py + 9 * pz]);
  }
  double Rx[2][9], Ry[4][3];  // a corner low or high along an axis is in two of its three types
#pragma unroll
  for (int q = 0; q < 9; q++)
#pragma unroll
    for (int i = 0; i < 2; i++) Rx[i][q] = M[3 * q + i] + M[3 * q + i + 1];
#pragma unroll
  for (int pz = 0; pz < 3; pz++)
#pragma unroll
    for (int a = 0; a < 4; a++) Ry[a][pz] = Rx[a & 1][3 * pz + (a >> 1)] + Rx[a & 1][3 * pz + (a >> 1) + 1];
#pragma unroll
  for (int a = 0; a < 8; a++) R[a] = vol * (Ry[a & 3][a >> 2] + Ry[a & 3][(a >> 2) + 1]);
  const double kx = mat.Gc / E.atcv * .5 * E.epsilon * vol;
  const double ix = kx * ih[0] * ih[0], iy = kx * ih[1] * ih[1], iz = kx * ih[2] * ih[2];
  constexpr double st[3] = {1., -1., 1.}, ms[3] = {1. / 3., 1. / 6., 1. / 3.};
#pragma unroll
  for (int pz = 0; pz < 3; pz++)
#pragma unroll
    for (int py = 0; py < 3; py++)
#pragma unroll
      for (int x = 0; x < 3; x++) {
        const double k = fma(ix, st[x] * ms[py] * ms[pz], fma(iy, ms[x] * st[py] * ms[pz], iz * (ms[x] * ms[py] * st[pz])));
        M[x + 3 * py + 9 * pz] = fma(vol, M[x + 3 * py + 9 * pz], k);
      }
}

// Assembles the couplings.  A block owns 31 x 7 node columns and the 32 x 8 cell columns
// around them, and marches up a chunk of node planes: per element layer each thread writes its
// cell's 27 entries to shared memory, then its node gathers them from the 4 cells around it
// (entry high-high in z of layer k - 1 carried in registers), so every coupling is summed in
// one fixed order with no atomics and no colours.  The cells on the seams of the blocks are
// computed twice (18 %).  FP64 issue bounds it.  It replaces the 27 coefficients per cell (in
// both precisions) and the diagonal's 8 coloured passes over them: 0.60 ms per StepV at
// 129^3, 0.41 ms now.
constexpr int VM_NX = 31, VM_NY = 7;
__global__ void __launch_bounds__(256, 1) v_assemble_kernel(const __grid_constant__ ElemArgs E,
                                                            const double* __restrict__ u,
                                                            const double* __restrict__ theta,
                                                            const double* __restrict__ thetaRef,
                                                            double* __restrict__ a64,
                                                            float* __restrict__ a32, int64_t stride, int gx,
                                                            int zc) {
  extern __shared__ double vm_s[];  // [27 + 8][8][32]
  const int l = threadIdx.x, w = threadIdx.y;
  const int nx = E.nx, ny = E.ny, nz = E.nz;
  const int ex = (int)(blockIdx.x % gx) * VM_NX - 1 + l, ey = (int)(blockIdx.x / gx) * VM_NY - 1 + w;
  const bool cell = ex >= 0 && ex < nx - 1 && ey >= 0 && ey < ny - 1;
  const bool node = l > 0 && w > 0 && ex < nx && ey < ny;  // owns node column (ex, ey)
  const int z0 = blockIdx.y * zc, z1 = min(z0 + zc, nz);
  const int64_t plane = (int64_t)nx * ny;
  const int64_t base = cell ? (int64_t)ey * nx + ex : 0;
  double f[3][8], th8[8], carry[6];  // of the couplings within the plane, and of the row sum
#pragma unroll
  for (int q = 0; q < 6; q++) carry[q] = 0.;
  auto load4 = [&](int k) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int64_t n = base + k * plane + (j >> 1) * nx + (j & 1);
#pragma unroll
      for (int c = 0; c < 3; c++) f[c][4 + j] = cell ? u[3 * n + c] : 0.;
      th8[4 + j] = (cell && theta) ? theta[n] - (thetaRef ? thetaRef[n] : 0.) : 0.;
    }
  };
  const int k0 = max(z0 - 1, 0);
  load4(k0);
  for (int k = k0; k < z1; k++) {
    double* s = vm_s + w * 32 + l;
    if (k < nz - 1) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
#pragma unroll
        for (int c = 0; c < 3; c++) f[c][j] = f[c][4 + j];
        th8[j] = th8[4 + j];
      }
      load4(k + 1);
      double M[27], R[8];
      if (cell) {
        double m[3][8], mth[8];
#pragma unroll
        for (int c = 0; c < 3; c++) modal_of(f[c], m[c]);
        modal_of(th8, mth);
        v_cell_types(E, cell_mat(E, ex, ey, k), m, mth, M, R);
      } else {
#pragma unroll
        for (int t = 0; t < 27; t++) M[t] = 0.;
#pragma unroll
        for (int a = 0; a < 8; a++) R[a] = 0.;
      }
#pragma unroll
      for (int t = 0; t < 27; t++) s[t * 256] = M[t];
#pragma unroll
      for (int a = 0; a < 8; a++) s[(27 + a) * 256] = R[a];
    }
    __syncthreads();
    if (node) {
      // the coupling (dx, dy) of z type pz over the 4 cells: lanes l - 1 (the node is the
      // cell's high x corner) and l, rows w - 1 and w
      auto gather = [&](int dx, int dy, int pz) {
        double r = 0.;
#pragma unroll
        for (int yy = 0; yy < 2; yy++) {
          if ((yy == 0 && dy > 0) || (yy == 1 && dy < 0)) continue;
          const int py = dy ? 1 : (yy == 0 ? 2 : 0);
#pragma unroll
          for (int xx = 0; xx < 2; xx++) {
            if ((xx == 0 && dx > 0) || (xx == 1 && dx < 0)) continue;
            const int px = dx ? 1 : (xx == 0 ? 2 : 0);
            r += s[(px + 3 * py + 9 * pz) * 256 + (yy - 1) * 32 + xx - 1];
          }
        }
        return r;
      };
      // the row sum's share of the 4 cells in which the node is low (0) or high (1) in z
      auto gather_sum = [&](int hz) {
        return (s[(27 + 3 + 4 * hz) * 256 - 33] + s[(27 + 2 + 4 * hz) * 256 - 32]) +
               (s[(27 + 1 + 4 * hz) * 256 - 1] + s[(27 + 4 * hz) * 256]);
      };
      const bool layer = k < nz - 1;
      if (k >= z0) {
        const int64_t n = (int64_t)k * plane + (int64_t)ey * nx + ex;
        auto put = [&](int d, double v) {
          a64[d * stride + n] = v;
          if (a32) a32[d * stride + n] = (float)v;
        };
#pragma unroll
        for (int q = 0; q < 5; q++)
          put(q, carry[q] + (layer ? gather(kVForward[q][0], kVForward[q][1], 0) : 0.));
#pragma unroll
        for (int q = 5; q < kVCouplings; q++)
          put(q, layer ? gather(kVForward[q][0], kVForward[q][1], 1) : 0.);
        put(kVRowSum, carry[5] + (layer ? gather_sum(0) : 0.));
      }
      if (layer) {
#pragma unroll
        for (int q = 0; q < 5; q++) carry[q] = gather(kVForward[q][0], kVForward[q][1], 2);
        carry[5] = gather_sum(1);
      }
    }
    __syncthreads();  // the next layer rewrites the entries
  }
}

// V load (VF_ResidualVAT1/AT23D_local and VF_ResidualVCrackPressure3D_local,
// VFMech.c:2294-2384) in tensor form: the AT term coef sum_g w phi_a = coef vol / 8 per
// node, the crack-pressure term sum_g w p (u . grad phi_a) as face moments of p u_c in closed form.
struct VRhsCell {
  static constexpr int NF = 4, NV = 1, MINB = 2;
  const double *__restrict__ u, *__restrict__ p;
  double* __restrict__ b;
  bool pressure;  // p given and crack pressure on
  __device__ __forceinline__ void load(int64_t n, double (&q)[NF]) const {
#pragma unroll
    for (int c = 0; c < 3; c++) q[c] = pressure ? u[3 * n + c] : 0.;
    q[3] = pressure ? p[n] : 0.;
  }
  __device__ __forceinline__ void put(int64_t n, const double (&y)[NV]) const { b[n] = y[0]; }
  __device__ __forceinline__ void cell(const ElemArgs& E, int ei, int ej, int ek, const double (&fld)[NF][8],
                                       double (&out)[8][NV]) const {
    const CellMat m = cell_mat(E, ei, ej, ek);
    const double vol = E.hx * E.hy * E.hz;
    const double coef = m.Gc / E.atcv / E.epsilon * (E.atnum == 1 ? .25 : .5);
#pragma unroll
    for (int a = 0; a < 8; a++) out[a][0] = coef * vol * 0.125;
    if (pressure) {
      double pm[8];
      modal_of(fld[3], pm);
      const double ih[3] = {1. / E.hx, 1. / E.hy, 1. / E.hz};
#pragma unroll
      for (int c = 0; c < 3; c++) {
        double um[8], F[2][2];
        modal_of(fld[c], um);
        product_face(pm, um, c, F);
        const double w = vol * ih[c];
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
          for (int j = 0; j < 2; j++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
              const int t = c == 0 ? i : (c == 1 ? j : k);
              const double m = F[c == 0 ? j : i][c == 2 ? j : k];
              out[i + 2 * j + 4 * k][0] = fma(t ? w : -w, m, out[i + 2 * j + 4 * k][0]);
            }
      }
    }
  }
};

// One pass of an element vector: a block owns 31 x 7 node columns and the 32 x 8 cell columns
// around them, and marches up a chunk of node planes.  Per element layer each thread evaluates
// its cell (C::cell); its corners' values are summed over x by a shuffle, over y through
// shared memory (two buffers, one barrier per layer) and over z in registers, so every node is
// written once, in one fixed order.  The cells on the seams of the blocks are computed
// twice.  8 launches of a parity colour each read and wrote the result 8 times, a cache line
// for every second node: at 129^3 U load 466 us, diagonal 234, V load 215; now 206, 118 and 125
// (a chain of loads, element and exchange per layer at 8 or 16 warps per SM; fetching a plane
// further ahead changed nothing); 65^3 74 -> 54, 47 -> 27, 50 -> 30; the diagonals of the coarse
// levels 47 -> 6 to 9.
constexpr int CG_NX = 31, CG_NY = 7;
template <class C>
__global__ void __launch_bounds__(256, C::MINB)
    cell_gather_kernel(const __grid_constant__ ElemArgs E, const C op, int gx, int zc) {
  constexpr int NF = C::NF, NV = C::NV;
  __shared__ double sh[2][2 * NV][256];
  const int l = threadIdx.x, w = threadIdx.y, t = w * 32 + l;
  const int nx = E.nx, ny = E.ny, nz = E.nz;
  const int bx = blockIdx.x % gx, by = blockIdx.x / gx;
  const int ex = bx * CG_NX - 1 + l, ey = by * CG_NY - 1 + w;
  const bool cell = ex >= 0 && ex < nx - 1 && ey >= 0 && ey < ny - 1;
  const bool node = l > 0 && w > 0 && ex < nx && ey < ny;  // owns node column (ex, ey)
  const int z0 = blockIdx.y * zc, z1 = min(z0 + zc, nz), k0 = max(z0 - 1, 0);
  const int64_t plane = (int64_t)nx * ny, base = cell ? (int64_t)ey * nx + ex : 0;
  double q[NF][8], carry[NV];
#pragma unroll
  for (int c = 0; c < NV; c++) carry[c] = 0.;
  auto load4 = [&](int k) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      double f[NF];
      op.load(cell ? base + k * plane + (j >> 1) * nx + (j & 1) : 0, f);
#pragma unroll
      for (int i = 0; i < NF; i++) q[i][4 + j] = f[i];
    }
  };
  load4(k0);
  for (int k = k0; k < z1; k++) {
    const int b = (k - k0) & 1;
    const bool layer = k < nz - 1;
    double xs[2][2][NV];  // [j][kk]: this cell's and its left neighbour's share of column ex
    if (layer) {
#pragma unroll
      for (int i = 0; i < NF; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) q[i][j] = q[i][4 + j];
      load4(k + 1);
      double out[8][NV];
      if (cell) {
        op.cell(E, ex, ey, k, q, out);
      } else {
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
          for (int c = 0; c < NV; c++) out[a][c] = 0.;
      }
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int kk = 0; kk < 2; kk++)
#pragma unroll
          for (int c = 0; c < NV; c++)
            xs[j][kk][c] = __shfl_up_sync(0xffffffffu, out[1 + 2 * j + 4 * kk][c], 1) + out[2 * j + 4 * kk][c];
#pragma unroll
      for (int kk = 0; kk < 2; kk++)
#pragma unroll
        for (int c = 0; c < NV; c++) sh[b][kk * NV + c][t] = xs[1][kk][c];
    }
    __syncthreads();
    if (!node) continue;
    double y[NV], up[NV];
#pragma unroll
    for (int c = 0; c < NV; c++) {
      y[c] = layer ? carry[c] + (sh[b][c][t - 32] + xs[0][0][c]) : carry[c];
      up[c] = layer ? sh[b][NV + c][t - 32] + xs[0][1][c] : 0.;
    }
    if (k >= z0) op.put((int64_t)k * plane + (int64_t)ey * nx + ex, y);
#pragma unroll
    for (int c = 0; c < NV; c++) carry[c] = up[c];
  }
}

// Node planes of a marching block's chunk: four waves of one block per SM on large grids
// (each chunk evaluates the layer below it again), at least `least` planes on small ones, at
// most 65535 chunks.
int march_planes(int64_t columns, int nz, int least) {
  const int zc = (int)std::max<int64_t>(least, (columns * nz + 591) / 592);
  return std::max(std::min(zc, nz), ceil_div(nz, 65535));
}

// Neumaier-compensated accumulation.
struct KSum {
  double s = 0., c = 0.;
  __device__ void add(double x) {
    const double t = s + x;
    c += fabs(s) >= fabs(x) ? (s - t) + x : (x - t) + s;
    s = t;
  }
  __device__ double value() const { return s + c; }
};

constexpr int EN_THREADS = 128, EN_BLOCKS = 888;  // 6 blocks per SM of 148

// Value and gradient of a modal form (modal_of) at the point t = (tx, ty, tz).
__device__ __forceinline__ double mval_t(const double (&m)[8], double tx, double ty, double tz) {
  return fma(fma(fma(m[7], tx, m[6]), ty, fma(m[5], tx, m[4])), tz,
             fma(fma(m[3], tx, m[2]), ty, fma(m[1], tx, m[0])));
}
__device__ __forceinline__ double mdx_t(const double (&m)[8], double ty, double tz, double ih) {
  return ih * fma(fma(m[7], tz, m[3]), ty, fma(m[5], tz, m[1]));
}
__device__ __forceinline__ double mdy_t(const double (&m)[8], double tx, double tz, double ih) {
  return ih * fma(fma(m[7], tz, m[3]), tx, fma(m[6], tz, m[2]));
}
__device__ __forceinline__ double mdz_t(const double (&m)[8], double tx, double ty, double ih) {
  return ih * fma(fma(m[7], ty, m[5]), tx, fma(m[6], ty, m[4]));
}

// NOCOMPRESSION: all four quantities point by point.
// One thread per element (grid-stride, fixed assignment), per-thread compensated
// sums, pairwise tree in shared memory, per-block partials: deterministic.  The fields
// at the 27 points come from their modal forms (the trilinear interpolants the
// reference's basis-function sums evaluate); the point loop is not unrolled, which
// keeps the thread at < 170 registers (3 blocks per SM).
__global__ void __launch_bounds__(EN_THREADS, 3) energy_kernel(
    const __grid_constant__ ElemArgs E, const double* __restrict__ u, const double* __restrict__ v,
    const double* __restrict__ theta, const double* __restrict__ thetaRef,
    const double* __restrict__ p, double* __restrict__ partial, double* __restrict__ cellcov) {
  __shared__ double red[4][EN_THREADS];
  const int64_t NCELL = (int64_t)(E.nx - 1) * (E.ny - 1) * (E.nz - 1);
  const double ihx = 1. / E.hx, ihy = 1. / E.hy, ihz = 1. / E.hz;
  const double vol = E.hx * E.hy * E.hz;
  KSum acc[4];
  for (int64_t cell = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; cell < NCELL;
       cell += (int64_t)gridDim.x * blockDim.x) {
    const int ei = (int)(cell % (E.nx - 1));
    const int ej = (int)((cell / (E.nx - 1)) % (E.ny - 1));
    const int ek = (int)(cell / ((int64_t)(E.nx - 1) * (E.ny - 1)));
    int64_t n[8];
    cell_nodes(E, ei, ej, ek, n);
    const CellMat m = cell_mat(E, ei, ej, ek);
    double mu3[3][8], mv[8], mp[8], mth[8];
    {
      double f[3][8], v8[8], th8[8], p8[8];
#pragma unroll
      for (int a = 0; a < 8; a++) {
#pragma unroll
        for (int c = 0; c < 3; c++) f[c][a] = u[3 * n[a] + c];
        v8[a] = v[n[a]];
        th8[a] = theta ? theta[n[a]] - (thetaRef ? thetaRef[n[a]] : 0.) : 0.;
        p8[a] = p ? p[n[a]] : 0.;
      }
#pragma unroll
      for (int c = 0; c < 3; c++) modal_of(f[c], mu3[c]);
      modal_of(v8, mv);
      modal_of(p8, mp);
      modal_of(th8, mth);
    }
    const double threekappa = 3. * m.lambda + 2. * m.mu, coefbeta = m.beta / threekappa;
    const double scoef = m.Gc / E.atcv * .25;
    double el = 0., pw = 0., se = 0., cv = 0., wsum = 0.;
#pragma unroll 1
    for (int g = 0; g < 27; g++) {
      const int gx = g % 3, gy = (g / 3) % 3, gz = g / 9;
      const double tx = gx == 1 ? 0. : (gx == 0 ? -VF_TAU : VF_TAU);
      const double ty = gy == 1 ? 0. : (gy == 0 ? -VF_TAU : VF_TAU);
      const double tz = gz == 1 ? 0. : (gz == 0 ? -VF_TAU : VF_TAU);
      const double w = vol * (w1(gx) * w1(gy) * w1(gz));
      double D11 = mdx_t(mu3[0], ty, tz, ihx), D22 = mdy_t(mu3[1], tx, tz, ihy);
      double D33 = mdz_t(mu3[2], tx, ty, ihz);
      const double D12 = (mdx_t(mu3[1], ty, tz, ihx) + mdy_t(mu3[0], tx, tz, ihy)) * .5;
      const double D23 = (mdy_t(mu3[2], tx, tz, ihy) + mdz_t(mu3[1], tx, ty, ihz)) * .5;
      const double D13 = (mdx_t(mu3[2], ty, tz, ihx) + mdz_t(mu3[0], tx, ty, ihz)) * .5;
      const double ve = mval_t(mv, tx, ty, tz), pe = mval_t(mp, tx, ty, tz);
      const double te = mval_t(mth, tx, ty, tz);
      const double gv0 = mdx_t(mv, ty, tz, ihx), gv1 = mdy_t(mv, tx, tz, ihy), gv2 = mdz_t(mv, tx, ty, ihz);
      // VF_ElasticEnergy3D_local (VFMech.c:725-809), quirk Q2: v^2 (1+eta) on the deviator
      const double tr = D11 + D22 + D33;
      D11 -= tr / 3.;
      D22 -= tr / 3.;
      D33 -= tr / 3.;
      el += (D11 * D11 + D22 * D22 + D33 * D33 + (D12 * D12 + D23 * D23 + D13 * D13) * 2.) * ve * ve *
            (1. + E.eta) * m.mu * w;
      // NOCOMPRESSION (VF_ElasticEnergyNoCompression3D_local, VFMech.c:819-908): the
      // spherical factor is 1 instead of v where tr < 0
      const double sph = tr < 0. ? 1. : ve;
      const double WD = (tr / 3. - m.alpha * te) * sph - coefbeta * pe;
      el += 3. * threekappa / 2. * WD * WD * w;
      el += threekappa / 6. * tr * tr * E.eta * w;
      const double udv = mval_t(mu3[0], tx, ty, tz) * gv0 + mval_t(mu3[1], tx, ty, tz) * gv1 +
                         mval_t(mu3[2], tx, ty, tz) * gv2;
      // VF_PressureWork3D_local (VFMech.c:920-974)
      if (E.hasCrackPressure) pw += w * pe * udv;
      // VF_AT1/AT2SurfaceEnergy3D_local (VFMech.c:2394-2465)
      const double g2 = gv0 * gv0 + gv1 * gv1 + gv2 * gv2;
      const double om = 1. - ve;
      se += w * ((E.atnum == 1 ? om : om * om) / E.epsilon + g2 * E.epsilon) * scoef;
      // VolumetricCrackOpening3D_local (VFPermfield.c:15-73)
      cv += udv * w;
      wsum += w;
    }
    if (cellcov) cellcov[cell] = cv / wsum;
    acc[0].add(el);
    acc[1].add(pw);
    acc[2].add(se);
    acc[3].add(cv);
  }
  for (int q = 0; q < 4; q++) red[q][threadIdx.x] = acc[q].value();
  __syncthreads();
  for (int st = EN_THREADS / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st)
      for (int q = 0; q < 4; q++) red[q][threadIdx.x] += red[q][threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x < 4) partial[blockIdx.x * 4 + threadIdx.x] = red[threadIdx.x][0];
}

// out[q] = compensated sum of partial[4 b + q] over the blocks: one warp per quantity, lane
// l takes blocks l, l + 32, ..., the lanes join in a fixed tree.  (One thread per quantity
// walking all 888 partials was a serial chain of 77 us.)
__global__ void __launch_bounds__(128) energy_final_kernel(const double* __restrict__ partial,
                                                           int nblocks, double* __restrict__ out) {
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  KSum s;
  for (int b = lane; b < nblocks; b += 32) s.add(partial[b * 4 + q]);
  double r = s.value();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
  if (lane == 0) out[q] = r;
}

// ---- energies by Gauss rows (the plain model).  Along a Gauss row (fixed gy, gz) every
// trilinear field is linear in t = tx, so each integrand is a polynomial of degree <= 4 in
// t and its 3-point sum follows from sum w = 1, sum w t^2 = 1/12, sum w t^4 = 1/80 (odd
// sums vanish): the same Gauss sum as point by point from 9 rows instead of 27 points.
// Where the 8 nodal v of the cell are equal and neither theta nor the Biot term enters,
// v leaves the sum and the elastic terms are squares of polynomials of degree <= 1 per
// axis, whose Gauss sums are closed (mean of t^2 = 1/12 per axis): no row is evaluated.
// WANT selects the quantities a caller asked for (kEnElastic ...), so that each entry
// point pays for its own.  A thread marches kEnLayers cells up a column and keeps the
// nodes shared with the cell below.
// The point-by-point kernel took 1.05 ms at 129^3 for every entry point (FP64 issue: 3500
// operations per cell; 77 us more in a serial final sum); the three entry points one after
// the other, each with its host read, measured 3.42 ms with it and 0.327 ms with these.
constexpr int kEnLayers = 4;

// Squared norm over the cell of a polynomial with coefficients c[m] of the monomials
// m = px + 2 py + 4 pz of degree <= 1 per axis: weights 1, 1/12, 1/144 (no xyz term).
__device__ __forceinline__ double en_sq(const double (&c)[7]) {
  return fma(c[0], c[0],
             fma(fma(c[1], c[1], fma(c[2], c[2], c[4] * c[4])), 1.0 / 12.0,
                 fma(c[3], c[3], fma(c[5], c[5], c[6] * c[6])) * (1.0 / 144.0)));
}

template <int WANT>
__global__ void __launch_bounds__(EN_THREADS, (WANT & kEnElastic) ? 3 : 4) energy_rows_kernel(
    const __grid_constant__ ElemArgs E, const double* __restrict__ u, const double* __restrict__ v,
    const double* __restrict__ theta, const double* __restrict__ thetaRef,
    const double* __restrict__ p, double* __restrict__ partial, double* __restrict__ cellcov) {
  constexpr bool EL = (WANT & kEnElastic) != 0, PW = EL, SU = (WANT & kEnSurface) != 0,
                 CV = (WANT & kEnOpening) != 0, U = EL || CV;
  __shared__ double red[4][EN_THREADS];
  const int nex = E.nx - 1, ney = E.ny - 1, nez = E.nz - 1;
  const int64_t ncol = (int64_t)nex * ney, nitem = ncol * ((nez + kEnLayers - 1) / kEnLayers);
  const int64_t plane = (int64_t)E.nx * E.ny;
  const double ih[3] = {1. / E.hx, 1. / E.hy, 1. / E.hz};
  const double vol = E.hx * E.hy * E.hz;
  KSum acc[4];
  for (int64_t it = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; it < nitem;
       it += (int64_t)gridDim.x * blockDim.x) {
    const int64_t col = it % ncol;
    const int ei = (int)(col % nex), ej = (int)(col / nex);
    const int k0 = (int)(it / ncol) * kEnLayers, k1 = min(k0 + kEnLayers, nez);
    double f[3][8], v8[8], th8[8], p8[8];  // [4 + j]: the upper nodes
    auto load4 = [&](int k) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int64_t n = k * plane + (int64_t)(ej + (j >> 1)) * E.nx + ei + (j & 1);
        if constexpr (U) {
#pragma unroll
          for (int c = 0; c < 3; c++) f[c][4 + j] = u[3 * n + c];
        }
        v8[4 + j] = v[n];
        if constexpr (EL) {
          th8[4 + j] = theta ? theta[n] - (thetaRef ? thetaRef[n] : 0.) : 0.;
          p8[4 + j] = p ? p[n] : 0.;
        }
      }
    };
    load4(k0);
#pragma unroll 1
    for (int ek = k0; ek < k1; ek++) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if constexpr (U) {
#pragma unroll
          for (int c = 0; c < 3; c++) f[c][j] = f[c][4 + j];
        }
        v8[j] = v8[4 + j];
        if constexpr (EL) {
          th8[j] = th8[4 + j];
          p8[j] = p8[4 + j];
        }
      }
      load4(ek + 1);
      const CellMat mat = cell_mat(E, ei, ej, ek);
      bool cst = true;
#pragma unroll
      for (int a = 1; a < 8; a++) cst = cst && v8[a] == v8[0];
      double mv[8];
      modal_of(v8, mv);
      if constexpr (SU) {  // VF_AT1/AT2SurfaceEnergy3D_local (VFMech.c:2394-2465)
        const double om = 1. - mv[0];
        double lin = om;
        if (E.atnum != 1)
          lin = fma(om, om, (mv[1] * mv[1] + mv[2] * mv[2] + mv[4] * mv[4]) * (1. / 12.) +
                                (mv[3] * mv[3] + mv[5] * mv[5] + mv[6] * mv[6]) * (1. / 144.) +
                                mv[7] * mv[7] * (1. / 1728.));
        auto g2 = [&](int a, int b, int c, double i) {
          return i * i * (mv[a] * mv[a] + (mv[b] * mv[b] + mv[c] * mv[c]) * (1. / 12.) +
                          mv[7] * mv[7] * (1. / 144.));
        };
        const double gr = (g2(1, 3, 5, ih[0]) + g2(2, 3, 6, ih[1])) + g2(4, 5, 6, ih[2]);
        acc[2].add(vol * (lin / E.epsilon + gr * E.epsilon) * (mat.Gc / E.atcv * .25));
      }
      if constexpr (U) {
        double m[3][8];
#pragma unroll
        for (int c = 0; c < 3; c++) modal_of(f[c], m[c]);
        const double threekappa = 3. * mat.lambda + 2. * mat.mu;
        const double cb = EL ? mat.beta / threekappa : 0.;
        bool closed = cst;
        if constexpr (EL) {
          closed = closed && cb == 0.;
#pragma unroll
          for (int a = 0; a < 8; a++) closed = closed && th8[a] == 0.;
        }
        double el = 0., pw = 0., cv = 0.;
        if (closed) {
          if constexpr (EL) {
            // gradient coefficients: d/dx of component c has the monomials 1, y, z, yz
            // (modes 1, 3, 5, 7), d/dy 1, x, z, xz (2, 3, 6, 7), d/dz 1, x, y, xy (4, 5, 6, 7)
            const double x1 = m[0][1] * ih[0], xy = m[0][3] * ih[0], xz = m[0][5] * ih[0], xyz = m[0][7] * ih[0];
            const double y1 = m[1][2] * ih[1], yx = m[1][3] * ih[1], yz = m[1][6] * ih[1], yxz = m[1][7] * ih[1];
            const double z1 = m[2][4] * ih[2], zx = m[2][5] * ih[2], zy = m[2][6] * ih[2], zxy = m[2][7] * ih[2];
            const double tr[7] = {(x1 + y1) + z1, yx + zx, xy + zy, zxy, xz + yz, yxz, xyz};
            double d0[7], d1[7], d2[7];
            const double e0[7] = {x1, 0., xy, 0., xz, 0., xyz}, e1[7] = {y1, yx, 0., 0., yz, yxz, 0.};
            const double e2[7] = {z1, zx, zy, zxy, 0., 0., 0.};
#pragma unroll
            for (int q = 0; q < 7; q++) {
              d0[q] = fma(tr[q], -1. / 3., e0[q]);
              d1[q] = fma(tr[q], -1. / 3., e1[q]);
              d2[q] = fma(tr[q], -1. / 3., e2[q]);
            }
            // twice the shear strains: 12 = d/dx u_y + d/dy u_x, ...
            const double s0[7] = {fma(m[1][1], ih[0], m[0][2] * ih[1]), m[0][3] * ih[1], m[1][3] * ih[0], 0.,
                                  fma(m[1][5], ih[0], m[0][6] * ih[1]), m[0][7] * ih[1], m[1][7] * ih[0]};
            const double s1[7] = {fma(m[2][2], ih[1], m[1][4] * ih[2]), fma(m[2][3], ih[1], m[1][5] * ih[2]),
                                  m[1][6] * ih[2], m[1][7] * ih[2], m[2][6] * ih[1], m[2][7] * ih[1], 0.};
            const double s2[7] = {fma(m[2][1], ih[0], m[0][4] * ih[2]), m[0][5] * ih[2],
                                  fma(m[2][3], ih[0], m[0][6] * ih[2]), m[0][7] * ih[2], m[2][5] * ih[0], 0.,
                                  m[2][7] * ih[0]};
            const double dev = (en_sq(d0) + en_sq(d1)) + en_sq(d2) + .5 * ((en_sq(s0) + en_sq(s1)) + en_sq(s2));
            const double tt = en_sq(tr), vv = v8[0] * v8[0];
            el = vol * (dev * vv * (1. + E.eta) * mat.mu + threekappa / 6. * tt * (vv + E.eta));
            // p only multiplies grad v = 0 here; a value that is not finite still shows
#pragma unroll
            for (int a = 0; a < 8; a++) pw += p8[a];
            pw = 0. * pw;
            el += pw;
          }
          if constexpr (CV) {  // u . grad v = 0; a displacement that is not finite still shows
            double t = 0.;
#pragma unroll
            for (int c = 0; c < 3; c++) t += m[c][0];
            cv = 0. * t;
          }
        } else {
          double mp[8], mth[8];
          if constexpr (EL) {
            modal_of(p8, mp);
            modal_of(th8, mth);
          }
#pragma unroll 1
          for (int gz = 0; gz < 3; gz++) {
            const double tz = gz == 1 ? 0. : (gz == 0 ? -VF_TAU : VF_TAU);
#pragma unroll 1
            for (int gy = 0; gy < 3; gy++) {
              const double ty = gy == 1 ? 0. : (gy == 0 ? -VF_TAU : VF_TAU);
              const double wr = vol * (w1(gy) * w1(gz));
              // value and slope of a trilinear field along the row
              auto row = [&](const double (&q)[8], double& r0, double& r1) {
                r0 = fma(fma(q[6], tz, q[2]), ty, fma(q[4], tz, q[0]));
                r1 = fma(fma(q[7], tz, q[3]), ty, fma(q[5], tz, q[1]));
              };
              // y and z derivatives along the row (value, slope)
              auto dy = [&](const double (&q)[8], double& r0, double& r1) {
                r0 = ih[1] * fma(q[6], tz, q[2]);
                r1 = ih[1] * fma(q[7], tz, q[3]);
              };
              auto dz = [&](const double (&q)[8], double& r0, double& r1) {
                r0 = ih[2] * fma(q[6], ty, q[4]);
                r1 = ih[2] * fma(q[7], ty, q[5]);
              };
              double v0, v1;
              row(mv, v0, v1);
              double gy0, gy1, gz0, gz1;
              dy(mv, gy0, gy1);
              dz(mv, gz0, gz1);
              const double gx0 = ih[0] * v1;
              double ux0, ux1, uy0, uy1, uz0, uz1;
              row(m[0], ux0, ux1);
              row(m[1], uy0, uy1);
              row(m[2], uz0, uz1);
              // u . grad v = c0 + c1 t + c2 t^2
              const double c0 = fma(ux0, gx0, fma(uy0, gy0, uz0 * gz0));
              const double c2 = fma(uy1, gy1, uz1 * gz1);
              if constexpr (CV) cv = fma(wr, fma(c2, 1. / 12., c0), cv);  // VolumetricCrackOpening3D_local
              if constexpr (EL) {
                double p0, p1, th0, th1;
                row(mp, p0, p1);
                row(mth, th0, th1);
                if (E.hasCrackPressure) {  // VF_PressureWork3D_local (VFMech.c:920-974)
                  const double c1 = fma(ux1, gx0, (uy0 * gy1 + uy1 * gy0) + (uz0 * gz1 + uz1 * gz0));
                  pw = fma(wr, fma(c0, p0, fma(c1, p1, c2 * p0) * (1. / 12.)), pw);
                }
                // VF_ElasticEnergy3D_local (VFMech.c:725-809): v^2 (1 + eta) on the deviator
                double ay[3], by[3], az[3], bz[3];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                  dy(m[c], ay[c], by[c]);
                  dz(m[c], az[c], bz[c]);
                }
                const double X0 = ih[0] * ux1, X1 = ih[0] * uy1, X2 = ih[0] * uz1;
                const double T0 = (X0 + ay[1]) + az[2], T1 = by[1] + bz[2];
                const double t0 = T0 * (1. / 3.), t1 = T1 * (1. / 3.);
                const double d00 = X0 - t0, d11 = ay[1] - t0, d22 = az[2] - t0;
                const double f11 = by[1] - t1, f22 = bz[2] - t1;
                const double s01 = X1 + ay[0], s02 = X2 + az[0], s12 = ay[2] + az[1];
                const double r12 = by[2] + bz[1];
                const double q0 = fma(d00, d00, fma(d11, d11, d22 * d22)) +
                                  .5 * fma(s01, s01, fma(s02, s02, s12 * s12));
                const double q1 = 2. * (fma(d11, f11, d22 * f22) - d00 * t1) +
                                  fma(s01, by[0], fma(s02, bz[0], s12 * r12));
                const double q2 = fma(t1, t1, fma(f11, f11, f22 * f22)) +
                                  .5 * fma(by[0], by[0], fma(bz[0], bz[0], r12 * r12));
                const double a0 = v0 * v0, a1 = 2. * v0 * v1, a2 = v1 * v1;
                const double dv = fma(a0, q0, fma(fma(a0, q2, fma(a1, q1, a2 * q0)), 1. / 12., a2 * q2 * (1. / 80.)));
                // WD = (tr / 3 - alpha theta) v - cb p along the row
                const double f0 = fma(-mat.alpha, th0, t0), f1 = fma(-mat.alpha, th1, t1);
                const double b0 = fma(f0, v0, -(cb * p0)), b1 = fma(f0, v1, fma(f1, v0, -(cb * p1))), b2 = f1 * v1;
                const double wd = fma(b0, b0, fma(fma(b1, b1, 2. * b0 * b2), 1. / 12., b2 * b2 * (1. / 80.)));
                const double t2 = fma(T0, T0, T1 * T1 * (1. / 12.));
                el = fma(wr, (dv * (1. + E.eta)) * mat.mu + fma(1.5 * threekappa, wd, threekappa / 6. * t2 * E.eta), el);
              }
            }
          }
        }
        if constexpr (EL) acc[0].add(el);
        if constexpr (PW) acc[1].add(E.hasCrackPressure ? pw : 0.);
        if constexpr (CV) {
          if (cellcov) cellcov[((int64_t)ek * ney + ej) * nex + ei] = cv / vol;
          acc[3].add(cv);
        }
      }
    }
  }
  for (int q = 0; q < 4; q++) red[q][threadIdx.x] = acc[q].value();
  __syncthreads();
  for (int st = EN_THREADS / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st)
      for (int q = 0; q < 4; q++) red[q][threadIdx.x] += red[q][threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x < 4) partial[blockIdx.x * 4 + threadIdx.x] = red[threadIdx.x][0];
}

template <class C> cudaError_t cell_gather(const ElemArgs& E, const C& op, cudaStream_t s) {
  const int gx = ceil_div(E.nx, CG_NX), gy = ceil_div(E.ny, CG_NY);
  const int zc = march_planes((int64_t)gx * gy, E.nz, 2);
  cell_gather_kernel<C><<<dim3(gx * gy, ceil_div(E.nz, zc)), dim3(32, 8), 0, s>>>(E, op, gx, zc);
  return cudaGetLastError();
}

template <typename K, typename... Args>
cudaError_t colours(const ElemArgs& E, K kernel, cudaStream_t s, Args... args) {
  for (int color = 0; color < 8; color++) {
    const int cx = color & 1, cy = (color >> 1) & 1, cz = color >> 2;
    const int64_t cnt = (int64_t)((E.nx - 1 - cx + 1) / 2) * ((E.ny - 1 - cy + 1) / 2) *
                        ((E.nz - 1 - cz + 1) / 2);
    if (cnt == 0) continue;
    kernel<<<(int)((cnt + 127) / 128), 128, 0, s>>>(E, color, args...);
  }
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_u_rhs(const ElemArgs& E, const double* v, const double* theta,
                         const double* thetaRef, const double* p, double* f, cudaStream_t s,
                         const double* u0) {
  if (!E.unilateral) return cell_gather(E, URhsCell{v, theta, thetaRef, p, f}, s);
  const int64_t N = (int64_t)E.nx * E.ny * E.nz;
  cudaError_t e = cudaMemsetAsync(f, 0, 3 * N * sizeof(double), s);
  if (e != cudaSuccess) return e;
  return colours(E, u_rhs_kernel, s, v, theta, thetaRef, p, f, u0);
}

cudaError_t launch_nc_flags(const ElemArgs& E, const double* u, uint32_t* flags, cudaStream_t s) {
  const int64_t NCELL = (int64_t)(E.nx - 1) * (E.ny - 1) * (E.nz - 1);
  nc_flags_kernel<<<(int)((NCELL + 127) / 128), 128, 0, s>>>(E, u, flags);
  return cudaGetLastError();
}

cudaError_t launch_u_diag(const ElemArgs& E, const double* v, const uint8_t* bcbits, double* d,
                          cudaStream_t s, const double* u0) {
  if (!E.unilateral) return cell_gather(E, UDiagCell{v, bcbits, d}, s);
  const int64_t N = (int64_t)E.nx * E.ny * E.nz;
  cudaError_t e = cudaMemsetAsync(d, 0, 3 * N * sizeof(double), s);
  if (e == cudaSuccess) e = colours(E, u_diag_kernel, s, v, d, u0);
  if (e == cudaSuccess && bcbits) {
    bc_diag_kernel<<<(int)std::min<int64_t>((N + 255) / 256, 2368), 256, 0, s>>>(bcbits, d, N);
    e = cudaGetLastError();
  }
  return e;
}

cudaError_t launch_v_assemble(const ElemArgs& E, const double* u, const double* theta,
                              const double* thetaRef, double* a64, float* a32, cudaStream_t s) {
  constexpr size_t smem = (27 + 8) * 256 * sizeof(double);
  cudaError_t e = cudaFuncSetAttribute(v_assemble_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int gx = ceil_div(E.nx, VM_NX), gy = ceil_div(E.ny, VM_NY);
  const int zc = march_planes((int64_t)gx * gy, E.nz, 4);
  v_assemble_kernel<<<dim3(gx * gy, ceil_div(E.nz, zc)), dim3(32, 8), smem, s>>>(
      E, u, theta, thetaRef, a64, a32, vmat_stride((int64_t)E.nx * E.ny * E.nz), gx, zc);
  return cudaGetLastError();
}

cudaError_t launch_v_rhs(const ElemArgs& E, const double* u, const double* p, double* b,
                         cudaStream_t s) {
  return cell_gather(E, VRhsCell{u, p, b, E.hasCrackPressure && p}, s);
}

int energy_blocks() { return EN_BLOCKS; }

cudaError_t launch_energies(const ElemArgs& E, int want, const double* u, const double* v,
                            const double* theta, const double* thetaRef, const double* p,
                            double* partial, double* out, double* cellcov, cudaStream_t s) {
  int blocks = EN_BLOCKS;
  if (E.unilateral) {  // the spherical factor switches per point: point by point
    energy_kernel<<<EN_BLOCKS, EN_THREADS, 0, s>>>(E, u, v, theta, thetaRef, p, partial, cellcov);
  } else {
    const int64_t items = (int64_t)(E.nx - 1) * (E.ny - 1) * ((E.nz - 1 + kEnLayers - 1) / kEnLayers);
    blocks = (int)std::min<int64_t>(EN_BLOCKS, (items + EN_THREADS - 1) / EN_THREADS);
    switch (want) {
      case kEnElastic:
        energy_rows_kernel<kEnElastic><<<blocks, EN_THREADS, 0, s>>>(E, u, v, theta, thetaRef, p, partial, cellcov);
        break;
      case kEnSurface:
        energy_rows_kernel<kEnSurface><<<blocks, EN_THREADS, 0, s>>>(E, u, v, theta, thetaRef, p, partial, cellcov);
        break;
      case kEnOpening:
        energy_rows_kernel<kEnOpening><<<blocks, EN_THREADS, 0, s>>>(E, u, v, theta, thetaRef, p, partial, cellcov);
        break;
      default: return cudaErrorInvalidValue;
    }
  }
  energy_final_kernel<<<1, 128, 0, s>>>(partial, blocks, out);
  return cudaGetLastError();
}

}  // namespace vfgpu
