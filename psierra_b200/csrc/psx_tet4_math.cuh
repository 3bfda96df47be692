// Tet4 geometry and kinematics shared by the Tet4 kernels (assembly, K.v, adjoint,
// hyper-reduced evaluation).  element/tet4_base.py:34-67 and
// element/tet4_total_lagrangian.py:44-46 restated.
#pragma once

#include "psx_common.cuh"

namespace psx {

struct Tet4Geom {
  double g[4][3];  // shape-function gradients
  double V;        // reference volume
  double detD;     // det of [X1-X0 X2-X0 X3-X0] = det [1 X] of the reference
};

__device__ __forceinline__ void load_nodes(const double* __restrict__ A, int4 c, double out[4][3]) {
  const int ids[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const double* p = A + 3 * (int64_t)ids[b];
    out[b][0] = __ldg(p);
    out[b][1] = __ldg(p + 1);
    out[b][2] = __ldg(p + 2);
  }
}

// tet4_base.py:34-67 (A = [1 X], V = det A / 6, H = rows of A^-1) in the form
// D = [X1-X0 X2-X0 X3-X0], g_b = row b-1 of D^-1 (b >= 1), g_0 = -(g_1+g_2+g_3).
__device__ __forceinline__ void tet4_geometry(const double Xn[4][3], Tet4Geom& G) {
  double D[3][3], Di[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) D[i][j] = dsub(Xn[j + 1][i], Xn[0][i]);
  G.detD = inv3(D, Di);
  G.V = dmul(G.detD, kSixth);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    G.g[1][j] = Di[0][j];
    G.g[2][j] = Di[1][j];
    G.g[3][j] = Di[2][j];
    G.g[0][j] = -dadd(dadd(Di[0][j], Di[1][j]), Di[2][j]);
  }
}

// Displacement gradient l = sum_b (u_b - u_0) g_b^T (exactly zero for a rigid translation).
__device__ __forceinline__ void tet4_grad(const double Un[4][3], const Tet4Geom& G, double l[3][3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      l[i][j] = ddot3(dsub(Un[1][i], Un[0][i]), G.g[1][j], dsub(Un[2][i], Un[0][i]), G.g[2][j],
                      dsub(Un[3][i], Un[0][i]), G.g[3][j]);
    }
}

// Explicitly rounded operations in the tangent's type (dmul / fmul etc. of psx_common.cuh).
__device__ __forceinline__ double xmul(double a, double b) { return dmul(a, b); }
__device__ __forceinline__ float xmul(float a, float b) { return fmul(a, b); }
__device__ __forceinline__ double xadd(double a, double b) { return dadd(a, b); }
__device__ __forceinline__ float xadd(float a, float b) { return fadd(a, b); }
__device__ __forceinline__ double xfma(double a, double b, double c) { return dfma(a, b, c); }
__device__ __forceinline__ float xfma(float a, float b, float c) { return ffma(a, b, c); }
template <typename T>
__device__ __forceinline__ T xdot3(T a0, T b0, T a1, T b1, T a2, T b2) {
  return xfma(a0, b0, xfma(a1, b1, xmul(a2, b2)));
}

// Arguments of the Tet4 sweeps (psx_tet4_assemble and its relatives).
struct Tet4Args {
  const int32_t* conn;
  const double* X;
  const double* U;
  const double* Vv;  // vector of the matrix-free product (PSX_KV) / cotangent (adjoint)
  double* dmu;       // adjoint: d(w.f)/d mu_e (E), or null
  double* dkappa;    // adjoint: d(w.f)/d kappa_e (E), or null
  const double* mu_e;
  const double* kappa_e;
  double mu0, kappa0, lam0;
  Status* st;
  // effective tangent (kModeEff): K_eff = c_t K_T + c_m M + c_0 K_0, M the consistent mass
  // of density rho, K_0 the small-strain stiffness (lam0, mu0, or per element
  // lambda = kappa_e - 2/3 mu_e, mu_e)
  double c_t, c_m, c_0, rho;
  // element records in the global ring (store_planes): the ring length (set by run_tet4)
  int64_t plane = 0;
};

constexpr int kModeDR = 16;       // internal: PSX_KV with the fused dynamic-relaxation epilogue
constexpr int kModeAdjoint = 64;  // internal: vector-Jacobian product of f_int
constexpr int kModeEff = 128;     // internal: c_t K_T + c_m M + c_0 K_0 (dynamic effective tangent)

// f_a = V P g_a of the element's four nodes.
__device__ __forceinline__ void tet4_force(const PointState& ps, const Tet4Geom& G, double fr[12]) {
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int i = 0; i < 3; ++i)
      fr[3 * a + i] = dmul(G.V, ddot3(ps.P[i][0], G.g[a][0], ps.P[i][1], G.g[a][1], ps.P[i][2], G.g[a][2]));
}

// p_a = F^-T g_a and q_a = F g_a of the element's four nodes, in the tangent's type.
template <typename KT>
__device__ __forceinline__ void tet4_pq(const PointState& ps, const KT gk[4][3], KT p[4][3], KT q[4][3]) {
  KT Fi[3][3], Fm[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      Fi[i][j] = (KT)ps.Finv[i][j];
      Fm[i][j] = (KT)ps.F[i][j];
    }
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      p[b][k] = xdot3(Fi[0][k], gk[b][0], Fi[1][k], gk[b][1], Fi[2][k], gk[b][2]);
      q[b][k] = xdot3(Fm[k][0], gk[b][0], Fm[k][1], gk[b][1], Fm[k][2], gk[b][2]);
    }
}

// Block K_ab = A p_a p_b^T + hb p_b p_a^T + p_a y_b^T + y_a p_b^T + phi (g_a.g_b) I of an element
// (y = c q; phi g_a.g_b = -3/2 p_a.y_b), in the association of tet4_element.
template <typename KT>
__device__ __forceinline__ void point_block(const KT pa[3], const KT ya[3], const KT pb[3], const KT yb[3], KT A, KT hb,
                                            KT v[9]) {
  const KT s = xmul((KT)-1.5, xdot3(pa[0], yb[0], pa[1], yb[1], pa[2], yb[2]));
  KT w[3], h[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    w[k] = xfma(A, pb[k], yb[k]);
    h[k] = xmul(hb, pa[k]);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const KT last = k == m ? xfma(ya[k], pb[m], s) : xmul(ya[k], pb[m]);
      v[3 * k + m] = xfma(pa[k], w[m], xfma(pb[k], h[m], last));
    }
}

// Sums over the element's nodes of a vector v that the product K_e v and the adjoint use:
// alpha = sum_b w_b.v_b (w = A p + c q), beta = sum_b p_b.v_b, Pv = sum_b p_b v_b^T,
// Gv = sum_b g_b v_b^T.
template <typename KT>
struct Tet4Sums {
  KT alpha, beta, Pv[3][3], Gv[3][3];
};
template <typename KT>
__device__ __forceinline__ void tet4_sums(const TangentCoef<KT>& tc, const KT p[4][3], const KT q[4][3],
                                          const KT gk[4][3], const double Vn[4][3], Tet4Sums<KT>& S) {
  KT vk[4][3];
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int k = 0; k < 3; ++k) vk[b][k] = (KT)Vn[b][k];
  KT alpha = 0, beta = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int m = 0; m < 3; ++m) S.Pv[k][m] = S.Gv[k][m] = (KT)0;
#pragma unroll
  for (int b = 0; b < 4; ++b) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      alpha = xfma(xfma(tc.A, p[b][k], xmul(tc.c, q[b][k])), vk[b][k], alpha);
      beta = xfma(p[b][k], vk[b][k], beta);
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        S.Pv[k][m] = xfma(p[b][k], vk[b][m], S.Pv[k][m]);
        S.Gv[k][m] = xfma(gk[b][k], vk[b][m], S.Gv[k][m]);
      }
    }
  }
  S.alpha = alpha;
  S.beta = beta;
}

// y_a = sum_b K_ab v_b = alpha p_a + Pv h_a + beta (c q_a) + phi (sum_b (g_a.g_b) v_b)
template <typename KT>
__device__ __forceinline__ void tet4_product(const TangentCoef<KT>& tc, const KT p[4][3], const KT q[4][3],
                                             const KT gk[4][3], const Tet4Sums<KT>& S, double yr[12]) {
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      KT t = xfma(S.alpha, p[a][k], xmul(xmul(S.beta, tc.c), q[a][k]));
#pragma unroll
      for (int m = 0; m < 3; ++m)
        t = xadd(t, xfma(S.Pv[k][m], xmul(tc.hb, p[a][m]), xmul(xmul(tc.phi, gk[a][m]), S.Gv[m][k])));
      yr[3 * a + k] = (double)t;
    }
}

// Vector-Jacobian product of w.f_e with f_e,a = V P g_a (the adjoint of
// tet4_total_lagrangian.py:136-137 w.r.t. X, mu, kappa): the coordinates' part into yr, the
// moduli's into A.dmu[e], A.dkappa[e].  L_w = sum_b w_b g_b^T,
// VM = V dP/dF[L_w] = alpha F^-T + hb Pv F^-T + beta c F + phi Gv^T.
__device__ __forceinline__ void tet4_vjp(const Tet4Args& A, int64_t e, const PointState& ps,
                                         const double l[3][3], const Tet4Geom& G, const double Un[4][3],
                                         const double Vn[4][3], const TangentCoef<double>& tc,
                                         const Tet4Sums<double>& S, double yr[12]) {
  double VM[3][3], Lw[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Lw[i][j] = 0.0;
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Lw[i][j] += Vn[b][i] * G.g[b][j];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      // (F^-T)[k][m] = Finv[m][k]
      double t = S.alpha * ps.Finv[m][k] + S.beta * tc.c * ps.F[k][m] + tc.phi * S.Gv[m][k];
#pragma unroll
      for (int j = 0; j < 3; ++j) t += S.Pv[k][j] * tc.hb * ps.Finv[m][j];
      VM[k][m] = t;
    }
  // h_b = VM^T u_b + V P^T w_b  (vectors conjugate to dg_b)
  double h[4][3];
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double t = 0.0;
#pragma unroll
      for (int i = 0; i < 3; ++i) t += VM[i][j] * Un[b][i] + G.V * ps.P[i][j] * Vn[b][i];
      h[b][j] = t;
    }
  double PL = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) PL += ps.P[i][j] * Lw[i][j];
  // dL/dD = PL V G^T - G^T Hm G^T with G = D^-1 (rows g_1..g_3), Hm rows h_b - h_0
  double Gm[3][3], Hm[3][3], T1[3][3], Z[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      Gm[r][j] = G.g[r + 1][j];
      Hm[r][j] = h[r + 1][j] - h[0][j];
    }
#pragma unroll
  for (int i = 0; i < 3; ++i)  // T1 = G^T Hm
#pragma unroll
    for (int j = 0; j < 3; ++j) T1[i][j] = Gm[0][i] * Hm[0][j] + Gm[1][i] * Hm[1][j] + Gm[2][i] * Hm[2][j];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      Z[i][j] = PL * G.V * Gm[j][i] - (T1[i][0] * Gm[j][0] + T1[i][1] * Gm[j][1] + T1[i][2] * Gm[j][2]);
  // D[i][j] = X_{j+1}[i] - X_0[i]
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    yr[i] = -(Z[i][0] + Z[i][1] + Z[i][2]);
#pragma unroll
    for (int j = 0; j < 3; ++j) yr[3 * (j + 1) + i] = Z[i][j];
  }
  // parameter gradients: dP/dmu = 2 J^-2/3 F^-T dev E, dP/dkappa = ln J F^-T
  if (A.dmu || A.dkappa) {
    double E[3][3], trE = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double ltl = l[0][i] * l[0][j] + l[1][i] * l[1][j] + l[2][i] * l[2][j];
        E[i][j] = 0.5 * (l[i][j] + l[j][i] + ltl);
      }
    trE = E[0][0] + E[1][1] + E[2][2];
    const double jm23 = exp((-2.0 / 3.0) * ps.lnJ);
    double FTL = 0.0, FDL = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        FTL += ps.Finv[j][i] * Lw[i][j];
        double fd = 0.0;  // (F^-T dev E)[i][j]
#pragma unroll
        for (int k = 0; k < 3; ++k) fd += ps.Finv[k][i] * (E[k][j] - (k == j ? trE * kThird : 0.0));
        FDL += fd * Lw[i][j];
      }
    if (A.dmu) A.dmu[e] = G.V * 2.0 * jm23 * FDL;
    if (A.dkappa) A.dkappa[e] = G.V * ps.lnJ * FTL;
  }
}

}  // namespace psx
