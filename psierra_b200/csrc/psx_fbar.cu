// Tet4 F-bar (nodal volume averaging) element and assembly for sm_100a.
//
// Restates psierra element/tet4_fbar.py: the nodal averages (:213-243)
//   v0_a = sum_{e in E_a} V_e / 4,   J_node_a = (sum_{e in E_a} V_e J_e / 4) / v0_a,
//   J_bar_e = mean of J_node over the element's nodes,
// the element force and deviatoric tangent at F_bar = (J_bar / J)^(1/3) F (:147-211,
// :375-410) and the nodal volumetric blocks kappa v0_a g_a g_a^T (:420-459).
//
// Closed forms (r = (J_bar/J)^(1/3); F, p_b = F^-T g_b, q_b = F g_b of the element's own
// deformation; S_bar, phi_bar = mu J_bar^(-2/3), I1_bar = tr(F_bar^T F_bar) at F_bar):
//   f_b = V F [r^2 S_bar + (1 - r^2) tr(S_bar)/3 I] g_b          (B_bar^T S_bar_voigt V)
//   K_bc = V [A' s_b s_c^T + B' (1/2 (p_b.p_c) I + 1/2 p_c p_b^T - 1/3 (t_b q_c^T + q_b t_c^T)
//             + 1/9 tr(C^-2) q_b q_c^T) + (g_b^T S_bar g_c) I]
// with s_b = p_b - tr(C^-1)/3 q_b, t_b = (F F^T)^-1 p_b, A' = kappa + 2/9 phi_bar I1_bar,
// B' = 2/3 phi_bar I1_bar - 2 kappa ln J_bar.  The reference's ratio^4 B_dev^T (C - kappa
// m m^T) B_dev contracts to this: B_dev maps to traceless strains, so kappa m m^T and the
// C^-1 (x) I terms of the NeoHookean tangent drop out, and the C^-1 scalings of C_bar
// cancel r^4.  The volumetric "div_e" rows (B_0 + B_1 + B_2) are q_b.
//
// Kernels (one thread per element, node, one-ring entry or two-ring block; every sum in a
// fixed order, the reference's ascending element / patch node but for the longest lists,
// which a warp adds as a tree).  Measured on 162,000 elements, us, in the order below: 11,
// 9, 30, 54, 111, 59.  What bounds them: the volumetric pass its
// instructions and gathered loads, the element pass 12 warps per SM and its 134 MB of records,
// the gather the latency of their loads.
//   fbar_pre     V_e, J_e, q_e (and the inversion status)
//   fbar_nodes   v0_a, J_node_a
//   fbar_patch   g_a[b] = sum_{e in E_a, b in e} (V_e J_e / (4 v0_a)) q_e,b
//   fbar_element element record: 6 pair blocks, 4 diagonal blocks, 12 forces
//   fbar_vol     two-ring blocks = sum_a kappa v0_a g_a[b] g_a[c]^T
//   fbar_gather  one-ring blocks += and f = fixed-order sums of the records
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "psx_common.cuh"

namespace psx {
namespace {

constexpr int kFbThreads = 128;
// Element record, in planes over the elements: per pair block two quads and its ninth value,
// per node f (a quad), the diagonal block's xx xy xz yy (a quad) and yz zz (a pair).  Whole
// sectors for the stores of a warp, three loads per item; one 800-byte record per element,
// staged through shared memory, took five (element pass 75 us, gather 76; now 54 and 59).
constexpr int kFbRec = 96;  // doubles per element: 94 in whole 32-byte sectors
__device__ __forceinline__ int64_t fb_quad(int64_t E, int i, int64_t e) { return (i * E + e) * 4; }
__device__ __forceinline__ int64_t fb_ninth(int64_t E, int slot, int64_t e) { return (80 + slot) * E + e; }
__device__ __forceinline__ int64_t fb_pair(int64_t E, int a, int64_t e) { return 86 * E + (a * E + e) * 2; }

struct FbarArgs {
  const int32_t* conn;      // E x 4
  const double* X;
  const double* U;
  double mu, kappa;
  const int32_t* inc_ptr;   // N + 1: node -> incident elements, ascending
  const int32_t* inc_elem;
  const int32_t* nbr_ptr;   // one-ring graph (self included)
  const int32_t* nbr;
  const int32_t* blk_ptr;   // per one-ring entry: (e * 4 + a) * 4 + b, ascending e
  const int32_t* blk_src;
  const double* jbar_in;    // optional per-element J_bar (overrides the nodal average)
  double* V;                // E
  double* J;                // E
  double* q;                // 16 E: (V_e J_e / 4) q_e,b, four doubles per node
  double* v0;               // N
  double* Jn;               // N
  double* Jbar;             // E (output: the J_bar used)
  double* g;                // 4 x one-ring entries: g_a[b], kappa v0_a
  double* rec;              // kFbRec x E
  Status* st;
  int64_t E, N;
};

__device__ __forceinline__ void fb_nodes(const double* __restrict__ A, int4 c, double out[4][3]) {
  const int ids[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int k = 0; k < 3; ++k) out[b][k] = A[3 * (int64_t)ids[b] + k];
}

// D = [X1-X0, X2-X0, X3-X0]; g_b = rows of D^-1 (b >= 1), g_0 = -sum; V = det D / 6
__device__ __forceinline__ double fb_geometry(const double Xn[4][3], double g[4][3], double& detD) {
  double D[3][3], Di[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) D[i][j] = Xn[j + 1][i] - Xn[0][i];
  detD = inv3(D, Di);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    g[1][j] = Di[0][j];
    g[2][j] = Di[1][j];
    g[3][j] = Di[2][j];
    g[0][j] = -(Di[0][j] + Di[1][j] + Di[2][j]);
  }
  return detD / 6.0;
}

__device__ __forceinline__ void fb_F(const double Un[4][3], const double g[4][3], double F[3][3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double v = 0.0;
#pragma unroll
      for (int b = 1; b < 4; ++b) v += (Un[b][i] - Un[0][i]) * g[b][j];
      F[i][j] = (i == j ? 1.0 : 0.0) + v;
    }
}

// Copy a block's records (n x len doubles, staged in shared memory with `stride` doubles per
// record) to consecutive global memory, whole lines at a time.
// `at(j)`: place of value j in the record of LEN doubles.
template <int VALS, int STRIDE, int LEN, typename At>
__device__ __forceinline__ void fb_copy_records(double* __restrict__ out, const double* s, int n, At at) {
  for (int k = threadIdx.x; k < n * VALS; k += blockDim.x) {
    const int r = k / VALS, j = k - r * VALS;
    out[r * LEN + at(j)] = s[r * STRIDE + j];
  }
}

// The node of entry t0 + lane for the kernels with one thread per entry of ptr's runs: the
// warp finds the node of t0 by a 32-way search (three dependent loads for 30,000 nodes; a
// binary search per thread took fifteen), then the lanes step over the run ends among their
// 32 entries.  Runs of unused nodes may be empty.
__device__ __forceinline__ int64_t fb_node_of(const int32_t* __restrict__ ptr, int64_t N, int64_t t0, int lane) {
  int64_t lo = 0, hi = N;  // ptr[lo] <= t0 < ptr[hi]
  while (hi - lo > 1) {
    const int64_t step = (hi - lo + 31) / 32;
    const int64_t at = lo + step * (lane + 1);
    const unsigned m = __ballot_sync(0xffffffffu, at < hi && __ldg(ptr + at) <= t0);
    const int c = __popc(m);  // the true lanes are the first ones
    hi = min(hi, lo + step * (c + 1));
    lo += step * c;
  }
  int64_t node = lo;
  for (int64_t k = lo + 1; k < N; ++k) {  // the same for all lanes: runs that start inside the warp's entries
    const int32_t p = __ldg(ptr + k);
    if (p >= t0 + 32) break;
    if (p <= t0 + lane) node = k;
  }
  return node;
}
// Entries with more terms than this are summed by the whole warp, a term per lane (a node's
// entry with itself has 15 or 24, most have one to eight); the others by their own lane.
constexpr int kFbLong = 8;
__device__ __forceinline__ double fb_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(kFbThreads) fbar_pre(FbarArgs A) {
  __shared__ double s_q[kFbThreads * 13];
  for (int64_t e0 = blockIdx.x * (int64_t)kFbThreads; e0 < A.E; e0 += (int64_t)gridDim.x * kFbThreads) {
    const int64_t e = e0 + threadIdx.x;
    __syncthreads();
    if (e < A.E) {
      const int4 cn = reinterpret_cast<const int4*>(A.conn)[e];
      double Xn[4][3], Un[4][3], g[4][3], F[3][3], detD;
      fb_nodes(A.X, cn, Xn);
      fb_nodes(A.U, cn, Un);
      const double V = fb_geometry(Xn, g, detD);
      if (!(detD > 0.0)) flag_bad_element(A.st, e, true);
      fb_F(Un, g, F);
      const double J = det3(F);
      if (detD > 0.0 && !(J > 0.0)) flag_bad_element(A.st, e, false);
      A.V[e] = V;
      A.J[e] = J;
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            s_q[13 * threadIdx.x + 3 * b + k] = 0.25 * V * J * (F[k][0] * g[b][0] + F[k][1] * g[b][1] + F[k][2] * g[b][2]);
    }
    __syncthreads();
    fb_copy_records<12, 13, 16>(A.q + 16 * e0, s_q, (int)min((int64_t)kFbThreads, A.E - e0),
                                [](int j) { return j + j / 3; });
  }
}

// np.bincount of 0.25 V_e and 0.25 V_e J_e over the element-major node list (ascending e)
__global__ void __launch_bounds__(kFbThreads) fbar_nodes(FbarArgs A) {
  for (int64_t a = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; a < A.N; a += (int64_t)gridDim.x * blockDim.x) {
    double v0 = 0.0, v = 0.0;
    for (int32_t s = A.inc_ptr[a]; s < A.inc_ptr[a + 1]; ++s) {
      const int32_t e = A.inc_elem[s];
      const double w = 0.25 * A.V[e];
      v0 += w;
      v += w * A.J[e];
    }
    A.v0[a] = v0;
    A.Jn[a] = v / v0;  // isolated nodes never enter an element average
  }
}

// g_a[b] for every one-ring entry t (node a and its neighbour b), one thread per entry.
__global__ void __launch_bounds__(kFbThreads) fbar_patch(FbarArgs A) {
  const int lane = threadIdx.x & 31;
  const int64_t n1 = __ldg(A.nbr_ptr + A.N);
  for (int64_t t0 = blockIdx.x * (int64_t)kFbThreads + (threadIdx.x & ~31); t0 < n1; t0 += (int64_t)gridDim.x * kFbThreads) {
    const int64_t t = t0 + lane;
    const int32_t s0 = __ldg(A.blk_ptr + min(t, n1)), s1 = __ldg(A.blk_ptr + min(t + 1, n1));
    const double v0 = A.v0[fb_node_of(A.nbr_ptr, A.N, t0, lane)];
    double g[3] = {0.0, 0.0, 0.0};
    auto term = [&](int32_t s) {
      const int32_t code = __ldg(A.blk_src + s);
      return ld_quad_nc(A.q + 16 * (int64_t)(code >> 4) + 4 * (code & 3));
    };
    if (s1 - s0 <= kFbLong) {
#pragma unroll 4
      for (int32_t s = s0; s < s1; ++s) {
        const Quad x = term(s);
        g[0] += x.x;
        g[1] += x.y;
        g[2] += x.z;
      }
    }
    for (unsigned m = __ballot_sync(0xffffffffu, s1 - s0 > kFbLong); m; m &= m - 1) {
      const int k = __ffs(m) - 1;
      const int32_t a0 = __shfl_sync(0xffffffffu, s0, k), a1 = __shfl_sync(0xffffffffu, s1, k);
      double h[3] = {0.0, 0.0, 0.0};
      for (int32_t s = a0 + lane; s < a1; s += 32) {
        const Quad x = term(s);
        h[0] += x.x;
        h[1] += x.y;
        h[2] += x.z;
      }
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        h[j] = fb_warp_sum(h[j]);
        if (lane == k) g[j] = h[j];
      }
    }
    if (t < n1) {
      double2* o = reinterpret_cast<double2*>(A.g + 4 * t);
      o[0] = make_double2(g[0] / v0, g[1] / v0);
      o[1] = make_double2(g[2] / v0, A.kappa * v0);
    }
  }
}

// Register target: 168, 12 warps per SM (148 bytes spilled).  F-bar sweep of 162,000 elements:
// 312 us, with 209 registers and 8 warps 318.
constexpr int kFbElemThreads = 64;
__global__ void __launch_bounds__(kFbElemThreads, 6) fbar_element(FbarArgs A) {
  const int64_t e = blockIdx.x * (int64_t)kFbElemThreads + threadIdx.x;
  if (e < A.E) {
    const int4 cn = reinterpret_cast<const int4*>(A.conn)[e];
    double Xn[4][3], Un[4][3], g[4][3], F[3][3], detD;
    fb_nodes(A.X, cn, Xn);
    fb_nodes(A.U, cn, Un);
    const double V = fb_geometry(Xn, g, detD);
    fb_F(Un, g, F);
    const double J = det3(F);
    const double jbar = A.jbar_in ? A.jbar_in[e] : (A.Jn[cn.x] + A.Jn[cn.y] + A.Jn[cn.z] + A.Jn[cn.w]) / 4.0;
    A.Jbar[e] = jbar;
    const double r = pow(jbar / J, 1.0 / 3.0);
    // NeoHookean at F_bar = r F (neohookean.py:74-92): S_bar = C_bar^-1 (2 phi dev E_bar + beta I)
    double Fb[3][3], Fbi[3][3], Fi[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Fb[i][j] = r * F[i][j];
    const double Jb = inv3(Fb, Fbi);
    inv3(F, Fi);
    double Eb[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double c = Fb[0][i] * Fb[0][j] + Fb[1][i] * Fb[1][j] + Fb[2][i] * Fb[2][j];
        Eb[i][j] = 0.5 * (c - (i == j ? 1.0 : 0.0));
      }
    const double I1b = 3.0 + 2.0 * (Eb[0][0] + Eb[1][1] + Eb[2][2]);
    const double lnJb = log(Jb);
    const double phib = A.mu * exp((-2.0 / 3.0) * lnJb);
    const double betab = A.kappa * lnJb;
    const double trEb = Eb[0][0] + Eb[1][1] + Eb[2][2];
    double T[3][3], Cbi[3][3], Sb[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        T[i][j] = 2.0 * phib * (Eb[i][j] - (i == j ? trEb / 3.0 : 0.0)) + (i == j ? betab : 0.0);
        Cbi[i][j] = Fbi[i][0] * Fbi[j][0] + Fbi[i][1] * Fbi[j][1] + Fbi[i][2] * Fbi[j][2];
      }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Sb[i][j] = Cbi[i][0] * T[0][j] + Cbi[i][1] * T[1][j] + Cbi[i][2] * T[2][j];
    // symmetrise (S_bar is symmetric; the product above is exact up to rounding)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i + 1; j < 3; ++j) {
        const double m = 0.5 * (Sb[i][j] + Sb[j][i]);
        Sb[i][j] = m;
        Sb[j][i] = m;
      }
    const double trS = Sb[0][0] + Sb[1][1] + Sb[2][2];
    // g_b^T S_bar g_c of the ten blocks, and f: g, S_bar and F are not needed after them
    // f_b = V F [r^2 S_bar + (1 - r^2) tr(S_bar)/3 I] g_b
    double gsg[10];
#pragma unroll
    for (int a = 0, at = 0; a < 4; ++a)
#pragma unroll
      for (int b = a; b < 4; ++b, ++at) {
        gsg[at] = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) gsg[at] += g[a][i] * Sb[i][j] * g[b][j];
      }
    const double r2 = r * r;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      double w[3], f[3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
        w[i] = r2 * (Sb[i][0] * g[b][0] + Sb[i][1] * g[b][1] + Sb[i][2] * g[b][2]) +
               (1.0 - r2) * (trS / 3.0) * g[b][i];
#pragma unroll
      for (int k = 0; k < 3; ++k) f[k] = V * (F[k][0] * w[0] + F[k][1] * w[1] + F[k][2] * w[2]);
      st_quad(A.rec + fb_quad(A.E, 12 + b, e), Quad{f[0], f[1], f[2], 0.0});
    }
    // per node: p = F^-T g, q = F g, t = (F F^T)^-1 p = F^-T F^-1 p, s = p - tr(C^-1)/3 q
    double p[4][3], qv[4][3], t[4][3], s[4][3];
    double Ci[3][3];  // C^-1 = F^-1 F^-T
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Ci[i][j] = Fi[i][0] * Fi[j][0] + Fi[i][1] * Fi[j][1] + Fi[i][2] * Fi[j][2];
    const double trCi = Ci[0][0] + Ci[1][1] + Ci[2][2];
    double trCi2 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) trCi2 += Ci[i][j] * Ci[j][i];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      double fp[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        p[b][k] = Fi[0][k] * g[b][0] + Fi[1][k] * g[b][1] + Fi[2][k] * g[b][2];
        qv[b][k] = F[k][0] * g[b][0] + F[k][1] * g[b][1] + F[k][2] * g[b][2];
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) fp[k] = Fi[k][0] * p[b][0] + Fi[k][1] * p[b][1] + Fi[k][2] * p[b][2];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        t[b][k] = Fi[0][k] * fp[0] + Fi[1][k] * fp[1] + Fi[2][k] * fp[2];
        s[b][k] = p[b][k] - (trCi / 3.0) * qv[b][k];
      }
    }
    const double Ap = A.kappa + (2.0 / 9.0) * phib * I1b;
    const double Bp = (2.0 / 3.0) * phib * I1b - 2.0 * A.kappa * lnJb;
    const int gid[4] = {cn.x, cn.y, cn.z, cn.w};
    int slot = 0;
#pragma unroll
    for (int a = 0, at = 0; a < 4; ++a)
#pragma unroll
      for (int b = a; b < 4; ++b, ++at) {
        double pp = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) pp += p[a][i] * p[b][i];
        double v[3][3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            double x = Ap * s[a][k] * s[b][m] +
                       Bp * (0.5 * p[b][k] * p[a][m] - (t[a][k] * qv[b][m] + qv[a][k] * t[b][m]) / 3.0 +
                             (trCi2 / 9.0) * qv[a][k] * qv[b][m]);
            if (k == m) x += Bp * 0.5 * pp + gsg[at];
            v[k][m] = V * x;
          }
        if (a == b) {
          st_quad(A.rec + fb_quad(A.E, 16 + a, e), Quad{v[0][0], v[0][1], v[0][2], v[1][1]});
          *reinterpret_cast<double2*>(A.rec + fb_pair(A.E, a, e)) = make_double2(v[1][2], v[2][2]);
        } else {
          const bool swap = gid[a] > gid[b];  // rows = the node of smaller global id
          double o[9];
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int m = 0; m < 3; ++m) o[3 * k + m] = swap ? v[m][k] : v[k][m];
          st_quad(A.rec + fb_quad(A.E, 2 * slot, e), Quad{o[0], o[1], o[2], o[3]});
          st_quad(A.rec + fb_quad(A.E, 2 * slot + 1, e), Quad{o[4], o[5], o[6], o[7]});
          A.rec[fb_ninth(A.E, slot, e)] = o[8];
          ++slot;
        }
      }
  }
}

struct FbarGather {
  const int32_t* pair_info2;  // 4 per one-ring pair: positions in the two-ring CSR
  const int32_t* pair_ptr;
  const int32_t* pair_src;    // e * 64 + local pair slot
  const int32_t* node_info2;
  const int32_t* node_ptr;
  const int32_t* node_src;    // e * 16 + local node
  int64_t n_pairs, n_nodes, E;
};

__device__ __forceinline__ int4 fb_info(const int32_t* p) { return make_int4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3)); }

// The one-ring blocks are added to the volumetric part, which fbar_vol has written (two
// terms: the same bits in either order).  kBatch records are loaded together; each sum stays
// in ascending element order.
constexpr int kFbBatch = 2;
__global__ void __launch_bounds__(kFbThreads) fbar_gather(FbarGather G, const double* __restrict__ rec,
                                                          double* __restrict__ k_out, double* __restrict__ f_out) {
  const int64_t pairs = (G.n_pairs + 31) / 32 * 32;  // whole warps per kind
  for (int64_t it = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; it < pairs + G.n_nodes;
       it += (int64_t)gridDim.x * blockDim.x) {
    if (it < pairs) {
      if (!k_out || it >= G.n_pairs) continue;
      const int4 info = fb_info(G.pair_info2 + 4 * it);
      const int32_t s1 = __ldg(G.pair_ptr + it + 1);
      double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      for (int32_t s = __ldg(G.pair_ptr + it); s < s1; s += kFbBatch) {
        double v[kFbBatch][9];
#pragma unroll
        for (int b = 0; b < kFbBatch; ++b)
          if (s + b < s1) {
            const int32_t c = __ldg(G.pair_src + s + b);
            const int slot = c & 63;
            const int64_t e = c >> 6;
            const Quad x = ld_quad_nc(rec + fb_quad(G.E, 2 * slot, e)), y = ld_quad_nc(rec + fb_quad(G.E, 2 * slot + 1, e));
            v[b][0] = x.x; v[b][1] = x.y; v[b][2] = x.z; v[b][3] = x.w;
            v[b][4] = y.x; v[b][5] = y.y; v[b][6] = y.z; v[b][7] = y.w;
            v[b][8] = __ldg(rec + fb_ninth(G.E, slot, e));
          }
#pragma unroll
        for (int b = 0; b < kFbBatch; ++b)
          if (s + b < s1) {
#pragma unroll
            for (int j = 0; j < 9; ++j) acc[j] += v[b][j];
          }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) add3(k_out + info.x + (int64_t)info.y * k, acc[3 * k], acc[3 * k + 1], acc[3 * k + 2]);
#pragma unroll
      for (int m = 0; m < 3; ++m) add3(k_out + info.z + (int64_t)info.w * m, acc[m], acc[3 + m], acc[6 + m]);
    } else {
      const int64_t n = it - pairs;
      const int4 info = fb_info(G.node_info2 + 4 * n);
      const int32_t s1 = __ldg(G.node_ptr + n + 1);
      double d[6] = {0, 0, 0, 0, 0, 0}, f[3] = {0, 0, 0};
      for (int32_t s = __ldg(G.node_ptr + n); s < s1; s += kFbBatch) {
        double v[kFbBatch][9];
#pragma unroll
        for (int b = 0; b < kFbBatch; ++b)
          if (s + b < s1) {
            const int32_t c = __ldg(G.node_src + s + b);
            const int a = c & 15;
            const int64_t e = c >> 4;
            const Quad x = ld_quad_nc(rec + fb_quad(G.E, 12 + a, e)), y = ld_quad_nc(rec + fb_quad(G.E, 16 + a, e));
            const double2 z = __ldg(reinterpret_cast<const double2*>(rec + fb_pair(G.E, a, e)));
            v[b][0] = y.x; v[b][1] = y.y; v[b][2] = y.z; v[b][3] = y.w;
            v[b][4] = z.x; v[b][5] = z.y;
            v[b][6] = x.x; v[b][7] = x.y; v[b][8] = x.z;
          }
#pragma unroll
        for (int b = 0; b < kFbBatch; ++b)
          if (s + b < s1) {
#pragma unroll
            for (int j = 0; j < 6; ++j) d[j] += v[b][j];
#pragma unroll
            for (int k = 0; k < 3; ++k) f[k] += v[b][6 + k];
          }
      }
      if (k_out && info.y > 0) {
        const double full[9] = {d[0], d[1], d[2], d[1], d[3], d[4], d[2], d[4], d[5]};
#pragma unroll
        for (int k = 0; k < 3; ++k)
          add3(k_out + info.x + (int64_t)info.y * k, full[3 * k], full[3 * k + 1], full[3 * k + 2]);
      }
      if (f_out) store3(f_out + 3 * (int64_t)info.z, f[0], f[1], f[2]);
    }
  }
}

// two-ring block (b, c): K = sum_a (kappa v0_a) (g_a[b] g_a[c]^T), a ascending.  One thread
// per two-ring entry t (the block of node b and its t-th two-ring neighbour).  A warp's blocks
// are exchanged through shared memory and leave row by row, 32 consecutive values per store.
__global__ void __launch_bounds__(kFbThreads) fbar_vol(int64_t N, const int32_t* __restrict__ nbr2_ptr,
                                                       const int32_t* __restrict__ vol_ptr,
                                                       const int32_t* __restrict__ vol_src,
                                                       const double* __restrict__ g, double* __restrict__ k_out) {
  __shared__ double s_all[kFbThreads / 32][32 * 9];
  __shared__ int64_t s_pos[kFbThreads / 32][32];
  __shared__ int32_t s_stride[kFbThreads / 32][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double* s_k = s_all[w];
  const int64_t n2 = __ldg(nbr2_ptr + N);
  for (int64_t t0 = blockIdx.x * (int64_t)kFbThreads + 32 * w; t0 < n2; t0 += (int64_t)gridDim.x * kFbThreads) {
    const int64_t t = t0 + lane;
    const int32_t s0 = __ldg(vol_ptr + min(t, n2)), s1 = __ldg(vol_ptr + min(t + 1, n2));
    const int64_t b = fb_node_of(nbr2_ptr, N, t0, lane);
    const int32_t p0 = __ldg(nbr2_ptr + b), p1 = __ldg(nbr2_ptr + b + 1);
    s_stride[w][lane] = 3 * (p1 - p0);
    s_pos[w][lane] = 9 * (int64_t)p0 + 3 * (t - p0);
    auto add = [&](double acc[9], int32_t s) {
      const int32_t* v = vol_src + 3 * (int64_t)s;
      const Quad gb = ld_quad_nc(g + 4 * (int64_t)__ldg(v + 1)), gc = ld_quad_nc(g + 4 * (int64_t)__ldg(v + 2));
      const double b3[3] = {gb.x, gb.y, gb.z}, c3[3] = {gc.x, gc.y, gc.z};
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int m = 0; m < 3; ++m) acc[3 * k + m] += gb.w * (b3[k] * c3[m]);
    };
    double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (s1 - s0 <= kFbLong) {
#pragma unroll 2
      for (int32_t s = s0; s < s1; ++s) add(acc, s);
    }
#pragma unroll
    for (int j = 0; j < 9; ++j) s_k[9 * lane + j] = acc[j];
    for (unsigned m = __ballot_sync(0xffffffffu, s1 - s0 > kFbLong); m; m &= m - 1) {
      const int e = __ffs(m) - 1;
      const int32_t a0 = __shfl_sync(0xffffffffu, s0, e), a1 = __shfl_sync(0xffffffffu, s1, e);
      double sum[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      for (int32_t s = a0 + lane; s < a1; s += 32) add(sum, s);
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        const double x = fb_warp_sum(sum[j]);
        if (lane == e) s_k[9 * e + j] = x;
      }
    }
    __syncwarp();
    const int n = (int)min((int64_t)32, n2 - t0);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      for (int c = lane; c < 3 * n; c += 32) {
        const int i = c / 3, m = c - 3 * i;
        __stcs(k_out + s_pos[w][i] + (int64_t)s_stride[w][i] * k + m, s_k[9 * i + 3 * k + m]);
      }
    __syncwarp();
  }
}

// Single elements with given J_bar (Tet4Fbar.compute_nonlinear_force_and_tangent_stiffness,
// element/tet4_fbar.py:147-211): k = B_bar^T C B_bar V + G^T (I (x) S_bar) G V with the full
// Voigt tangent C of NeoHookean at F_bar (material/neohookean.py:95-120, Voigt order
// xx yy zz xy yz zx), B the nonlinear strain-displacement matrix and
// B_bar = r^2 (B - m b_vol^T) + m b_vol^T.  An API-compatibility path: one thread per
// element, explicit 6 x 12 products.
__global__ void __launch_bounds__(kFbThreads) fbar_single(int64_t n, const double* __restrict__ Xe,
                                                          const double* __restrict__ Ue,
                                                          const double* __restrict__ jbar, double mu, double kappa,
                                                          double* __restrict__ k_out, double* __restrict__ f_out,
                                                          Status* st) {
  constexpr int vi[6] = {0, 1, 2, 0, 1, 2}, vj[6] = {0, 1, 2, 1, 2, 0};
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    double Xn[4][3], Un[4][3], g[4][3], F[3][3], detD;
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        Xn[b][k] = Xe[12 * e + 3 * b + k];
        Un[b][k] = Ue[12 * e + 3 * b + k];
      }
    const double V = fb_geometry(Xn, g, detD);
    if (!(detD > 0.0)) flag_bad_element(st, e, true);
    fb_F(Un, g, F);
    const double J = det3(F);
    if (detD > 0.0 && !(J > 0.0)) flag_bad_element(st, e, false);
    const double r = pow(jbar[e] / J, 1.0 / 3.0);
    double Fb[3][3], C[3][3], Ci[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Fb[i][j] = r * F[i][j];
    const double Jb = det3(Fb);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) C[i][j] = Fb[0][i] * Fb[0][j] + Fb[1][i] * Fb[1][j] + Fb[2][i] * Fb[2][j];
    inv3(C, Ci);
    const double I1 = C[0][0] + C[1][1] + C[2][2];
    const double fac = mu * pow(Jb, -2.0 / 3.0);
    const double lnJ = log(Jb);
    double S[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) S[i][j] = fac * ((i == j ? 1.0 : 0.0) - I1 / 3.0 * Ci[i][j]) + kappa * lnJ * Ci[i][j];
    double Cv[6][6];
    for (int a = 0; a < 6; ++a)
      for (int b = 0; b < 6; ++b) {
        const int i = vi[a], j = vj[a], k = vi[b], l = vj[b];
        const double oo = Ci[i][j] * Ci[k][l];
        const double ii = 0.5 * (Ci[i][k] * Ci[j][l] + Ci[i][l] * Ci[j][k]);
        const double ci = Ci[i][j] * (k == l ? 1.0 : 0.0) + (i == j ? 1.0 : 0.0) * Ci[k][l];
        Cv[a][b] = kappa * oo - 2.0 * kappa * lnJ * ii - (2.0 / 3.0) * fac * ci + (2.0 / 9.0) * fac * I1 * oo +
                   (2.0 / 3.0) * fac * I1 * ii;
      }
    double Bb[6][12];
    for (int b = 0; b < 4; ++b)
      for (int k = 0; k < 3; ++k) {
        double col[6];
        for (int a = 0; a < 6; ++a) {
          const int i = vi[a], j = vj[a];
          col[a] = i == j ? F[k][i] * g[b][i] : F[k][i] * g[b][j] + F[k][j] * g[b][i];
        }
        const double bvol = (col[0] + col[1] + col[2]) / 3.0;
        for (int a = 0; a < 6; ++a) {
          const double m = a < 3 ? 1.0 : 0.0;
          Bb[a][3 * b + k] = r * r * (col[a] - m * bvol) + m * bvol;
        }
      }
    double CB[6][12];
    for (int a = 0; a < 6; ++a)
      for (int c = 0; c < 12; ++c) {
        double x = 0.0;
        for (int b = 0; b < 6; ++b) x += Cv[a][b] * Bb[b][c];
        CB[a][c] = x;
      }
    const double Sv[6] = {S[0][0], S[1][1], S[2][2], S[0][1], S[1][2], S[2][0]};
    for (int c = 0; c < 12; ++c) {
      double fv = 0.0;
      for (int a = 0; a < 6; ++a) fv += Bb[a][c] * Sv[a];
      f_out[12 * e + c] = fv * V;
      for (int d = 0; d < 12; ++d) {
        double x = 0.0;
        for (int a = 0; a < 6; ++a) x += Bb[a][c] * CB[a][d];
        double geo = 0.0;
        if (c % 3 == d % 3) {
          const int pa = c / 3, pb = d / 3;
          for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) geo += g[pa][i] * S[i][j] * g[pb][j];
        }
        k_out[144 * e + 12 * c + d] = x * V + geo * V;
      }
    }
  }
}

inline int fb_grid(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + kFbThreads - 1) / kFbThreads, 148 * 16)); }

}  // namespace
}  // namespace psx

extern "C" int psx_fbar_element(int64_t n, const double* X_elem, const double* u_elem, const double* jbar, double mu,
                                double kappa, double* k_out, double* f_out, void* status, void* stream) {
  using namespace psx;
  if (n <= 0 || !X_elem || !u_elem || !jbar || !k_out || !f_out || !status) return PSX_ERR_ARG;
  fbar_single<<<fb_grid(n), kFbThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      n, X_elem, u_elem, jbar, mu, kappa, k_out, f_out, static_cast<Status*>(status));
  PSX_CUDA_CHECK_LAUNCH();
  return PSX_OK;
}

extern "C" int64_t psx_fbar_work_doubles(int64_t E, int64_t N, int64_t n_nbr) {
  return 4 * E + 2 * N + 16 * E + 4 * n_nbr + (int64_t)psx::kFbRec * E + 3;  // + 3: 32-byte alignment of q, g and records
}

extern "C" int psx_fbar_assemble(const int32_t* conn, int64_t E, int64_t N, const double* X, const double* u,
                                 double mu, double kappa, const int32_t* inc_ptr, const int32_t* inc_elem,
                                 const int32_t* nbr_ptr, const int32_t* nbr, int64_t n_nbr, const int32_t* blk_ptr,
                                 const int32_t* blk_src, int64_t n_pairs, const int32_t* pair_info2,
                                 const int32_t* pair_ptr, const int32_t* pair_src, const int32_t* node_info2,
                                 const int32_t* node_ptr, const int32_t* node_src, const int32_t* nbr2_ptr,
                                 const int32_t* vol_ptr, const int32_t* vol_src, const double* jbar_in,
                                 double* f_out, double* k_out, int64_t nnz2, double* jbar_out, double* work,
                                 int64_t work_doubles, void* status, void* stream) {
  using namespace psx;
  if (!conn || E <= 0 || N <= 0 || !X || !u || !inc_ptr || !inc_elem || !nbr_ptr || !nbr || !blk_ptr || !blk_src ||
      !pair_info2 || !pair_ptr || !pair_src || !node_info2 || !node_ptr || !node_src || !nbr2_ptr || !vol_ptr ||
      !vol_src || !work || !status || (!f_out && !k_out))
    return PSX_ERR_ARG;
  if (work_doubles < psx_fbar_work_doubles(E, N, n_nbr) || (k_out && nnz2 <= 0)) return PSX_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  FbarArgs A;
  A.conn = conn; A.X = X; A.U = u; A.mu = mu; A.kappa = kappa;
  A.inc_ptr = inc_ptr; A.inc_elem = inc_elem; A.nbr_ptr = nbr_ptr; A.nbr = nbr;
  A.blk_ptr = blk_ptr; A.blk_src = blk_src; A.jbar_in = jbar_in;
  double* w = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(work) + 31) / 32 * 32);
  A.rec = w; w += (int64_t)kFbRec * E;
  A.q = w; w += 16 * E;
  A.g = w; w += 4 * n_nbr;
  A.V = w; w += E;
  A.J = w; w += E;
  A.v0 = w; w += N;
  A.Jn = w; w += N;
  A.Jbar = jbar_out ? jbar_out : w;
  A.st = static_cast<Status*>(status);
  A.E = E; A.N = N;
  fbar_pre<<<fb_grid(E), kFbThreads, 0, s>>>(A);
  fbar_nodes<<<fb_grid(N), kFbThreads, 0, s>>>(A);
  if (k_out) fbar_patch<<<fb_grid(n_nbr), kFbThreads, 0, s>>>(A);  // one thread per one-ring entry
  // before the element pass, so that the records are still in L2 when they are gathered; the
  // two-ring CSR holds 9 values per entry
  if (k_out)
    fbar_vol<<<fb_grid(nnz2 / 9), kFbThreads, 0, s>>>(N, nbr2_ptr, vol_ptr, vol_src, A.g, k_out);
  if ((E + kFbElemThreads - 1) / kFbElemThreads > 0x7fffffff) return PSX_ERR_LIMIT;
  fbar_element<<<(unsigned)((E + kFbElemThreads - 1) / kFbElemThreads), kFbElemThreads, 0, s>>>(A);
  FbarGather G{pair_info2, pair_ptr, pair_src, node_info2, node_ptr, node_src, n_pairs, N, E};
  fbar_gather<<<fb_grid(n_pairs + N), kFbThreads, 0, s>>>(G, A.rec, k_out, f_out);
  PSX_CUDA_CHECK_LAUNCH();
  return PSX_OK;
}
