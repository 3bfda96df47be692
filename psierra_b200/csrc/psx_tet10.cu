// Tet10 Total-Lagrangian NeoHookean assembly for sm_100a.
//
// Replaces the element loops of SolidDomain (psierra domain/solid.py:172-207, 230-325)
// around Tet10TotalLagrangian.compute_nonlinear_force_and_tangent_stiffness
// (element/tet10_total_lagrangian.py:63-136; shape gradients element/tet10_base.py:118-179,
// VTK edge order 4:(0,1) 5:(1,2) 6:(2,0) 7:(0,3) 8:(1,3) 9:(2,3); 4-point rule
// element/quadrature.py:36-49 with weight 1/24) and the COO->CSR / np.add.at scatter.
//
// Element tiles of up to 8 elements are evaluated by one warp in two phases:
//   1. lane 4*le + q handles element le of the tile at quadrature point q: Jacobian
//      J = X^T dN, det J, H = dN J^-1, the displacement gradient, the NeoHookean point
//      (psx_common.cuh), the nodal force contributions (reduced over the 4 q-lanes of
//      the element in a fixed tree) and, per node, p = F^-T H_a, q = F H_a, H_a into
//      shared memory with the weighted tangent coefficients;
//   2. the warp spreads the 8 x 55 3x3 blocks (45 node pairs + 10 diagonals) over its
//      lanes; each sums its block over the 4 quadrature points with the closed form of
//      psx_common.cuh and writes it into the element's record.
// The records are then gathered by the shared owner-computes queue (psx_gather.cuh).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "psx_common.cuh"
#include "psx_gather.cuh"

namespace psx {
namespace {

constexpr int kThreads10 = 128;
constexpr int kTile10 = 8;  // elements per warp task (one per 4 lanes)
using L10 = RecLayout<10>;

// local node pairs (a < b) in slot order, then the 10 diagonals
struct PairTable {
  int8_t a[55], b[55];
};
__constant__ PairTable c_pairs = {
    {0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 1, 1, 1, 1, 2, 2, 2, 2, 2, 2, 2, 3, 3, 3, 3, 3, 3, 4, 4, 4, 4, 4, 5, 5, 5, 5,
     6, 6, 6, 7, 7, 8, 0, 1, 2, 3, 4, 5, 6, 7, 8, 9},
    {1, 2, 3, 4, 5, 6, 7, 8, 9, 2, 3, 4, 5, 6, 7, 8, 9, 3, 4, 5, 6, 7, 8, 9, 4, 5, 6, 7, 8, 9, 5, 6, 7, 8, 9, 6, 7, 8, 9,
     7, 8, 9, 8, 9, 9, 0, 1, 2, 3, 4, 5, 6, 7, 8, 9}};

// Consistent mass of the 10-node tetrahedron with straight edges: M_ab = rho V m_ab / 2520
// times the 3x3 identity, m_ab the exact integrals of N_a N_b over the reference element
// (VTK node order; element/tet10_base.py:11-27, 344-372).
__constant__ int16_t c_mass10[10][10] = {
    {36, 6, 6, 6, -24, -36, -24, -24, -36, -36},   {6, 36, 6, 6, -24, -24, -36, -36, -24, -36},
    {6, 6, 36, 6, -36, -24, -24, -36, -36, -24},   {6, 6, 6, 36, -36, -36, -36, -24, -24, -24},
    {-24, -24, -36, -36, 192, 96, 96, 96, 96, 48}, {-36, -24, -24, -36, 96, 192, 96, 48, 96, 96},
    {-24, -36, -24, -36, 96, 96, 192, 96, 48, 96}, {-24, -36, -36, -24, 96, 48, 96, 192, 96, 96},
    {-36, -24, -36, -24, 96, 96, 48, 96, 192, 96}, {-36, -36, -24, -24, 48, 96, 96, 96, 96, 192}};

// Barycentric coordinates (L1, L2, L3) of the 4-point rule: a = (5 - sqrt 5)/20,
// b = (5 + 3 sqrt 5)/20.
__device__ __forceinline__ void qp_coords(int q, double& L1, double& L2, double& L3) {
  const double a = 0.13819660112501051517954131656344, b = 0.58541019662496845446137605030969;
  L1 = q == 1 ? b : a;
  L2 = q == 2 ? b : a;
  L3 = q == 3 ? b : a;
}

// dN_a / d(xi, eta, zeta) at (L1, L2, L3); tet10_base.py:137-177.
__device__ __forceinline__ void shape_grad(int a, double L1, double L2, double L3, double d[3]) {
  const double L0 = 1.0 - L1 - L2 - L3;
  switch (a) {
    case 0: d[0] = d[1] = d[2] = -(4.0 * L0 - 1.0); break;
    case 1: d[0] = 4.0 * L1 - 1.0; d[1] = 0.0; d[2] = 0.0; break;
    case 2: d[0] = 0.0; d[1] = 4.0 * L2 - 1.0; d[2] = 0.0; break;
    case 3: d[0] = 0.0; d[1] = 0.0; d[2] = 4.0 * L3 - 1.0; break;
    case 4: d[0] = 4.0 * (L0 - L1); d[1] = -4.0 * L1; d[2] = -4.0 * L1; break;
    case 5: d[0] = 4.0 * L2; d[1] = 4.0 * L1; d[2] = 0.0; break;
    case 6: d[0] = -4.0 * L2; d[1] = 4.0 * (L0 - L2); d[2] = -4.0 * L2; break;
    case 7: d[0] = -4.0 * L3; d[1] = -4.0 * L3; d[2] = 4.0 * (L0 - L3); break;
    case 8: d[0] = 4.0 * L3; d[1] = 0.0; d[2] = 4.0 * L1; break;
    default: d[0] = 0.0; d[1] = 4.0 * L3; d[2] = 4.0 * L2; break;
  }
}

struct Tet10Args {
  const int32_t* conn;
  const double* X;
  const double* U;
  const double* mu_e;
  const double* kappa_e;
  double mu0, kappa0, lam0;
  Status* st;
};

// Shared-memory scratch of one warp: per (element, qp, node) a 48-byte record, per (element,
// qp) the weighted tangent coefficients.  FP32: p, q, H as three 16-byte vectors.  FP64: p and
// q as three pairs; H_a.H_b is formed as p_a.q_b (p = F^-T H, q = F H), which left the error of
// the blocks against extended precision where it was (3.5e-14 of their norm at strains of
// 0.2).  The block phase was bound by its 22 scalar loads per block and point (84% of the
// kernel's shared-memory cycles, FP64); three vector loads per node take a third of them, and
// 48 bytes keep consecutive nodes on distinct banks.  f + K, 162,000 elements, one launch:
// 1035 -> 863 us FP64, 652 -> 639 us FP32; with H kept beside them 5 vectors: 797 us against
// 736 (two passes).
template <typename KT>
struct Tet10Smem;
template <>
struct Tet10Smem<float> {
  float4 v[kTile10][4][10][3];
  float4 c[kTile10][4];  // A, hb, c, phi (times w det J)
  __device__ __forceinline__ void put(int e, int q, int a, const float p[3], const float qv[3], const float h[3]) {
    v[e][q][a][0] = make_float4(p[0], p[1], p[2], 0.f);
    v[e][q][a][1] = make_float4(qv[0], qv[1], qv[2], 0.f);
    v[e][q][a][2] = make_float4(h[0], h[1], h[2], 0.f);
  }
  __device__ __forceinline__ void node(int e, int q, int a, float p[3], float qv[3], float h[3]) const {
    const float4 x = v[e][q][a][0], y = v[e][q][a][1], z = v[e][q][a][2];
    p[0] = x.x; p[1] = x.y; p[2] = x.z;
    qv[0] = y.x; qv[1] = y.y; qv[2] = y.z;
    h[0] = z.x; h[1] = z.y; h[2] = z.z;
  }
  __device__ __forceinline__ void put_coef(int e, int q, const TangentCoef<float>& t) {
    c[e][q] = make_float4(t.A, t.hb, t.c, t.phi);
  }
  __device__ __forceinline__ TangentCoef<float> coef(int e, int q) const {
    const float4 x = c[e][q];
    return TangentCoef<float>{x.x, x.y, x.z, x.w};
  }
  static __device__ __forceinline__ float gram(const float[3], const float[3], const float ha[3], const float hb[3]) {
    return ha[0] * hb[0] + ha[1] * hb[1] + ha[2] * hb[2];
  }
};
template <>
struct Tet10Smem<double> {
  double2 v[kTile10][4][10][3];
  double2 c[kTile10][4][2];
  __device__ __forceinline__ void put(int e, int q, int a, const double p[3], const double qv[3], const double[3]) {
    v[e][q][a][0] = make_double2(p[0], p[1]);
    v[e][q][a][1] = make_double2(p[2], qv[0]);
    v[e][q][a][2] = make_double2(qv[1], qv[2]);
  }
  __device__ __forceinline__ void node(int e, int q, int a, double p[3], double qv[3], double[3]) const {
    const double2 x = v[e][q][a][0], y = v[e][q][a][1], z = v[e][q][a][2];
    p[0] = x.x; p[1] = x.y; p[2] = y.x;
    qv[0] = y.y; qv[1] = z.x; qv[2] = z.y;
  }
  __device__ __forceinline__ void put_coef(int e, int q, const TangentCoef<double>& t) {
    c[e][q][0] = make_double2(t.A, t.hb);
    c[e][q][1] = make_double2(t.c, t.phi);
  }
  __device__ __forceinline__ TangentCoef<double> coef(int e, int q) const {
    const double2 x = c[e][q][0], y = c[e][q][1];
    return TangentCoef<double>{x.x, x.y, y.x, y.y};
  }
  static __device__ __forceinline__ double gram(const double pa[3], const double qb[3], const double[3], const double[3]) {
    return pa[0] * qb[0] + pa[1] * qb[1] + pa[2] * qb[2];
  }
};

template <typename KT, int MODE>
__device__ __forceinline__ void tet10_tile(const Tet10Args& A, const int4& task, int64_t ring_mask,
                                           KT* __restrict__ krec, double* __restrict__ frec, Tet10Smem<KT>& sm) {
  constexpr bool kLinear = (MODE & PSX_LINEAR) != 0;
  constexpr bool kWantF = (MODE & PSX_WANT_F) != 0 && !kLinear;
  constexpr bool kWantK = (MODE & PSX_WANT_K) != 0 || kLinear;
  const int lane = threadIdx.x & 31;
  if constexpr ((MODE & PSX_MASS) != 0) {
    // consistent mass (density in lam0) with the element volume of the mesh, |det| / 6 of
    // the corner tetrahedron (domain/solid.py:209-228): one 3x3 block per lane
    const int n = (int)(task.w - task.z);
    for (int t = lane; t < n * 55; t += 32) {
      const int me = t / 55, slot = t - me * 55;
      const int a = c_pairs.a[slot], b = c_pairs.b[slot];
      const int64_t em = task.z + me;
      double Xc[4][3];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const double* x = A.X + 3 * (int64_t)__ldg(A.conn + 10 * em + c);
#pragma unroll
        for (int i = 0; i < 3; ++i) Xc[c][i] = __ldg(x + i);
      }
      double D[3][3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) D[i][j] = Xc[j + 1][i] - Xc[0][i];
      const double V = fabs(det3(D)) / 6.0;
      const KT m = (KT)(A.lam0 * V * (double)c_mass10[a][b] / 2520.0);
      KT* rec = krec + (em & ring_mask) * L10::kK;
      if (slot < 45) {
        const KT blk[9] = {m, (KT)0, (KT)0, (KT)0, m, (KT)0, (KT)0, (KT)0, m};
        store_pair_block<KT>(rec + L10::pair_off(slot), blk, false);
      } else {
        const KT dg[6] = {m, (KT)0, (KT)0, m, (KT)0, m};
        store_diag_block<KT>(rec + L10::diag_off(slot - 45), dg);
      }
    }
    return;
  }
  const int le = lane >> 2, q = lane & 3;
  const int64_t e = task.z + (int64_t)le;
  const bool active = e < task.w;
  // ---- phase 1: one (element, quadrature point) per lane
  double L1, L2, L3;
  qp_coords(q, L1, L2, L3);
  int32_t nid[10];
  if (active) {
    const int2* c2 = reinterpret_cast<const int2*>(A.conn + 10 * e);  // 40-byte rows are 8-byte aligned
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const int2 t = __ldg(c2 + i);
      nid[2 * i] = t.x;
      nid[2 * i + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 10; ++i) nid[i] = 0;
  }
  double Jm[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
  for (int a = 0; a < 10; ++a) {
    double d[3];
    shape_grad(a, L1, L2, L3, d);
    const double* x = A.X + 3 * (int64_t)nid[a];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double xi = active ? __ldg(x + i) : (i == (a % 3) ? 1.0 : 0.0);
#pragma unroll
      for (int j = 0; j < 3; ++j) Jm[i][j] += xi * d[j];
    }
  }
  double Ji[3][3];
  const double detJ = inv3(Jm, Ji);
  if (active && !(detJ > 0.0)) flag_bad_element(A.st, e, true);
  const double w = detJ / 24.0;
  double mu = A.mu0, kappa = A.kappa0;
  if (active && A.mu_e) mu = A.mu_e[e];
  if (active && A.kappa_e) kappa = A.kappa_e[e];
  PointState ps;
  TangentCoef<KT> tc;
  if constexpr (kLinear) {
    tc.A = (KT)(w * A.lam0);
    tc.hb = (KT)(w * A.mu0);
    tc.c = (KT)0;
    tc.phi = (KT)(w * A.mu0);
  } else {
    double l[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    double u0[3] = {0, 0, 0};
    if (active) {
      const double* up = A.U + 3 * (int64_t)nid[0];
      u0[0] = __ldg(up);
      u0[1] = __ldg(up + 1);
      u0[2] = __ldg(up + 2);
    }
#pragma unroll
    for (int a = 1; a < 10; ++a) {
      double d[3], H[3];
      shape_grad(a, L1, L2, L3, d);
#pragma unroll
      for (int j = 0; j < 3; ++j) H[j] = d[0] * Ji[0][j] + d[1] * Ji[1][j] + d[2] * Ji[2][j];
      const double* up = A.U + 3 * (int64_t)nid[a];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double du = active ? __ldg(up + i) - u0[i] : 0.0;
#pragma unroll
        for (int j = 0; j < 3; ++j) l[i][j] += du * H[j];
      }
    }
    neohookean_point(l, mu, kappa, ps);
    if (active && detJ > 0.0 && ps.Jm1 <= -1.0) flag_bad_element(A.st, e, false);
    tc = tangent_coef<KT>(ps, kappa, w);
  }
  KT Fi[3][3], Fm[3][3];
  if constexpr (!kLinear) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        Fi[i][j] = (KT)ps.Finv[i][j];
        Fm[i][j] = (KT)ps.F[i][j];
      }
  }
#pragma unroll
  for (int a = 0; a < 10; ++a) {
    double d[3], H[3];
    shape_grad(a, L1, L2, L3, d);
#pragma unroll
    for (int j = 0; j < 3; ++j) H[j] = d[0] * Ji[0][j] + d[1] * Ji[1][j] + d[2] * Ji[2][j];
    if constexpr (kWantF) {
      // f_a += w P H_a, summed over the element's 4 q-lanes in a fixed tree
      double fa[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        double v = active ? w * (ps.P[i][0] * H[0] + ps.P[i][1] * H[1] + ps.P[i][2] * H[2]) : 0.0;
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        fa[i] = v;
      }
      if (active && q == 0) {
        double* fr = frec + (e & ring_mask) * L10::kF + 3 * a;
        st_ring(fr, fa[0]);
        st_ring(fr + 1, fa[1]);
        st_ring(fr + 2, fa[2]);
      }
    }
    if constexpr (kWantK) {
      const KT Hk[3] = {(KT)H[0], (KT)H[1], (KT)H[2]};
      if constexpr (kLinear) {
        sm.put(le, q, a, Hk, Hk, Hk);
      } else {
        KT pk[3], qk[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          pk[k] = Fi[0][k] * Hk[0] + Fi[1][k] * Hk[1] + Fi[2][k] * Hk[2];
          qk[k] = Fm[k][0] * Hk[0] + Fm[k][1] * Hk[1] + Fm[k][2] * Hk[2];
        }
        sm.put(le, q, a, pk, qk, Hk);
      }
    }
  }
  if constexpr (kWantK) {
    sm.put_coef(le, q, tc);
    __syncwarp();
    // ---- phase 2: blocks of the tile, summed over the 4 quadrature points
    const int n = (int)(task.w - task.z);
    for (int t = lane; t < n * 55; t += 32) {
      const int me = t / 55, slot = t - me * 55;
      const int a = c_pairs.a[slot], b = c_pairs.b[slot];
      KT acc[9];
#pragma unroll
      for (int j = 0; j < 9; ++j) acc[j] = (KT)0;
#pragma unroll
      for (int qq = 0; qq < 4; ++qq) {
        const TangentCoef<KT> co = sm.coef(me, qq);
        KT pa[3], qa[3], xa[3], pb[3], qb[3], xb[3], ha[3], ya[3], wb[3];
        sm.node(me, qq, a, pa, qa, xa);
        sm.node(me, qq, b, pb, qb, xb);
        const KT s = co.phi * Tet10Smem<KT>::gram(pa, qb, xa, xb);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          ha[k] = co.hb * pa[k];
          ya[k] = co.c * qa[k];
          wb[k] = co.A * pb[k] + co.c * qb[k];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int m = 0; m < 3; ++m) acc[3 * k + m] += pa[k] * wb[m] + pb[k] * ha[m] + ya[k] * pb[m] + (k == m ? s : (KT)0);
      }
      const int64_t em = task.z + me;
      KT* rec = krec + (em & ring_mask) * L10::kK;
      if (slot < 45) {
        const int32_t ga = __ldg(A.conn + 10 * em + a), gb = __ldg(A.conn + 10 * em + b);
        store_pair_block<KT>(rec + L10::pair_off(slot), acc, ga > gb);
      } else {
        const KT dg[6] = {acc[0], acc[1], acc[2], acc[4], acc[5], acc[8]};
        store_diag_block<KT>(rec + L10::diag_off(slot - 45), dg);
      }
    }
  }
}

template <typename KT, int MODE>
__global__ void __launch_bounds__(kThreads10, 2)
tet10_persistent_kernel(Tet10Args A, GatherArgs g, QueueArgs Q, KT* __restrict__ krec, double* __restrict__ frec,
                        KT* __restrict__ k_out, double* __restrict__ f_out) {
  constexpr bool kWantF = (MODE & PSX_WANT_F) != 0;
  constexpr bool kWantK = (MODE & (PSX_WANT_K | PSX_LINEAR | PSX_MASS)) != 0;
  extern __shared__ __align__(16) unsigned char s_raw[];
  Tet10Smem<KT>& sm = reinterpret_cast<Tet10Smem<KT>*>(s_raw)[threadIdx.x >> 5];
  auto element_tile = [&](const int4& task) { tet10_tile<KT, MODE>(A, task, g.ring_mask, krec, frec, sm); };
  drain_queue<KT, 10, kWantK, kWantF, false, false>(g, Q, A.st, krec, frec, k_out, f_out, DRArgs{}, element_tile);
}

// Two passes, as psx_tet4.cu: element tiles (8 elements per one-warp block), then one thread
// per pair / node.  The queue kept every SM at 8 warps (252 registers) for both phases and
// its gathers, latency bound, waited on element tiles; split, a tile takes 168 registers and
// no task (12 warps per SM), and the gathers run at their own occupancy with cached 32-byte
// loads.  Kuhn cubes, us, queue / two passes: f + K FP64 384 elements 35 / 23,
// 10,368 79 / 56, 162,000 1035 / 685, 750,000 4041 / 3280; FP32 162,000 652 / 493; f 384
// elements 16 / 11, 162,000 200 / 76.  Tiles: 8 warps per SM 730 us (FP64 f + K, batches of
// 2), 9 and more 708.  Pass 1 is bound by shared memory and FP64 latency, pass 2 by DRAM
// (1.66 GB of records and values at 67% of the measured copy rate).
template <typename KT, int MODE>
constexpr int tiles10_blocks() {
  return (MODE & PSX_MASS) != 0 ? 16 : sizeof(KT) == 8 && (MODE & (PSX_WANT_K | PSX_LINEAR)) != 0 ? 9 : 11;
}
template <typename KT, int MODE>
__global__ void __launch_bounds__(32, (tiles10_blocks<KT, MODE>()))
tet10_tiles_kernel(Tet10Args A, int64_t ring_mask, int64_t n_elements, KT* __restrict__ krec, double* __restrict__ frec) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  const int64_t e0 = kTile10 * (int64_t)blockIdx.x;
  tet10_tile<KT, MODE>(A, make_int4(0, 0, (int)e0, (int)min(e0 + kTile10, n_elements)), ring_mask, krec, frec,
                       *reinterpret_cast<Tet10Smem<KT>*>(s_raw));
}

// Records in flight per thread: 3 (FP64 / FP32 f + K, 162,000 elements: 685 / 493 us; 1: 715 /
// 510, 2: 697 / 504, 4: 686 / 493).
constexpr int kItemThreads10 = 128, kItemBatch10 = 3;
template <typename KT, int MODE>
__global__ void __launch_bounds__(kItemThreads10)
tet10_items_kernel(GatherArgs g, int32_t n_pairs, int32_t n_nodes, const KT* __restrict__ krec,
                   const double* __restrict__ frec, KT* __restrict__ k_out, double* __restrict__ f_out) {
  constexpr bool kWantF = (MODE & PSX_WANT_F) != 0;
  constexpr bool kWantK = (MODE & (PSX_WANT_K | PSX_LINEAR | PSX_MASS)) != 0;
  const int32_t pairs = kWantK ? (n_pairs + 31) / 32 * 32 : 0;  // whole warps per kind
  const int32_t i = blockIdx.x * kItemThreads10 + threadIdx.x;
  if (i < pairs) {
    if constexpr (kWantK)
      if (i < n_pairs) gather_pair<KT, 10, false, kWantF, kItemBatch10, true, true>(g, pair_head<false>(g, i), krec, k_out);
  } else if (i - pairs < n_nodes) {
    gather_node<KT, 10, kWantK, kWantF, false, false, kItemBatch10, true, true>(g, node_head<false>(g, i - pairs), krec,
                                                                                frec, k_out, f_out);
  }
}

// det J and det F at the 4 quadrature points of one element (error messages).
__global__ void tet10_dets_kernel(const int32_t* __restrict__ conn, const double* __restrict__ X,
                                  const double* __restrict__ U, int64_t e, double* out8) {
  const int q = threadIdx.x;
  if (q >= 4) return;
  double L1, L2, L3;
  qp_coords(q, L1, L2, L3);
  double Jm[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, Fm[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
  for (int a = 0; a < 10; ++a) {
    double d[3];
    shape_grad(a, L1, L2, L3, d);
    const int64_t n = conn[10 * e + a];
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) Jm[i][j] += X[3 * n + i] * d[j];
  }
  double Ji[3][3];
  const double detJ = inv3(Jm, Ji);
  if (U) {
    for (int a = 0; a < 10; ++a) {
      double d[3], H[3];
      shape_grad(a, L1, L2, L3, d);
      for (int j = 0; j < 3; ++j) H[j] = d[0] * Ji[0][j] + d[1] * Ji[1][j] + d[2] * Ji[2][j];
      const int64_t n = conn[10 * e + a];
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) Fm[i][j] += U[3 * n + i] * H[j];
    }
  }
  out8[2 * q] = detJ;
  out8[2 * q + 1] = det3(Fm);
}

template <typename KT, int MODE>
int run_tet10(const psx_plan_t* P, const Tet10Args& A, const WorkLayout& W, KT* k_out, double* f_out,
              cudaStream_t stream) {
  constexpr bool kWantK = (MODE & (PSX_WANT_K | PSX_LINEAR | PSX_MASS)) != 0;
  const GatherArgs g = gather_args(P, W.ring_elems);
  if (kWantK ? P->two_pass_k : P->two_pass) {
    // f and the mass matrix stage nothing
    const size_t smem = (MODE & (PSX_WANT_K | PSX_LINEAR)) != 0 ? sizeof(Tet10Smem<KT>) : 0;
    tet10_tiles_kernel<KT, MODE><<<(unsigned)((P->n_elements + kTile10 - 1) / kTile10), 32, smem, stream>>>(
        A, g.ring_mask, P->n_elements, static_cast<KT*>(W.krec), W.frec);
    const int64_t items = (kWantK ? (P->n_pairs + 31) / 32 * 32 : 0) + P->n_nodes;
    tet10_items_kernel<KT, MODE><<<(unsigned)((items + kItemThreads10 - 1) / kItemThreads10), kItemThreads10, 0, stream>>>(
        g, (int32_t)P->n_pairs, (int32_t)P->n_nodes, static_cast<const KT*>(W.krec), W.frec, k_out, f_out);
    PSX_CUDA_CHECK_LAUNCH();
    return PSX_OK;
  }
  const QueueArgs Q = queue_args(P, W, kWantK);
  if (cudaMemsetAsync(W.counters, 0, W.counter_bytes, stream) != cudaSuccess) return PSX_ERR_CUDA;
  const size_t smem = sizeof(Tet10Smem<KT>) * (kThreads10 / 32);
  static unsigned long long s_smem_set = 0;
  if (set_dynamic_smem_once(tet10_persistent_kernel<KT, MODE>, (int)smem, &s_smem_set) != cudaSuccess)
    return PSX_ERR_CUDA;
  tet10_persistent_kernel<KT, MODE><<<W.grid, kThreads10, smem, stream>>>(A, g, Q, static_cast<KT*>(W.krec),
                                                                          W.frec, k_out, f_out);
  PSX_CUDA_CHECK_LAUNCH();
  return PSX_OK;
}

}  // namespace
}  // namespace psx

extern "C" int psx_tet10_assemble(const psx_plan_t* plan, const double* X, const double* u, const double* mu_e,
                                  const double* kappa_e, double mu, double kappa, double lam, int mode,
                                  int precision, double* f_out, void* k_out, void* work, int64_t work_bytes,
                                  void* status, void* stream) {
  using namespace psx;
  if (!plan || plan->npe != 10 || !X || !status || !work || plan->tile != kTile10) return PSX_ERR_ARG;
  const bool wantF = (mode & PSX_WANT_F) != 0, wantK = (mode & PSX_WANT_K) != 0,
             mass = (mode & PSX_MASS) != 0, linear = (mode & PSX_LINEAR) != 0 || mass;
  if (mode & ~(PSX_WANT_F | PSX_WANT_K | PSX_LINEAR | PSX_MASS)) return PSX_ERR_ARG;
  if ((mode & PSX_LINEAR) && mass) return PSX_ERR_ARG;
  if (linear && (wantF || wantK || !k_out)) return PSX_ERR_ARG;
  if (!linear && (!(wantF || wantK) || !u)) return PSX_ERR_ARG;
  if (wantF && !f_out) return PSX_ERR_ARG;
  if (wantK && !k_out) return PSX_ERR_ARG;
  WorkLayout W;
  int rc = work_layout(plan, precision, work, &W, 2, wantK || linear);
  if (rc != PSX_OK) return rc;
  if (work_bytes < W.total_bytes) return PSX_ERR_ARG;
  Tet10Args A{plan->conn, X, u, mu_e, kappa_e, mu, kappa, lam, static_cast<Status*>(status)};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define PSX_T10(KT, M) run_tet10<KT, M>(plan, A, W, static_cast<KT*>(k_out), f_out, s)
  if (mass) return precision == PSX_FP64 ? PSX_T10(double, PSX_MASS) : PSX_T10(float, PSX_MASS);
  if (linear) return precision == PSX_FP64 ? PSX_T10(double, PSX_LINEAR) : PSX_T10(float, PSX_LINEAR);
  if (wantF && wantK)
    return precision == PSX_FP64 ? PSX_T10(double, PSX_WANT_F | PSX_WANT_K)
                                 : PSX_T10(float, PSX_WANT_F | PSX_WANT_K);
  if (wantK) return precision == PSX_FP64 ? PSX_T10(double, PSX_WANT_K) : PSX_T10(float, PSX_WANT_K);
  return PSX_T10(double, PSX_WANT_F);
#undef PSX_T10
}

extern "C" int psx_tet10_element_dets(const int32_t* conn, const double* X, const double* u, int64_t e,
                                      double* out8, void* stream) {
  if (!conn || !X || !out8 || e < 0) return PSX_ERR_ARG;
  psx::tet10_dets_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(conn, X, u, e, out8);
  PSX_CUDA_CHECK_LAUNCH();
  return PSX_OK;
}
