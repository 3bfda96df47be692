// Hyper-reduced (ECSW) Tet4 evaluation for sm_100a.
//
// Restates HyperReducedECSWModel.evaluate_forces_and_stiffness (psierra
// hyperreduction/model.py:254-318): on the reduced integration domain (p elements with
// cubature weights w_e and modal sub-bases Phi_e, 12 x r),
//   u_e = Phi_e u_r,  f_r = sum_e w_e Phi_e^T f_e(u_e),  K_r = sum_e w_e Phi_e^T k_e(u_e) Phi_e,
//   K_r <- (K_r + K_r^T) / 2.
// Three launches:
//   ecsw_elements  one warp per element: u_e, the NeoHookean point, and the columns of
//                  T_e = w_e [k_e Phi_e | f_e], lane by lane through the matrix-free product
//                  k_e v of the assembly kernels (about 150 multiply-adds a column, where
//                  forming k_e and multiplying takes 144 and the 12 x 12 matrix);
//   ecsw_gemm      Phi^T T over all 12 n rows, split over the rows: one block per 32 x 32
//                  tile of the result and run of elements, partial sums to the workspace;
//   ecsw_sum       the partial sums of every entry in a fixed order, and the symmetrisation.
// Every sum has a fixed order.  1,500 elements and 30 modes: 60 us a call, 20 of them in the
// kernels; what bounds it is the host's part and three launches.  One thread per entry of K_r
// over all elements takes 5.2 ms there: a serial chain of 36,000 multiply-adds on a few warps.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "psx_common.cuh"
#include "psx_tet4_math.cuh"

namespace psx {
namespace {

constexpr int kEcThreads = 128;
constexpr int kEcTile = 32;   // result tile of one block of ecsw_gemm
constexpr int kEcStep = 24;   // rows (two elements) staged at a time

__global__ void __launch_bounds__(kEcThreads) ecsw_elements(int64_t n, int32_t r, const double* __restrict__ Xe,
                                                            const double* __restrict__ phi,
                                                            const double* __restrict__ w,
                                                            const double* __restrict__ ur,
                                                            const double* __restrict__ mu_e,
                                                            const double* __restrict__ kappa_e, double mu0,
                                                            double kappa0, double* __restrict__ T, Status* st) {
  const int lane = threadIdx.x & 31;
  const int64_t e = blockIdx.x * (int64_t)(kEcThreads / 32) + (threadIdx.x >> 5);
  if (e >= n) return;
  const double* P = phi + (int64_t)12 * r * e;  // row-major 12 x r
  double u[12];
#pragma unroll
  for (int d = 0; d < 12; ++d) u[d] = 0.0;
  for (int j = lane; j < r; j += 32) {
    const double c = __ldg(ur + j);
#pragma unroll
    for (int d = 0; d < 12; ++d) u[d] += __ldg(P + d * r + j) * c;
  }
  double Xn[4][3], Un[4][3];
#pragma unroll
  for (int d = 0; d < 12; ++d) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) u[d] += __shfl_xor_sync(0xffffffffu, u[d], o);
    Un[d / 3][d % 3] = u[d];
    Xn[d / 3][d % 3] = __ldg(Xe + 12 * e + d);
  }
  Tet4Geom G;
  tet4_geometry(Xn, G);
  if (!(G.detD > 0.0) && lane == 0) flag_bad_element(st, e, true);
  double l[3][3];
  tet4_grad(Un, G, l);
  PointState ps;
  const double mu = mu_e ? mu_e[e] : mu0, kappa = kappa_e ? kappa_e[e] : kappa0;
  neohookean_point(l, mu, kappa, ps);
  if (G.detD > 0.0 && ps.Jm1 <= -1.0 && lane == 0) flag_bad_element(st, e, false);
  const double we = w[e];
  const TangentCoef<double> tc = tangent_coef<double>(ps, kappa, G.V);
  double p[4][3], q[4][3];
  tet4_pq<double>(ps, G.g, p, q);
  double* Te = T + (int64_t)12 * (r + 1) * e;  // row-major 12 x (r + 1), f_e last
  for (int j = lane; j <= r; j += 32) {
    double y[12];
    if (j < r) {
      double v[4][3];
#pragma unroll
      for (int d = 0; d < 12; ++d) v[d / 3][d % 3] = __ldg(P + d * r + j);
      Tet4Sums<double> S;
      tet4_sums<double>(tc, p, q, G.g, v, S);
      tet4_product<double>(tc, p, q, G.g, S, y);
    } else {
      tet4_force(ps, G, y);
    }
#pragma unroll
    for (int d = 0; d < 12; ++d) Te[d * (r + 1) + j] = we * y[d];
  }
}

// part[s] (r x (r + 1)) = Phi^T T over the rows of run s
__global__ void __launch_bounds__(kEcThreads) ecsw_gemm(int64_t n, int32_t r, int32_t runs, const double* __restrict__ phi,
                                                        const double* __restrict__ T, double* __restrict__ part) {
  __shared__ double sa[kEcStep][kEcTile], sb[kEcStep][kEcTile];
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;  // outputs 2 x 4 per thread
  const int i0 = blockIdx.x * kEcTile, j0 = blockIdx.y * kEcTile, run = blockIdx.z;
  const int64_t row0 = 12 * (n * run / runs), row1 = 12 * (n * (run + 1) / runs);
  double acc[2][4];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
  for (int64_t k0 = row0; k0 < row1; k0 += kEcStep) {
#pragma unroll
    for (int c = 0; c < kEcStep * kEcTile / kEcThreads; ++c) {
      const int k = (c * kEcThreads + tid) / kEcTile, m = tid % kEcTile;
      const bool in = k0 + k < row1;
      sa[k][m] = in && i0 + m < r ? __ldg(phi + (k0 + k) * r + i0 + m) : 0.0;
      sb[k][m] = in && j0 + m <= r ? __ldg(T + (k0 + k) * (r + 1) + j0 + m) : 0.0;
    }
    __syncthreads();
#pragma unroll 6
    for (int k = 0; k < kEcStep; ++k) {
      const double a0 = sa[k][ty], a1 = sa[k][ty + 16];
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const double v = sb[k][tx + 8 * b];
        acc[0][b] += a0 * v;
        acc[1][b] += a1 * v;
      }
    }
    __syncthreads();
  }
  double* out = part + (int64_t)run * r * (r + 1);
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = i0 + ty + 16 * a, j = j0 + tx + 8 * b;
      if (i < r && j <= r) out[(int64_t)i * (r + 1) + j] = acc[a][b];
    }
}

// Entries of K_r and f_r from the partial sums: 16 threads per 8 entries of consecutive
// columns, each a fixed share of the runs, their shares added in order.
constexpr int kEcShares = 16;
__global__ void __launch_bounds__(kEcThreads) ecsw_sum(int32_t r, int32_t runs, const double* __restrict__ part,
                                                       double* __restrict__ f_r, double* __restrict__ K_r) {
  __shared__ double s[2][kEcShares][kEcThreads / kEcShares];
  constexpr int kPer = kEcThreads / kEcShares;
  const int tid = threadIdx.x, col = tid % kPer, share = tid / kPer;
  const int64_t size = (int64_t)r * (r + 1), t = blockIdx.x * (int64_t)kPer + col;
  const int i = (int)(t / (r + 1)), j = (int)(t % (r + 1));
  double x = 0.0, y = 0.0;
  if (t < size) {
    const int s0 = runs * share / kEcShares, s1 = runs * (share + 1) / kEcShares;
    const double* p = part + t;
    const double* q = part + (j < r ? (int64_t)j * (r + 1) + i : t);  // the transposed entry
#pragma unroll 4
    for (int k = s0; k < s1; ++k) {
      x += __ldg(p + k * size);
      y += __ldg(q + k * size);
    }
  }
  s[0][share][col] = x;
  s[1][share][col] = y;
  __syncthreads();
  if (share != 0 || t >= size) return;
  double a = 0.0, b = 0.0;
#pragma unroll
  for (int k = 0; k < kEcShares; ++k) {
    a += s[0][k][col];
    b += s[1][k][col];
  }
  if (j < r)
    K_r[(int64_t)i * r + j] = 0.5 * (a + b);
  else
    f_r[i] = a;
}

// Runs of elements whose partial sums are kept apart: a few elements each, and about four
// blocks per SM over the tiles of the result (1,500 elements, 30 modes: 375 runs of 4).
inline int32_t ec_runs(int64_t n, int32_t r) {
  const int64_t tiles = (int64_t)((r + kEcTile - 1) / kEcTile) * ((r + kEcTile) / kEcTile);
  return (int32_t)std::max<int64_t>(1, std::min<int64_t>((n + 3) / 4, 592 / tiles));
}

}  // namespace
}  // namespace psx

extern "C" int64_t psx_ecsw_work_doubles(int64_t n, int32_t r) {
  return n <= 0 || r <= 0 ? 0 : (int64_t)12 * (r + 1) * n + psx::ec_runs(n, r) * (int64_t)r * (r + 1);
}

extern "C" int psx_ecsw_evaluate(int64_t n, int32_t r, const double* X_elem, const double* phi_elem,
                                 const double* weights, const double* u_r, const double* mu_e, const double* kappa_e,
                                 double mu, double kappa, double* f_r, double* K_r, double* work,
                                 int64_t work_doubles, void* status, void* stream) {
  using namespace psx;
  if (n <= 0 || r <= 0 || !X_elem || !phi_elem || !weights || !u_r || !f_r || !K_r || !work || !status)
    return PSX_ERR_ARG;
  if ((mu_e == nullptr) != (kappa_e == nullptr)) return PSX_ERR_ARG;
  if (work_doubles < psx_ecsw_work_doubles(n, r)) return PSX_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if ((n + 3) / 4 > 0x7fffffff || (r + kEcTile) / kEcTile > 0xffff) return PSX_ERR_LIMIT;
  double* T = work;
  double* part = work + (int64_t)12 * (r + 1) * n;
  const int32_t runs = ec_runs(n, r);
  constexpr int kWarps = kEcThreads / 32, kPer = kEcThreads / kEcShares;
  ecsw_elements<<<(unsigned)((n + kWarps - 1) / kWarps), kEcThreads, 0, s>>>(
      n, r, X_elem, phi_elem, weights, u_r, mu_e, kappa_e, mu, kappa, T, static_cast<Status*>(status));
  ecsw_gemm<<<dim3((r + kEcTile - 1) / kEcTile, (r + kEcTile) / kEcTile, runs), kEcThreads, 0, s>>>(n, r, runs, phi_elem,
                                                                                               T, part);
  ecsw_sum<<<(unsigned)(((int64_t)r * (r + 1) + kPer - 1) / kPer), kEcThreads, 0, s>>>(r, runs, part, f_r, K_r);
  PSX_CUDA_CHECK_LAUNCH();
  return PSX_OK;
}
