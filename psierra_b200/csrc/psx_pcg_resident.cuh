// Preconditioned CG in one launch (included by psx_pcg.cu).
//
// Three launches per iteration leave a system of some 10^5 unknowns waiting: on 207,000
// unknowns (FP32 values, 36 MB, in L2) the iteration takes 44 us, of which the updates of
// 1.6 MB vectors are 22 and the launches and their drains most of the rest.  Here one
// block per SM runs the whole solve.  A block owns a range of nodes (or rows) and keeps their
// x, r, p, q and preconditioner in shared memory; only p goes to global memory, padded to 32
// bytes per node, for the neighbours' products.  The blocks meet three times per iteration:
// p is written / p.q / r.r and r.z.  At a meeting each block posts its partial sums, waits
// for everybody's and adds them in block order, so all blocks hold the same bits and the
// result is reproducible.
//   Blocks of one thread-block cluster (16, on small systems) meet by the cluster barrier
// and post into each other's shared memory; more blocks (a cooperative launch, so all are
// resident) count their arrivals in global memory.  Polls are bounded: a block that gives up
// ends without arriving again, so the others' next meeting gives up too, and block 0 sets status
// flag bit 0.
// Measured (block-Jacobi, FP32 values), us per iteration, three launches -> one:
//   2,187 unknowns 20 -> 5.5, 6,591 21.2 -> 8.5, 46,875 25.6 -> 9.8, 206,763 44.4 -> 18.5.
// What bounds it: small systems, the meetings; 207,000 unknowns, the product's loads.

// Threads of a block: 1,024 in the grid form (207,000 unknowns 18.5 us, 512 with two nodes of
// a group in flight 20.6), 512 in the cluster form, whose blocks hold few rows each (2,187
// unknowns 5.5 us against 6.4).
template <bool CLUSTER>
constexpr int res_threads() { return CLUSTER ? 512 : 1024; }
constexpr int kResLanes = 8;               // lanes per node / row of the product, as in spmv_node
// State of a block's own nodes.  With it the block takes up to 196 KB of the SM's memory (960 bytes
// of its own and 1 KB of the system's besides), which leaves the gathers of p 60 KB of L1.  The next
// carve-out, 228 KB, leaves 28, and the neighbours' p no longer stay: Kuhn cubes, block-Jacobi and
// nodal rows, us per iteration, one launch / three: 499,125 unknowns (193 KB) FP32 50 / 60, FP64
// 67 / 99; 526,848 (204 KB) 81 / 63 and 118 / 101.  Jacobi, rows: 714,984 (189 KB) FP64 114 / 127,
// 750,141 (198 KB) 197 / 135.
constexpr int kResSmem = 194 * 1024;
constexpr int kResClusterMax = 16;
// Rows up to which one cluster is faster than a block per SM: its meetings take a third of
// the time, its product runs on 16 SMs (us per iteration, cluster and grid: 2,187 rows 5.5 and
// 8.4, 6,591 rows 9.2 and 8.5, 17,496 rows 13.1 and 8.7).
constexpr int64_t kResClusterRows = 6144;
constexpr int32_t kResSpins = 1 << 21;     // default polls of one meeting: a second or two

// What the blocks of the grid form meet on: a count of arrivals, and the sums that each
// block posts before it arrives, in two sets in turn (a block can be one meeting ahead).
// One thread per block polls the one count: with a thread per posted epoch word (148 polling
// 148) a meeting took 6 us.
struct ResBoard {
  unsigned int arrived;
  unsigned int pad[7];
  double posted[2][256][3];
};
static_assert(sizeof(ResBoard) <= sizeof(double) * 3 * kGridMax, "the board fits the partial sums' place");

__device__ __forceinline__ void res_arrive(unsigned int* p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ unsigned int res_arrived(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <bool CLUSTER>
struct Meeting {
  ResBoard* board;              // grid form
  double (*all)[kResClusterMax][3];  // 2 x 16 x 3 in shared memory (cluster form)
  double (*warp)[3];            // 32 x 3: a block's warps
  double (*eight)[3];           // 8 x 3: the first warps' sums of what the blocks posted
  const int32_t& limit;         // polls of one meeting, in the kernel's parameters
  unsigned int epoch;

  // Every thread's v summed over all threads of all blocks; false when a wait gave up.
  template <int NV>
  __device__ __forceinline__ bool sum(double v[3]) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    ++epoch;
    const int set = (int)(epoch & 1);
    if constexpr (NV > 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const double t = warp_sum(v[i]);
        if (lane == 0) warp[w][i] = t;
      }
    }
    __syncthreads();  // also orders the block's own writes before its post
    double b[3] = {0.0, 0.0, 0.0};
    if (w == 0) {
#pragma unroll
      for (int i = 0; i < NV; ++i) b[i] = warp_sum(lane < res_threads<CLUSTER>() / 32 ? warp[lane][i] : 0.0);
    }
    if constexpr (CLUSTER) {
      if constexpr (NV > 0) {
        if (w == 0 && lane < (int)gridDim.x) {
          // lane = the block that receives this block's sums
          const unsigned mine = (unsigned)__cvta_generic_to_shared(&all[set][blockIdx.x][0]);
          unsigned there;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(mine), "r"(lane));
#pragma unroll
          for (int i = 0; i < NV; ++i)
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(there + 8 * i), "d"(b[i]) : "memory");
        }
      }
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      if constexpr (NV > 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          // a tree over the blocks (absent ones are zero)
          double t[kResClusterMax];
#pragma unroll
          for (int k = 0; k < kResClusterMax; ++k) t[k] = all[set][k][i];
#pragma unroll
          for (int o = kResClusterMax / 2; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < o; ++k) t[k] += t[k + o];
          v[i] = t[0];
        }
      }
      return true;
    } else {
      bool gave_up = false;
      if (tid == 0) {
        if constexpr (NV > 0) {
          double* mine = board->posted[set][blockIdx.x];
#pragma unroll
          for (int i = 0; i < NV; ++i) __stcg(mine + i, b[i]);
        }
        res_arrive(&board->arrived);
        const unsigned int want = epoch * gridDim.x;
        for (int32_t spins = 0; (int)(res_arrived(&board->arrived) - want) < 0;)
          if (++spins > limit) {
            gave_up = true;
            break;
          }
      }
      const bool ok = !__syncthreads_or(gave_up);
      if constexpr (NV > 0) {
        // at most 256 blocks: the first eight warps add what they posted
        if (w < 8) {
#pragma unroll
          for (int i = 0; i < NV; ++i) {
            const double x = warp_sum(tid < (int)gridDim.x ? __ldcg(&board->posted[set][tid][i]) : 0.0);
            if (lane == 0) eight[w][i] = x;
          }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          double t[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) t[k] = eight[k][i];
          v[i] = ((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]));
        }
      }
      return ok;
    }
  }
};

struct ResArgs {
  int64_t n;
  int64_t units;        // nodes, or rows
  int32_t per_block;    // units of one block
  const int32_t* indptr;
  const int32_t* indices;
  const void* vals;
  const double* b;
  double* x;
  double* p;            // 4 per node (NODAL), else n
  ResBoard* board;
  Status* st;
  double rtol, atol;
  int32_t maxiter, identity, spins;
};

// Matrix values and columns, each read once per product: not kept in L1, which is p's.
__device__ __forceinline__ float res_once(const float* p) {
  float v;
  asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double res_once(const double* p) {
  double v;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int32_t res_once(const int32_t* p) {
  int32_t v;
  asm("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// The arguments stay in the parameter space: with the poll limit in one of the grid form's 64
// registers an iteration of 206,763 unknowns takes 19.1 us, read from there 18.8 (18.7 with a
// constant limit).
template <typename VT, bool BLOCK, bool NODAL, bool CLUSTER>
__global__ void __launch_bounds__(res_threads<CLUSTER>(), 1) pcg_resident(const __grid_constant__ ResArgs A) {
  constexpr int kThreads = res_threads<CLUSTER>();
  constexpr bool kNode = BLOCK || NODAL;  // a unit is a node (three rows) or a row
  constexpr int kD = kNode ? 3 : 1;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double s_all[2][kResClusterMax][3], s_warp[32][3], s_eight[8][3];
  const int tid = threadIdx.x;
  const int cap = A.per_block;
  double* s_x = reinterpret_cast<double*>(smem);  // [component][unit]
  double* s_r = s_x + kD * cap;
  double* s_p = s_r + kD * cap;
  double* s_q = s_p + kD * cap;  // q, then z
  double* s_m = s_q + kD * cap;
  int32_t* s_row = reinterpret_cast<int32_t*>(s_m + (BLOCK ? 9 : kD) * cap);  // NODAL: first value and length of the node's first row
  const VT* vals = static_cast<const VT*>(A.vals);
  if constexpr (CLUSTER) {
    for (int k = tid; k < 2 * kResClusterMax * 3; k += kThreads) (&s_all[0][0][0])[k] = 0.0;  // absent blocks
  }
  const int64_t u0 = (int64_t)blockIdx.x * cap;
  const int own = (int)max((int64_t)0, min((int64_t)cap, A.units - u0));
  Meeting<CLUSTER> meet{A.board, s_all, s_warp, s_eight, A.spins, 0};

  // p of an own unit to global memory, where the neighbours read it
  auto publish = [&](int k, const double* from) {
    if constexpr (NODAL) {
      double* o = A.p + 4 * (u0 + k);
      *reinterpret_cast<double2*>(o) = make_double2(from[k], from[cap + k]);
      o[2] = from[2 * cap + k];
    } else {
#pragma unroll
      for (int d = 0; d < kD; ++d) A.p[kD * (u0 + k) + d] = from[d * cap + k];
    }
  };
  // q = A p over the own rows
  auto product = [&]() {
    const int lane = tid & (kResLanes - 1), group = tid / kResLanes;
    constexpr int kGroups = kThreads / kResLanes;
    if constexpr (NODAL) {
      for (int k0 = 0; k0 < own; k0 += kGroups) {
        const int k = k0 + group;
        const int r0 = k < own ? s_row[2 * k] : 0, len = k < own ? s_row[2 * k + 1] : 0;
        double a[3] = {0.0, 0.0, 0.0};
        for (int b3 = 3 * lane; b3 < len; b3 += 3 * kResLanes) {
          const int32_t c = res_once(A.indices + r0 + b3);
          const VT* q = vals + r0 + b3;
          VT v[9];
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            v[m] = res_once(q + m);
            v[3 + m] = res_once(q + len + m);
            v[6 + m] = res_once(q + 2 * len + m);
          }
          // a plain (L1) load: the meeting before the product acquires the other blocks'
          // writes, and a node's p is read by its neighbours in this block as well
          const Quad x = ld_quad(A.p + 4 * (int64_t)(c / 3));
#pragma unroll
          for (int m = 0; m < 3; ++m)
            a[m] += (double)v[3 * m] * x.x + (double)v[3 * m + 1] * x.y + (double)v[3 * m + 2] * x.z;
        }
#pragma unroll
        for (int m = 0; m < 3; ++m) {
#pragma unroll
          for (int o = kResLanes / 2; o > 0; o >>= 1) a[m] += __shfl_xor_sync(0xffffffffu, a[m], o);
          if (lane == 0 && k < own) s_q[m * cap + k] = a[m];
        }
      }
    } else {
      for (int k0 = 0; k0 < kD * own; k0 += kGroups) {
        const int k = k0 + group;  // own row
        double a = 0.0;
        if (k < kD * own) {
          const int64_t row = kD * u0 + k;
          const int32_t j1 = __ldg(A.indptr + row + 1);
          for (int32_t j = __ldg(A.indptr + row) + lane; j < j1; j += kResLanes) {
            double x;
            asm volatile("ld.global.f64 %0, [%1];" : "=d"(x) : "l"(A.p + res_once(A.indices + j)));
            a += (double)res_once(vals + j) * x;
          }
        }
#pragma unroll
        for (int o = kResLanes / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0 && k < kD * own) s_q[(k % kD) * cap + k / kD] = a;
      }
    }
  };
  auto precond = [&](int k, const double r[3], double z[3]) {
    if constexpr (BLOCK) {
#pragma unroll
      for (int d = 0; d < 3; ++d)
        z[d] = s_m[(3 * d) * cap + k] * r[0] + s_m[(3 * d + 1) * cap + k] * r[1] + s_m[(3 * d + 2) * cap + k] * r[2];
    } else {
#pragma unroll
      for (int d = 0; d < kD; ++d) z[d] = s_m[d * cap + k] * r[d];
    }
  };

  // ---- setup: preconditioner, x, r = b - A x, z
  for (int k = tid; k < own; k += kThreads) {
    const int64_t u = u0 + k;
    if constexpr (NODAL) {
      s_row[2 * k] = __ldg(A.indptr + 3 * u);
      s_row[2 * k + 1] = __ldg(A.indptr + 3 * u + 1) - s_row[2 * k];
    }
    if constexpr (BLOCK) {
      double B[3][3], Bi[3][3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) B[i][j] = csr_at(A.indptr, A.indices, A.vals, sizeof(VT) == 4, 3 * u + i, 3 * u + j);
      const double det = inv3(B, Bi);
      const bool ok = fabs(det) > 1e-300 && isfinite(det);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) s_m[(3 * i + j) * cap + k] = ok ? Bi[i][j] : (i == j ? 1.0 : 0.0);
    } else {
#pragma unroll
      for (int d = 0; d < kD; ++d) {
        const double v = A.identity ? 0.0 : csr_at(A.indptr, A.indices, A.vals, sizeof(VT) == 4, kD * u + d, kD * u + d);
        s_m[d * cap + k] = fabs(v) > 1e-14 ? 1.0 / v : 1.0;
      }
    }
#pragma unroll
    for (int d = 0; d < kD; ++d) s_x[d * cap + k] = A.x[kD * u + d];
    publish(k, s_x);
  }
  double v[3] = {0.0, 0.0, 0.0};
  auto report = [&](int32_t iters, int32_t flags, double rr) {
    if (blockIdx.x == 0 && tid == 0) {
      A.st->iters = iters;
      A.st->flags = flags;
      A.st->value = sqrt(rr);
    }
  };
  if (!meet.template sum<0>(v)) {
    report(0, 1, 0.0);
    return;
  }
  product();
  __syncthreads();
  v[0] = v[1] = v[2] = 0.0;
  for (int k = tid; k < own; k += kThreads) {
    double r[3], z[3];
#pragma unroll
    for (int d = 0; d < kD; ++d) {
      const double bd = A.b[kD * (u0 + k) + d];
      r[d] = bd - s_q[d * cap + k];
      s_r[d * cap + k] = r[d];
      v[2] += bd * bd;
    }
    precond(k, r, z);
#pragma unroll
    for (int d = 0; d < kD; ++d) {
      s_q[d * cap + k] = z[d];
      v[0] += r[d] * r[d];
      v[1] += r[d] * z[d];
    }
  }
  bool ok = meet.template sum<3>(v);
  double rr = v[0], rho = v[1], rho_prev = 0.0;
  const double tol = fmax(A.atol, A.rtol * sqrt(v[2])), tol2 = tol * tol;
  bool converged = v[2] == 0.0 || sqrt(rr) < tol;
  int32_t iters = 0, breakdown = 0;

  for (int32_t it = 0; it < A.maxiter && ok && !converged && !breakdown; ++it) {
    const double beta = iters == 0 ? 0.0 : rho / rho_prev;
    for (int k = tid; k < own; k += kThreads) {
#pragma unroll
      for (int d = 0; d < kD; ++d) {
        const double z = s_q[d * cap + k];
        s_p[d * cap + k] = iters == 0 ? z : z + beta * s_p[d * cap + k];
      }
      publish(k, s_p);
    }
    ok = meet.template sum<0>(v);
    if (!ok) break;
    product();
    __syncthreads();
    v[0] = 0.0;
    for (int k = tid; k < own; k += kThreads)
#pragma unroll
      for (int d = 0; d < kD; ++d) v[0] += s_p[d * cap + k] * s_q[d * cap + k];
    ok = meet.template sum<1>(v);
    if (!ok) break;
    if (!(v[0] != 0.0) || !isfinite(v[0])) {
      breakdown = 1;
      break;
    }
    const double alpha = rho / v[0];
    v[0] = v[1] = 0.0;
    for (int k = tid; k < own; k += kThreads) {
      double r[3], z[3];
#pragma unroll
      for (int d = 0; d < kD; ++d) {
        s_x[d * cap + k] += alpha * s_p[d * cap + k];
        r[d] = s_r[d * cap + k] - alpha * s_q[d * cap + k];
        s_r[d * cap + k] = r[d];
      }
      precond(k, r, z);
#pragma unroll
      for (int d = 0; d < kD; ++d) {
        s_q[d * cap + k] = z[d];
        v[0] += r[d] * r[d];
        v[1] += r[d] * z[d];
      }
    }
    ok = meet.template sum<2>(v);
    if (!ok) break;
    rho_prev = rho;
    rr = v[0];
    rho = v[1];
    ++iters;
    // scipy checks the residual at the top of each of its maxiter iterations, so a
    // residual reached by the last allowed update still reports non-convergence
    if (!isfinite(rr)) breakdown = 1;
    else if (iters >= A.maxiter) breakdown = 2;
    else if (rr < tol2) converged = true;
  }
  for (int k = tid; k < own; k += kThreads)
#pragma unroll
    for (int d = 0; d < kD; ++d) A.x[kD * (u0 + k) + d] = s_x[d * cap + k];
  report(iters, !ok ? 1 : converged ? 0 : breakdown == 2 ? 2 : 4, rr);
}

// Units per block and blocks of a system, or 0 when its state does not fit the GPU's shared
// memory.
struct ResShape {
  int blocks = 0, per_block = 0;
  size_t smem = 0;
};
inline ResShape res_shape(int64_t units, int doubles_per_unit, int blocks) {
  ResShape s;
  const int64_t per = (units + blocks - 1) / blocks;
  const int64_t bytes = per * 8 * doubles_per_unit;
  if (bytes > kResSmem) return s;
  s.per_block = (int)per;
  s.blocks = (int)((units + per - 1) / per);
  s.smem = (size_t)bytes;
  return s;
}

inline void res_cluster_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int blocks, size_t smem, cudaStream_t s) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = blocks;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg->gridDim = dim3(blocks);
  cfg->blockDim = dim3(res_threads<true>());
  cfg->dynamicSmemBytes = smem;
  cfg->stream = s;
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

// Blocks of the cluster form on this device: 16 where such a cluster fits with a block's whole
// shared memory, else 8, else 0; -1 on a CUDA error.  Asked once per kernel and device: the
// kernels differ in registers but not in type, so each caller keeps its own answers (1 + blocks,
// 0 = not asked).
template <typename K>
inline int res_cluster_blocks(K* kernel, int dev, int answers[64]) {
  int* answer = answers + (dev & 63);
  const int known = __atomic_load_n(answer, __ATOMIC_ACQUIRE);
  if (known) return known - 1;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem) != cudaSuccess)
    return -1;
  int found = 0;
  for (int blocks = kResClusterMax; blocks >= 8 && !found; blocks /= 2) {
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg{};
    res_cluster_config(&cfg, at, blocks, kResSmem, nullptr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) cudaGetLastError();
    else if (clusters > 0) found = blocks;
  }
  __atomic_store_n(answer, 1 + found, __ATOMIC_RELEASE);
  return found;
}

// 1: solved here; 0: not this system (too large, or the launch is refused, as a cooperative one is
// where the process has a part of the SMs); -1: a CUDA error.  A refusal's error is cleared and the
// next form tried; an error of earlier work stays, and the next form's own checks report it.
template <typename VT, bool BLOCK, bool NODAL>
int run_pcg_resident(int64_t n, const int32_t* indptr, const int32_t* indices, const VT* vals, const double* b, double* x,
                     double rtol, double atol, int32_t maxiter, const PcgWork& w, Status* st, cudaStream_t s,
                     int identity, int32_t spins) {
  constexpr bool kNode = BLOCK || NODAL;
  constexpr int kD = kNode ? 3 : 1, kDoubles = 4 * kD + (BLOCK ? 9 : kD) + (NODAL ? 1 : 0);
  const int64_t units = n / kD;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return -1;
  if (sms > 256) sms = 256;
  ResArgs A{n, units, 0, indptr, indices, vals, b, x, w.z, reinterpret_cast<ResBoard*>(w.partial), st, rtol, atol, maxiter,
            identity, spins > 0 ? spins : kResSpins};
  // one cluster on small systems, else one block per SM
  static unsigned long long s_grid = 0;
  static int s_cluster[64];
  const int64_t rows = units * kD;
  if (rows <= kResClusterRows) {
    auto* kernel = pcg_resident<VT, BLOCK, NODAL, true>;
    const int blocks = res_cluster_blocks(kernel, dev, s_cluster);
    const ResShape c = res_shape(units, kDoubles, blocks > 0 ? blocks : 1);
    if (blocks > 0 && c.per_block > 0) {
      A.per_block = c.per_block;
      cudaLaunchAttribute at[1];
      cudaLaunchConfig_t cfg{};
      res_cluster_config(&cfg, at, blocks, c.smem, s);
      if (cudaLaunchKernelEx(&cfg, kernel, A) == cudaSuccess) return 1;
    }
    if (blocks != 0) cudaGetLastError();
  }
  const ResShape g = res_shape(units, kDoubles, sms);
  if (g.blocks <= 0) return 0;
  auto* kernel = pcg_resident<VT, BLOCK, NODAL, false>;
  A.per_block = g.per_block;
  void* args[] = {&A};
  if (cudaMemsetAsync(A.board, 0, sizeof(unsigned int), s) != cudaSuccess) return -1;
  if (set_dynamic_smem_once(kernel, kResSmem, &s_grid) == cudaSuccess &&
      cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(g.blocks), dim3(res_threads<false>()), args, g.smem,
                                  s) == cudaSuccess)
    return 1;
  cudaGetLastError();
  return 0;
}
