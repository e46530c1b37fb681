// Jacobi-PCG of a small system on one thread-block cluster.
//
// A k_pcg iteration takes 8.8 us from 1000 rows to 85 000: latency, in two grid-wide all-reduces
// through an atomic counter in L2 and three dependent rounds of L2 loads (columns, the gathered
// vectors, the partials).  Up to PCG_CL_MAX_ROWS rows, this kernel runs the same iteration on one
// cluster of up to 16 blocks: the search direction and the operator stay in shared memory,
// neighbours' rows are read over distributed shared memory, and an iteration's three waits are
// hardware cluster barriers.  The recurrences, the null-space handling and the stopping rule are
// those of k_pcg (src/solver/pressure_backend_petsc.c:816-876); only the order of the sums over
// blocks differs.  The direction p is published before the product (one more barrier than k_pcg,
// which forms its neighbours' p from z and the old p): half the bytes gathered from shared memory,
// which bound the kernel at 2000 rows per block and more.  Microseconds per iteration, here and
// k_pcg: 1000 rows 3.5 / 9.4, 9216 rows 4.0 / 8.9, 32 768 rows 4.9 / 8.8, 35 937 rows 5.7 / 8.9;
// beyond 40 960 rows more of the operator than its last slot would have to come from L2 (44 880 rows
// 8.2 / 8.8, 50 400 rows 10.6 / 8.8).
//
// Its waits need no poll limit: the blocks of a cluster are scheduled together, and every thread
// reaches every barrier.  Scheduled together does not mean started: a block's shared memory may be
// accessed only once that block runs, so each block arrives at a cluster barrier on entry and waits
// there after staging its operator, before the first store to another block.
#pragma once
#include <algorithm>

#include "pcg.cuh"

namespace dpm {
namespace gpu {

constexpr int PCG_CL_BLOCKS = 16;
constexpr int PCG_CL_TPB = 512;  // s_w below holds 16 warps
constexpr int PCG_CL_CPT = 5;
constexpr int PCG_CL_MAX_ROWS = PCG_CL_BLOCKS * PCG_CL_TPB * PCG_CL_CPT;

__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cl_map(unsigned addr, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ double cl_ld(unsigned addr) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cl_st(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_barrier() {
  cl_arrive();
  cl_wait();
}

// Sums over a warp of four values at once: two exchange steps leave each lane one value's partial
// sum, three more add it over the eight lanes that hold it.  Lane l returns the sum of value l >> 3
// (6 double shuffles instead of 20: with 32 warps, the shuffles are a good part of an all-reduce).
__device__ __forceinline__ double warp_sum4(double v0, double v1, double v2, double v3) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, q = lane & 8;
  const double a0 = __shfl_xor_sync(0xffffffffu, h ? v0 : v2, 16);
  const double a1 = __shfl_xor_sync(0xffffffffu, h ? v1 : v3, 16);
  const double k0 = (h ? v2 : v0) + a0, k1 = (h ? v3 : v1) + a1;
  double t = (q ? k1 : k0) + __shfl_xor_sync(0xffffffffu, q ? k0 : k1, 8);
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// Sum of four values over the cluster, the same bits in every thread: warps, then the block's warps
// and after the barrier the blocks, each by one warp in a fixed order.  Two buffers alternate.
__device__ __forceinline__ void cl_allreduce(const double (&v)[4], double (&res)[4], unsigned rank, unsigned nblk,
                                             unsigned& gen) {
  __shared__ double s_w[PCG_CL_TPB / 32][4];
  __shared__ double s_part[2][PCG_CL_BLOCKS][4];
  __shared__ double s_res[4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, k = lane >> 3, j = lane & 7;
  double(*part)[4] = s_part[gen & 1u];
  {
    const double t = warp_sum4(v[0], v[1], v[2], v[3]);
    if (j == 0) s_w[w][k] = t;
  }
  __syncthreads();
  if (w == 0) {
    double t = s_w[j][k] + s_w[j + 8][k];
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    const unsigned at = (unsigned)__cvta_generic_to_shared(&part[rank][k]);
    if (j < (int)nblk) cl_st(cl_map(at, j), t);
    if (j + 8 < (int)nblk) cl_st(cl_map(at, j + 8), t);
  }
  cl_barrier();
  if (w == 0) {
    double t = j < (int)nblk ? part[j][k] : 0.0;
    if (j + 8 < (int)nblk) t += part[j + 8][k];
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (j == 0) s_res[k] = t;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) res[q] = s_res[q];
  ++gen;
}

// Block `rank` owns rows [rank C, rank C + size).  CPT: rows per thread; WT: row width (7 on
// hexahedral meshes, 0: runtime width <= 16); WS: slots of the operator kept in shared memory.
template <int CPT, int WT>
__global__ void __launch_bounds__(PCG_CL_TPB, 1) k_pcg_cluster(PcgArgs<double> a, int C, int WS) {
  extern __shared__ double cl_smem[];
  cl_arrive();                            // this block runs; cl_wait below: all blocks do
  constexpr int CH = WT > 0 ? WT : 4;     // slots whose loads are in flight together
  const int n = a.n, WA = WT > 0 ? WT : a.WA;
  const unsigned rank = cl_rank(), nblk = gridDim.x;
  const int base = (int)rank * C, size = max(0, min(C, n - base));
  const unsigned magic = 0xffffffffu / (unsigned)C + 1u;  // row / C by high product, exact for rows < 2^17
  double* s_p = cl_smem;                                  // [C]
  double* s_val = s_p + C;                                // [WS][C]
  unsigned* s_adr = reinterpret_cast<unsigned*>(s_val + (size_t)WS * C);  // [WS][C] address of the entry's p
  const unsigned p0 = (unsigned)__cvta_generic_to_shared(s_p);
  unsigned gen = 0;
  auto address = [&](int c) {
    const unsigned r = C > 1 ? __umulhi((unsigned)c, magic) : (unsigned)c;
    const unsigned at = p0 + 8u * ((unsigned)c - r * (unsigned)C);
    return r == rank ? at : cl_map(at, r);
  };
  // row l (of this block) of A times the published vector
  auto product = [&](int l) {
    const int i = base + l;
    double s = 0.0;
    for (int w0 = 0; w0 < WA; w0 += CH) {
      unsigned ad[CH];
      double v[CH], x[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int w = w0 + u;
        if (WT > 0 || w < WA) {
          if (w < WS) {
            ad[u] = s_adr[w * C + l];
            v[u] = s_val[w * C + l];
          } else {
            ad[u] = address(__ldg(&a.col[(size_t)w * n + i]));
            v[u] = __ldg(&a.val[(size_t)w * n + i]);
          }
        } else {
          ad[u] = p0 + 8u * l;
          v[u] = 0.0;
        }
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) x[u] = cl_ld(ad[u]);
#pragma unroll
      for (int u = 0; u < CH; ++u) s += v[u] * x[u];
    }
    return s;
  };
#define CL_OWN(k) (threadIdx.x + (k) * PCG_CL_TPB < size)
#define CL_ROW(k) ((int)threadIdx.x + (k) * PCG_CL_TPB)
  for (int w = 0; w < WS; ++w)
    for (int l = threadIdx.x; l < size; l += PCG_CL_TPB) {
      s_adr[w * C + l] = address(__ldg(&a.col[(size_t)w * n + base + l]));
      s_val[w * C + l] = __ldg(&a.val[(size_t)w * n + base + l]);
    }
  cl_wait();
  double rx[CPT], rr[CPT], rp[CPT], rq[CPT], rd[CPT];
  // ---- b' = b - mean(b) when the constant null space is active; x published
  double mb = 0.0;
  {
    double v[4] = {0, 0, 0, 0}, t[4];
#pragma unroll
    for (int k = 0; k < CPT; ++k)
      if (CL_OWN(k)) {
        const int i = base + CL_ROW(k);
        const double x0 = a.guess_zero ? 0.0 : a.x[i];
        rr[k] = a.b[i];
        rp[k] = 0.0;
        rx[k] = x0;
        rd[k] = __ldg(&a.dinv[i]);
        s_p[CL_ROW(k)] = x0;
        v[0] += rr[k];
      }
    cl_allreduce(v, t, rank, nblk, gen);
    mb = a.nullsp ? t[0] / (double)n : 0.0;
  }
  // ---- r = b' - A x
  double v2[4] = {0, 0, 0, 0}, t2[4];
#pragma unroll
  for (int k = 0; k < CPT; ++k)
    if (CL_OWN(k)) {
      const double bp = a.nullsp ? rr[k] - mb : rr[k];
      rr[k] = bp - product(CL_ROW(k));
      v2[0] += rr[k] * rr[k];
      v2[1] += bp * bp;
    }
  cl_allreduce(v2, t2, rank, nblk, gen);
  double dp = sqrt(t2[0]);
  const double sn = sqrt(t2[1]);
  const double rnorm0 = a.guess_zero ? dp : (sn == 0.0 ? dp : sn);
  const double ttol = fmax(a.rtol * rnorm0, a.atol);
  int reason = classify(dp, ttol, a.atol, rnorm0);
  int its = 0;
  if (!reason) {
    double v4[4] = {0, 0, 0, 0}, t4[4];
#pragma unroll
    for (int k = 0; k < CPT; ++k)
      if (CL_OWN(k)) {
        const double z = rr[k] * rd[k];
        v4[0] += z; v4[1] += rr[k]; v4[2] += z * rr[k];
      }
    cl_allreduce(v4, t4, rank, nblk, gen);
    double mz = a.nullsp ? t4[0] / (double)n : 0.0;
    double beta = a.nullsp ? t4[2] - mz * t4[1] : t4[2];
    double betaold = 0.0, dpi = 0.0, dpiold = 0.0, bb = 0.0;
    int it = 0;
    const double rn = 1.0 / (double)n;
    do {
      its = it + 1;
      if (beta == 0.0) { reason = 3; break; }
      if (it > 0 && beta * betaold < 0.0) { reason = -8; break; }
      // ---- p, q = A p, p.q
#pragma unroll
      for (int k = 0; k < CPT; ++k)
        if (CL_OWN(k)) {
          double p = rr[k] * rd[k] - mz;
          if (it > 0) p = p + bb * rp[k];
          rp[k] = p;
          s_p[CL_ROW(k)] = p;
        }
      cl_barrier();
      double v1[4] = {0, 0, 0, 0}, t1[4];
#pragma unroll
      for (int k = 0; k < CPT; ++k)
        if (CL_OWN(k)) {
          rq[k] = product(CL_ROW(k));
          v1[0] += rp[k] * rq[k];
        }
      cl_allreduce(v1, t1, rank, nblk, gen);
      dpiold = dpi;
      dpi = t1[0];
      betaold = beta;
      if (dpi == 0.0 || (it > 0 && ((dpi > 0) - (dpi < 0)) * ((dpiold > 0) - (dpiold < 0)) < 0)) {
        reason = dpi == 0.0 ? 3 : -10;
        break;
      }
      const double al = beta / dpi;
      // ---- x, r, z and the four sums
      double w4[4] = {0, 0, 0, 0}, s4[4];
#pragma unroll
      for (int k = 0; k < CPT; ++k)
        if (CL_OWN(k)) {
          rx[k] += al * rp[k];
          rr[k] = rr[k] - al * rq[k];
          const double z = rr[k] * rd[k];
          w4[0] += rr[k] * rr[k]; w4[1] += z; w4[2] += rr[k]; w4[3] += z * rr[k];
        }
      cl_allreduce(w4, s4, rank, nblk, gen);
      // the root of the stopping test and the quotient of the next direction side by side
      dp = sqrt(s4[0]);
      mz = a.nullsp ? s4[1] * rn : 0.0;
      beta = a.nullsp ? s4[3] - mz * s4[2] : s4[3];
      bb = beta / betaold;
      reason = classify(dp, ttol, a.atol, rnorm0);
      if (reason) break;
      it++;
    } while (it < a.maxit);
    if (!reason && it >= a.maxit) reason = -3;
  }
  // ---- x, then the true residual ||b - A x|| with the caller's b (every product of the loop was
  // followed by a barrier, so the published vector may be overwritten)
#pragma unroll
  for (int k = 0; k < CPT; ++k)
    if (CL_OWN(k)) {
      a.x[base + CL_ROW(k)] = rx[k];
      s_p[CL_ROW(k)] = rx[k];
    }
  cl_barrier();
  double v1[4] = {0, 0, 0, 0}, t1[4];
#pragma unroll
  for (int k = 0; k < CPT; ++k)
    if (CL_OWN(k)) {
      const double d = a.b[base + CL_ROW(k)] - product(CL_ROW(k));
      v1[0] += d * d;
    }
  cl_allreduce(v1, t1, rank, nblk, gen);  // also keeps every block's shared memory until all have read it
  if (rank == 0 && threadIdx.x == 0) {
    a.dout[0] = sqrt(t1[0]);
    a.dout[1] = dp;
    a.dout[2] = sn;
    a.status[0] = reason;
    a.status[1] = its;
  }
#undef CL_OWN
#undef CL_ROW
}

// The cluster kernel for a system: its instantiation, blocks, rows per block, staged slots and shared
// memory; kernel null when the system is too large or the device cannot hold such a cluster.
struct PcgCluster {
  void* kernel = nullptr;
  int blocks = 0, C = 0, WS = 0;
  size_t smem = 0;

  template <int CPT>
  static void* pick_cpt(int cpt, int width) {
    if constexpr (CPT < PCG_CL_CPT)
      if (cpt > CPT) return pick_cpt<CPT + 1>(cpt, width);
    return width == 7 ? (void*)k_pcg_cluster<CPT, 7> : (void*)k_pcg_cluster<CPT, 0>;
  }
  static void* pick(int cpt, int width) { return pick_cpt<1>(cpt, width); }
  cudaLaunchConfig_t config(cudaLaunchAttribute* at, cudaStream_t st) const {
    cudaLaunchConfig_t c{};
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = (unsigned)blocks;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    c.gridDim = dim3((unsigned)blocks);
    c.blockDim = dim3(PCG_CL_TPB);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = at;
    c.numAttrs = 1;
    return c;
  }
  // Attributes of an instantiation: loads it, and allows clusters of 16 and max_smem of shared memory.
  static bool prepare(const void* k) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
           cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem) == cudaSuccess;
  }
  static constexpr int max_smem = 224 * 1024;  // of 227 KB per block; the reductions' buffers take 2 KB

  void plan(int n, int width) {
    kernel = nullptr;
    if (n < 1 || n > PCG_CL_MAX_ROWS || width > 16) return;
    blocks = 1;
    while (blocks < PCG_CL_BLOCKS && blocks * PCG_CL_TPB < n) blocks *= 2;
    C = (n + blocks - 1) / blocks;
    const int cpt = (C + PCG_CL_TPB - 1) / PCG_CL_TPB;
    const size_t fixed = 8 * (size_t)C;
    WS = (int)std::min<size_t>(width, (max_smem - fixed) / (12 * (size_t)C));
    smem = fixed + 12 * (size_t)C * WS;
    void* k = pick(cpt, width);
    int clusters = 0;
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t c = config(&at, nullptr);
    if (prepare(k) && cudaOccupancyMaxActiveClusters(&clusters, k, &c) == cudaSuccess && clusters > 0) kernel = k;
    else cudaGetLastError();
  }
  cudaError_t launch(PcgArgs<double> a, cudaStream_t st) const {
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t c = config(&at, st);
    int rows = C, slots = WS;
    void* args[] = {&a, &rows, &slots};
    return cudaLaunchKernelExC(&c, kernel, args);
  }
};

}  // namespace gpu
}  // namespace dpm
