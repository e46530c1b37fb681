// Jacobi-preconditioned conjugate gradients as one persistent, cooperatively launched kernel.
//
// The reference solves A phi = rhs with PETSc KSPCG: unpreconditioned residual norm, convergence
// when ||r|| <= max(rtol ||b||, atol), nonzero initial guess, constant null space removed from the
// right-hand side and from every preconditioned residual when no Dirichlet row exists
// (src/solver/pressure_backend_petsc.c:381-463, 816-876).  This kernel runs the same recurrence
// with the whole solve on the device:
//
//   phase A: p = (z - mean z) + (beta/beta_old) p_old, built on the fly for neighbour cells
//            (ping-pong p buffers), q = A p, partial p.q            -> grid all-reduce
//   phase B: x += a p, r -= a q, z = D^-1 r, partials r.r, sum z, sum r, z.r  -> grid all-reduce
//
// Rows of A are stored ELL [width][n] with sorted columns and padded to a fixed width with
// (self, 0) entries.  k_pcg_staged up to 1024 rows per SM; k_pcg beyond: up to 4096 with each thread's
// x, r, z and p in registers (CPT cells per thread), then with grid-stride loops.  The vectors that
// neighbours read (z, p) go through L2 (ld.cg), where other SMs' writes are visible.  Grid all-reduces
// are deterministic (see grid_allreduce).  The launches are cooperative, which guarantees co-residency
// of all blocks; every wait is bounded.
#pragma once
#include <algorithm>

#include "common.cuh"

namespace dpm {
namespace gpu {

#ifndef DPM_BARRIER_SPIN_LIMIT
#define DPM_BARRIER_SPIN_LIMIT (1u << 26)
#endif

constexpr int PCG_TPB = 1024;

// Poll limit of a grid-wide wait: status[3] when the host set it (a failure-detection test makes
// the wait run out this way), else DPM_BARRIER_SPIN_LIMIT.  Read by the waiting thread before it
// arrives, so the load overlaps the arrival.
__device__ __forceinline__ unsigned spin_limit(const int* status) {
  const unsigned o = (unsigned)__ldcg(&status[3]);
  return o ? o : (unsigned)DPM_BARRIER_SPIN_LIMIT;
}

template <class V>
struct PcgArgs {
  int n, WA;
  const int* col;      // [WA][n] sorted columns, PADI padded
  const V* val;        // [WA][n]
  const V* dinv;       // 1 / diag
  const V* b;          // right-hand side
  V* x;                // initial guess in, solution out
  V *r, *z, *p0, *p1, *q, *bp;
  double* partials;    // [2][nblocks][4]
  unsigned* bar;       // [0] monotonic arrival counter
  int* status;         // [0] reason, [1] iterations, [2] barrier timeout, [3] poll limit (0: default)
  double* dout;        // [0] true residual ||b - A x||, [1] last ||r||, [2] ||b'||
  double rtol, atol;
  int maxit, nullsp, guess_zero;
};

__device__ __forceinline__ double ld_cg(const double* p) { return __ldcg(p); }
__device__ __forceinline__ double ld_cg_if(const double* p, int on) {  // 0 when off
  double v = 0.0;
  asm volatile("{ .reg .pred t; setp.ne.s32 t, %2, 0; @t ld.global.cg.f64 %0, [%1]; }" : "+d"(v) : "l"(p), "r"(on) : "memory");
  return v;
}
__device__ __forceinline__ float ld_cg(const float* p) { return __ldcg(p); }

// Grid-wide deterministic all-reduce + barrier.  Each block reduces its NV values (fixed shuffle
// trees; warp k takes value k), writes them into the partial buffer of this barrier (two buffers
// alternate) and thread 0 arrives on a monotonic counter; once all blocks have arrived, warp k of
// every block reads value k of all partials with a fixed lane-to-block mapping, all of a lane's
// loads of a round issued together, and reduces them with the same shuffle tree, so all blocks
// hold bit-identical totals.  The wait is bounded and returns false on timeout.
template <int NV>
__device__ __forceinline__ bool grid_allreduce(double (&v)[NV], double* partials, unsigned* bar, unsigned& gen,
                                               int* status, double (&res)[NV]) {
  constexpr int RB = 5;  // blocks per lane per round of the post-barrier read (one round up to 160 blocks)
  __shared__ double sh[32][4];
  __shared__ double shr[4];
  __shared__ int s_ok;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int P = gridDim.x;
  double* buf = partials + (size_t)(gen & 1u) * 4 * gridDim.x;
#pragma unroll
  for (int k = 0; k < NV; ++k)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[w][k] = v[k];
  __syncthreads();
  if (w < NV) {  // warp w: value w over the block's warps
    double t = lane < nw ? sh[lane][w] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) buf[blockIdx.x * 4 + w] = t;
  }
  __syncthreads();  // the partial stores precede thread 0's release below
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned target = (gen + 1u) * gridDim.x;
    const unsigned lim = spin_limit(status);
    __threadfence();
    atomicAdd(&bar[0], 1u);
    unsigned spins = 0;
    for (;;) {
      unsigned cur;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(&bar[0]) : "memory");
      if ((int)(cur - target) >= 0) break;
      if (++spins > lim) { ok = 0; atomicExch(&status[2], 1); break; }
      if (spins > 32) __nanosleep(20);
    }
    // the acquiring load orders what the block reads after the next barrier: a fence here as well cost
    // 0.4 us per wait (393 216 rows: 12.9 us per iteration with it, 12.0 without)
    s_ok = ok;
  }
  __syncthreads();
  if (s_ok && w < NV) {  // warp w: value w over the blocks, lane l sums blocks l, l + 32, ... in order
    double u = 0.0;
    for (int b0 = lane; b0 < P; b0 += 32 * RB) {
      double pv[RB];
#pragma unroll
      for (int h = 0; h < RB; ++h) pv[h] = b0 + 32 * h < P ? __ldcg(&buf[(b0 + 32 * h) * 4 + w]) : 0.0;
#pragma unroll
      for (int h = 0; h < RB; ++h) u += pv[h];
    }
    for (int o = 16; o > 0; o >>= 1) u += __shfl_down_sync(0xffffffffu, u, o);
    if (lane == 0) shr[w] = u;
  }
  __syncthreads();
  gen = gen + 1u;
#pragma unroll
  for (int k = 0; k < NV; ++k) res[k] = s_ok ? shr[k] : 0.0;
  return s_ok != 0;
}

__device__ __forceinline__ int classify(double dp, double ttol, double atol, double rnorm0) {
  if (!(fabs(dp) <= 1.7976931348623157e308)) return -9;   // KSP_DIVERGED_NANORINF
  if (dp <= ttol) return dp < atol ? 3 : 2;               // KSP_CONVERGED_ATOL / _RTOL
  if (dp >= 1.0e5 * rnorm0) return -4;                    // KSP_DIVERGED_DTOL
  return 0;
}

// Row i of A times the vector v (ELL, padded rows: no early exit, all loads independent).
template <class V, int WT>
__device__ __forceinline__ double spmv_row(const PcgArgs<V>& a, int i, const V* v) {
  const int n = a.n;
  constexpr int W = WT > 0 ? WT : 16;
  const int WA = WT > 0 ? WT : a.WA;
  int c[W];
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (w < WA) c[w] = __ldg(&a.col[w * n + i]);
  double x[W];
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (w < WA) x[w] = (double)ld_cg(&v[c[w]]);
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (w < WA) s += (double)__ldcg(&a.val[w * n + i]) * x[w];
  return s;
}

// Row i of A times p = (z - mz) + bb p_old (first iteration: p = z - mz), p formed on the fly.
template <class V, int WT>
__device__ __forceinline__ double spmv_row_p(const PcgArgs<V>& a, int i, const V* pold, double mz, double bb,
                                             bool first) {
  const int n = a.n;
  constexpr int W = WT > 0 ? WT : 16;
  const int WA = WT > 0 ? WT : a.WA;
  int c[W];
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (w < WA) c[w] = __ldg(&a.col[w * n + i]);
  double zz[W], pp[W];
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (w < WA) {
      zz[w] = (double)ld_cg(&a.z[c[w]]);
      pp[w] = first ? 0.0 : (double)ld_cg(&pold[c[w]]);
    }
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (w < WA) {
      double pj = zz[w] - mz;
      if (!first) pj = pj + bb * pp[w];
      s += (double)__ldcg(&a.val[w * n + i]) * (double)(V)pj;
    }
  return s;
}

// CPT > 0: at most CPT cells per thread, own x, r, z, p held in registers
//          (requires n <= grid * blockDim * CPT).
// CPT == 0: grid-stride loops with the own-cell vectors in global memory (any n).
// WT: fixed padded row width (7 on hexahedral meshes), 0 = runtime width <= 16.
template <class V, int CPT, int WT>
__global__ void __launch_bounds__(PCG_TPB, 1) k_pcg(PcgArgs<V> a) {
  const int n = a.n;
  const int stride = gridDim.x * blockDim.x;
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned gen = 0;
  constexpr int NR = CPT > 0 ? CPT : 1;
  double rx[NR], rr_[NR], rz[NR], rp[NR], rq[NR], rd[NR];

  // ---- b' = b - mean(b) when the constant null space is active
  double mb = 0.0;
  if (a.nullsp) {
    double v[1] = {0.0}, t[1];
    for (int i = i0; i < n; i += stride) v[0] += (double)a.b[i];
    if (!grid_allreduce<1>(v, a.partials, a.bar, gen, a.status, t)) return;
    mb = t[0] / (double)n;
  }
  if (a.guess_zero) {
    for (int i = i0; i < n; i += stride) a.x[i] = (V)0;
    double v[1] = {0.0}, t[1];
    if (!grid_allreduce<1>(v, a.partials, a.bar, gen, a.status, t)) return;
  }
  // ---- r = b' - A x
  double v2[2] = {0.0, 0.0}, t2[2];
  if (CPT > 0) {
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      int i = i0 + k * stride;
      if (i < n) {
        double bi = (double)a.b[i];
        double bpi = (double)(V)(a.nullsp ? bi - mb : bi);
        double ri = bpi - spmv_row<V, WT>(a, i, a.x);
        rx[k] = (double)a.x[i];
        rr_[k] = (double)(V)ri;
        rd[k] = (double)__ldg(&a.dinv[i]);
        v2[0] += rr_[k] * rr_[k];
        v2[1] += bpi * bpi;
      }
    }
  } else {
    for (int i = i0; i < n; i += stride) {
      double bi = (double)a.b[i];
      double bpi = (double)(V)(a.nullsp ? bi - mb : bi);
      double ri = (double)(V)(bpi - spmv_row<V, WT>(a, i, a.x));
      a.r[i] = (V)ri;
      v2[0] += ri * ri;
      v2[1] += bpi * bpi;
    }
  }
  if (!grid_allreduce<2>(v2, a.partials, a.bar, gen, a.status, t2)) return;
  double dp = sqrt(t2[0]);
  const double sn = sqrt(t2[1]);
  const double rnorm0 = a.guess_zero ? dp : (sn == 0.0 ? dp : sn);
  const double ttol = fmax(a.rtol * rnorm0, a.atol);
  int reason = classify(dp, ttol, a.atol, rnorm0);
  int its = 0;
  if (!reason) {
    // ---- z = D^-1 r
    double v4[4] = {0, 0, 0, 0}, t4[4];
    if (CPT > 0) {
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        int i = i0 + k * stride;
        if (i < n) {
          rz[k] = (double)(V)(rr_[k] * rd[k]);
          a.z[i] = (V)rz[k];
          v4[0] += rz[k]; v4[1] += rr_[k]; v4[2] += rz[k] * rr_[k];
        }
      }
    } else {
      for (int i = i0; i < n; i += stride) {
        double ri = (double)a.r[i];
        double zi = (double)(V)(ri * (double)__ldg(&a.dinv[i]));
        a.z[i] = (V)zi;
        v4[0] += zi; v4[1] += ri; v4[2] += zi * ri;
      }
    }
    if (!grid_allreduce<4>(v4, a.partials, a.bar, gen, a.status, t4)) return;
    double mz = a.nullsp ? t4[0] / (double)n : 0.0;
    double beta = a.nullsp ? t4[2] - mz * t4[1] : t4[2];
    double betaold = 0.0, dpi = 0.0, dpiold = 0.0;
    V* pold = a.p0;
    V* pnew = a.p1;
    int it = 0;
    do {
      its = it + 1;
      if (beta == 0.0) { reason = 3; break; }
      if (it > 0 && beta * betaold < 0.0) { reason = -8; break; }
      const double bb = it == 0 ? 0.0 : beta / betaold;
      const bool first = it == 0;
      // ---- phase A: p, q = A p, p.q
      double v1[1] = {0.0}, t1[1];
      if (CPT > 0) {
#pragma unroll
        for (int k = 0; k < NR; ++k) {
          int i = i0 + k * stride;
          if (i < n) {
            double pi = rz[k] - mz;
            if (!first) pi = pi + bb * rp[k];
            rp[k] = (double)(V)pi;
            pnew[i] = (V)rp[k];
            rq[k] = (double)(V)spmv_row_p<V, WT>(a, i, pold, mz, bb, first);
            v1[0] += rp[k] * rq[k];
          }
        }
      } else {
        for (int i = i0; i < n; i += stride) {
          double pi = (double)a.z[i] - mz;
          if (!first) pi = pi + bb * (double)pold[i];
          pi = (double)(V)pi;
          pnew[i] = (V)pi;
          double qi = (double)(V)spmv_row_p<V, WT>(a, i, pold, mz, bb, first);
          a.q[i] = (V)qi;
          v1[0] += pi * qi;
        }
      }
      if (!grid_allreduce<1>(v1, a.partials, a.bar, gen, a.status, t1)) return;
      dpiold = dpi;
      dpi = t1[0];
      betaold = beta;
      if (dpi == 0.0 || (it > 0 && ((dpi > 0) - (dpi < 0)) * ((dpiold > 0) - (dpiold < 0)) < 0)) {
        reason = dpi == 0.0 ? 3 : -10;
        break;
      }
      const double al = beta / dpi;
      // ---- phase B: x, r, z and the four sums
      double w4[4] = {0, 0, 0, 0}, s4[4];
      if (CPT > 0) {
#pragma unroll
        for (int k = 0; k < NR; ++k) {
          int i = i0 + k * stride;
          if (i < n) {
            rx[k] = (double)(V)(rx[k] + al * rp[k]);
            rr_[k] = (double)(V)(rr_[k] - al * rq[k]);
            rz[k] = (double)(V)(rr_[k] * rd[k]);
            a.z[i] = (V)rz[k];
            w4[0] += rr_[k] * rr_[k]; w4[1] += rz[k]; w4[2] += rr_[k]; w4[3] += rz[k] * rr_[k];
          }
        }
      } else {
        for (int i = i0; i < n; i += stride) {
          double pi = (double)pnew[i];
          a.x[i] = (V)((double)a.x[i] + al * pi);
          double ri = (double)(V)((double)a.r[i] - al * (double)a.q[i]);
          a.r[i] = (V)ri;
          double zi = (double)(V)(ri * (double)__ldg(&a.dinv[i]));
          a.z[i] = (V)zi;
          w4[0] += ri * ri; w4[1] += zi; w4[2] += ri; w4[3] += zi * ri;
        }
      }
      if (!grid_allreduce<4>(w4, a.partials, a.bar, gen, a.status, s4)) return;
      dp = sqrt(s4[0]);
      reason = classify(dp, ttol, a.atol, rnorm0);
      if (reason) break;
      mz = a.nullsp ? s4[1] / (double)n : 0.0;
      beta = a.nullsp ? s4[3] - mz * s4[2] : s4[3];
      V* t = pold; pold = pnew; pnew = t;
      it++;
    } while (it < a.maxit);
    if (!reason && it >= a.maxit) reason = -3;
  }
  // ---- write back x, then the true residual ||b - A x|| with the caller's b (KSPBuildResidual)
  if (CPT > 0) {
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      int i = i0 + k * stride;
      if (i < n) a.x[i] = (V)rx[k];
    }
  }
  double v1[1] = {0.0}, t1[1];
  if (!grid_allreduce<1>(v1, a.partials, a.bar, gen, a.status, t1)) return;
  for (int i = i0; i < n; i += stride) {
    double d = (double)a.b[i] - spmv_row<V, WT>(a, i, a.x);
    v1[0] += d * d;
  }
  if (!grid_allreduce<1>(v1, a.partials, a.bar, gen, a.status, t1)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.dout[0] = sqrt(t1[0]);
    a.dout[1] = dp;
    a.dout[2] = sn;
    a.status[0] = reason;
    a.status[1] = its;
  }
}

// The scalars that an iteration of the staged form carries over, with KSPCG's tests.
struct PcgScalars {
  double beta, betaold = 0.0, dpi = 0.0, bb = 0.0, mz;
  // before p: KSP_DIVERGED_INDEFINITE_PC on a sign change of z.r; 0 when the iteration goes on
  __device__ int top(int it) const {
    if (beta == 0.0) return 3;
    return it > 0 && beta * betaold < 0.0 ? -8 : 0;
  }
  // p.q: KSP_DIVERGED_INDEFINITE_MAT on a sign change
  __device__ int curvature(int it, double pq) {
    const double old = dpi;
    dpi = pq;
    betaold = beta;
    if (dpi == 0.0) return 3;
    return it > 0 && ((dpi > 0) - (dpi < 0)) * ((old > 0) - (old < 0)) < 0 ? -10 : 0;
  }
  // the sums (r.r, sum z, sum r, z.r) after the update
  __device__ void next(const double (&s)[4], int nullsp, int n) {
    mz = nullsp ? s[1] / (double)n : 0.0;
    beta = nullsp ? s[3] - mz * s[2] : s[3];
    bb = beta / betaold;
  }
};

// Staged form: block b owns the consecutive rows [b C, b C + size) and keeps their operator (200 B per
// row of 16, the widest) and its part of p in shared memory, x, r, p, q and 1/diag in registers.  The
// entries of a row that lie in the block's own rows - five of seven on a hexahedral mesh - read p
// there; the others form p_j from z_j and the old p_j in L2, as k_pcg does for all.
// us per iteration (of two solves that differ by 100), here and in the form that reads all of it through
// L2: 44 880 rows 6.0 / 8.45, 66 600 rows 6.1 / 8.5, 85 050 rows 6.6 / 8.6, 131 072 rows 6.7 / 8.8.
// With more than two rows per thread the few warps no longer cover the loads from other blocks' rows, one
// row after the other (393 216 rows, six rows per thread: 15.5 / 12.7), and the register form with 32 warps
// takes over.
// CPT: rows per thread.
constexpr int PCG_ST_TPB = 512;
constexpr int PCG_ST_CPT = 2;
template <int CPT, int WT>
__global__ void __launch_bounds__(PCG_ST_TPB, 1) k_pcg_staged(PcgArgs<double> a, int C) {
  extern __shared__ double st_smem[];
  constexpr int CH = WT > 0 ? WT : 4;  // slots whose loads are in flight together
  const int n = a.n, WA = WT > 0 ? WT : a.WA;
  const int base = (int)blockIdx.x * C, size = max(0, min(C, n - base));
  double* s_p = st_smem;                               // [C]
  double* s_val = s_p + C;                             // [WA][C]
  int* s_col = reinterpret_cast<int*>(s_val + (size_t)WA * C);  // [WA][C] own row l, or ~global column
  unsigned gen = 0;
  auto code = [&](int c) { return (unsigned)(c - base) < (unsigned)size ? c - base : ~c; };
  // row l of this block times the vector that is s_p on its own rows and elsewhere z - m + f po (no f:
  // z - m).  Both loads are predicated, not branched over, so that a row's are in flight together.
  auto product = [&](int l, const double* z, const double* po, double m, double f, int with_po) {
    double s = 0.0;
    for (int w0 = 0; w0 < WA; w0 += CH) {
      int cc[CH];
      double v[CH], x[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int w = w0 + u;
        const bool on = WT > 0 || w < WA;
        cc[u] = on ? s_col[w * C + l] : l;
        v[u] = on ? s_val[w * C + l] : 0.0;
      }
      double zz[CH], pp[CH];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int j = cc[u] < 0 ? ~cc[u] : 0;
        zz[u] = ld_cg_if(z + j, cc[u] < 0);
        pp[u] = ld_cg_if(po + j, cc[u] < 0 && with_po);
      }
#pragma unroll
      for (int u = 0; u < CH; ++u) x[u] = s_p[max(cc[u], 0)];
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        if (cc[u] < 0) {
          x[u] = zz[u] - m;
          if (with_po) x[u] = x[u] + f * pp[u];
        }
        s += v[u] * x[u];
      }
    }
    return s;
  };
#define ST_OWN(k) ((int)threadIdx.x + (k) * PCG_ST_TPB < size)
#define ST_ROW(k) ((int)threadIdx.x + (k) * PCG_ST_TPB)
  for (int w = 0; w < WA; ++w)
    for (int l = threadIdx.x; l < size; l += PCG_ST_TPB) {
      s_col[w * C + l] = code(__ldg(&a.col[(size_t)w * n + base + l]));
      s_val[w * C + l] = __ldg(&a.val[(size_t)w * n + base + l]);
    }
  double rx[CPT], rr[CPT], rp[CPT], rq[CPT], rd[CPT];
  // ---- b' = b - mean(b) when the constant null space is active; the guess
  double mb = 0.0;
  {
    double v[1] = {0.0}, t[1];
#pragma unroll
    for (int k = 0; k < CPT; ++k)
      if (ST_OWN(k)) {
        const int i = base + ST_ROW(k);
        rx[k] = a.guess_zero ? 0.0 : a.x[i];
        rr[k] = a.b[i];
        rd[k] = __ldg(&a.dinv[i]);
        rp[k] = 0.0;
        s_p[ST_ROW(k)] = rx[k];
        v[0] += rr[k];
      }
    if (!grid_allreduce<1>(v, a.partials, a.bar, gen, a.status, t)) return;
    mb = a.nullsp ? t[0] / (double)n : 0.0;
  }
  // ---- r = b' - A x (the caller's x: nobody writes it before the end)
  double v2[2] = {0.0, 0.0}, t2[2];
#pragma unroll
  for (int k = 0; k < CPT; ++k)
    if (ST_OWN(k)) {
      const double bp = a.nullsp ? rr[k] - mb : rr[k];
      rr[k] = bp - (a.guess_zero ? 0.0 : product(ST_ROW(k), a.x, a.x, 0.0, 0.0, 0));
      v2[0] += rr[k] * rr[k];
      v2[1] += bp * bp;
    }
  if (!grid_allreduce<2>(v2, a.partials, a.bar, gen, a.status, t2)) return;
  double dp = sqrt(t2[0]);
  const double sn = sqrt(t2[1]);
  const double rnorm0 = a.guess_zero ? dp : (sn == 0.0 ? dp : sn);
  const double ttol = fmax(a.rtol * rnorm0, a.atol);
  int reason = classify(dp, ttol, a.atol, rnorm0);
  int its = 0;
  if (!reason) {
    // ---- z = D^-1 r
    double v4[4] = {0, 0, 0, 0}, t4[4];
#pragma unroll
    for (int k = 0; k < CPT; ++k)
      if (ST_OWN(k)) {
        const double z = rr[k] * rd[k];
        a.z[base + ST_ROW(k)] = z;
        v4[0] += z; v4[1] += rr[k]; v4[2] += z * rr[k];
      }
    if (!grid_allreduce<4>(v4, a.partials, a.bar, gen, a.status, t4)) return;
    PcgScalars c;
    c.mz = a.nullsp ? t4[0] / (double)n : 0.0;
    c.beta = a.nullsp ? t4[2] - c.mz * t4[1] : t4[2];
    double* pold = a.p0;
    double* pnew = a.p1;
    int it = 0;
    do {
      its = it + 1;
      if ((reason = c.top(it))) break;
      const bool first = it == 0;
      // ---- p, q = A p, p.q
#pragma unroll
      for (int k = 0; k < CPT; ++k)
        if (ST_OWN(k)) {
          double p = rr[k] * rd[k] - c.mz;
          if (!first) p = p + c.bb * rp[k];
          rp[k] = p;
          s_p[ST_ROW(k)] = p;
          pnew[base + ST_ROW(k)] = p;
        }
      __syncthreads();
      double v1[1] = {0.0}, t1[1];
#pragma unroll
      for (int k = 0; k < CPT; ++k)
        if (ST_OWN(k)) {
          rq[k] = product(ST_ROW(k), a.z, pold, c.mz, c.bb, !first);
          v1[0] += rp[k] * rq[k];
        }
      if (!grid_allreduce<1>(v1, a.partials, a.bar, gen, a.status, t1)) return;
      if ((reason = c.curvature(it, t1[0]))) break;
      const double al = c.beta / c.dpi;
      // ---- x, r, z and the four sums
      double w4[4] = {0, 0, 0, 0}, s4[4];
#pragma unroll
      for (int k = 0; k < CPT; ++k)
        if (ST_OWN(k)) {
          rx[k] = rx[k] + al * rp[k];
          rr[k] = rr[k] - al * rq[k];
          const double z = rr[k] * rd[k];
          a.z[base + ST_ROW(k)] = z;
          w4[0] += rr[k] * rr[k]; w4[1] += z; w4[2] += rr[k]; w4[3] += z * rr[k];
        }
      if (!grid_allreduce<4>(w4, a.partials, a.bar, gen, a.status, s4)) return;
      dp = sqrt(s4[0]);
      c.next(s4, a.nullsp, n);
      reason = classify(dp, ttol, a.atol, rnorm0);
      if (reason) break;
      double* t = pold; pold = pnew; pnew = t;
      it++;
    } while (it < a.maxit);
    if (!reason && it >= a.maxit) reason = -3;
  }
  // ---- x, then the true residual ||b - A x|| with the caller's b (KSPBuildResidual)
#pragma unroll
  for (int k = 0; k < CPT; ++k)
    if (ST_OWN(k)) {
      a.x[base + ST_ROW(k)] = rx[k];
      s_p[ST_ROW(k)] = rx[k];
    }
  double v1[1] = {0.0}, t1[1];
  if (!grid_allreduce<1>(v1, a.partials, a.bar, gen, a.status, t1)) return;
#pragma unroll
  for (int k = 0; k < CPT; ++k)
    if (ST_OWN(k)) {
      const double d = a.b[base + ST_ROW(k)] - product(ST_ROW(k), a.x, a.x, 0.0, 0.0, 0);
      v1[0] += d * d;
    }
  if (!grid_allreduce<1>(v1, a.partials, a.bar, gen, a.status, t1)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.dout[0] = sqrt(t1[0]);
    a.dout[1] = dp;
    a.dout[2] = sn;
    a.status[0] = reason;
    a.status[1] = its;
  }
#undef ST_OWN
#undef ST_ROW
}

constexpr size_t pcg_staged_smem(int rows, int width) { return (size_t)rows * (8 + 12 * (size_t)width); }

// The cooperative launch of a system: kernel, blocks, rows per block, shared memory.
struct PcgGrid {
  void* kernel = nullptr;
  int grid = 0, tpb = 0, C = 0;
  size_t smem = 0;
  static constexpr int max_smem = 223 * 1024;  // of 227 KB per block; the all-reduces' buffers take 3 KB
  static_assert(pcg_staged_smem(PCG_ST_TPB * PCG_ST_CPT, 16) <= max_smem, "the widest operator is staged whole");

  template <int CPT>
  static void* pick_cpt(int cpt, int width) {
    if constexpr (CPT < PCG_ST_CPT)
      if (cpt > CPT) return pick_cpt<CPT + 1>(cpt, width);
    return width == 7 ? (void*)k_pcg_staged<CPT, 7> : (void*)k_pcg_staged<CPT, 0>;
  }
  static void* staged(int cpt, int width) { return pick_cpt<1>(cpt, width); }
  static void* regs(int cpt, int width) {  // cpt 2..4: register-resident, else grid-stride
    const bool w7 = width == 7;
    switch (cpt) {
      case 2: return w7 ? (void*)k_pcg<double, 2, 7> : (void*)k_pcg<double, 2, 0>;
      case 3: return w7 ? (void*)k_pcg<double, 3, 7> : (void*)k_pcg<double, 3, 0>;
      case 4: return w7 ? (void*)k_pcg<double, 4, 7> : (void*)k_pcg<double, 4, 0>;
      default: return w7 ? (void*)k_pcg<double, 0, 7> : (void*)k_pcg<double, 0, 0>;
    }
  }
  // Loads the kernel and sets its shared memory, or for the other forms the largest L1.
  static bool prepare(const void* k, bool is_staged) {
    return (is_staged ? cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem)
                      : cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 5)) == cudaSuccess;
  }
  // 256 rows per block at least: fewer blocks have less to wait for
  bool plan(int n, int width, int sms) {
    kernel = nullptr;
    grid = std::max(1, std::min(sms, (n + 255) / 256));
    C = (n + grid - 1) / grid;
    const int cpt = (C + PCG_ST_TPB - 1) / PCG_ST_TPB;
    const bool st = cpt <= PCG_ST_CPT;
    tpb = st ? PCG_ST_TPB : PCG_TPB;
    smem = st ? pcg_staged_smem(C, width) : 0;
    const int rows = (C + PCG_TPB - 1) / PCG_TPB;  // of a thread in the register form
    void* k = st ? staged(cpt, width) : regs(rows >= 2 && rows <= 4 ? rows : 0, width);
    int per_sm = 0;
    if (!prepare(k, st) || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, tpb, smem) != cudaSuccess ||
        per_sm < 1)
      return false;
    kernel = k;
    return true;
  }
  cudaError_t launch(PcgArgs<double> a, cudaStream_t st) const {
    int rows = C;
    void* staged_args[] = {&a, &rows};
    return cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(tpb), staged_args, smem, st);  // k_pcg takes the first
  }
};

}  // namespace gpu
}  // namespace dpm
