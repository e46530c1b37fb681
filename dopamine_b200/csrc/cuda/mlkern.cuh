// The multilevel flexible-CG solve as a sequence of standalone kernels, for large meshes.
//
// k_mlcg keeps the whole solve in one persistent cooperative kernel: no launch gaps, but every
// phase runs at two 512-thread blocks per SM under a 64-register cap, and on a fine level of
// millions of rows its sweeps reach ~40 % of HBM bandwidth (long-scoreboard stalls; more rows per
// lane, a register software pipeline and shared-memory staging of the row data were all measured
// slower).  The same sweep as a standalone kernel - one row per thread, 32 registers, full
// occupancy - streams a 19.3M-row, 6-neighbour level at the measured copy bandwidth (0.21 ms,
// 6.6 TB/s).  So each phase is its own kernel: Chebyshev sweep, residual, restriction, dense coarse
// solve, prolongation, w = A z with per-block partial sums, the FCG scalars (the partials reduced in
// a fixed order, the stopping rule applied by the block that arrives last), and the vector update.
// The Krylov state lives in device memory (MlkState); once a solve has stopped, every kernel returns
// at its first instruction, so the host enqueues the next iteration before it reads the stop flag of
// the last one.  An iteration is one captured graph whose kernels follow each other with
// programmatic launches (mlk_enter): single launches of 3-60 us each had left 4-5 us between them.  At
// Chebyshev degree 2 an iteration of L smoothed levels is 6 L + 4 launches: 16, 22 or 28.
//
// The hierarchy is smoothed aggregation (SaLevel, csrc/host/multilevel.hpp).  The unsmoothed one of
// k_mlcg moves a quarter fewer bytes per iteration, but its two-grid contraction is 0.4-0.5 whatever
// the cycle on the coarse levels (K- and W-cycles 24-30 iterations, V 33-36 on the 2.4M-cell urban
// operator), against 0.17-0.36 here: 12 iterations per solve instead of 31 there (Poisson 45.1 ->
// 18.0 ms per step), 13.7 instead of 36 at 8.2M cells (127 -> 57 ms), 22 instead of 29 on the
// graded 1.06M-cell Rayleigh-Benard mesh (24.7 -> 14.3 ms).
// Bounds (ncu, 2.4M rows): the finest level's sweeps stream 68 B per row, 33 us at 5.0 of the 6.47 TB/s
// a copy reaches, the FP64 w = A z 4.0 and the update 5.4 TB/s; the first coarse level's rows (37 entries)
// are bound by the latency of their gathers, 28 us per sweep of 304k rows at 3.8 TB/s: they are laid out
// as slices with a row per thread (22 us when the two were compared, 41 with eight lanes per row); levels
// below ~20k rows cost their launch and latency, 4-10 us.
// The recurrences, the null-space handling, the stall guard and the stopping rule are those of
// k_mlcg and k_fcg (src/solver/pressure_backend_petsc.c:816-876 for the rule itself); only the
// order of the reductions' sums differs.
#pragma once
#include "mlcg.cuh"

namespace dpm {
namespace gpu {

constexpr int MLK_TPB = 256;
constexpr int MLK_NV = 8;            // sums reduced per iteration
constexpr int MLK_RED_BLOCKS = 2368; // grid of the reducing kernels (16 blocks per SM)

struct MlkState {
  double mb, rnorm0, ttol, rtol, atol, dp, sn, dp_mark, pq_old, alpha, beta, m, true_res;
  int its, reason, done, maxit, nullsp, guess_zero, stall_window;
  unsigned folded;  // blocks of k_mlk_rule that have arrived
  double stall_ratio;
  double* x;        // the iterate, here so that a captured iteration serves every caller's array
};

// The kernels of an iteration are launched with programmatic stream serialization: each lets the
// next one's blocks come in as its own drain, and waits here for the one before to have completed
// (its stores visible) before it touches memory.  A kernel is thus resident while the arrays that it
// reads are still being written: those are read by mlk_ld, __ldcg or plain loads, which stay behind the
// wait, never by __ldg (the non-coherent load wants data that nobody writes while the kernel lives, and
// may be moved up) nor through __restrict__ pointers (which the clobbers above do not cover).  __ldg
// is for what the set-up wrote: operators, transfers, diagonals, the inverse, omega.
__device__ __forceinline__ void mlk_enter() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// A cached load of such a value; not reordered with mlk_enter.
__device__ __forceinline__ float mlk_ld(const float* p) {
  float v;
  asm volatile("ld.global.ca.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float mlk_ld_if(const float* p, bool on) {  // 0 when off
  float v = 0.0f;
  asm volatile("{ .reg .pred t; setp.ne.s32 t, %2, 0; @t ld.global.ca.f32 %0, [%1]; }" : "+f"(v) : "l"(p), "r"((int)on));
  return v;
}
__device__ __forceinline__ float4 mlk_ld(const float4* p) {
  float4 v;
  asm volatile("ld.global.ca.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// Block sum of NV values per thread into part[block][NV] (fixed shuffle tree, then warps in order).
template <int NV>
__device__ __forceinline__ void mlk_block_partials(double (&v)[NV], double* part) {
  __shared__ double sh[MLK_TPB / 32][NV];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double t = v[k];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) sh[w][k] = t;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double t = 0.0;
    for (int j = 0; j < MLK_TPB / 32; ++j) t += sh[j][threadIdx.x];
    part[(size_t)blockIdx.x * NV + threadIdx.x] = t;
  }
}

// Totals of the per-block partials (one block of 32 * NV threads: warp k sums value k over the
// blocks, lane l taking blocks l, l + 32, ... in order, then a fixed shuffle tree).
template <int NV>
__device__ __forceinline__ void mlk_totals(int nparts, const double* part, double (&tot)[NV]) {
  __shared__ double s_t[NV];
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (k < NV) {
    double t = 0.0;
    for (int j = lane; j < nparts; j += 32) t += __ldcg(&part[(size_t)j * NV + k]);
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) s_t[k] = t;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NV; ++q) tot[q] = s_t[q];
}

// Sparse rows of the smoothed-aggregation hierarchy on the device: entries are (index, FP32 bits)
// pairs, one 8-byte load each.  lg >= 0: compressed rows, off [rows+1], 2^lg lanes share a row.
// lg < 0: slices of 32 rows, off [slices+1] in entries, entry k of the slice's row r at
// off[slice] + 32 k + r, short rows padded with (own first index, 0).
struct MlkRows {
  const int* off;
  const int2* ent;
  int lg;
};

// One level of the smoothed-aggregation hierarchy (csrc/host/multilevel.hpp, SaLevel), passed to
// the kernels by value.
struct MlkLevel {
  int n, n_next;
  int W;             // finest level: ELL width of the scaled off-diagonals
  const int* col;    // [W][n]
  const void* sv;    // [W][n] FP32 or binary16 bits
  MlkRows A, P, R;   // other levels' scaled off-diagonals; prolongation; restriction (rows of the next level)
  const float *g, *diag, *dinv;
  float oc;                  // factor of the coarse correction
  float *b, *x0, *x1, *d;    // scaled right-hand side, iterate (two buffers), Chebyshev direction
  float inv_theta, c1[ML_DEG], c2[ML_DEG];
};

// The scaled right-hand side of level L.  The first Chebyshev step from a zero iterate is
// x = d = inv_theta b: it is not stored, the sweep of STEP_SECOND forms it from b (deg > 1) or k_mlk_first writes it.
__device__ __forceinline__ void mlk_start(const MlkLevel& L, int i, float ri) { L.b[i] = ri * __ldg(&L.dinv[i]); }

// A smoothing step of one row.  STEP_SECOND: the second step from a zero iterate (the gathered
// vector is b, so x = d = inv_theta b); STEP_NEXT: a later step; STEP_UP: the first step after the
// coarse correction; STEP_RESID: the unscaled residual.  keep: the direction is read again.
enum MlkStep { STEP_SECOND, STEP_NEXT, STEP_UP, STEP_RESID };
__device__ __forceinline__ void mlk_step(const MlkLevel& L, int step, int keep, float c1, float c2, int i, float acc,
                                         float x, float* xo, float add) {
  const float b = __ldcg(&L.b[i]), g = __ldg(&L.g[i]);
  if (step == STEP_RESID) {
    xo[i] = __ldg(&L.diag[i]) * (b - fmaf(g, x, acc));
    return;
  }
  float rs, d;
  if (step == STEP_SECOND) {  // x is b here, acc = S b
    x = L.inv_theta * x;
    rs = b - fmaf(g, x, L.inv_theta * acc);
    d = fmaf(c1, x, c2 * rs);
  } else {
    rs = b - fmaf(g, x, acc);
    d = step == STEP_UP ? L.inv_theta * rs : fmaf(c1, __ldcg(&L.d[i]), c2 * rs);
  }
  if (keep) L.d[i] = d;
  xo[i] = x + d + add * b;
}
// degree 1: the only step from a zero iterate
static __global__ void __launch_bounds__(256) k_mlk_first(MlkLevel L, const MlkState* S) {
  mlk_enter();
  if (S->done) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < L.n) L.x0[i] = L.inv_theta * __ldcg(&L.b[i]);
}

// Row sum of val * v[index] for the row of this thread (SELL: thread = row; else 2^lg lanes per
// row, every lane of the row returning the sum, added over the lanes by a fixed butterfly).  A
// lane's loads are in flight together, eight or four at a time.  The gathers go through L1:
// neighbouring rows share most of their columns.
template <bool SELL>
__device__ __forceinline__ float mlk_rowsum(const MlkRows& m, int t, int rows, const float* v) {
  float s = 0.0f;
  if (SELL) {
    if (t >= rows) return s;
    const int e0 = __ldg(&m.off[t >> 5]), w = (__ldg(&m.off[(t >> 5) + 1]) - e0) >> 5;
    const int2* q = m.ent + e0 + (t & 31);
    int k = 0;
    for (; k + 8 <= w; k += 8) {
      int2 e[8];
      float x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) e[u] = __ldg(&q[32 * (k + u)]);
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = mlk_ld(&v[e[u].x]);
#pragma unroll
      for (int u = 0; u < 8; ++u) s = fmaf(__int_as_float(e[u].y), x[u], s);
    }
    for (; k < w; ++k) {
      const int2 e = __ldg(&q[32 * k]);
      s = fmaf(__int_as_float(e.y), mlk_ld(&v[e.x]), s);
    }
    return s;
  }
  const int i = t >> m.lg, G = 1 << m.lg, sub = t & (G - 1);
  const bool ok = i < rows;
  const int e0 = ok ? __ldg(&m.off[i]) : 0, e1 = ok ? __ldg(&m.off[i + 1]) : 0;
  for (int e = e0 + sub; e < e1; e += 4 * G) {
    int2 q[4];
    float x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) q[u] = e + u * G < e1 ? __ldg(&m.ent[e + u * G]) : make_int2(-1, 0);
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = mlk_ld_if(v + max(q[u].x, 0), q[u].x >= 0);
#pragma unroll
    for (int u = 0; u < 4; ++u) s = fmaf(__int_as_float(q[u].y), x[u], s);
  }
  for (int o = G >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
// Row of thread t, or -1 for a lane that only helps (or lies beyond the rows).
template <bool SELL>
__device__ __forceinline__ int mlk_row_of(const MlkRows& m, int t, int rows) {
  const int i = SELL ? t : t >> m.lg;
  return i < rows && (SELL || (t & ((1 << m.lg) - 1)) == 0) ? i : -1;
}

// ---- start: b' = b - mean(b) (null space), r = b' - A x
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_init_sum(int n, const double* __restrict__ b, double* x,
                                                          int guess_zero, double* part) {
  double v[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (guess_zero) x[i] = 0.0;
    v[0] += b[i];
  }
  mlk_block_partials<1>(v, part);
}
static __global__ void k_mlk_init_mean(int n, int nparts, const double* part, MlkState* S) {
  double t[1];
  mlk_totals<1>(nparts, part, t);
  if (threadIdx.x == 0) S->mb = S->nullsp ? t[0] / (double)n : 0.0;
}
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_init_resid(MlArgs a, MlkLevel L0, const MlkState* S,
                                                            double* part) {
  const double mb = S->mb;
  double v[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
    const double bp = a.b[i] - mb;
    const double ri = bp - ml_row64(a, i, (const double*)a.x);
    a.r[i] = ri;
    a.p[i] = 0.0;
    a.q[i] = 0.0;
    v[0] += ri * ri;
    v[1] += bp * bp;
    mlk_start(L0, i, (float)ri);
  }
  mlk_block_partials<2>(v, part);
}
static __global__ void k_mlk_init_rule(int nparts, const double* part, MlkState* S) {
  double t[2];
  mlk_totals<2>(nparts, part, t);
  if (threadIdx.x == 0) {
    const double dp = sqrt(t[0]), sn = sqrt(t[1]);
    S->dp = dp;
    S->sn = sn;
    S->rnorm0 = S->guess_zero ? dp : (sn == 0.0 ? dp : sn);
    S->ttol = fmax(S->rtol * S->rnorm0, S->atol);
    int reason = classify(dp, S->ttol, S->atol, S->rnorm0);
    if (!reason && S->maxit <= 0) reason = -3;
    S->reason = reason;
    S->its = 0;
    S->pq_old = 1.0;
    S->dp_mark = dp;
    S->done = reason != 0;
  }
}

// ---- V-cycle phases.  Finest level: one row per thread (ELL).  Bound by HBM: a sweep reads
// columns, values, g, b, x and d and writes d and x.
template <class SV>
__device__ __forceinline__ float mlk_row0(const MlkLevel& L, int i, const float* x) {
  const SV* sv = static_cast<const SV*>(L.sv);
  float s = 0.0f;
  for (int k0 = 0; k0 < L.W; k0 += ML_CHUNK) {
    int c[ML_CHUNK];
    float v[ML_CHUNK], xv[ML_CHUNK];
#pragma unroll
    for (int u = 0; u < ML_CHUNK; ++u) {
      const size_t e = (size_t)(k0 + u) * L.n + i;
      c[u] = k0 + u < L.W ? __ldg(&L.col[e]) : i;
      v[u] = k0 + u < L.W ? ml_sval(&sv[e]) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < ML_CHUNK; ++u) xv[u] = mlk_ld(&x[c[u]]);
#pragma unroll
    for (int u = 0; u < ML_CHUNK; ++u) s = fmaf(v[u], xv[u], s);
  }
  return s;
}
template <class SV>
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_sweep(MlkLevel L, int step, int keep, float c1, float c2,
                                                       const float* xi, float* xo,
                                                       const float* om, float gam, const MlkState* S) {
  mlk_enter();
  if (S->done) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= L.n) return;
  const float acc = mlk_row0<SV>(L, i, xi);
  mlk_step(L, step, keep, c1, c2, i, acc, mlk_ld(&xi[i]), xo, om ? gam * __ldg(&om[i]) : 0.0f);
}
// Other levels, 30-110 entries per row: a row per thread in 32-row slices while the level has the
// rows to fill the chip (neighbouring rows' columns lie close together, so a warp's gathers touch
// few sectors), else 2^lg lanes per row.
template <bool SELL>
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_csweep(MlkLevel L, int step, int keep, float c1, float c2,
                                                        const float* xi, float* xo,
                                                        const MlkState* S) {
  mlk_enter();
  if (S->done) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const float acc = mlk_rowsum<SELL>(L.A, t, L.n, xi);
  const int i = mlk_row_of<SELL>(L.A, t, L.n);
  if (i >= 0) mlk_step(L, step, keep, c1, c2, i, acc, mlk_ld(&xi[i]), xo, 0.0f);
}
// restriction P^T r: the next level's scaled right-hand side (or the coarsest one, unscaled)
template <bool SELL>
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_restrict(MlkLevel L, const float* r, MlkLevel N,
                                                          float* bC, const MlkState* S) {
  mlk_enter();
  if (S->done) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const float s = mlk_rowsum<SELL>(L.R, t, L.n_next, r);
  const int c = mlk_row_of<SELL>(L.R, t, L.n_next);
  if (c < 0) return;
  if (bC) bC[c] = s;
  else mlk_start(N, c, s);
}
// coarsest level: x_C = A_C^-1 b_C, one warp per row; rows of the inverse and b_C padded with zeros
// to a multiple of 4 (16-byte loads)
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_coarse(int nC, int nC4, const float4* cinv,
                                                        const float4* bC, float* xC,
                                                        const MlkState* S) {
  mlk_enter();
  if (S->done) return;
  const int lane = threadIdx.x & 31;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= nC) return;
  const float4* q = cinv + (size_t)row * nC4;
  float s = 0.0f;
#pragma unroll 4
  for (int k = lane; k < nC4; k += 32) {
    const float4 c = __ldg(&q[k]), b = mlk_ld(&bC[k]);
    s = fmaf(c.x, b.x, s);
    s = fmaf(c.y, b.y, s);
    s = fmaf(c.z, b.z, s);
    s = fmaf(c.w, b.w, s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) xC[row] = s;
}
// prolongation in place: x_i += oc (P x_c)_i
template <bool SELL>
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_prolong(MlkLevel L, float* x,
                                                         const float* xc, const MlkState* S) {
  mlk_enter();
  if (S->done) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const float s = mlk_rowsum<SELL>(L.P, t, L.n, xc);
  const int i = mlk_row_of<SELL>(L.P, t, L.n);
  if (i >= 0) x[i] = fmaf(L.oc, s, x[i]);
}

// training-sample recording of the learned term (as in k_mlcg): every rec_stride-th iteration
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_record(MlArgs a, const float* z, const float* b0,
                                                        const MlkState* S) {
  mlk_enter();
  if (S->done) return;
  const int its = S->its;
  if (a.rec_stride <= 0 || its % a.rec_stride != 0 || a.rec_base + its / a.rec_stride >= a.rec_max) return;
  const size_t off = (size_t)(a.rec_base + its / a.rec_stride) * a.n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
    const size_t o = off + __ldg(&a.pinv[i]);
    a.rec_r[o] = __ldcg(&a.r[i]);
    a.rec_z[o] = (double)__ldcg(&z[i]);
    a.rec_u[o] = (double)__ldcg(&b0[i]);
    a.rec_x[o] = __ldcg(&S->x[i]);
  }
}

// ---- w = A z (FP64 operator) and the eight sums of the iteration: one row per thread (as the
// sweeps; a grid-stride loop over ~32 rows per thread ran at half the bandwidth), per-block
// partials folded by k_mlk_rule
template <class ZT>
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_wz(MlArgs a, const ZT* z, double* part,
                                                    const MlkState* S) {
  mlk_enter();
  if (S->done) return;
  double v[MLK_NV];
#pragma unroll
  for (int k = 0; k < MLK_NV; ++k) v[k] = 0.0;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.n) {
    const double wi = ml_row64(a, i, z);
    const double zi = (double)__ldcg(&z[i]), qi = __ldcg(&a.q[i]), ri = __ldcg(&a.r[i]);
    a.w[i] = wi;
    v[0] += zi * ri;
    v[1] += zi * qi;
    v[2] += zi * wi;
    v[3] += zi;
    v[4] += ri * ri;
    v[5] += ri;
    v[6] += qi;
    v[7] += wi;
  }
  mlk_block_partials<MLK_NV>(v, part);
}
// Block b sums partials b*256 .. b*256+255 (fixed order); the block that arrives last then sums
// the blocks' values (fixed order), forms the FCG scalars and applies the stopping rule (k_mlcg's,
// after its reduce-and-gather).  The iteration counted here is the one k_mlk_update ends; the cap
// stops the solve at the next rule (KSP_DIVERGED_ITS).
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_rule(int n, int nparts, const double* in,
                                                      double* part, MlkState* S) {
  mlk_enter();
  if (S->done) return;
  {
    double v[MLK_NV];
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
    for (int k = 0; k < MLK_NV; ++k) v[k] = j < nparts ? __ldcg(&in[(size_t)j * MLK_NV + k]) : 0.0;
    mlk_block_partials<MLK_NV>(v, part);
  }
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&S->folded, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double t[MLK_NV];
  mlk_totals<MLK_NV>((int)gridDim.x, part, t);
  if (threadIdx.x != 0) return;
  S->folded = 0;
  const int its = S->its;
  if (its >= S->maxit) {
    S->reason = -3;
    S->done = 1;
    return;
  }
  const double dp = sqrt(t[4]);
  S->dp = dp;
  int reason = classify(dp, S->ttol, S->atol, S->rnorm0);
  if (!reason && S->stall_window > 0 && its > 0 && its % S->stall_window == 0) {
    if (dp > S->stall_ratio * S->dp_mark) reason = -20;
    else S->dp_mark = dp;
  }
  if (!reason) {
    const double m = S->nullsp ? t[3] / (double)n : 0.0;
    const double zr = t[0] - m * t[5], zq = t[1] - m * t[6], zw = t[2] - m * t[7];
    const double beta = its == 0 ? 0.0 : -zq / S->pq_old;
    const double pq = zw + 2.0 * beta * zq + beta * beta * S->pq_old;
    if (!(pq > 0.0)) {
      reason = pq == 0.0 ? 3 : -10;
    } else {
      S->m = m;
      S->beta = beta;
      S->alpha = zr / pq;
      S->pq_old = pq;
      S->its = its + 1;
    }
  }
  if (reason) {
    S->reason = reason;
    S->done = 1;
  }
}
// p = (z - m) + beta p, q = w + beta q, x += alpha p, r -= alpha q, then level 0's scaled
// right-hand side
template <class ZT>
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_update(MlArgs a, const ZT* z, MlkLevel L0,
                                                        const MlkState* S) {
  mlk_enter();
  if (S->done) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const double m = S->m, beta = S->beta, al = S->alpha;
  const double pi = ((double)__ldcg(&z[i]) - m) + beta * __ldcg(&a.p[i]);
  const double qi = __ldcg(&a.w[i]) + beta * __ldcg(&a.q[i]);
  const double ri = __ldcg(&a.r[i]) - al * qi;
  a.p[i] = pi;
  a.q[i] = qi;
  S->x[i] = __ldcg(&S->x[i]) + al * pi;
  a.r[i] = ri;
  mlk_start(L0, i, (float)ri);
}
// ---- true residual ||b - A x|| and the outcome in the status / result words
static __global__ void __launch_bounds__(MLK_TPB) k_mlk_true_resid(MlArgs a, double* part) {
  double v[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
    const double di = a.b[i] - ml_row64(a, i, (const double*)a.x);
    v[0] += di * di;
  }
  mlk_block_partials<1>(v, part);
}
static __global__ void k_mlk_finish(int nparts, const double* part, const MlkState* S, int* status, double* dout) {
  double t[1];
  mlk_totals<1>(nparts, part, t);
  if (threadIdx.x == 0) {
    dout[0] = sqrt(t[0]);
    dout[1] = S->dp;
    dout[2] = S->sn;
    status[0] = S->reason;
    status[1] = S->its;
  }
}

}  // namespace gpu
}  // namespace dpm
