// Set-up of the aggregation multigrid preconditioner used by the multilevel flexible-CG
// pressure solve.
//
// Levels are built by pairwise aggregation along the strongest negative coupling (each pass
// pairs every still-unpaired row with its strongest unpaired neighbour, so a pass roughly
// halves the rows and follows the mesh anisotropy; `passes` passes make one level), with the
// Galerkin operator A_{l+1} = T^T A_l T of the piecewise-constant prolongation T.  Each
// smoothed level keeps its operator in FP32 padded ELL, 1/diagonal, the aggregate of every row
// and the member rows of every aggregate; the coarsest level keeps a dense FP32 inverse
// (regularised by the constant vector when the operator is singular).  No counterpart in the
// reference, whose pressure solve is PETSc CG with BoomerAMG or (block-)Jacobi
// (src/solver/pressure_backend_petsc.c:381-463); the Krylov stopping rule is kept identical.
#pragma once
#include <cstdint>
#include <memory>
#include <vector>

namespace dpm {

// Arrays that are filled in parallel right after they are sized: resize leaves them uninitialised,
// so that their pages are first touched by the threads that fill them.
template <class T>
struct RawAlloc : std::allocator<T> {
  template <class U>
  struct rebind {
    using other = RawAlloc<U>;
  };
  template <class U>
  void construct(U*) noexcept {}
  template <class U, class A, class... R>
  void construct(U* p, A&& a, R&&... r) {
    ::new ((void*)p) U(std::forward<A>(a), std::forward<R>(r)...);
  }
};
template <class T>
using Raw = std::vector<T, RawAlloc<T>>;

// An entry of a compressed row as the device reads it.
struct SaEntry {
  int col;
  float val;
};

constexpr int ML_MAX_LEVELS = 12;
constexpr int ML_MAX_DEGREE = 8;

struct MlLevel {
  int n = 0, W = 0, M = 0;        // rows, widest row (diagonal included), members per aggregate
  std::vector<float> dinv;        // [n]
  // The same operator as the smoother reads it: off-diagonal entries only, scaled by the row's
  // diagonal (D^-1 A = G + S), in ELL [Wo][n] padded with (own row, 0).  sv32 holds s_ij in FP32,
  // sv16 the IEEE binary16 bits of s_ij (round to nearest even); g32 / g16 the diagonal term of
  // the scaled row, 1 + sum_j (s_ij - stored s_ij), so that every stored row sums to the same
  // value as the exact one (a rounded off-diagonal would otherwise shift the near-null space).
  int Wo = 0;
  std::vector<int> ocol;          // [Wo][n]
  std::vector<float> sv32;        // [Wo][n]
  std::vector<unsigned short> sv16;  // [Wo][n]
  std::vector<float> g32, g16;    // [n]
  std::vector<float> diag;        // [n] a_ii
  std::vector<int> agg;           // [n] row of the next level this row belongs to
  std::vector<int> mem;           // [M][n_next] rows of this level in each aggregate, -1 padded
  double lmax = 0.0;              // estimate of the largest eigenvalue of D^-1 A
};

struct Multilevel {
  std::vector<MlLevel> lv;        // smoothed levels (level 0 = the fine operator)
  int nC = 0;                     // rows of the coarsest (directly solved) level
  std::vector<float> cinv;        // [nC][nC]
  std::vector<int> sizes;         // rows per level, coarsest last
  std::vector<int64_t> nnz;       // non-zeros per level, coarsest last
};

// One level of the smoothed-aggregation hierarchy, which the standalone-kernel form of the solve
// uses.  The transfer to the next level is P = (I - (omega / lmax) D^-1 A_F) T: the piecewise-
// constant prolongation T of the same pairwise aggregates, smoothed by one Jacobi step on A_F, the
// operator whose weak entries (-a_ij < theta max_k(-a_ik)) are lumped on the diagonal; the next
// operator is the Galerkin product P^T A P of the stored FP32 P, so no over-correction is needed.
// The aggregates of every level come from the unsmoothed Galerkin operators, which stay sparse.  The smoother reads
// the operator in the scaled off-diagonal form of MlLevel: the finest level in ELL, the others
// (about 30-40 entries per row) in compressed rows.
struct SaLevel {
  int n = 0, n_next = 0;
  int Wo = 0;                            // finest level: ELL width, ocol / sv32 / sv16 as in MlLevel
  Raw<int> ocol;
  Raw<float> sv32;
  Raw<unsigned short> sv16;
  Raw<int> off;                          // other levels: off-diagonal rows, s_ij = a_ij / a_ii
  Raw<SaEntry> ent;
  Raw<float> g, diag, dinv;              // [n] as in MlLevel (g for the stored values in use)
  Raw<int> poff;                         // P by rows of this level
  Raw<SaEntry> pent;
  Raw<int> roff;                         // P^T by rows of the next level, fine rows ascending
  Raw<SaEntry> rent;
  float oc = 1.0f;                       // factor of the coarse correction (1.6: unsmoothed transfer)
  double lmax = 0.0;
};

struct SaMultilevel {
  std::vector<SaLevel> lv;
  int nC = 0;
  std::vector<float> cinv;               // [nC][nC]
  std::vector<int> sizes;
};

// A as for build_multilevel.  passes: pairwise passes of the first coarsening (deeper levels take
// one more); with fewer than three, or where the smoothed Galerkin operator would hold more
// entries than the level itself, the transfer stays unsmoothed with the over-correction oc.
// half: the finest level's off-diagonals in binary16.  Coarsening stops at <= ncoarse rows.
// Fluid regions that do not touch one another and hold no Dirichlet row each have their own constant in the
// null space: the dense inverse lifts every one of them, and a region that has shrunk to one row gets no
// coarse correction (its 1/diagonal and its row of the inverse are zero).
int build_smoothed_multilevel(int n, int WA, const int* A_col, const double* A_val, bool nullsp, int passes,
                              double beta, double oc, bool half, int ncoarse, SaMultilevel& M);

// Compressed rows to slices of 32 rows, as wide as the slice's longest row: entry k of the slice's
// row r at soff[slice] + 32 k + r, short rows padded with (their first column, 0).  False when the
// slices do not fit 31-bit offsets.
bool slice_rows(int rows, const Raw<int>& off, const Raw<SaEntry>& ent, Raw<int>& soff, Raw<SaEntry>& sent);

// A in padded ELL [WA][n] (padding = (own row, 0)); nullsp = the operator has the constant null
// space.  Coarsening stops at <= ncoarse rows; returns 0, or a negative code when the coarsening
// stalls above max_dense rows or a factorisation fails.
int build_multilevel(int n, int WA, const int* A_col, const double* A_val, bool nullsp, int passes, double beta,
                     int ncoarse, int max_dense, Multilevel& M);

}  // namespace dpm
