#include "multilevel.hpp"

#include <algorithm>
#include <cmath>

namespace dpm {
namespace {

// Compressed rows with ascending columns (diagonal included).
struct Csr {
  int n = 0;
  std::vector<int64_t> off;
  Raw<int> col;
  Raw<double> val;
};

// Rows are independent: counted in parallel, then filled in parallel at their prefix offsets.
Csr csr_from_ell(int n, int WA, const int* col, const double* val) {
  Csr A;
  A.n = n;
  A.off.assign(n + 1, 0);
  auto row_entries = [&](int i, int* cj, double* vj) {  // sorted, equal columns summed
    int m = 0;
    for (int s = 0; s < WA; ++s) {
      const int j = col[(size_t)s * n + i];
      const double v = val[(size_t)s * n + i];
      if (!(j == i || v != 0.0)) continue;
      int t = m++;
      while (t > 0 && cj[t - 1] > j) { cj[t] = cj[t - 1]; vj[t] = vj[t - 1]; --t; }  // stable
      cj[t] = j;
      vj[t] = v;
    }
    int u = 0;
    for (int k = 0; k < m; ++k) {
      if (u > 0 && cj[u - 1] == cj[k]) {  // padding slots share the own column
        vj[u - 1] += vj[k];
        continue;
      }
      cj[u] = cj[k];
      vj[u] = vj[k];
      ++u;
    }
    return u;
  };
  std::vector<int> cnt(n);
#pragma omp parallel for schedule(static)
  for (int i = 0; i < n; ++i) {
    int cj[64];
    double vj[64];
    cnt[i] = row_entries(i, cj, vj);
  }
  for (int i = 0; i < n; ++i) A.off[i + 1] = A.off[i] + cnt[i];
  A.col.resize(A.off[n]);
  A.val.resize(A.off[n]);
#pragma omp parallel for schedule(static)
  for (int i = 0; i < n; ++i) {
    int cj[64];
    double vj[64];
    const int u = row_entries(i, cj, vj);
    for (int k = 0; k < u; ++k) {
      A.col[A.off[i] + k] = cj[k];
      A.val[A.off[i] + k] = vj[k];
    }
  }
  return A;
}

// One pass of pairwise aggregation: rows in order; an unpaired row takes its strongest unpaired
// neighbour j (largest -a_ij, first in column order on ties) if -a_ij >= beta * max_k(-a_ik).
int pairwise(const Csr& A, double beta, std::vector<int>& agg) {
  agg.assign(A.n, -1);
  int na = 0;
  for (int i = 0; i < A.n; ++i) {
    if (agg[i] >= 0) continue;
    double mx = 0.0;
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k)
      if (A.col[k] != i) mx = std::max(mx, -A.val[k]);
    int best = -1;
    double bv = 0.0;
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
      const int j = A.col[k];
      if (j == i || agg[j] >= 0) continue;
      const double s = -A.val[k];
      if (s >= beta * mx && s > bv) {
        bv = s;
        best = j;
      }
    }
    agg[i] = na;
    if (best >= 0) agg[best] = na;
    ++na;
  }
  // A row left alone (its strong neighbours were all taken, typically around one strongly
  // coupled row) joins the aggregate of its strongest neighbour if that holds fewer than 3 rows,
  // so that a pass keeps coarsening on irregular meshes; 3 passes then give at most 27 rows.
  std::vector<int> size(na, 0);
  for (int i = 0; i < A.n; ++i) size[agg[i]]++;
  for (int i = 0; i < A.n; ++i) {
    if (size[agg[i]] != 1) continue;
    int best = -1;
    double bv = 0.0;
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
      const int j = A.col[k];
      if (j == i || size[agg[j]] >= 3 || -A.val[k] <= bv) continue;
      bv = -A.val[k];
      best = j;
    }
    if (best < 0) continue;
    size[agg[i]] = 0;
    agg[i] = agg[best];
    size[agg[best]]++;
  }
  // renumber the aggregates densely, in order of first appearance
  std::vector<int> remap(na, -1);
  int m = 0;
  for (int i = 0; i < A.n; ++i) {
    if (remap[agg[i]] < 0) remap[agg[i]] = m++;
    agg[i] = remap[agg[i]];
  }
  return m;
}

// Member rows of every aggregate, ascending.
void members(const std::vector<int>& agg, int na, std::vector<int64_t>& moff, std::vector<int>& mrow) {
  moff.assign(na + 1, 0);
  for (int a : agg) moff[a + 1]++;
  for (int a = 0; a < na; ++a) moff[a + 1] += moff[a];
  mrow.assign(agg.size(), 0);
  std::vector<int64_t> fill(moff.begin(), moff.end() - 1);
  for (size_t i = 0; i < agg.size(); ++i) mrow[fill[agg[i]]++] = (int)i;
}

// A_c = T^T A T for the aggregation T (row i -> column agg[i]); entries summed in the order
// (aggregate member ascending, fine column ascending), so the result is reproducible.
Csr galerkin(const Csr& A, const std::vector<int>& agg, int na) {
  std::vector<int64_t> moff;
  std::vector<int> mrow;
  members(agg, na, moff, mrow);
  Csr C;
  C.n = na;
  C.off.assign(na + 1, 0);
  // one aggregate's row: columns in order of first appearance, summed, then sorted by column
  auto agg_row = [&](int a, std::vector<int64_t>& pos, std::vector<int>& cols, std::vector<double>& vals,
                     std::vector<int>& order) {
    cols.clear();
    vals.clear();
    for (int64_t m = moff[a]; m < moff[a + 1]; ++m) {
      const int i = mrow[m];
      for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
        const int c = agg[A.col[k]];
        if (pos[c] < 0) {
          pos[c] = (int64_t)cols.size();
          cols.push_back(c);
          vals.push_back(0.0);
        }
        vals[pos[c]] += A.val[k];
      }
    }
    order.resize(cols.size());
    for (size_t k = 0; k < order.size(); ++k) order[k] = (int)k;
    std::sort(order.begin(), order.end(), [&](int x, int y) { return cols[x] < cols[y]; });
    for (int c : cols) pos[c] = -1;
  };
  std::vector<int64_t> cnt(na);
#pragma omp parallel
  {
    std::vector<int64_t> pos(na, -1);
    std::vector<int> cols, order;
    std::vector<double> vals;
#pragma omp for schedule(static)
    for (int a = 0; a < na; ++a) {
      agg_row(a, pos, cols, vals, order);
      cnt[a] = (int64_t)cols.size();
    }
  }
  for (int a = 0; a < na; ++a) C.off[a + 1] = C.off[a] + cnt[a];
  C.col.resize(C.off[na]);
  C.val.resize(C.off[na]);
#pragma omp parallel
  {
    std::vector<int64_t> pos(na, -1);
    std::vector<int> cols, order;
    std::vector<double> vals;
#pragma omp for schedule(static)
    for (int a = 0; a < na; ++a) {
      agg_row(a, pos, cols, vals, order);
      int64_t o = C.off[a];
      for (int k : order) {
        C.col[o] = cols[k];
        C.val[o] = vals[k];
        ++o;
      }
    }
  }
  return C;
}

// Largest eigenvalue of D^-1 A by `steps` power steps from a fixed start vector.  The norms are summed
// over fixed chunks of rows, then the chunks in order: the same value on any number of threads.
// noise: a hashed start vector; the smooth default start is close to the operator's constant mode and
// takes its 30 steps to leave it.
double lambda_max(const Csr& A, const std::vector<double>& dinv, int steps = 30, bool noise = false) {
  constexpr int CH = 16384;
  const int n = A.n, nch = (n + CH - 1) / CH;
  std::vector<double> v(n), w(n), pv(nch), pw(nch);
#pragma omp parallel for schedule(static)
  for (int i = 0; i < n; ++i)
    v[i] = noise ? (double)((uint32_t)i * 2654435761u >> 8) / 8388608.0 - 1.0 : 1.0 + 0.5 * std::sin(0.7 * i + 0.3);
  double lam = 0.0;
  for (int it = 0; it < steps; ++it) {
#pragma omp parallel for schedule(static)
    for (int c = 0; c < nch; ++c) {
      double nv = 0.0, nw = 0.0;
      const int i1 = std::min(n, (c + 1) * CH);
      for (int i = c * CH; i < i1; ++i) {
        double s = 0.0;
        for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) s += A.val[k] * v[A.col[k]];
        w[i] = dinv[i] * s;
        nv += v[i] * v[i];
        nw += w[i] * w[i];
      }
      pv[c] = nv;
      pw[c] = nw;
    }
    double nv = 0.0, nw = 0.0;
    for (int c = 0; c < nch; ++c) { nv += pv[c]; nw += pw[c]; }
    if (!(nw > 0.0)) return 1.0;
    lam = std::sqrt(nw / nv);
    const double sc = 1.0 / std::sqrt(nw);
#pragma omp parallel for schedule(static)
    for (int i = 0; i < n; ++i) v[i] = w[i] * sc;
  }
  return lam;
}

// Lower Cholesky factor in place; each entry is one inner product over a fixed range, so the
// result does not depend on the thread count.
bool cholesky_lower(std::vector<double>& a, int n) {
  for (int j = 0; j < n; ++j) {
    const double* rj = &a[(size_t)j * n];
    double d = rj[j];
    for (int k = 0; k < j; ++k) d -= rj[k] * rj[k];
    if (!(d > 0.0)) return false;
    d = std::sqrt(d);
    a[(size_t)j * n + j] = d;
#pragma omp parallel for schedule(static) if (n - j > 128)
    for (int i = j + 1; i < n; ++i) {
      const double* ri = &a[(size_t)i * n];
      double s = ri[j];
      for (int k = 0; k < j; ++k) s -= ri[k] * rj[k];
      a[(size_t)i * n + j] = s / d;
    }
  }
  return true;
}

// region: of every row, where the operator falls apart into several (null: one region); lift: of every
// region, whether its constant is in the null space.  The rows of skip (null: none) are closed regions
// on their own: their rows of the inverse are zero.
int dense_inverse(const Csr& A, bool nullsp, std::vector<float>& out, const std::vector<int>* region = nullptr,
                  const std::vector<char>* lift = nullptr, const std::vector<char>* skip = nullptr) {
  const int n = A.n;
  std::vector<double> a((size_t)n * n, 0.0);
  double tr = 0.0;
  for (int i = 0; i < n; ++i)
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
      a[(size_t)i * n + A.col[k]] += A.val[k];
      if (A.col[k] == i) tr += A.val[k];
    }
  if (region) {  // every closed region's own constant, as below
    std::vector<double> trr(lift->size(), 0.0);
    std::vector<int> m(lift->size(), 0);
    for (int i = 0; i < n; ++i) {
      if ((*skip)[i]) a[(size_t)i * n + i] = 1.0;  // alone in its row
      trr[(*region)[i]] += a[(size_t)i * n + i];
      m[(*region)[i]]++;
    }
    for (int i = 0; i < n; ++i) {
      const int c = (*region)[i];
      if (!(*lift)[c] || (*skip)[i]) continue;
      for (int j = 0; j < n; ++j)
        if ((*region)[j] == c) a[(size_t)i * n + j] += trr[c] / ((double)m[c] * m[c]);
    }
  } else if (nullsp) {  // constant mode lifted to the mean diagonal: (A + s 1 1^T) 1 = (tr / n) 1
    const double s = tr / ((double)n * n);
    for (auto& x : a) x += s;
  }
  if (!cholesky_lower(a, n)) return -4;
  // rows of yt: the columns of L^-1 (L y = e_c, zero above c), then A^-1 = L^-T L^-1 by inner
  // products of those rows
  std::vector<double> yt((size_t)n * n, 0.0);
#pragma omp parallel for schedule(dynamic, 8)
  for (int c = 0; c < n; ++c) {
    double* y = &yt[(size_t)c * n];
    for (int i = c; i < n; ++i) {
      const double* ri = &a[(size_t)i * n];
      double s = i == c ? 1.0 : 0.0;
      for (int k = c; k < i; ++k) s -= ri[k] * y[k];
      y[i] = s / ri[i];
    }
  }
  out.assign((size_t)n * n, 0.0f);
#pragma omp parallel for schedule(dynamic, 8)
  for (int i = 0; i < n; ++i)
    for (int j = 0; j <= i; ++j) {
      const double *yi = &yt[(size_t)i * n], *yj = &yt[(size_t)j * n];
      double s = 0.0;
      for (int k = i; k < n; ++k) s += yi[k] * yj[k];
      out[(size_t)i * n + j] = (float)s;
      out[(size_t)j * n + i] = (float)s;
    }
  if (region)
    for (int i = 0; i < n; ++i)
      if ((*skip)[i]) out[(size_t)i * n + i] = 0.0f;
  return 0;
}

// IEEE binary16 bits of a finite double, round to nearest even (subnormals included; values
// beyond the largest finite half saturate to it).
unsigned short half_bits(double v) {
  const unsigned short sign = std::signbit(v) ? 0x8000 : 0;
  double a = std::fabs(v);
  if (a >= 65504.0) return sign | 0x7bff;
  if (a < std::ldexp(1.0, -24) * 0.5) return sign;
  int e;
  std::frexp(a, &e);  // a = m 2^e, m in [0.5, 1)
  int ex = e - 1;     // a = (1.f) 2^ex
  if (ex < -14) ex = -14;  // subnormal range: fixed exponent, 10-bit fraction of 2^-24 units
  const double q = std::ldexp(a, 10 - ex);  // value in units of the last place
  double r = std::nearbyint(q);             // round half to even (default rounding mode)
  unsigned mant = (unsigned)r;
  if (mant >= 2048) { mant >>= 1; ex += 1; }  // rounding carried into the next binade
  if (ex > 15) return sign | 0x7bff;
  if (mant < 1024) return sign | (unsigned short)mant;  // subnormal (ex == -14)
  return sign | (unsigned short)(((ex + 15) << 10) | (mant - 1024));
}

double half_value(unsigned short h) {
  const int e = (h >> 10) & 0x1f, f = h & 0x3ff;
  const double m = e == 0 ? std::ldexp((double)f, -24) : std::ldexp(1024.0 + f, e - 25);
  return (h & 0x8000) ? -m : m;
}

MlLevel make_level(const Csr& A, const std::vector<int>& agg, int na, int& rc) {
  MlLevel L;
  rc = 0;
  L.n = A.n;
  for (int i = 0; i < A.n; ++i) L.W = std::max<int>(L.W, (int)(A.off[i + 1] - A.off[i]));
  L.dinv.resize(A.n);
  std::vector<double> dinv(A.n, 0.0);
  int bad = 0;
#pragma omp parallel for schedule(static) reduction(| : bad)
  for (int i = 0; i < A.n; ++i) {
    double dg = 0.0;
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k)
      if (A.col[k] == i) dg = A.val[k];
    if (!(dg > 0.0)) bad = 1;
    dinv[i] = dg > 0.0 ? 1.0 / dg : 0.0;
    L.dinv[i] = (float)dinv[i];
  }
  if (bad) rc = -5;
  L.lmax = lambda_max(A, dinv);
  // scaled off-diagonal form of the smoother
  for (int i = 0; i < A.n; ++i) L.Wo = std::max<int>(L.Wo, (int)(A.off[i + 1] - A.off[i]) - 1);
  L.Wo = std::max(L.Wo, 1);
  L.ocol.resize((size_t)L.Wo * A.n);
  L.sv32.assign((size_t)L.Wo * A.n, 0.0f);
  L.sv16.assign((size_t)L.Wo * A.n, 0);
  L.g32.resize(A.n);
  L.g16.resize(A.n);
  L.diag.resize(A.n);
#pragma omp parallel for schedule(static)
  for (int i = 0; i < A.n; ++i) {
    int s = 0;
    double d32 = 1.0, d16 = 1.0;
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
      if (A.col[k] == i) continue;
      const double sij = A.val[k] * dinv[i];
      const float f = (float)sij;
      const unsigned short h = half_bits(sij);
      L.ocol[(size_t)s * A.n + i] = A.col[k];
      L.sv32[(size_t)s * A.n + i] = f;
      L.sv16[(size_t)s * A.n + i] = h;
      d32 += sij - (double)f;
      d16 += sij - half_value(h);
      ++s;
    }
    for (; s < L.Wo; ++s) L.ocol[(size_t)s * A.n + i] = i;
    L.g32[i] = (float)d32;
    L.g16[i] = (float)d16;
    L.diag[i] = (float)(dinv[i] > 0.0 ? 1.0 / dinv[i] : 0.0);
  }
  L.agg = agg;
  std::vector<int64_t> moff;
  std::vector<int> mrow;
  members(agg, na, moff, mrow);
  for (int a = 0; a < na; ++a) L.M = std::max<int>(L.M, (int)(moff[a + 1] - moff[a]));
  L.mem.assign((size_t)L.M * na, -1);
  for (int a = 0; a < na; ++a)
    for (int64_t m = moff[a]; m < moff[a + 1]; ++m) L.mem[(size_t)(m - moff[a]) * na + a] = mrow[m];
  return L;
}

// `passes` pairwise passes on A: the aggregate of every row and the operator T^T A T.
Csr aggregate(const Csr& A, double beta, int passes, std::vector<int>& agg_tot) {
  Csr Ac;
  for (int p = 0; p < passes; ++p) {
    std::vector<int> agg;
    const Csr& from = p == 0 ? A : Ac;
    const int na = pairwise(from, beta, agg);
    Csr next = galerkin(from, agg, na);
    if (p == 0) agg_tot = agg;
    else {
#pragma omp parallel for schedule(static)
      for (int i = 0; i < A.n; ++i) agg_tot[i] = agg[agg_tot[i]];
    }
    Ac = std::move(next);
  }
  return Ac;
}

// Smoothed prolongation by rows: row i of (I - w D^-1 A_F) T, columns in order of first appearance.
void smooth_prolongation(const Csr& A, const std::vector<double>& dinv, const std::vector<int>& agg, double w,
                         double theta, Raw<int>& off, Raw<SaEntry>& ent) {
  // one row into c / v; returns its entries
  auto row = [&](int i, std::vector<int>& c, std::vector<double>& v) {
    double mx = 0.0, dg = 0.0;
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k)
      if (A.col[k] != i) mx = std::max(mx, -A.val[k]);
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k)
      if (A.col[k] == i || -A.val[k] < theta * mx) dg += A.val[k];
    c.assign(1, agg[i]);
    v.assign(1, 1.0 - w * dg * dinv[i]);
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
      const int j = A.col[k];
      if (j == i || -A.val[k] < theta * mx) continue;
      size_t t = 0;
      while (t < c.size() && c[t] != agg[j]) ++t;
      if (t == c.size()) {
        c.push_back(agg[j]);
        v.push_back(0.0);
      }
      v[t] -= w * A.val[k] * dinv[i];
    }
    return (int)c.size();
  };
  off.resize((size_t)A.n + 1);
  off[0] = 0;
#pragma omp parallel
  {
    std::vector<int> c;
    std::vector<double> v;
#pragma omp for schedule(static)
    for (int i = 0; i < A.n; ++i) off[i + 1] = row(i, c, v);
  }
  for (int i = 0; i < A.n; ++i) off[i + 1] += off[i];
  ent.resize(off[A.n]);
#pragma omp parallel
  {
    std::vector<int> c;
    std::vector<double> v;
#pragma omp for schedule(static)
    for (int i = 0; i < A.n; ++i) {
      const int m = row(i, c, v);
      for (int k = 0; k < m; ++k) ent[off[i] + k] = {c[k], (float)v[k]};
    }
  }
}

// P^T by rows (fine rows ascending in each): slots taken concurrently, then every row sorted, so
// the result is the same on any thread count.
void transpose(int n, int na, const Raw<int>& off, const Raw<SaEntry>& ent, Raw<int>& toff, Raw<SaEntry>& tent) {
  std::vector<int> cnt(na, 0);
#pragma omp parallel for schedule(static)
  for (int k = 0; k < off[n]; ++k) {
#pragma omp atomic
    cnt[ent[k].col]++;
  }
  toff.resize((size_t)na + 1);
  toff[0] = 0;
  for (int a = 0; a < na; ++a) {
    toff[a + 1] = toff[a] + cnt[a];
    cnt[a] = toff[a];
  }
  tent.resize(off[n]);
#pragma omp parallel for schedule(static)
  for (int i = 0; i < n; ++i)
    for (int k = off[i]; k < off[i + 1]; ++k) {
      int slot;
#pragma omp atomic capture
      slot = cnt[ent[k].col]++;
      tent[slot] = {i, ent[k].val};
    }
#pragma omp parallel for schedule(static)
  for (int a = 0; a < na; ++a)
    std::sort(tent.begin() + toff[a], tent.begin() + toff[a + 1],
              [](const SaEntry& x, const SaEntry& y) { return x.col < y.col; });
}

// Rows formed one by one by fn(i, add), add(column, value) accumulating the row's entries: a chunk
// of rows per thread at a time, each row's columns sorted.  Every row is formed in a fixed order.
template <class Fn>
Csr accumulate_rows(int n, int ncol, Fn fn) {
  Csr C;
  C.n = n;
  const int CH = std::max(16, std::min(4096, n / 512));
  const int nch = (n + CH - 1) / CH;
  std::vector<Raw<int>> cc(nch);
  std::vector<Raw<double>> vv(nch);
  C.off.assign((size_t)n + 1, 0);
#pragma omp parallel
  {
    std::vector<int> pos(ncol, -1), cols, order;
    std::vector<double> vals;
    auto add = [&](int c, double v) {
      if (pos[c] < 0) {
        pos[c] = (int)cols.size();
        cols.push_back(c);
        vals.push_back(0.0);
      }
      vals[pos[c]] += v;
    };
#pragma omp for schedule(dynamic, 1)
    for (int ch = 0; ch < nch; ++ch) {
      const int i1 = std::min(n, (ch + 1) * CH);
      for (int i = ch * CH; i < i1; ++i) {
        cols.clear();
        vals.clear();
        fn(i, add);
        order = cols;
        std::sort(order.begin(), order.end());
        for (int c : order) {
          cc[ch].push_back(c);
          vv[ch].push_back(vals[pos[c]]);
        }
        for (int c : cols) pos[c] = -1;
        C.off[i + 1] = (int64_t)cols.size();
      }
    }
  }
  for (int i = 0; i < n; ++i) C.off[i + 1] += C.off[i];
  C.col.resize(C.off[n]);
  C.val.resize(C.off[n]);
#pragma omp parallel for schedule(dynamic, 1)
  for (int ch = 0; ch < nch; ++ch) {
    std::copy(cc[ch].begin(), cc[ch].end(), C.col.begin() + C.off[(size_t)ch * CH]);
    std::copy(vv[ch].begin(), vv[ch].end(), C.val.begin() + C.off[(size_t)ch * CH]);
  }
  return C;
}

// P^T A P.  Short rows of A (the finest level): in one product per coarse row, so that A P, the
// largest array, is never stored; long ones: P^T (A P), a quarter of the multiplications.
Csr galerkin_smoothed(const Csr& A, int na, const Raw<int>& poff, const Raw<SaEntry>& pent, const Raw<int>& roff,
                      const Raw<SaEntry>& rent) {
  if (A.off[A.n] < 16 * (int64_t)A.n)
    return accumulate_rows(na, na, [&](int a, auto& add) {
      for (int m = roff[a]; m < roff[a + 1]; ++m) {
        const int i = rent[m].col;
        for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
          const double w = (double)rent[m].val * A.val[k];
          const int j = A.col[k];
          for (int q = poff[j]; q < poff[j + 1]; ++q) add(pent[q].col, w * (double)pent[q].val);
        }
      }
    });
  const Csr AP = accumulate_rows(A.n, na, [&](int i, auto& add) {
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
      const int j = A.col[k];
      for (int q = poff[j]; q < poff[j + 1]; ++q) add(pent[q].col, A.val[k] * (double)pent[q].val);
    }
  });
  return accumulate_rows(na, na, [&](int a, auto& add) {
    for (int m = roff[a]; m < roff[a + 1]; ++m) {
      const int i = rent[m].col;
      for (int64_t k = AP.off[i]; k < AP.off[i + 1]; ++k) add(AP.col[k], (double)rent[m].val * AP.val[k]);
    }
  });
}

// The smoother's scaled off-diagonal form of A: ELL (finest level) or compressed rows.
int scaled_rows(const Csr& A, const std::vector<double>& dinv, bool ell, bool half, SaLevel& L) {
  const int n = A.n;
  L.n = n;
  L.g.resize(n);
  L.diag.resize(n);
  L.dinv.resize(n);
  if (ell) {
    L.Wo = 1;
    for (int i = 0; i < n; ++i) L.Wo = std::max<int>(L.Wo, (int)(A.off[i + 1] - A.off[i]) - 1);
    L.ocol.resize((size_t)L.Wo * n);
    if (half) L.sv16.resize((size_t)L.Wo * n);
    else L.sv32.resize((size_t)L.Wo * n);
  } else {
    if (A.off[n] - n > 2000000000LL) return -6;
    L.off.resize((size_t)n + 1);
    for (int i = 0; i <= n; ++i) L.off[i] = (int)(A.off[i] - i);  // one diagonal entry per row left out
    L.ent.resize(L.off[n]);
  }
#pragma omp parallel for schedule(static)
  for (int i = 0; i < n; ++i) {
    int s = 0;
    double d = 1.0;
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
      if (A.col[k] == i) continue;
      const double sij = A.val[k] * dinv[i];
      if (ell) {
        const size_t e = (size_t)s * n + i;
        L.ocol[e] = A.col[k];
        if (half) {
          L.sv16[e] = half_bits(sij);
          d += sij - half_value(L.sv16[e]);
        } else {
          L.sv32[e] = (float)sij;
          d += sij - (double)L.sv32[e];
        }
      } else {
        const size_t e = (size_t)L.off[i] + s;
        L.ent[e] = {A.col[k], (float)sij};
        d += sij - (double)L.ent[e].val;
      }
      ++s;
    }
    if (ell)
      for (; s < L.Wo; ++s) {
        const size_t e = (size_t)s * n + i;
        L.ocol[e] = i;
        if (half) L.sv16[e] = 0;
        else L.sv32[e] = 0.0f;
      }
    L.g[i] = (float)d;
    L.diag[i] = dinv[i] > 0.0 ? (float)(1.0 / dinv[i]) : 0.0f;  // 0: a closed region on its own
    L.dinv[i] = (float)dinv[i];
  }
  return 0;
}

// A region whose sum of entries is this small a part of its diagonals is closed: no Dirichlet row holds
// its constant.  The sums of closed regions are rounding (below 1e-15); one Dirichlet face on a region
// of 10^7 cells is about 1e-8.
constexpr double CLOSED = 1e-11;

// Of every row of U = T^T A T: whether it is a closed region on its own; empty when no row is.  before:
// the same of A's rows (their diagonals are rounding already).
std::vector<char> closed_rows(const Csr& A, const Csr& U, const std::vector<int>& agg,
                              const std::vector<char>& before) {
  std::vector<char> closed;
  auto alone = [](const Csr& C, int i) { return C.off[i + 1] - C.off[i] == 1; };
  for (int c = 0; c < U.n; ++c)
    if (alone(U, c) && closed.empty()) closed.assign(U.n, 0);
  if (closed.empty()) return closed;
  std::vector<double> dg(U.n, 0.0);
  for (int i = 0; i < A.n; ++i)
    for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k)
      if (A.col[k] == i) dg[agg[i]] += A.val[k];
  for (int c = 0; c < U.n; ++c)
    closed[c] = alone(U, c) && U.val[U.off[c]] <= CLOSED * dg[c];
  for (size_t i = 0; i < before.size(); ++i)
    if (before[i]) closed[agg[i]] = 1;
  return closed;
}

// Regions of A that do not touch one another, numbered in order of their first row.
int regions(const Csr& A, std::vector<int>& region) {
  region.assign(A.n, -1);
  int nr = 0;
  std::vector<int> todo;
  for (int r = 0; r < A.n; ++r) {
    if (region[r] >= 0) continue;
    region[r] = nr;
    todo.assign(1, r);
    while (!todo.empty()) {
      const int i = todo.back();
      todo.pop_back();
      for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k)
        if (region[A.col[k]] < 0) {
          region[A.col[k]] = nr;
          todo.push_back(A.col[k]);
        }
    }
    ++nr;
  }
  return nr;
}

}  // namespace

int build_smoothed_multilevel(int n, int WA, const int* A_col, const double* A_val, bool nullsp, int passes,
                              double beta, double oc, bool half, int ncoarse, SaMultilevel& M) {
  constexpr double OMEGA = 1.5, THETA = 0.25;
  if (n < 1 || WA < 1 || WA > 64 || passes < 1 || ncoarse < 1) return -1;
  M = SaMultilevel{};
  Csr A = csr_from_ell(n, WA, A_col, A_val), U;  // U: the unsmoothed Galerkin operator of this level
  // Rows that are closed regions on their own (empty: none).  Such a row's constant is all it has, which no
  // level can correct: its 1/diagonal is taken as zero.
  std::vector<char> closed;
  for (;;) {
    const Csr& from = M.lv.empty() ? A : U;
    M.sizes.push_back(A.n);
    if (A.n <= ncoarse) break;
    if ((int)M.lv.size() >= ML_MAX_LEVELS) return -3;
    std::vector<double> dinv(A.n, 0.0);
    int bad = 0;
    double bound = 0.0;
#pragma omp parallel for schedule(static) reduction(| : bad) reduction(max : bound)
    for (int i = 0; i < A.n; ++i) {
      double dg = 0.0, s = 0.0;
      int nd = 0;
      for (int64_t k = A.off[i]; k < A.off[i + 1]; ++k) {
        s += std::fabs(A.val[k]);
        if (A.col[k] == i) {
          dg = A.val[k];
          ++nd;
        }
      }
      if (!closed.empty() && closed[i]) continue;
      if (!(dg > 0.0) || nd != 1) {
        bad = 1;
        continue;
      }
      dinv[i] = 1.0 / dg;
      bound = std::max(bound, s * dinv[i]);
    }
    if (bad) return -5;
    SaLevel L;
    // The finest level's rows are diagonally dominant, where Gershgorin's bound is close (2 against
    // 1.85-1.99 on the hex meshes); on the others (2-4 against 1.3-2) power steps, which have been
    // seen to stop up to 15 % short of the largest eigenvalue.  Chebyshev steps on 1.1 lmax still
    // damp up to 1.21 lmax.
    L.lmax = M.lv.empty() ? 0.97 * bound : 1.08 * lambda_max(A, dinv, 20, true);
    int rc = scaled_rows(A, dinv, M.lv.empty(), half, L);
    if (rc) return rc;
    std::vector<int> agg;
    int np = passes;
    if (!M.lv.empty()) {
      np = passes + 1;
      // a coarsening that can reach the dense level does: on a 300 000-cell mesh 15 iterations of 16
      // launches instead of 13 of 22, when every launch on the coarse levels costs its latency
      if (A.n <= 32 * ncoarse)
        for (np = 1; np < 5 && (A.n >> np) > ncoarse;) ++np;
    }
    Csr Un = aggregate(from, beta, np, agg);
    const int na = Un.n;
    if (na > 0.85 * A.n) return -2;
    Csr C;
    bool smoothed = passes >= 3;
    if (smoothed) {
      smooth_prolongation(A, dinv, agg, OMEGA / L.lmax, THETA, L.poff, L.pent);
      transpose(A.n, na, L.poff, L.pent, L.roff, L.rent);
      C = galerkin_smoothed(A, na, L.poff, L.pent, L.roff, L.rent);
      smoothed = C.off[na] <= A.off[A.n];
    }
    if (!smoothed) {
      L.oc = (float)oc;
      L.poff.resize((size_t)A.n + 1);
      L.pent.resize(A.n);
      for (int i = 0; i <= A.n; ++i) L.poff[i] = i;
      for (int i = 0; i < A.n; ++i) L.pent[i] = {agg[i], 1.0f};
      transpose(A.n, na, L.poff, L.pent, L.roff, L.rent);
      C = galerkin(A, agg, na);
    }
    L.n_next = na;
    closed = closed_rows(from, Un, agg, closed);
    M.lv.push_back(std::move(L));
    A = std::move(C);
    U = std::move(Un);
  }
  M.nC = A.n;
  const Csr& from = M.lv.empty() ? A : U;
  std::vector<int> region;
  const int nr = regions(from, region);
  if (nr == 1) return dense_inverse(A, nullsp, M.cinv);
  std::vector<double> sum(nr, 0.0), dg(nr, 0.0);
  for (int i = 0; i < A.n; ++i)
    for (int64_t k = from.off[i]; k < from.off[i + 1]; ++k) {
      sum[region[i]] += from.val[k];
      if (from.col[k] == i) dg[region[i]] += from.val[k];
    }
  std::vector<char> lift(nr);
  for (int c = 0; c < nr; ++c) lift[c] = sum[c] <= CLOSED * dg[c];
  closed.resize(A.n, 0);
  return dense_inverse(A, nullsp, M.cinv, &region, &lift, &closed);
}

bool slice_rows(int rows, const Raw<int>& off, const Raw<SaEntry>& ent, Raw<int>& soff, Raw<SaEntry>& sent) {
  const int ns = (rows + 31) / 32;
  soff.resize((size_t)ns + 1);
  int64_t total = 0;
  for (int s = 0; s < ns; ++s) {
    int w = 0;
    for (int i = 32 * s; i < std::min(rows, 32 * s + 32); ++i) w = std::max(w, off[i + 1] - off[i]);
    soff[s] = (int)total;
    total += 32 * (int64_t)w;
    if (total > 2147483647) return false;
  }
  soff[ns] = (int)total;
  sent.resize(total);
#pragma omp parallel for schedule(static)
  for (int s = 0; s < ns; ++s) {
    const int w = (soff[s + 1] - soff[s]) / 32;
    for (int r = 0; r < 32; ++r) {
      const int i = 32 * s + r, m0 = i < rows ? off[i] : 0, mn = i < rows ? off[i + 1] - m0 : 0;
      for (int k = 0; k < w; ++k)
        sent[soff[s] + 32 * (int64_t)k + r] = k < mn ? ent[m0 + k] : SaEntry{mn > 0 ? ent[m0].col : 0, 0.0f};
    }
  }
  return true;
}

int build_multilevel(int n, int WA, const int* A_col, const double* A_val, bool nullsp, int passes, double beta,
                     int ncoarse, int max_dense, Multilevel& M) {
  if (n < 1 || WA < 1 || WA > 64 || passes < 1 || ncoarse < 1) return -1;
  M = Multilevel{};
  Csr A = csr_from_ell(n, WA, A_col, A_val);
  for (;;) {
    M.sizes.push_back(A.n);
    M.nnz.push_back((int64_t)A.col.size());
    if (A.n <= ncoarse) break;
    if ((int)M.lv.size() >= ML_MAX_LEVELS) {
      if (A.n > max_dense) return -3;
      break;
    }
    std::vector<int> agg_tot;
    Csr Ac;
    for (int p = 0; p < passes; ++p) {
      std::vector<int> agg;
      const Csr& from = p == 0 ? A : Ac;
      const int na = pairwise(from, beta, agg);
      Csr next = galerkin(from, agg, na);
      if (p == 0) agg_tot = agg;
      else
        for (int i = 0; i < A.n; ++i) agg_tot[i] = agg[agg_tot[i]];
      Ac = std::move(next);
    }
    if (Ac.n > 0.85 * A.n) {  // coarsening stalled: solve this level directly if it is small enough
      if (A.n > max_dense) return -2;
      break;
    }
    int rc = 0;
    M.lv.push_back(make_level(A, agg_tot, Ac.n, rc));
    if (rc) return rc;
    A = std::move(Ac);
  }
  M.nC = A.n;
  return dense_inverse(A, nullsp, M.cinv);
}

}  // namespace dpm
