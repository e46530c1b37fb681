// C entry points to the smoothed-aggregation builder (dopamine_b200/csrc/host/multilevel.cpp) for
// test_smoothed_multilevel_host.py: the hierarchy is built, then its arrays are read one by one.
#include "../dopamine_b200/csrc/host/multilevel.hpp"

namespace {
dpm::SaMultilevel M;
template <class V>
const void* give(const V& v, long long* n) {
  *n = (long long)v.size();
  return v.data();
}
}  // namespace

extern "C" {
int sa_build(int n, int width, const int* col, const double* val, int nullsp, int passes, int half, int* levels,
             int* rows_coarse) {
  const int rc = dpm::build_smoothed_multilevel(n, width, col, val, nullsp != 0, passes, 0.25, 1.6, half != 0, 1200, M);
  *levels = (int)M.lv.size();
  *rows_coarse = M.nC;
  return rc;
}
// n, n_next, ELL width; oc, lmax
void sa_level(int l, int* sizes, double* scalars) {
  const dpm::SaLevel& L = M.lv[l];
  sizes[0] = L.n; sizes[1] = L.n_next; sizes[2] = L.Wo;
  scalars[0] = L.oc; scalars[1] = L.lmax;
}
const void* sa_array(int l, int which, long long* n) {
  if (which == 0) return give(M.cinv, n);
  const dpm::SaLevel& L = M.lv[l];
  switch (which) {
    case 1: return give(L.ocol, n);
    case 2: return give(L.sv32, n);
    case 3: return give(L.sv16, n);
    case 4: return give(L.off, n);
    case 5: return give(L.ent, n);
    case 6: return give(L.g, n);
    case 7: return give(L.diag, n);
    case 8: return give(L.dinv, n);
    case 9: return give(L.poff, n);
    case 10: return give(L.pent, n);
    case 11: return give(L.roff, n);
    default: return give(L.rent, n);
  }
}
}
