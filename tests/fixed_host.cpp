// Host build of single operations of periodic-lbm_gb300/csrc (hybrid.cuh, fixed.cuh,
// df64.cuh) for test_fixed_host.py.
#include <stdint.h>
#include "hybrid.cuh"
using namespace plbm;

extern "C" double fx_to_double(int64_t T, int exact) {
  return exact ? hy::fixed_to_double_tr<hy::kScale, true>(T) : hy::fixed_to_double_tr(T);
}
// The shifted BGK of a cell, as the plugin's kernel and its out-of-line path take it: 0 in the
// kernel, 1 out of line in the fixed point, 2 left to the binary64 operator.
extern "C" int fx_bgk_shifted(double* f, double omega) {
  const double w[3] = {4.0 / 9.0, 1.0 / 9.0, 1.0 / 36.0};
  const hy::BgkParams p = hy::bgk_fma_params(omega, w);
  double v[9];
  for (int q = 0; q < 9; q++) v[q] = f[q];
  bool bad = false;
  hy::bgk_fma<true>(v, p, bad);
  if (bad) {
    for (int q = 0; q < 9; q++) v[q] = f[q];
    if (!hy::bgk_rest(v, p)) return 2;
  }
  for (int q = 0; q < 9; q++) f[q] = v[q];
  return bad;
}
// The nine shifted populations in units of 2^-59, as TRT and RR load them; 0 where one is out of range.
extern "C" int fx_load_shifted(const double* f, int64_t* F) {
  double v[9];
  int64_t G[9];
  bool bad = false, small;
  for (int q = 0; q < 9; q++) v[q] = f[q];
  hy::load_fixed<true, true>(v, G, bad, small);
  for (int q = 0; q < 9; q++) F[q] = G[q];
  return !bad;
}
