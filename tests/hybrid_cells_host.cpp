// Host build of the fixed-point binary64 collisions of
// periodic-lbm_gb300/csrc/hybrid.cuh for the CPU tests in
// test_hybrid_cells_host.py: the same source the kernels compile.
#include <stdint.h>
#include "hybrid.cuh"
using namespace plbm;

// One cell, kind 0 BGK, 1 TRT, 2 RR; returns 1 when the cell is out of range.
extern "C" int hc_collide(int kind, int shifted, double* f, double omega, double lambda_d) {
  const double w[3] = {4.0 / 9.0, 1.0 / 9.0, 1.0 / 36.0};
  double v[9];
  for (int q = 0; q < 9; q++) v[q] = f[q];
  bool bad = false;
  if (kind == 0) {
    const hy::BgkParams p = hy::bgk_fma_params(omega, w);
    if (shifted) hy::bgk_fma<true>(v, p, bad);
    else hy::bgk_fma<false>(v, p, bad);
  } else if (kind == 1) {
    const hy::TrtFmaParams p = hy::trt_fma_params(omega, lambda_d, w);
    if (shifted) hy::trt_fma<true>(v, p, bad);
    else hy::trt_fma<false>(v, p, bad);
  } else {
    const hy::BgkParams p = hy::bgk_fma_params(1.0, w);
    const hy::RrParams r = hy::rr_fma_params(omega);
    if (shifted) hy::rr_fma<true>(v, r, p, bad);
    else hy::rr_fma<false>(v, r, p, bad);
  }
  for (int q = 0; q < 9; q++) f[q] = v[q];
  return bad;
}
// The unshifted forms that end in hy::finish.
extern "C" int hc_collide_quick(int kind, double* f, double omega, double lambda_d) {
  const double w[3] = {4.0 / 9.0, 1.0 / 9.0, 1.0 / 36.0};
  double v[9];
  for (int q = 0; q < 9; q++) v[q] = f[q];
  bool bad = false;
  if (kind == 0) hy::bgk_fma<false, true>(v, hy::bgk_fma_params(omega, w), bad);
  else if (kind == 1) hy::trt_fma<false, true>(v, hy::trt_fma_params(omega, lambda_d, w), bad);
  else hy::rr_fma<false, true>(v, hy::rr_fma_params(omega), hy::bgk_fma_params(1.0, w), bad);
  for (int q = 0; q < 9; q++) f[q] = v[q];
  return bad;
}
extern "C" int64_t hc_mulh64(int64_t a, int64_t b) { return hy::mulh64(a, b); }
extern "C" int64_t hc_recip(int64_t R) { return hy::recip_fixed(R); }
