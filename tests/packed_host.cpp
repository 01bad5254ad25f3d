// Host build of the binary32 operators that the kernels run on one cell or a pair
// (periodic-lbm_gb300/csrc/f32x2.cuh, df64.cuh) and of the fixed point's reciprocal,
// for test_packed_host.py.  SEED_ULPS: how far the reciprocal's seed, which the hardware
// gives within 1 ulp, is off the rounded quotient.
#include <math.h>
#include <stdint.h>
#include <string.h>
static float seed(float x) {
  const float r = 1.0f / x;
  int32_t b;
  memcpy(&b, &r, 4);
  b += SEED_ULPS;
  float s;
  memcpy(&s, &b, 4);
  return s;
}
#define PLBM_HOST_SEED(x) seed(x)
#include "f32x2.cuh"
#include "fixed.cuh"
using namespace plbm;

extern "C" void pk_rcp(const float* x, float* r, long n) {
  for (long i = 0; i < n; i++) r[i] = vrcp(x[i]);
}
extern "C" void pk_quot(const float* a, const float* x, float* q, long n) {
  for (long i = 0; i < n; i++) q[i] = vquot(a[i], x[i], vrcp(x[i]));
}
extern "C" int64_t pk_recip_fixed(int64_t R) { return hy::recip_fixed(R); }
extern "C" void pk_bgk(float* h, float omega, int f16) {
  float v[9];
  for (int q = 0; q < 9; q++) v[q] = h[q];
  if (f16) bgk_f16(v, omega);
  else bgk_dev(v, omega);
  for (int q = 0; q < 9; q++) h[q] = v[q];
}
