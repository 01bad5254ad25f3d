// f32x2.cuh -- a pair of binary32 values in one 64-bit register, with the packed
// operations of sm_100 and later (one instruction for both, each value rounded
// as by the scalar operation), and the same operations on a single float, so that
// one template serves a kernel with one cell per thread and one with two and gives
// the same bits in both.  GB300 retires the packed operations at half the issue
// slots of the scalar ones and the same 128 values per clock and SM (measured).
#pragma once
#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif
#include <stdint.h>
#include "df64.cuh"

namespace plbm {

struct f32x2 {
  unsigned long long v;
};
DF_HD f32x2 pack2(float lo, float hi) {
  return {((unsigned long long)df::f2u(hi) << 32) | (unsigned long long)df::f2u(lo)};
}
template <>
DF_HD f32x2 vset<f32x2>(float c) { return pack2(c, c); }
#ifdef __CUDACC__
__device__ __forceinline__ float lo2(f32x2 a) {
  return __uint_as_float((unsigned)a.v);
}
__device__ __forceinline__ float hi2(f32x2 a) {
  return __uint_as_float((unsigned)(a.v >> 32));
}

__device__ __forceinline__ f32x2 vadd(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32x2 vsub(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32x2 vmul(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f32x2 vfma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// a b, not to be contracted into a sum that follows: ptxas fuses a packed product and
// sum, .rn or not; a fused product and sum of its own is left alone (+ -0 changes no
// product, not even the sign of a zero).
__device__ __forceinline__ f32x2 vprod(f32x2 a, f32x2 b) { return vfma(a, b, vset<f32x2>(-0.0f)); }
__device__ __forceinline__ f32x2 rcp_seed(f32x2 x) { return pack2(rcp_seed(lo2(x)), rcp_seed(hi2(x))); }
#endif
DF_HD float vprod(float a, float b) { return vmul(a, b); }

// a / x with r = vrcp(x): the product and its exact residual added back
// (Markstein 1990), within half an ulp and a hair.
template <typename V>
DF_HD V vquot(V a, V x, V r) {
  const V q = vmul(a, r);
  const V e = vfma(vsub(vset<V>(0.0f), x), q, a);
  return vfma(e, r, q);
}

// BGK of the shifted populations h = f - w in binary32 (sim/sim.F90:445-499
// with collide_bgk's equilibrium), h' = h + omega (heq - h).  With j = rho u,
//   heq_q = w_q (dr + 4.5 (c.j)(c.u) - 1.5 j.u + 3 c.j),  dr = sum h:
// the even part of a pair (q, -q) once, the odd part added and subtracted; 66
// operations.  The O(h) terms come from dr and j themselves, not from rho - 1 and
// rho u, which lose dr's low bits to the rounding of rho = 1 + dr.
template <typename V>
DF_HD void bgk_dev(V (&h)[9], float omega) {
  // the three binary32 weights share one relative error, 7e-9, with which mass and
  // momentum drift; 3 w c.j with a rounded 3 w would drift four times as fast
  const float w0 = 4.0f / 9.0f, ws = 1.0f / 9.0f, wd = 1.0f / 36.0f;
  const V s13 = vadd(h[1], h[3]), s24 = vadd(h[2], h[4]), s57 = vadd(h[5], h[7]), s68 = vadd(h[6], h[8]);
  const V d13 = vsub(h[1], h[3]), d24 = vsub(h[2], h[4]), d57 = vsub(h[5], h[7]), d86 = vsub(h[8], h[6]);
  const V dr = vadd(vadd(vadd(s57, s68), vadd(s13, s24)), h[0]);
  const V jx = vadd(vadd(d57, d86), d13), jy = vadd(vsub(d57, d86), d24);
  const V rho = vadd(dr, vset<V>(1.0f));
  const V r = vrcp(rho);
  const V ux = vquot(jx, rho, r), uy = vquot(jy, rho, r);
  const V base = vfma(vset<V>(-1.5f), vfma(jy, uy, vmul(jx, ux)), dr);
  // h' = h - omega (h - w heq'), all fused: no plain product feeds a sum or a
  // difference (ptxas contracts a packed product and difference, .rn or not).
  const V mom = vset<V>(-omega);
  h[0] = vfma(mom, vfma(vset<V>(-w0), base, h[0]), h[0]);
  auto pair = [&](int a, int b, V u, V j, float w) {
    const V even = vfma(vmul(vset<V>(4.5f), j), u, base);
    const V ha = vfma(vset<V>(3.0f), j, even), hb = vfma(vset<V>(-3.0f), j, even);
    h[a] = vfma(mom, vfma(vset<V>(-w), ha, h[a]), h[a]);
    h[b] = vfma(mom, vfma(vset<V>(-w), hb, h[b]), h[b]);
  };
  pair(1, 3, ux, jx, ws);
  pair(2, 4, uy, jy, ws);
  pair(5, 7, vadd(ux, uy), vadd(jx, jy), wd);
  pair(8, 6, vsub(ux, uy), vsub(jx, jy), wd);
}

// BGK on binary16 deviations kept in their stored scale, H = 2^15 h: the scale
// enters the constants instead of 18 multiplies per cell.  rho = 1 + 2^-15 sum H,
// u = j / rho, and H' = (1 - omega) H + omega Heq with Heq = w (sum H + 2^15 rho P),
// P = -1.5 u^2 + 3 c.u + 4.5 (c.u)^2 -- the shifted equilibrium of coll_bgk_shift,
// scaled, with omega w folded into the two per-cell factors; 64 operations and the
// division.  u takes the approximate division (2 ulp): binary16 storage rounds the
// populations to 2^-11 relative, far above it.  Each operation rounds on its own, so
// that one cell per thread, two per thread and a pass of several steps give the same
// bits: an operator that rounds otherwise lands on another binary16 value now and
// then, 2^-11 of h apart.
DF_HD float f16_inv_rho(float rho) {
#ifdef __CUDA_ARCH__
  return __fdividef(1.0f / 32768.0f, rho);
#else
  return 1.0f / 32768.0f / rho;
#endif
}
#ifdef __CUDACC__
__device__ __forceinline__ f32x2 f16_inv_rho(f32x2 rho) { return pack2(f16_inv_rho(lo2(rho)), f16_inv_rho(hi2(rho))); }
#endif
template <typename V>
DF_HD void bgk_f16(V (&H)[9], float omega) {
  const V s13 = vadd(H[1], H[3]), s24 = vadd(H[2], H[4]), s57 = vadd(H[5], H[7]), s68 = vadd(H[6], H[8]);
  const V d13 = vsub(H[1], H[3]), d24 = vsub(H[2], H[4]), d57 = vsub(H[5], H[7]), d86 = vsub(H[8], H[6]);
  const V dh = vadd(vadd(vadd(s57, s68), vadd(s13, s24)), H[0]);
  const V rho = vfma(dh, vset<V>(1.0f / 32768.0f), vset<V>(1.0f));
  const V r = f16_inv_rho(rho);
  const V ux = vprod(vadd(vadd(d57, d86), d13), r), uy = vprod(vadd(vsub(d57, d86), d24), r);
  const V uxx = vprod(ux, ux), uyy = vprod(uy, uy);
  const V indp = vmul(vset<V>(-1.5f), vadd(uxx, uyy));
  const V sr = vmul(vset<V>(32768.0f), rho), omb = vset<V>(vsub(1.0f, omega));
  const V three = vset<V>(3.0f), mthree = vset<V>(-3.0f);
  const V a0 = vset<V>(vmul(omega, 4.0f / 9.0f));
  H[0] = vfma(omb, H[0], vfma(vmul(a0, sr), indp, vmul(a0, dh)));
  auto pair = [&](int a, int b, V u, V even, V k1, V k0) {
    H[a] = vfma(omb, H[a], vfma(k1, vfma(three, u, even), k0));
    H[b] = vfma(omb, H[b], vfma(k1, vfma(mthree, u, even), k0));
  };
  const V as = vset<V>(vmul(omega, 1.0f / 9.0f)), k1s = vmul(as, sr), k0s = vmul(as, dh);
  pair(1, 3, ux, vfma(vset<V>(4.5f), uxx, indp), k1s, k0s);
  pair(2, 4, uy, vfma(vset<V>(4.5f), uyy, indp), k1s, k0s);
  const V ad = vset<V>(vmul(omega, 1.0f / 36.0f)), k1d = vmul(ad, sr), k0d = vmul(ad, dh);
  const V up = vadd(ux, uy), um = vsub(ux, uy);
  pair(5, 7, up, vfma(vmul(vset<V>(4.5f), up), up, indp), k1d, k0d);
  pair(8, 6, um, vfma(vmul(vset<V>(4.5f), um), um, indp), k1d, k0d);
}

}  // namespace plbm
