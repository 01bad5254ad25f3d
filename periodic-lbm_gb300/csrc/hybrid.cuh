// hybrid.cuh -- binary64 collisions with the binary64 pipe reserved for the
// one operation per population that needs its precision.
//
// GB300 issues binary64 at 1/64 of the binary32 rate, so a straight binary64
// BGK (about 70 FP64 instructions per cell) is bound by the FP64 pipe at ~15 %
// of HBM bandwidth.  These forms keep every term whose size is O(f) exact, and
// do the rest on the integer, XU and binary32 pipes.
//
// Common part:
//   F_q       = f_q * 2^59 as int64 (exact for |f_q| >= 2^-7; below that
//               rounded to nearest, error <= 2^-60)
//   R, JX, JY = sum F_q, sum cx F_q, sum cy F_q          exact integer sums
//   f'_q      = fma(c_q, Y_q 2^-59, f_q)                  ONE binary64 FMA
// where Y_q is an integer bracket holding the whole update of population q
// (the linear part exact, the nonlinear part from fixed-point products), c_q a power-of-two multiple
// of one rounded relaxation constant, so that the brackets of the nine
// populations sum to zero with the weights exactly: mass and momentum change
// only by the nine final roundings, plus the drift the reference's own
// binary64 weights cause (sums 1 - 2^-54), which is restored in the integers.
//
//   BGK (bgk_fma, src/collision_bgk.F90:58-71 with the equilibrium of
//     src/fvm_bardow.F90:99-126): the nonlinear terms of all nine populations
//     are integer combinations of three products j_a u_b.
//   TRT (trt_fma, incompressible, src/collision_trt.F90:98-152): symmetric
//     and antisymmetric brackets of each pair, joined by one product r D
//     (r = lambda_d / lambda_e scaled) rounded to nearest.
//   RR (rr_fma, src/collision_regularized.F90:72-194): the six merged Hermite
//     coefficients of the equilibrium and the regularized part.
// The products are fixed-point (mulh64, recip_fixed of fixed.cuh), each within
// ~2^-60: the error of a collision is the nine final roundings, below that of
// the straight binary64 operators (random cells at |u| <= 0.05, against 113-bit
// arithmetic, norm-wise: BGK 1.3e-16 against 1.4e-16, TRT 1.3e-16 / 1.4e-16, RR
// 1.2e-16 / 1.2e-16; largest error of a population over its weight 3e-16 against
// 1e-15).  Products in double-float, with conversions to and from the fixed
// point, erred by 1e-15 of the weight at |u| = 0.05 and took more instructions;
// 8192^2, ms per step, with them / as fixed-point products / with every product
// written as 32 x 32 -> 64 multiply-adds (mulh64 17 instructions, then 9; trt_rate
// in place of an exact 128-bit product): BGK 1.76 / 1.70 / 1.58 (1.43 with the
// columns copied ahead), TRT - / 1.89 / 1.79 (1.67), RR 2.60 / 2.24 / 2.05.  Bound by
// the integer pipes; BGK at 97 % of the copy bandwidth.
// Each states its range; a cell outside it reports `bad`, and the kernels then
// evaluate that cell with the binary64 operator of the reference instead.
// Populations stored shifted (h = f - w, the plugin's storage) take the same
// forms with DH = sum h = rho - 1 in place of R in the linear brackets.
#pragma once
#include <math.h>
#include "fixed.cuh"

namespace plbm {
namespace hy {

using df::df64;

constexpr int kScale = 59;  // fixed-point scale 2^59


DF_HD double fma_d(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return ::fma(a, b, c);
#endif
}

DF_HD int clz64(uint64_t a) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)a);
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}

// m / 2^rs rounded to nearest, ties to even (1 <= rs; 0 for rs >= 64).
DF_HD uint64_t shr_rne(uint64_t m, int rs) {
  if (rs >= 64) return 0;
  const uint64_t q = m >> rs, rem = m - (q << rs), half = 1ull << (rs - 1);
  return q + (uint64_t)((rem > half) | ((rem == half) & (q & 1ull)));
}

// binary64 -> int64 fixed point, scale 2^59, rounded to nearest even below
// 2^-59.  `bad` is set when the biased exponent of d exceeds emax
// (emax <= 1023), or d is not finite.
DF_HD int64_t to_fixed_lim(double d, int emax, bool& bad) {
  const uint64_t u = df::d2u(d);
  const int e = (int)((u >> 52) & 0x7FF);
  if (e > emax) {
    bad = true;
    return 0;
  }
  const int64_t m = (int64_t)((u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull);
  const int sh = e - 1075 + kScale;  // value = m * 2^(e-1075)
  int64_t F;
  if (e == 0) F = 0;
  else if (sh >= 0) F = m << sh;
  else F = (int64_t)shr_rne((uint64_t)m, -sh);
  return (u >> 63) ? -F : F;
}


// ---- fast paths for the ranges lattice states live in --------------------
// The general conversions are called out of line from the fast paths, so that
// the compiler branches around them instead of predicating them in.
#ifdef __CUDACC__
#define PLBM_NOINLINE static __host__ __device__ __noinline__
#else
#define PLBM_NOINLINE static __attribute__((noinline))
#endif

// High word of (hi:lo) << sh, 0 <= sh <= 31.
DF_HD uint32_t funnel_l(uint32_t lo, uint32_t hi, uint32_t sh) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, sh);
#else
  return sh ? (hi << sh) | (lo >> (32 - sh)) : hi;
#endif
}



// ---- shifted populations h = f - w (the plugin path) -------------------------
// With h in place of f the exact sums give DH = sum h = rho - 1 and the same
// J; every linear bracket keeps its form with DH in place of R (the w terms
// cancel), and rho = 1 + DH where the nonlinear terms need it.  The range
// limits apply to |h|.

// binary64 h (either sign, |h| < 2^(EMAX-1022)) -> int64 fixed point, scale
// 2^59; below 2^-59 rounded to nearest with ties toward +inf (an arithmetic
// shift of the signed value plus half a unit).  Most h = f - w are below 2^-7,
// where bits drop out.  Truncating toward zero shrank them by half a unit on
// average, and with h of the sign of c.u that damped |J| by ~1e-16 per step
// (2e-12 in u over 10,000 plugin steps); a bias that does not depend on the
// sign of h leaves every odd moment alone.
template <int EMAX>
DF_HD int64_t to_fixed_signed(double d, bool& bad) {
  const uint64_t u = df::d2u(d);
  const int e = (int)((u >> 52) & 0x7FF);
  if (e > EMAX) {
    bad = true;
    return 0;
  }
  const uint64_t m = (u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const int sh = e - 1016;  // value * 2^59 = m * 2^(e - 1016)
  const int64_t s = (u >> 63) ? -(int64_t)m : (int64_t)m;
  if (sh >= 0) return (int64_t)((uint64_t)s << sh);
  const int rs = -sh;
  return rs < 64 ? (s + ((int64_t)1 << (rs - 1))) >> rs : 0;
}

// int64 fixed point (any value) -> binary64, rounded to nearest with ties
// away from zero, branch-free apart from zero.  Ties are common (the integers
// are sums of binary64 images whose low bits are often zero) and in the
// shifted forms these values carry the sign of c.J, so the tie rule nudges |J|
// up: 1.5e-13 in u over 10,000 plugin steps (256 x 192 TGV), against 9e-14
// with ties to even, which costs 7 % of the plugin step.
DF_HD double fixed_to_double_any(int64_t T) {
  if (T == 0) return 0.0;
  const uint64_t neg = (uint64_t)T >> 63;
  const uint64_t a = neg ? (uint64_t)(-T) : (uint64_t)T;
  const int lz = clz64(a);
  const uint64_t n = a << lz;                      // bit 63 set
  const uint64_t m = (n >> 11) + ((n >> 10) & 1);  // <= 2^53; 2^53 carries into the exponent
  const uint64_t ex = (uint64_t)(1086 - lz - kScale);
  return df::u2d((neg << 63) | ((ex << 52) + (m - (1ull << 52))));
}

constexpr int64_t kOne = (int64_t)1 << kScale;  // 1.0 in fixed point

DF_HD int64_t shl(int64_t a, int s) { return (int64_t)((uint64_t)a << s); }
// a / 2^s rounded to nearest (ties toward +infinity).
DF_HD int64_t round_shr(int64_t a, int s) { return (a + ((int64_t)1 << (s - 1))) >> s; }
// |a| / 2^32, within one unit.
DF_HD uint32_t uabs_hi(int64_t a) {
  const int32_t h = (int32_t)(a >> 32);
  return (uint32_t)(h ^ (h >> 31));
}

// a k / 2^64 rounded to nearest, for the constant corrections below
// (|a| < 2^63, |k| < 2^31; a's low 32 bits do not take part).
DF_HD int64_t scale_2m64(int64_t a, int32_t k) {
  return mad_wide((int32_t)(a >> 32), k, (int64_t)1 << 31) >> 32;
}


// ---- conversions shaped for the GB300 pipes ----------------------------------
// Measured issue rates per SM and clock: integer add/logic/shift and
// I2F.F32.S32 go to the ALU pipe (64 lanes), IMAD and binary32 arithmetic to
// the FMA pipes (64 / 128), F2I, FRND and FLO (clz) to the XU pipe (16), and
// every conversion to or from a 64-bit type to the binary64 pipe (~2).  The
// one-FMA BGK is bound by its ALU work, so these forms move work to the FMA
// and XU pipes.

// 32-bit count of leading zeros (XU pipe).
DF_HD uint32_t clz32(uint32_t a) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__clz((int)a);
#else
  return a ? (uint32_t)__builtin_clz(a) : 32u;
#endif
}
// Low word of (hi:lo) >> sh, 0 <= sh <= 31.
DF_HD uint32_t funnel_r(uint32_t lo, uint32_t hi, uint32_t sh) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, sh);
#else
  return sh ? (lo >> sh) | (hi << (32 - sh)) : lo;
#endif
}
DF_HD int32_t f2i_trunc(float v) {
#ifdef __CUDA_ARCH__
  return __float2int_rz(v);
#else
  return (int32_t)v;
#endif
}
DF_HD float i2f(int32_t v) {
#ifdef __CUDA_ARCH__
  return __int2float_rn(v);
#else
  return (float)v;
#endif
}


DF_HD constexpr double pow2_const(int e) { return e == 0 ? 1.0 : (e > 0 ? 2.0 * pow2_const(e - 1) : 0.5 * pow2_const(e + 1)); }
PLBM_NOINLINE double fixed_to_double_any_slow(int64_t T) { return fixed_to_double_any(T); }

// int64 v > 0 (scale 2^SCALE) -> binary64 rounded to nearest, ties away from
// zero (10 instructions; the carry of the rounding runs into the exponent).
template <int SCALE>
DF_HD double pos_fixed_to_double(int64_t v) {
  const int lz = clz64((uint64_t)v);
  const uint64_t n = ((uint64_t)v << lz) + 0x400u;  // bit 63 set, or 2^64 -> 0 on a carry
  const uint64_t m = (n >> 11) | ((uint64_t)(n < 0x400u) << 53);
  return df::u2d(((uint64_t)(uint32_t)(1085 - SCALE - lz) << 52) + m);
}

// int64 fixed point (scale 2^SCALE) -> binary64 for |T| >= 2^32 (others out of
// line, exactly): the magnitude taken in one's complement (a negative T comes
// out 2^-59 smaller in magnitude) and truncated to 53 bits.  The error is below
// 2^-52 relative plus 2^-59 absolute -- for the non-equilibrium brackets it
// converts, negligible against the binary64 rounding of the populations.  (Selecting the
// words without a branch put more on the ALU pipe, which binds: 8192^2 TRT 33.3
// GLUPS against 36.)  EXACT: a negative T's own magnitude, for sums over many T, in which
// half of a unit on average adds up.
template <int SCALE = kScale, bool EXACT = false>
DF_HD double fixed_to_double_tr(int64_t T) {
  uint32_t hi = (uint32_t)((uint64_t)T >> 32), lo = (uint32_t)(uint64_t)T;
  const uint32_t s = (uint32_t)((int32_t)hi >> 31);  // 0 or ~0
  if (EXACT) {
    const uint64_t m = (uint64_t)T + (((uint64_t)s << 32) | s);  // -T = ~(T - 1)
    hi = (uint32_t)(m >> 32), lo = (uint32_t)m;
  }
  const uint32_t ah = hi ^ s, al = lo ^ s;
  if (ah == 0u) return fixed_to_double_any_slow(T) * pow2_const(kScale - SCALE);
  const uint32_t lz = clz32(ah);  // 0..31
  const uint32_t nh = funnel_l(al, ah, lz), nl = al << lz;  // bit 63 of (nh:nl) set
  const uint32_t mh = nh >> 11, ml = funnel_r(nl, nh, 11);  // 53 bits, leading one at bit 52
  // value = (nh:nl) 2^(-lz - SCALE): biased exponent 1086 - SCALE - lz; the leading
  // one of mh (bit 20) adds the final 1 to the exponent field
  const uint32_t eh = (1085u - (uint32_t)SCALE - lz) * 0x100000u + mh;
  return df::u2d(((uint64_t)(eh | (s & 0x80000000u)) << 32) | (uint64_t)ml);
}

// ---- the new populations -------------------------------------------------------
// f'_q = f_q + k_q c Y_q 2^-59 rounded to nearest, in the last places of f_q: with
// the biased exponent E of f_q one place is 2^(E - 1075), so the change is
// k_q c Y_q 2^(1016 - E) places, one fixed-point product (c at 2^66) and a right
// shift, added to f_q's bits.  That is f'_q while its exponent is E; a cell with a
// population that changes binade converts them all from 2^-61 (about one cell in
// twenty of a flow of |u| = 0.05), one with a population below 2^-7 or a sign change
// takes the binary64 FMAs out of line.  Against an integer-to-binary64 conversion
// (sign, leading zeros, two shifts, a branch for small Y) and an FMA: no binary64
// instruction, no branch per population.  The product is within 2 units of 2^-61
// (diagonal) or 2^-59 (axis, rest; places of 2^-56 and 2^-54).  Norm-wise error
// against 113-bit arithmetic as with the FMAs: BGK 1.31e-16 / 1.33e-16, TRT
// 1.31e-16 / 1.32e-16, RR 1.16e-16 / 1.17e-16.
// Rate: omega (TRT: lambda_e) in [0, 2], where c fits 2^66 and every new population of a
// cell in range 2^61; a launch with another rate takes the binary64 FMAs.
inline bool finish_takes(double omega) { return omega >= 0.0 && omega <= 2.0; }
PLBM_NOINLINE void finish_slow(double* f, const int64_t* Y, double c0, double cs, double cd) {
  for (int q = 0; q < 9; q++) f[q] = fma_d(q == 0 ? c0 : (q < 5 ? cs : cd), fixed_to_double_tr(Y[q]), f[q]);
}
// KS: log2 of k_q of the axis populations (2 BGK and RR, 1 TRT; k_0 = 4, k_diag =
// 1).  c0, cs, cd: k_q c; small: a population below 2^-7 (load_fixed).
template <int KS>
DF_HD void finish(double (&f)[9], const int64_t (&Y)[9], int64_t c, double c0, double cs, double cd, bool small) {
  uint64_t b[9];
  int64_t m[9];
  uint32_t moved = small ? 0x100000u : 0u;
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const uint64_t u = df::d2u(f[q]);
    const uint32_t sh = ((uint32_t)(u >> 52) - 1014u - (q == 0 ? 2u : (q < 5 ? (uint32_t)KS : 0u))) & 31u;
    m[q] = mulh64(Y[q], c);  // 4 c Y
    b[q] = u + (uint64_t)((m[q] + (int64_t)((1u << sh) >> 1)) >> sh);
    moved |= (uint32_t)((b[q] ^ u) >> 32);
  }
  if (moved >> 20) {
    int64_t low = small ? 0 : 1;
#pragma unroll
    for (int q = 0; q < 9; q++) {  // the populations at 2^-61
      const uint64_t u = df::d2u(f[q]);
      const int64_t F = shl((int64_t)((u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull), (int)((u >> 52) - 1014u) & 31);
      m[q] = F + shl(m[q], q == 0 ? 2 : (q < 5 ? KS : 0));
      low = m[q] < low ? m[q] : low;
    }
    if (low <= 0) {
      double g[9];
      int64_t Z[9];
#pragma unroll
      for (int q = 0; q < 9; q++) g[q] = f[q], Z[q] = Y[q];
      finish_slow(g, Z, c0, cs, cd);
#pragma unroll
      for (int q = 0; q < 9; q++) f[q] = g[q];
    } else {
#pragma unroll
      for (int q = 0; q < 9; q++) f[q] = pos_fixed_to_double<61>(m[q]);
    }
  } else {
#pragma unroll
    for (int q = 0; q < 9; q++) f[q] = df::u2d(b[q]);
  }
}

// ---- BGK with one binary64 FMA per population --------------------------------
// f'_q = f_q + omega (feq_q - f_q), feq_q = w_q T_q, T_q = R + 3 c_q.J + C_q,
// C_q = rho (4.5 (c_q.u)^2 - 1.5 u^2) (src/collision_bgk.F90:58-71 with the
// equilibrium of src/fvm_bardow.F90:99-126, rearranged).  The nonlinear terms
// of all nine populations are integer combinations of three products,
//   A = 1.5 jx^2 / rho,  B = 1.5 jy^2 / rho,  X = 4.5 jx jy / rho,
//   C_0 = -(A + B),  C_x = 2A - B,  C_y = 2B - A,  C_(+-diag) = 2 (A + B) +- 2X,
// evaluated as fixed-point products and taken to 2^-59 once each.  With
// every F_q and the C images integers, 36 (w_q T_q - F_q) is an integer, and
//   rest      4 Y_0,  Y_0 = 4 (R + C_0) - 9 F_0
//   axis      4 Y_q,  Y_q = T_q - 9 F_q
//   diagonal    Y_q,  Y_q = T_q - 36 F_q
// so f'_q = fma(k_q c, Y_q 2^-59, f_q) with c = RN(omega / 36), k_q = 4 or 1:
// the only rounding of the linear part is the final one, and the integers
// satisfy sum k_q Y_q = 0 and sum k_q c_q Y_q = 0 exactly (the nonlinear
// combinations above sum to zero with the weights), so mass and momentum
// change only by the nine final roundings.  Y_q is taken to binary64 by
// integer instructions (53 leading bits); its error is relative to the small
// non-equilibrium term, not to f.
//
// The reference relaxes with its binary64 weights, whose sum W0 + 4 WS + 4 WD
// and first-moment factor 3 (2 WS + 4 WD) are both 1 - 2^-54: each step its
// mass and momentum lose omega 2^-54 of themselves, 1e-12 over 10,000 steps
// -- the size of the tolerance.  The same relaxation is restored in the
// integers: the rest bracket gains omega eps_m R / (4c) (mass_k), and the
// x-axis pair gains +- omega eps_j JX / (8c) (mom_k; the y pair likewise), so
// the mass changes by omega eps_m R and JX by omega eps_j JX per step.
//
// Range.  The loads take 0 <= f_0 < 1, 0 <= f_axis < 1/4, 0 <= f_diag < 1/8
// (biased exponents at most 1022, 1020, 1019), and the cell must satisfy
// A + B < 0.2 (7.5 rho |u|^2 < 1, which bounds every |C_q| below 1).  Then,
// in units of 2^59, R < 2.5, |JX|, |JY| < 1/2, |JX +- JY| < 3/4, and
// |Y_0| < 10, |Y_axis| < 7.25, |Y_diag| < 10.25: every bracket fits int64
// (intermediate products such as 4 R may wrap; two's complement sums of
// wrapped terms are exact when the result fits).  Other cells report `bad`.
struct BgkParams {
  double c1;       // RN(omega / 36)
  double c4;       // 4 RN(omega / 36), exact
  int32_t mass_k;  // omega eps_m / c4 2^64, rounded (bgk_fma_params)
  int32_t mom_k;   // omega eps_j / (2 c4) 2^64, rounded
  int64_t c_fx;    // c1 2^66
};

// a + b = s + e exactly (Knuth's two-sum).
inline void two_sum_d(double a, double b, double& s, double& e) {
  s = a + b;
  const double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// eps_m = W0 + 4 WS + 4 WD - 1 and eps_j = 3 (2 WS + 4 WD) - 1 of the binary64
// weights, evaluated without rounding error (both are -2^-54 for 4/9, 1/9,
// 1/36: the sums are within 2^-50 of 1, so the final subtraction is exact).
inline double weight_sum_error(const double (&w)[3]) {
  double s1, e1, s2, e2;
  two_sum_d(w[0], 4.0 * w[1], s1, e1);
  two_sum_d(s1, 4.0 * w[2], s2, e2);
  return (s2 - 1.0) + (e1 + e2);
}
inline double first_moment_error(const double (&w)[3]) {
  double s, e;
  two_sum_d(2.0 * w[1], 4.0 * w[2], s, e);
  const double p = 3.0 * s, ep = ::fma(3.0, s, -p);
  return (p - 1.0) + (ep + 3.0 * e);
}

inline BgkParams bgk_fma_params(double omega, const double (&w)[3]) {
  BgkParams p;
  p.c1 = omega / 36.0;
  p.c4 = 4.0 * p.c1;
  const double eps_m = weight_sum_error(w), eps_j = first_moment_error(w);
  const double km = ldexp(omega * eps_m / p.c4, 64), kj = ldexp(0.5 * omega * eps_j / p.c4, 64);
  p.mass_k = fabs(km) < 0x1p30 ? (int32_t)llrint(km) : 0;
  p.mom_k = fabs(kj) < 0x1p30 ? (int32_t)llrint(kj) : 0;
  p.c_fx = finish_takes(omega) ? llrint(ldexp(p.c1, 66)) : 0;
  return p;
}

// Exact fixed-point image of a non-negative population below 2^(EMAX-1022);
// `bad` for negative values, values past the limit and non-finite ones.
PLBM_NOINLINE int64_t to_fixed_nonneg_slow(double d, int emax, int* bad) {
  bool b = false;
  const int64_t r = to_fixed_lim(d, emax, b);
  if (b || r < 0) *bad = 1;
  return r;
}
template <int EMAX>
DF_HD int64_t to_fixed_nonneg(double d, bool& bad) {
  const uint64_t u = df::d2u(d);
  const uint32_t H = (uint32_t)(u >> 32), L = (uint32_t)u;
  const uint32_t sh = (H >> 20) - 1016u;  // a set sign bit makes this large
  if (sh <= (uint32_t)(EMAX - 1016)) {
    const uint32_t mh = (H & 0xFFFFFu) | 0x100000u;
    return (int64_t)(((uint64_t)funnel_l(L, mh, sh) << 32) | (uint64_t)(L << sh));
  }
  int b = 0;
  const int64_t r = to_fixed_nonneg_slow(d, EMAX, &b);
  if (b) bad = true;
  return r;
}

// The nine populations in the fixed point.  Unshifted: exact for
// 2^-7 <= f below the limits of bgk_fma (a biased exponent in [1016, EMAX], one
// shift of the significand); a cell with a smaller value goes through
// to_fixed_nonneg out of line, one with a value past the limits is reported
// before any further work (a 2048^2 lattice of density 3 in FMA arithmetic then
// takes the 624 us per BGK step of the binary64 kernel; 702 when reported last).  SHIFTED: the significand at 2^62, negated in
// one's complement, shifted right with half a unit added: rounded to nearest,
// an error whose mean does not depend on the sign of h.  (Rounded toward zero,
// h of the sign of c.u shrinks and |J| is damped by ~1e-16 per step, 2e-12 in u
// over 10,000 plugin steps; rounded toward -infinity, one instruction pair
// fewer, the error of one step is 1.4 times as large.)  The half unit is a 32-bit one, so that
// |h| < 2^-28 is rounded toward -infinity, unless NEAREST: then to the nearest as well, which costs
// TRT and RR 1.1 to 2.4 % (641 x 500 10.95 -> 11.08 us per step and 12.82 -> 13.01) and shows in flows of
// 1e-11 and less (40 x 36 vortex with noise of 1e-13, velocity after 400 steps: TRT 4.5e-4 off without and
// 1.6e-4 with it, RR 5.8e-3 and 2.2e-4).  BGK takes such cells out of line instead (bgk_tiny; 1 %
// rather than 1.9).
PLBM_NOINLINE void load_fixed_slow(const double* f, int64_t* F) {
  bool b = false;  // stays false: the caller has checked the limits
  F[0] = to_fixed_nonneg<1022>(f[0], b);
  for (int q = 1; q < 5; q++) F[q] = to_fixed_nonneg<1020>(f[q], b);
  for (int q = 5; q < 9; q++) F[q] = to_fixed_nonneg<1019>(f[q], b);
}
template <bool SHIFTED, bool NEAREST = false>
DF_HD void load_fixed(const double (&f)[9], int64_t (&F)[9], bool& bad, bool& small) {
  bool odd = false;
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const uint64_t u = df::d2u(f[q]);
    const uint32_t H = (uint32_t)(u >> 32), L = (uint32_t)u;
    const uint32_t mh = (H & 0xFFFFFu) | 0x100000u;
    if constexpr (SHIFTED) {
      const uint32_t e = (H >> 20) & 0x7FFu;
      odd |= e > (q == 0 ? 1021u : (q < 5 ? 1019u : 1018u));
      const uint64_t n = ((((uint64_t)mh << 32) | L) << 10) ^ (uint64_t)((int64_t)u >> 63);
      if constexpr (NEAREST) {
        const uint32_t rs = 1025u - e < 63u ? 1025u - e : 63u;  // to half units
        F[q] = (((int64_t)n >> rs) + 1) >> 1;
      } else {
        const uint32_t rs = 1026u - e < 63u ? 1026u - e : 63u;
        F[q] = (int64_t)(n + (1u << ((rs - 1u) & 31u))) >> rs;
      }
    } else {
      const uint32_t sh = (H >> 20) - 1016u;  // a set sign bit makes this large
      odd |= sh > (q == 0 ? 6u : (q < 5 ? 4u : 3u));
      F[q] = (int64_t)(((uint64_t)funnel_l(L, mh, sh & 31u) << 32) | (uint64_t)funnel_l(0u, L, sh & 31u));
    }
  }
  small = odd;
  if constexpr (SHIFTED) {
    bad |= odd;
  } else if (odd) {
    // past a limit, negative or not finite (a set sign bit included in H >> 20)
#pragma unroll
    for (int q = 0; q < 9; q++)
      bad |= (uint32_t)(df::d2u(f[q]) >> 52) > (q == 0 ? 1022u : (q < 5 ? 1020u : 1019u));
    if (bad) return;
    double g[9];
    int64_t G[9];
#pragma unroll
    for (int q = 0; q < 9; q++) g[q] = f[q];
    load_fixed_slow(g, G);
#pragma unroll
    for (int q = 0; q < 9; q++) F[q] = G[q];
  }
}

// rho outside [2^-2 + 2^-27, 4): the reciprocal's range.
DF_HD bool rho_out_of_range(int64_t R) { return (uint32_t)((uint64_t)R >> 32) - 0x2000001u > 0x1dfffffeu; }
constexpr int32_t kTurn02 = 26843545;    // 0.2 2^27

// SHIFTED: f holds h = f - w (the plugin's storage, sim/sim.F90:131).  The
// linear brackets then take DH = sum h = rho - 1 in place of R (the w terms
// cancel) and the nonlinear terms rho = 1 + DH.  Range for h: |h_0| < 1/2,
// |h_axis| < 1/8, |h_diag| < 1/16 (biased exponents at most 1021, 1019, 1018),
// rho >= 1/4 and A + B < 0.2; then |DH| < 1.25, |JX|, |JY| < 1/2,
// |JX +- JY| < 3/4 and |Y_0| < 10.3, |Y_axis| < 4.9, |Y_diag| < 6.75 (units of
// 2^59).  Small h are rounded to the fixed point with ties toward +infinity,
// a bias that leaves the odd moments alone (to_fixed_signed).
//
// bgk_brackets: Y of the fixed-point populations F, and u at 2^61.  lg: the shifted
// populations, R and J, Y and u are held 2^lg times as large.
template <bool SHIFTED>
DF_HD void bgk_brackets(const int64_t (&F)[9], const BgkParams& p, int64_t (&Y)[9], int64_t& U, int64_t& V, bool& bad,
                        int lg = 0) {
  // R: the zeroth moment of the stored values (rho, or DH when shifted)
  const int64_t R = (((F[5] + F[7]) + (F[6] + F[8])) + ((F[1] + F[3]) + (F[2] + F[4]))) + F[0];
  const int64_t d57 = F[5] - F[7], d86 = F[8] - F[6];
  const int64_t JX = (d57 + d86) + (F[1] - F[3]);
  const int64_t JY = (d57 - d86) + (F[2] - F[4]);
  const int64_t Rrho = SHIFTED ? (R >> (lg < 63 ? lg : 63)) + kOne : R;
  const int64_t I = recip_fixed(Rrho);                 // 2^61 / rho
  const int64_t jx = shl(JX, 5), jy = shl(JY, 5);      // 2^64 j
  U = mulh64(jx, I), V = mulh64(jy, I);                // 2^61 u
  const int sh = lg < 59 ? 3 + lg : 62;
  const int64_t Ai = round_shr(3 * mulh64(jx, U), sh), Bi = round_shr(3 * mulh64(jy, V), sh);
  const int64_t Xi = round_shr(9 * mulh64(jx, V), sh);
  const int64_t AB = Ai + Bi;
  bad |= rho_out_of_range(Rrho) | ((int32_t)(AB >> 32) >= kTurn02);
  Y[0] = 4 * (R - AB) - 9 * F[0] + scale_2m64(R, p.mass_k);
  const int64_t cx = R + (2 * Ai - Bi), cy = R + (2 * Bi - Ai);
  const int64_t jx3 = 3 * JX, jy3 = 3 * JY;
  const int64_t ax = jx3 + scale_2m64(JX, p.mom_k), ay = jy3 + scale_2m64(JY, p.mom_k);
  Y[1] = cx + ax - 9 * F[1];
  Y[3] = cx - ax - 9 * F[3];
  Y[2] = cy + ay - 9 * F[2];
  Y[4] = cy - ay - 9 * F[4];
  const int64_t dp = R + 2 * (AB + Xi), dm = R + 2 * (AB - Xi);
  const int64_t sp = jx3 + jy3, sm = jy3 - jx3;
  Y[5] = dp + sp - 36 * F[5];
  Y[7] = dp - sp - 36 * F[7];
  Y[6] = dm + sm - 36 * F[6];
  Y[8] = dm - sm - 36 * F[8];
}

template <bool SHIFTED>
DF_HD void bgk_brackets(const int64_t (&F)[9], const BgkParams& p, int64_t (&Y)[9], bool& bad) {
  int64_t U, V;
  bgk_brackets<SHIFTED>(F, p, Y, U, V, bad);
}

// A shifted cell of which every |h| < 2^-27, with h scaled to the upper end of the fixed
// point's range: in units of 2^-59 the errors stay absolute however small h is, and the load
// rounds |h| < 2^-28 toward -infinity.  A 40 x 36 vortex with noise, 400 steps, hybrid plugin,
// mean-square error of the velocity relative to it, at u = 1e-8, 1e-10 and 1e-13: 1.6e-9, 2.7e-7
// and 1.1e-3 in those units (2.1e-9, 1.5e-7 and 1.5e-4 when they were rounded to nearest),
// 6.3e-10, 6.2e-8 and 6.1e-5 here, which is the equilibrium it starts from; from the default
// arithmetic's equilibrium 3.6e-14 at each (binary64 operator 2.3e-8, 2.4e-6 and 2.1e-3).  Out of
// line; false: not such a cell.
PLBM_NOINLINE bool bgk_tiny(double* f, const BgkParams& p) {
  int e = 0;  // the largest biased exponent
  for (int q = 0; q < 9; q++) {
    const int eq = (int)(df::d2u(f[q]) >> 52) & 0x7FF;
    e = eq > e ? eq : e;
  }
  if (e > 995) return false;
  const int lg = 1017 - e;  // |g| < 2^-5
  const double up = df::u2d((uint64_t)(1023 + lg) << 52), down = df::u2d((uint64_t)(1023 - lg) << 52);
  double g[9];
  int64_t F[9], Y[9], U, V;
  bool bad = false, odd;
  for (int q = 0; q < 9; q++) g[q] = f[q] * up + 0.0;  // + 0: no -0, which the load takes for -2^-59
  load_fixed<true>(g, F, bad, odd);
  bgk_brackets<true>(F, p, Y, U, V, bad, lg);
  for (int q = 0; q < 9; q++) f[q] = fma_d(q < 5 ? p.c4 : p.c1, fixed_to_double_tr(Y[q]), g[q]) * down;
  return true;
}

// HINT: a shifted cell that may be bgk_tiny's is reported out of range, for bgk_rest to take
// (641 x 500: 9.99 us per step without the two tests, 10.07 with them; with every small h
// rounded to nearest in the load instead, 10.3).
template <bool SHIFTED = false, bool QUICK = false, bool HINT = SHIFTED>
DF_HD void bgk_fma(double (&f)[9], const BgkParams& p, bool& bad) {
  int64_t F[9], Y[9];
  bool small;
  load_fixed<SHIFTED>(f, F, bad, small);
  // two of them below 2^-27, and not +0 (at rest): perhaps all nine
  if constexpr (HINT)
    if ((uabs_hi(F[1]) | uabs_hi(F[2])) == 0) bad |= (df::d2u(f[1]) | df::d2u(f[2])) != 0;
  if (bad) return;
  bgk_brackets<SHIFTED>(F, p, Y, bad);
  if constexpr (SHIFTED || !QUICK) {
#pragma unroll
    for (int q = 0; q < 9; q++) f[q] = fma_d(q < 5 ? p.c4 : p.c1, fixed_to_double_tr(Y[q]), f[q]);
  } else {
    finish<2>(f, Y, p.c_fx, p.c4, p.c4, p.c1, small);
  }
}

// A shifted cell that bgk_fma reports: true where the fixed point takes it after all.
PLBM_NOINLINE bool bgk_rest(double* f, const BgkParams& p) {
  if (bgk_tiny(f, p)) return true;
  double g[9];
  bool bad = false;
  for (int q = 0; q < 9; q++) g[q] = f[q];
  bgk_fma<true, false, false>(g, p, bad);
  if (bad) return false;
  for (int q = 0; q < 9; q++) f[q] = g[q];
  return true;
}

// Recursive-regularized constant (rr_fma): 1 - omega at scale 2^63, for omega in [0, 2]
// (the ends 2^-63 inside it).  Another omega, or none, has no place in that scale: every
// cell is then out of range.
struct RrParams {
  int64_t omb;
  uint32_t limit;  // of 6 sum |M / 2| 2^30; 0: every cell
};
constexpr uint32_t kTurn06 = 644245094;  // 0.6 2^30
inline RrParams rr_fma_params(double omega) {
  RrParams r = {0, omega >= 0.0 && omega <= 2.0 ? kTurn06 : 0};
  const double b = r.limit ? ldexp(1.0 - omega, 63) : 0.0;
  r.omb = b >= 0x1p63 ? INT64_MAX : (b <= -0x1p63 ? INT64_MIN + 1 : (int64_t)llrint(b));
  return r;
}

// Recursive regularized collision with one binary64 FMA per population.
// f'_q = w_q (T_q + N_q), T_q = R + 3 c_q.J, N_q the Hermite combination of
// the six merged coefficients M = rho (u product) + (1 - omega) a of the
// second-, third- and fourth-order Hermite terms (the equilibrium's and the
// regularized non-equilibrium part's, src/collision_regularized.F90:99-194).
// With b = 1 - omega, B = b a and q = rho u u the recursion of the higher
// orders closes over the merged coefficients:
//   3 B_xx = b (3 P_xx - R - 3 q_xx), B_xy = b (P_xy - q_xy),  M = q + B,
//   M_xxy  = u_y M_xx + 2 u_x B_xy,   M_yyx = u_x M_yy + 2 u_y B_xy,
//   M_xxyy = u_y M_xxy + u_x (M_yyx - u_x q_yy)
// (a_xxyy of the reference is u_x a_yyx + u_y a_xxy), fifteen fixed-point
// products in all (mulh64) on exact integer moments.  Taken to integers of
// 2^-59 once each as X3 = 1.5 M_xx, Y3 = 1.5 M_yy, K = 9 M_xy, GY = 4.5 M_xxy,
// GX = 4.5 M_yyx and G = 4.5 M_xxyy, every 36 (f'_q - f_q) / k_q is an integer
// bracket:
//   rest      4 Y_0,  Y_0 = 4 R - 9 F_0 - 4 (X3 + Y3) + 2 G
//   axis      4 Y_q,  Y_q = T_q - 9 F_q + 2 X3 - Y3 - G -+ GX  (x; y alike)
//   diagonal    Y_q,  Y_q = T_q - 36 F_q + 2 (X3 + Y3) + 2 G +- K +- 2 (GY +- GX)
// and f'_q = fma(k_q RN(1/36), Y_q 2^-59, f_q).  The Hermite parts of the
// brackets sum to zero with the weights exactly, as T_q - 36 w_q F_q does; the
// reference's binary64 weights (sums 1 - 2^-54) take 2^-54 of the mass and
// momentum each step, restored by p.mass_k / p.mom_k (bgk_fma_params at
// omega = 1).  Range: omega in [0, 2], as bgk_fma, q_xx + q_yy < 0.2 and sum |M / 2| < 0.1: then the Hermite parts
// add at most 3, 0.9 and 1.8 (units of 2^59) to the rest, axis and diagonal
// brackets, which stay below 13 x 2^59, and no product's operand leaves int64.
template <bool SHIFTED>
DF_HD void rr_brackets(const int64_t (&F)[9], const RrParams& r, const BgkParams& p, int64_t (&Y)[9], bool& bad) {
  const int64_t s57 = F[5] + F[7], s68 = F[6] + F[8];
  const int64_t sd = s57 + s68;
  const int64_t R = (sd + ((F[1] + F[3]) + (F[2] + F[4]))) + F[0];
  const int64_t d57 = F[5] - F[7], d86 = F[8] - F[6];
  const int64_t JX = (d57 + d86) + (F[1] - F[3]);
  const int64_t JY = (d57 - d86) + (F[2] - F[4]);
  const int64_t PXX3 = 3 * ((F[1] + F[3]) + sd) - R;
  const int64_t PYY3 = 3 * ((F[2] + F[4]) + sd) - R;
  const int64_t PXY = s57 - s68;
  const int64_t Rrho = SHIFTED ? R + kOne : R;
  const int64_t I = recip_fixed(Rrho);                                                 // 2^61 / rho
  const int64_t jx = shl(JX, 5), jy = shl(JY, 5);                                      // 2^64 j
  const int64_t U = mulh64(jx, I), V = mulh64(jy, I);                                  // 2^61 u
  const int64_t qxx = mulh64(jx, U), qyy = mulh64(jy, V), qxy = mulh64(jx, V);         // 2^61 rho u u
  const int64_t u = shl(U, 2), v = shl(V, 2);                                          // 2^63 u
  // 3 M_xx, 3 M_yy, M_xy and B_xy, scale 2^60
  const int64_t mxx = round_shr(3 * qxx, 1) + mulh64(shl(PXX3, 2) - 3 * qxx, r.omb);
  const int64_t myy = round_shr(3 * qyy, 1) + mulh64(shl(PYY3, 2) - 3 * qyy, r.omb);
  const int64_t bxy = mulh64(shl(PXY, 2) - qxy, r.omb);
  const int64_t mxy = round_shr(qxy, 1) + bxy;
  // 3 M_xxy, 3 M_yyx, 3 M_xxyy, scale 2^62
  const int64_t mx3 = shl(mxx, 3), my3 = shl(myy, 3), b3 = shl(bxy, 3);
  const int64_t mxxy = mulh64(mx3, v) + 6 * mulh64(b3, u);
  const int64_t myyx = mulh64(my3, u) + 6 * mulh64(b3, v);
  const int64_t mxxyy = mulh64(shl(mxxy, 1), v) + mulh64(shl(myyx - 3 * mulh64(shl(qyy, 2), u), 1), u);
  // sum |M / 2| < 0.1, on the leading words
  const uint32_t sum2 = uabs_hi(mxx) + uabs_hi(myy) + 3 * uabs_hi(mxy);  // scale 6 2^28
  const uint32_t sum3 = uabs_hi(mxxy) + uabs_hi(myyx) + uabs_hi(mxxyy);  // scale 6 2^30
  bad |= rho_out_of_range(Rrho) | ((int32_t)((qxx + qyy) >> 34) >= kTurn02) | (sum2 >= kTurn06 / 4) |
         (4 * sum2 + sum3 >= r.limit);
  const int64_t X3 = round_shr(mxx, 2), Y3 = round_shr(myy, 2), K = round_shr(9 * mxy, 1);
  const int64_t GY = round_shr(3 * mxxy, 4), GX = round_shr(3 * myyx, 4), G = round_shr(3 * mxxyy, 4);
  Y[0] = 4 * (R - X3 - Y3) - 9 * F[0] + 2 * G + scale_2m64(R, p.mass_k);
  const int64_t jx3 = 3 * JX, jy3 = 3 * JY;
  const int64_t ax = jx3 + scale_2m64(JX, p.mom_k) - GX, ay = jy3 + scale_2m64(JY, p.mom_k) - GY;
  const int64_t cx = R + 2 * X3 - Y3 - G, cy = R + 2 * Y3 - X3 - G;
  Y[1] = cx + ax - 9 * F[1];
  Y[3] = cx - ax - 9 * F[3];
  Y[2] = cy + ay - 9 * F[2];
  Y[4] = cy - ay - 9 * F[4];
  // diagonal pairs without the momentum correction (the axis pairs carry it)
  const int64_t c = R + 2 * (X3 + Y3 + G), dp = c + K, dm = c - K;
  const int64_t sp = (jx3 + jy3) + 2 * (GY + GX), sm = (jy3 - jx3) + 2 * (GY - GX);
  Y[5] = dp + sp - 36 * F[5];
  Y[7] = dp - sp - 36 * F[7];
  Y[6] = dm + sm - 36 * F[6];
  Y[8] = dm - sm - 36 * F[8];
}

template <bool SHIFTED = false, bool QUICK = false>
DF_HD void rr_fma(double (&f)[9], const RrParams& r, const BgkParams& p, bool& bad) {
  int64_t F[9], Y[9];
  bool small;
  load_fixed<SHIFTED, SHIFTED>(f, F, bad, small);
  if (bad) return;
  rr_brackets<SHIFTED>(F, r, p, Y, bad);
  if constexpr (SHIFTED || !QUICK) {
#pragma unroll
    for (int q = 0; q < 9; q++) f[q] = fma_d(q < 5 ? p.c4 : p.c1, fixed_to_double_tr(Y[q]), f[q]);
  } else {
    finish<2>(f, Y, p.c_fx, p.c4, p.c4, p.c1, small);
  }
}

// (a b) / 2^sh, 0 < sh < 64, of the exact 128-bit product, rounded to nearest
// (ties toward +infinity); the caller keeps the result within int64.  Rounding
// toward -infinity instead biases every product by half a unit in one
// direction: in the antisymmetric brackets that is a uniform force on the flow
// (about 3e-19 per step in J), which grew to 2e-12 of the decaying u over
// 10,000 steps.
DF_HD int64_t mul_shr(int64_t a, int64_t b, int sh) {
#ifdef __CUDA_ARCH__
  int64_t hi = __mul64hi(a, b);
#else
  int64_t hi = (int64_t)(((__int128)a * b) >> 64);
#endif
  const uint64_t lo = (uint64_t)a * (uint64_t)b;
  const uint64_t lo2 = lo + (1ull << (sh - 1));
  hi += (int64_t)(lo2 < lo);
  return (int64_t)(((uint64_t)hi << (64 - sh)) | (lo2 >> sh));
}

// Incompressible TRT with one binary64 FMA per population
// (src/collision_trt.F90:98-152).  With c = RN(lambda_e / 18) and the exact
// integer brackets of the pairs (axis: weights 1/9, diagonal: 1/36; J2 = |J|^2,
// XY = JX JY as products taken to the fixed point)
//   axis x    Sb = 9 (F_1 + F_3) - 2 R - 6 JX^2 + 3 JY^2,   D = 3 (F_1 - F_3) - 2 JX
//   diagonal  Sb = 18 (F_5 + F_7) - R - 3 J2 -+ 9 XY,       D = 6 (F_5 - F_7) - (JX +- JY)
// the reference's sym = les (...) is c Sb (axis) and c/2 Sb (diagonal), its
// asym the same constants times r D with r = lambda_d / (6 c) (trt_rate, one
// product per pair), so
//   f'_p = fma(c_k, -(Sb + r D), f_p),  f'_m = fma(c_k, -(Sb - r D), f_m),
//   f'_0 = fma(2c, 4 R - 6 J2 - 9 F_0, f_0)
// (c_k = c on the axis pairs, c/2 on the diagonal ones).  The integer brackets
// sum to zero with the weights; the reference's binary64 weights relax the
// mass by lambda_e (sum w - 1) R per step (the sum is 1 - 2^-54), restored in
// the rest bracket (mass_k).  Range: the loads of bgk_fma, and |Sb| < 2^61,
// |D| < dmax = 2^61 / r (checked), so every bracket stays below 2^62.
struct TrtFmaParams {
  double c, c2, ch;    // RN(lambda_e / 18), 2c, c/2
  int64_t dmax;        // smallest |D| out of range: |r D| < 2^61, |D| < 2^60 (0: every cell falls back)
  int64_t r_round;     // half a unit of the product's discarded bits
  int32_t r_hi, r_lo;  // r = lambda_d / (6c) = (r_hi 2^31 + r_lo) 2^-(r_s + 31)
  int32_t r_s;
  int32_t mass_k;      // lambda_e eps_m / (2c) 2^64
  int32_t mom_k;       // lambda_d eps_j / (2c) 2^64
  int64_t c_fx;        // (c / 2) 2^66
};

inline TrtFmaParams trt_fma_params(double lambda_e, double lambda_d, const double (&w)[3]) {
  TrtFmaParams p;
  p.c = lambda_e / 18.0;
  p.c2 = 2.0 * p.c;
  p.ch = 0.5 * p.c;
  const double r = lambda_d / (6.0 * p.c);
  int e = 0;
  frexp(r, &e);  // r in [2^(e-1), 2^e)
  int sh = 61 - e;  // r 2^sh in [2^60, 2^61)
  if (sh > 63) sh = 63;
  const bool fits = r >= 0 && sh >= 33;
  const int64_t rf = fits ? (int64_t)llrint(ldexp(r, sh)) : 0;
  p.r_hi = (int32_t)(rf >> 31);
  p.r_lo = (int32_t)(rf & 0x7fffffff);
  p.r_s = fits ? sh - 31 : 2;
  p.r_round = (int64_t)1 << (p.r_s - 2);
  p.dmax = !fits ? 0 : (r > 0 ? (int64_t)fmin(0x1p61 / r, 0x1p60) : (int64_t)1 << 60);
  const double km = ldexp(lambda_e * weight_sum_error(w) / p.c2, 64);
  const double kj = ldexp(lambda_d * first_moment_error(w) / p.c2, 64);
  p.mass_k = fabs(km) < 0x1p30 ? (int32_t)llrint(km) : 0;
  p.mom_k = fabs(kj) < 0x1p30 ? (int32_t)llrint(kj) : 0;
  p.c_fx = finish_takes(lambda_e) ? llrint(ldexp(p.ch, 66)) : 0;
  return p;
}

DF_HD int64_t abs64(int64_t v) { return v < 0 ? -v : v; }

// r D rounded to nearest (the error's mean is below 2^-25 unit: a bias in the
// antisymmetric brackets is a uniform force, see mul_shr), |D| < 2^60: four 32 x 32
// products.
DF_HD int64_t trt_rate(int64_t D, const TrtFmaParams& p) {
  const int32_t dh = (int32_t)(D >> 32);
  const uint32_t dl = (uint32_t)D;
  const uint64_t low = mad_wide_u(dl, (uint32_t)p.r_hi, mad_wide_u(dl, (uint32_t)p.r_lo, 0) >> 31);
  const int64_t mid = mad_wide(dh, p.r_lo, p.r_round);  // + half a unit / 2
  const int64_t a = (int64_t)(low + ((uint64_t)mid << 1));
  return (a >> p.r_s) + (int64_t)((uint64_t)mad_wide(dh, p.r_hi, 0) << (32 - p.r_s));
}

DF_HD void trt_brackets(const int64_t (&F)[9], const TrtFmaParams& p, int64_t (&Y)[9], bool& bad) {
  const int64_t R = (((F[5] + F[7]) + (F[6] + F[8])) + ((F[1] + F[3]) + (F[2] + F[4]))) + F[0];
  const int64_t d57 = F[5] - F[7], d86 = F[8] - F[6];
  const int64_t JX = (d57 + d86) + (F[1] - F[3]);
  const int64_t JY = (d57 - d86) + (F[2] - F[4]);
  const int64_t jx = shl(JX, 5), jy = shl(JY, 5);  // 2^64 j
  const int64_t X2 = round_shr(mulh64(jx, jx), 5), Y2 = round_shr(mulh64(jy, jy), 5), XY = round_shr(mulh64(jx, jy), 5);
  const int64_t J2 = X2 + Y2;
  const int64_t sx = 9 * (F[1] + F[3]) - 2 * R - 6 * X2 + 3 * Y2, dx = 3 * (F[1] - F[3]) - 2 * JX;
  const int64_t sy = 9 * (F[2] + F[4]) - 2 * R - 6 * Y2 + 3 * X2, dy = 3 * (F[2] - F[4]) - 2 * JY;
  const int64_t sp = 18 * (F[5] + F[7]) - R - 3 * J2 - 9 * XY, dp = 6 * d57 - (JX + JY);
  const int64_t sm = 18 * (F[8] + F[6]) - R - 3 * J2 + 9 * XY, dm = 6 * d86 - (JX - JY);
  const int64_t lim = (int64_t)1 << 61;
  bad |= (abs64(sx) | abs64(sy) | abs64(sp) | abs64(sm)) >= lim;
  bad |= (abs64(dx) | abs64(dy) | abs64(dp) | abs64(dm)) >= p.dmax;
  Y[0] = 4 * R - 6 * J2 - 9 * F[0] + scale_2m64(R, p.mass_k);
  const int64_t rx = trt_rate(dx, p) - scale_2m64(JX, p.mom_k);
  const int64_t ry = trt_rate(dy, p) - scale_2m64(JY, p.mom_k);
  const int64_t rp = trt_rate(dp, p), rm = trt_rate(dm, p);
  Y[1] = -(sx + rx);
  Y[3] = rx - sx;
  Y[2] = -(sy + ry);
  Y[4] = ry - sy;
  Y[5] = -(sp + rp);
  Y[7] = rp - sp;
  Y[8] = -(sm + rm);
  Y[6] = rm - sm;
}

template <bool SHIFTED = false, bool QUICK = false>
DF_HD void trt_fma(double (&f)[9], const TrtFmaParams& p, bool& bad) {
  int64_t F[9], Y[9];
  bool small;
  load_fixed<SHIFTED, SHIFTED>(f, F, bad, small);
  if (bad) return;
  trt_brackets(F, p, Y, bad);
  if constexpr (SHIFTED || !QUICK) {
#pragma unroll
    for (int q = 0; q < 9; q++) f[q] = fma_d(q == 0 ? p.c2 : (q < 5 ? p.c : p.ch), fixed_to_double_tr(Y[q]), f[q]);
  } else {
    finish<1>(f, Y, p.c_fx, p.c2, p.c, p.ch, small);
  }
}

}  // namespace hy
}  // namespace plbm
