// fixed.cuh -- fixed-point building blocks of the binary64 collisions
// (hybrid.cuh): population loads to int64, the truncated 64 x 64-bit product,
// and the reciprocal of the density, all on the integer pipes with no 64-bit
// conversion.
//
// Values are int64 multiples of 2^-59 unless a scale is named.  Everything is
// __host__ __device__ so that the arithmetic can be checked on the CPU.
#pragma once
#include "df64.cuh"

namespace plbm {
namespace hy {

// a b + c, one 32 x 32 -> 64-bit multiply-add (the compiler does not always see
// one in the widened C++ product: mulh64 took 17 instructions instead of 9).
DF_HD int64_t mad_wide(int32_t a, int32_t b, int64_t c) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (int64_t)((uint64_t)((int64_t)a * b) + (uint64_t)c);
#endif
}
DF_HD uint64_t mad_wide_u(uint32_t a, uint32_t b, uint64_t c) {
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (uint64_t)a * b + c;
#endif
}

// (a b) / 2^64 of two int64, within (-2, 2) units and unbiased to 1/4 unit:
// the three upper partial products of 32-bit halves, each lower half without
// its last bit so that it is a non-negative 31-bit integer and every product
// is a signed 32 x 32 -> 64 multiply-add (IMAD.WIDE; 9 instructions, a
// quarter of the exact 128-bit product).  What is left out lies between -1
// and 3 units with mean 3/4, which the constant adds back.  |a|, |b| < 2^63
// and |a b| < 2^126.
DF_HD int64_t mulh64(int64_t a, int64_t b) {
  const int32_t ah = (int32_t)(a >> 32), bh = (int32_t)(b >> 32);
  const int32_t al = (int32_t)((uint32_t)a >> 1), bl = (int32_t)((uint32_t)b >> 1);
  const int64_t m = mad_wide(ah, bl, mad_wide(al, bh, 0x60000000));
  return mad_wide(ah, bh, m >> 31);
}

// 2^61 / rho of R = rho 2^59, 1/4 < rho < 4, relative error below 2^-59: a
// binary32 seed (24 bits), then the second-order step
// y (1 + e + e^2), e = 1 - rho y, in the integers.  Other R give a
// meaningless value (the callers report such cells as out of range).
DF_HD int64_t recip_fixed(int64_t R) {
  // rho 2^30 and 2^26 / rho
  const float y = rcp_seed((float)(uint32_t)(R >> 29));
#ifdef __CUDA_ARCH__
  const uint32_t Y = __float2uint_rz(y * 0x1p56f);
#else
  const float yf = y * 0x1p56f;
  const uint32_t Y = yf < 0x1p31f ? (uint32_t)yf : 0x7fffffffu;
#endif
  // rho y 2^62 = R Y / 2^23
  const uint64_t p = (mad_wide_u((uint32_t)(R >> 32), Y, 0) << 9) + (mad_wide_u((uint32_t)R, Y, 0) >> 23);
  const int64_t e = (int64_t)(((uint64_t)1 << 62) - p);  // |e| < 2^40
  const int32_t eh = (int32_t)(e >> 12);
  const int64_t t = e + (mad_wide(eh, eh, 0) >> 38);     // (e + e^2) 2^62
  // y (1 + t) 2^61 = Y 2^35 + Y t / 2^27
  const uint64_t ty = (uint64_t)mad_wide((int32_t)(t >> 32), (int32_t)Y, 0) + ((uint64_t)Y << 30);
  return (int64_t)((ty << 5) + (mad_wide_u((uint32_t)t, Y, 1u << 26) >> 27));
}

}  // namespace hy
}  // namespace plbm
