// step_df64.cu -- deviation-storage steps whose collision runs in more than
// binary32: compensated binary32 (PLBM_MATH_HYBRID), double-float
// (PLBM_MATH_DF64) or binary64 (PLBM_MATH_STRICT) arithmetic on h = f - w,
// stored back in binary32 / scaled binary16.
//
// Compiled with --fmad=false: the double-float error-free transformations
// need every + - * rounded on its own; the fused operations are explicit.
#include "coll_df64.cuh"
#include "f32x2.cuh"
#include "plbm_launch.h"

namespace plbm {
namespace {

// Deviation storage, BGK evaluated in double-float on h.
template <class S>
__global__ void __launch_bounds__(kBlock) k_step_dev_df(const typename S::elem* __restrict__ src,
                                                       typename S::elem* __restrict__ dst, int nx, int ny, int ld,
                                                       Rows rows, df::DfParams p) {
  chain_begin();
  int x, y;
  flat_cell(rows, x, y);
  if (x >= nx) return;
  df::df64 h[9];
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const int sx = wrap_add(x, -cx_of(q), nx), sy = wrap_add(y, -cy_of(q), ny);
    h[q] = df::make(S::load(src, YFast::off(sx, sy, q, nx, ny, ld)), 0.0f);
  }
  df::bgk(h, p);
#pragma unroll
  for (int q = 0; q < 9; q++) S::store(dst, YFast::off(x, y, q, nx, ny, ld), h[q].hi + h[q].lo);
}

// Deviation storage, BGK with the compensated binary32 operator, a cell per thread:
// binary16, and binary32 below packed_bgk's line.
template <class S, typename I>
__global__ void __launch_bounds__(kBlock) k_step_dev_comp_one(const typename S::elem* __restrict__ src,
                                                             typename S::elem* __restrict__ dst, int nx, int ny,
                                                             int ld, Rows rows, df::DevParams p) {
  chain_begin();
  int x, y;
  flat_cell(rows, x, y);
  if (x >= nx) return;
  const I L = (I)ld, P = (I)ld * (I)nx;
  const I c0 = (I)x * L, cm = (I)wrap_m(x, nx) * L, cp = (I)wrap_p(x, nx) * L;
  const I y0 = (I)y, ym = (I)wrap_m(y, ny), yp = (I)wrap_p(y, ny);
  float h[9];
  h[0] = S::load(src, c0 + y0);
  h[1] = S::load(src, P + cm + y0);
  h[2] = S::load(src, 2 * P + c0 + ym);
  h[3] = S::load(src, 3 * P + cp + y0);
  h[4] = S::load(src, 4 * P + c0 + yp);
  h[5] = S::load(src, 5 * P + cm + ym);
  h[6] = S::load(src, 6 * P + cp + ym);
  h[7] = S::load(src, 7 * P + cp + yp);
  h[8] = S::load(src, 8 * P + cm + yp);
  df::bgk_dev_comp_one(h, p);
  const I o = c0 + y0;
#pragma unroll
  for (int q = 0; q < 9; q++) S::store(dst, (I)q * P + o, h[q]);
}

// Deviation storage, BGK with the compensated binary32 operator, two cells of
// adjacent columns per thread in packed binary32 registers: the operator's 350
// operations per cell bound the one-cell kernel by issue (437 instructions per
// cell, 4.4 cycles per cell and SM against the memory's 3.2), packed they take
// half the slots (4096 x 3000: 185 -> 169 us per step; the packed pipe 70 % busy).
// I: offset type (32-bit when the lattice has fewer than 2^32 elements).
template <class S, typename I>
__global__ void __launch_bounds__(kBlock) k_step_dev_comp(const typename S::elem* __restrict__ src,
                                                         typename S::elem* __restrict__ dst, int nx, int ny, int ld,
                                                         Rows rows, df::DevParams p) {
  chain_begin();
  int x, y;
  flat_cell(rows, x, y);
  if (x >= (nx + 1) / 2) return;
  x *= 2;
  const I L = (I)ld, P = (I)ld * (I)nx;
  const int x2 = wrap_p(x, nx);  // the second column (column 0 again after an odd last one)
  const I ca = (I)x * L, cb = (I)x2 * L, cm = (I)wrap_m(x, nx) * L, cp = (I)wrap_p(x2, nx) * L;
  const I y0 = (I)y, ym = (I)wrap_m(y, ny), yp = (I)wrap_p(y, ny);
  f32x2 h[9];
  h[0] = pack2(S::load(src, ca + y0), S::load(src, cb + y0));
  h[1] = pack2(S::load(src, P + cm + y0), S::load(src, P + ca + y0));
  h[2] = pack2(S::load(src, 2 * P + ca + ym), S::load(src, 2 * P + cb + ym));
  h[3] = pack2(S::load(src, 3 * P + cb + y0), S::load(src, 3 * P + cp + y0));
  h[4] = pack2(S::load(src, 4 * P + ca + yp), S::load(src, 4 * P + cb + yp));
  h[5] = pack2(S::load(src, 5 * P + cm + ym), S::load(src, 5 * P + ca + ym));
  h[6] = pack2(S::load(src, 6 * P + cb + ym), S::load(src, 6 * P + cp + ym));
  h[7] = pack2(S::load(src, 7 * P + cb + yp), S::load(src, 7 * P + cp + yp));
  h[8] = pack2(S::load(src, 8 * P + cm + yp), S::load(src, 8 * P + ca + yp));
  df::bgk_dev_comp(h, p);
  const I oa = ca + y0, ob = cb + y0;
#pragma unroll
  for (int q = 0; q < 9; q++) S::store(dst, (I)q * P + oa, lo2(h[q]));
  if (x2 > x) {
#pragma unroll
    for (int q = 0; q < 9; q++) S::store(dst, (I)q * P + ob, hi2(h[q]));
  }
}

// Deviation storage, collision evaluated in binary64 on h (any kind but BGKI).
template <class S, int KIND>
__global__ void __launch_bounds__(kBlock) k_step_dev_d(const typename S::elem* __restrict__ src,
                                                      typename S::elem* __restrict__ dst, int nx, int ny, int ld,
                                                      Rows rows, CollParams p) {
  chain_begin();
  int x, y;
  flat_cell(rows, x, y);
  if (x >= nx) return;
  double h[9];
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const int sx = wrap_add(x, -cx_of(q), nx), sy = wrap_add(y, -cy_of(q), ny);
    h[q] = (double)S::load(src, YFast::off(sx, sy, q, nx, ny, ld));
  }
  collide_shift<KIND, double>(h, p);
#pragma unroll
  for (int q = 0; q < 9; q++) S::store(dst, YFast::off(x, y, q, nx, ny, ld), (float)h[q]);
}

df::df64 split_const(double d) {
  const float hi = (float)d;
  return df::make(hi, (float)(d - (double)hi));
}

}  // namespace

cudaError_t step_pull_dev_hi(int storage, int math, int kind, const Sweep& s, const CollParams& cp) {
  if (math == 2) {  // compensated binary32
    if (kind != K_BGK) return cudaErrorNotSupported;
    const df::DevParams p = df::dev_params(cp.omega);
    const bool small = (unsigned long long)s.ld * (unsigned long long)s.nx * 9ull < (1ull << 32);
    // binary16: the one-cell kernel at every size (packed_bgk)
    if (storage == ST_F16DEV)
      return small ? step_cells<k_step_dev_comp_one<StoreF16Dev, uint32_t>>(s, s.ny, s.nx, false, true, p)
                   : step_cells<k_step_dev_comp_one<StoreF16Dev, size_t>>(s, s.ny, s.nx, false, true, p);
    if (storage != ST_F32DEV) return cudaErrorInvalidValue;
    if (!packed_bgk(s.nx, s.ny))  // fewer than 2^32 elements unless the rows are mostly padding
      return small ? step_cells<k_step_dev_comp_one<StoreF32Dev, uint32_t>>(s, s.ny, s.nx, false, true, p)
                   : step_cells<k_step_dev_comp_one<StoreF32Dev, size_t>>(s, s.ny, s.nx, false, true, p);
    const int pairs = s.nx / 2 + (s.nx & 1);
    const bool flat = dev_flat(s.ny, pairs);
    return small ? step_cells<k_step_dev_comp<StoreF32Dev, uint32_t>>(s, s.ny, pairs, false, flat, p)
                 : step_cells<k_step_dev_comp<StoreF32Dev, size_t>>(s, s.ny, pairs, false, flat, p);
  }
  // As the straight binary64 kernels, blocks by the grid's size and an even share for each SM.  Rows in
  // chained blocks of 256: 300 x 257 strict BGK 50.6 us per binary16 step (42.2 with launches apart; 21.3 now),
  // double-float 7.9 (6.4; 3.9); 513 x 700 strict BGK 106.8 and 95.3; rows that fill such blocks lose at
  // most 0.4 us in double-float (256^2 3.6 and 3.9, 4.1 with launches apart) and gain elsewhere.
  const bool flat = !rows_fit(s.ny, s.nx, true);
  if (math == 3) {  // double-float
    if (kind != K_BGK) return cudaErrorNotSupported;
    df::DfParams p;
    p.om = split_const(cp.omega);
    p.omb = split_const(cp.omegabar);
    p.w0 = split_const(W0);
    p.ws = split_const(WS);
    p.wd = split_const(WD);
    p.ws3 = split_const(3.0 * WS);
    p.wd3 = split_const(3.0 * WD);
    if (storage == ST_F32DEV) return step_cells<k_step_dev_df<StoreF32Dev>>(s, s.ny, s.nx, true, flat, p);
    if (storage == ST_F16DEV) return step_cells<k_step_dev_df<StoreF16Dev>>(s, s.ny, s.nx, true, flat, p);
    return cudaErrorInvalidValue;
  }
#define PLBM_DEVD(S)                                                                           \
  switch (kind) {                                                                              \
    case K_BGK: return step_cells<k_step_dev_d<S, K_BGK>>(s, s.ny, s.nx, true, flat, cp);      \
    case K_TRT: return step_cells<k_step_dev_d<S, K_TRT>>(s, s.ny, s.nx, true, flat, cp);      \
    case K_RR: return step_cells<k_step_dev_d<S, K_RR>>(s, s.ny, s.nx, true, flat, cp);        \
    default: return cudaErrorNotSupported;                                                     \
  }
  if (storage == ST_F32DEV) PLBM_DEVD(StoreF32Dev)
  if (storage == ST_F16DEV) PLBM_DEVD(StoreF16Dev)
#undef PLBM_DEVD
  return cudaErrorInvalidValue;
}

}  // namespace plbm
