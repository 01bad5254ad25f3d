// step_hybrid.cu -- binary64-storage fused steps in the fixed-point arithmetic of
// hybrid.cuh (exact integer moments, one binary64 FMA per population), BGK, TRT
// and RR: the lattice step, the plugin's collide-and-push step and the
// finite-volume / finite-difference schemes.  They serve PLBM_MATH_HYBRID and,
// their error being no larger than the straight binary64 kernels' at a fraction
// of the binary64 instructions, PLBM_MATH_FMA.  Cells outside the fixed point's
// range are evaluated with the binary64 operator of the reference (hybrid grids
// also set the range flag); this file is compiled with FMA contraction, which
// concerns those cells only.
#include "hybrid.cuh"
#include "plbm_launch.h"
#include "schemes.cuh"

namespace plbm {

// Set to 1 by a hybrid kernel that met a cell outside its range.
__device__ int g_hybrid_range_flag = 0;

namespace {

// Constants of one hybrid launch: the hybrid operator's and the binary64
// operator's (for cells outside the hybrid range).
struct HybridArgs {
  hy::BgkParams bgk1;  // BGK (bgk_fma, populations or shifted populations)
  hy::BgkParams rr1;   // RR (rr_fma): the one-FMA constants at omega = 1
  hy::TrtFmaParams trt;  // TRT (trt_fma)
  hy::RrParams rr;
  CollParams ref;
  int report;  // set the range flag (PLBM_MATH_HYBRID)
};

// One cell outside the hybrid range: pull, the binary64 operator of the
// reference, store.  Out of line so that the hot kernel's registers and code
// are not shaped by this rarely taken path.
template <int KIND>
__device__ __noinline__ void hybrid_fallback_cell(const double* __restrict__ src, double* __restrict__ dst, int x,
                                                  int y, int nx, int ny, int ld, const CollParams& p, int report) {
  double f[9];
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const int sx = wrap_add(x, -cx_of(q), nx), sy = wrap_add(y, -cy_of(q), ny);
    f[q] = ld_chain(src + YFast::off(sx, sy, q, nx, ny, ld));
  }
  collide_ref<KIND>(f, p);
#pragma unroll
  for (int q = 0; q < 9; q++) dst[YFast::off(x, y, q, nx, ny, ld)] = f[q];
  if (report) g_hybrid_range_flag = 1;
}

// Resident CTAs per SM the one-cell kernels are compiled for: BGK (bgk_fma) and
// TRT (trt_fma) at 4, RR (rr_fma) at 3 (register caps 64 and 80).  Capped at
// 48 registers for 5 CTAs the BGK kernel spills and runs 2 % slower at 8192^2.
constexpr int hybrid_min_blocks(int kind) { return kind == K_RR ? 3 : 4; }

// I: index type of the lattice offsets; 32-bit when the whole lattice has
// fewer than 2^32 elements (one multiply-add per address instead of 64-bit
// arithmetic).  QUICK: see kQuickCells.
template <typename I, int KIND, bool QUICK>
__global__ void __launch_bounds__(kBlock, hybrid_min_blocks(KIND)) k_step_hybrid(const double* __restrict__ src,
                                                                                double* __restrict__ dst, int nx,
                                                                                int ny, int ld, Rows rows,
                                                                                HybridArgs a) {
  chain_begin();
  int x, y;
  flat_cell(rows, x, y);
  if (x >= nx) return;
  const I L = (I)ld, P = (I)ld * (I)nx;
  const I c0 = (I)x * L, cm = (I)wrap_m(x, nx) * L, cp = (I)wrap_p(x, nx) * L;
  const I y0 = (I)y, ym = (I)wrap_m(y, ny), yp = (I)wrap_p(y, ny);
  double f[9];
  // pull: f_q(x, y) = f_q(x - cx_q, y - cy_q) of the source lattice
  f[0] = ld_chain(src + (c0 + y0));
  f[1] = ld_chain(src + (P + cm + y0));
  f[2] = ld_chain(src + (2 * P + c0 + ym));
  f[3] = ld_chain(src + (3 * P + cp + y0));
  f[4] = ld_chain(src + (4 * P + c0 + yp));
  f[5] = ld_chain(src + (5 * P + cm + ym));
  f[6] = ld_chain(src + (6 * P + cp + ym));
  f[7] = ld_chain(src + (7 * P + cp + yp));
  f[8] = ld_chain(src + (8 * P + cm + yp));
  bool bad = false;
  if (KIND == K_TRT) hy::trt_fma<false, QUICK>(f, a.trt, bad);
  else if (KIND == K_RR) hy::rr_fma<false, QUICK>(f, a.rr, a.rr1, bad);
  else hy::bgk_fma<false, QUICK>(f, a.bgk1, bad);
  if (bad) {  // outside the hybrid range: the binary64 operator on the same inputs
    hybrid_fallback_cell<KIND>(src, dst, x, y, nx, ny, ld, a.ref, a.report);
    return;
  }
  const I o = c0 + y0;
#pragma unroll
  for (int q = 0; q < 9; q++) dst[(I)q * P + o] = f[q];
}

// The same step for large grids (BGK and TRT): a CTA keeps its 128 rows and walks
// along x over seg columns, each thread copying its own nine populations of the
// next column into shared memory (cp.async: no register held, no barrier, no
// latency waited for) while it collides the present ones.  One cell per thread
// leaves the loads' latency to the other CTAs of the SM, of which the registers
// allow four; here the memory stays busy.  8192^2, GLUPS: BGK 42.4 one cell per
// thread, 46.8 here (144 bytes per cell at the copy bandwidth: 48), TRT 37.5 and
// 40.0; 2048^2 BGK 40.8 and 43.8, TRT 36.3 and 37.5.  RR (32.6 and 32.9, 31.8 and
// 31.3) is bound by its instructions and keeps one cell per thread.  Three columns
// in flight take shared memory from the L1 cache that the neighbours' rows live
// in: slower.
constexpr int kAheadThreads = 128;
template <int KIND>
__global__ void __launch_bounds__(kAheadThreads, 8)
    k_step_ahead(const double* __restrict__ src, double* __restrict__ dst, int nx, int ny, int ld, int ytiles, int seg,
                 HybridArgs a) {
  __shared__ double sm[2][9][kAheadThreads];  // a thread reads what it copied itself
  chain_begin();
  const int bx = blockIdx.x / ytiles;
  const int y = (blockIdx.x - bx * ytiles) * kAheadThreads + threadIdx.x;
  if (y >= ny) return;
  const unsigned ym = wrap_m(y, ny), yp = wrap_p(y, ny);
  const size_t P = (size_t)ld * nx;
  const int x0 = bx * seg, x1 = min(x0 + seg, nx);
  auto copy_column = [&](int x, int stage) {
    const double *c0 = src + (size_t)x * ld, *cm = src + (size_t)wrap_m(x, nx) * ld, *cp = src + (size_t)wrap_p(x, nx) * ld;
    const unsigned s0 = (unsigned)__cvta_generic_to_shared(&sm[stage][0][threadIdx.x]);
    auto copy = [&](int q, const double* p) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s0 + q * (unsigned)(8 * kAheadThreads)), "l"(p)
                   : "memory");
    };
    copy(0, c0 + y);
    copy(1, cm + P + y);
    copy(2, c0 + 2 * P + ym);
    copy(3, cp + 3 * P + y);
    copy(4, c0 + 4 * P + yp);
    copy(5, cm + 5 * P + ym);
    copy(6, cp + 6 * P + ym);
    copy(7, cp + 7 * P + yp);
    copy(8, cm + 8 * P + yp);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  copy_column(x0, 0);
  int stage = 0;
#pragma unroll 1
  for (int x = x0; x < x1; x++) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    double f[9];
#pragma unroll
    for (int q = 0; q < 9; q++) f[q] = sm[stage][q][threadIdx.x];
    stage ^= 1;
    if (x + 1 < x1) copy_column(x + 1, stage);
    bool bad = false;
    if (KIND == K_TRT) hy::trt_fma(f, a.trt, bad);
    else hy::bgk_fma(f, a.bgk1, bad);
    if (bad) {
      hybrid_fallback_cell<KIND>(src, dst, x, y, nx, ny, ld, a.ref, a.report);
      continue;
    }
    double* o = dst + (size_t)x * ld;
#pragma unroll
    for (int q = 0; q < 9; q++) (o + q * P)[(unsigned)y] = f[q];
  }
}

// Whether a grid takes k_step_ahead: BGK from 2^20 cells (1024^2 37.3 GLUPS against
// 36.2 one cell per thread; 512^2 slower), TRT from 2^22 (2048^2 37.5 and 36.3;
// 1024^2 31.7 and 32.7), rows enough to fill half a CTA.
bool takes_ahead(int kind, const Sweep& s) {
  const long long cells = (long long)s.nx * s.ny;
  return s.ny >= kAheadThreads / 2 && ((kind == K_BGK && cells >= 1 << 20) || (kind == K_TRT && cells >= 1 << 22));
}

template <int KIND>
cudaError_t launch_ahead(const Sweep& s, const HybridArgs& a) {
  const int yt = (s.ny + kAheadThreads - 1) / kAheadThreads;
  // Columns per CTA: 4 keep the last wave short (2048^2 BGK 43.8 GLUPS against 43.2 with
  // 8), 8 where there are tens of waves (8192^2 46.8 against 46.5).
  const int seg = (long long)s.nx * s.ny >= 1 << 25 ? 8 : 4;
  const long long blocks = (long long)yt * ((s.nx + seg - 1) / seg);
  if (blocks <= 0 || blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  chained(k_step_ahead<KIND>, (unsigned)blocks, kAheadThreads, s.stream)(
      static_cast<const double*>(s.src), static_cast<double*>(s.dst), s.nx, s.ny, s.ld, yt, seg, a);
  return cudaGetLastError();
}

// A finite-volume / finite-difference streaming scheme in stencil form fused
// with the hybrid collision (binary64 storage).  Out-of-range cells take the
// binary64 collision (out of line, the stencil evaluated again).
template <int TAPS, int KIND>
__device__ __noinline__ void scheme_fallback_cell(const double* __restrict__ src, double* __restrict__ dst, int x,
                                                  int y, int nx, int ny, int ld, const sch::Stencil& st,
                                                  const CollParams& p, int report) {
  double f[9];
  sch::stencil_pull<YFast, TAPS>(src, x, y, nx, ny, ld, st, f);
  collide_ref<KIND>(f, p);
#pragma unroll
  for (int q = 0; q < 9; q++) dst[YFast::off(x, y, q, nx, ny, ld)] = f[q];
  if (report) g_hybrid_range_flag = 1;
}

template <int TAPS, int KIND>
__global__ void __launch_bounds__(kBlock) k_step_scheme_hybrid(const double* __restrict__ src,
                                                              double* __restrict__ dst, int nx, int ny, int ld,
                                                              int ftiles, sch::Stencil st, HybridArgs a) {
  chain_begin();
  const int x = blockIdx.x / ftiles;
  const int y = (blockIdx.x - x * ftiles) * blockDim.x + threadIdx.x;
  if (y >= ny) return;
  double f[9];
  sch::stencil_pull<YFast, TAPS>(src, x, y, nx, ny, ld, st, f);
  bool bad = false;
  if (KIND == K_TRT) hy::trt_fma(f, a.trt, bad);
  else if (KIND == K_RR) hy::rr_fma(f, a.rr, a.rr1, bad);
  else hy::bgk_fma(f, a.bgk1, bad);
  if (bad) {
    scheme_fallback_cell<TAPS, KIND>(src, dst, x, y, nx, ny, ld, st, a.ref, a.report);
    return;
  }
#pragma unroll
  for (int q = 0; q < 9; q++) dst[YFast::off(x, y, q, nx, ny, ld)] = f[q];
}

// ---- finite-difference streaming in the fixed point --------------------------
// Every scheme but the Gaussian-weighted ones is
//   f*_q = f_q - a1 D1 + a2 D2,
// D1 and D2 integer combinations of the 3x3 neighbourhood (first differences
// along c_q, second differences), so on int64 populations the sums are exact
// and two products per population remain where the stencil form takes 3 or 9
// binary64 FMAs (48 per cell for FVM / central FDM: the binary64 pipe's 25
// cycles per cell and SM).  A CTA converts the populations of a 32 x TX tile
// and its halo to the fixed point once, in shared memory.  The streamed
// population joins the collision as an integer, and the new one,
//   f'_q = F_q + (a2 D2 - a1 D1) + k_q c Y_q  (at 2^-61),
// is rounded to binary64 once: no binary64 instruction at all.
// Rule: LINE (Sofonea), CENTRAL (FVM, which expands to the same sums, and central
// FDM), ISO and WLS, while a1 and a2 are below 2^(shift - 4) (time steps up to
// about 1, the scheme's own stability limit); other schemes and steps keep the
// stencil form.  512^2, central FDM, BGK, dt = 0.3: 68 us per step in the stencil
// form with the binary64 collision, 33 us with the fixed-point collision, 16.8 us
// here (15.6 GLUPS; 2048^2 17.0 against 4.2 and 8.0); error against binary64
// arithmetic of the reference's expressions 4.4e-16 (stencil form 2.1e-15).
// Bound by the integer pipe: about 1,450 instructions per cell, the ALU pipe 70 % busy.
enum { FORM_LINE = 0, FORM_CENTRAL = 1, FORM_ISO = 2, FORM_WLS = 3 };
// Left shift of D1, D2 before the product: the largest for which |D| 2^shift stays
// below 2^63 for axis populations below 1/4 and diagonal ones below 1/8.
__host__ __device__ constexpr int form_shift(int form) { return form <= FORM_CENTRAL ? 3 : (form == FORM_ISO ? 1 : 2); }

struct SchemeFx {
  int64_t a1s, a2s, a1d, a2d;  // a1, a2 of axis and diagonal populations, 2^(66 - shift) a
  int64_t c;                   // 2^66 of the collision's constant (1/36 of the rate)
};

template <int FORM>
__device__ __forceinline__ void scheme_differences(const int64_t (&v)[9], int q, int64_t& d1, int64_t& d2) {
  using namespace sch;
  const int cx = cx_of(q), cy = cy_of(q);
  if (FORM == FORM_LINE || (FORM == FORM_CENTRAL && q <= 4)) {
    const int64_t u = v[nb(cx, cy)], d = v[nb(-cx, -cy)];
    d1 = u - d;
    d2 = u + d - 2 * v[C];
    return;
  }
  if (FORM == FORM_CENTRAL) {
    const int64_t dx = v[E] - v[W], dy = v[N] - v[S];
    const int64_t xy = (v[NE] + v[SW]) - (v[NW] + v[SE]);
    d1 = (cx > 0 ? dx : -dx) + (cy > 0 ? dy : -dy);
    d2 = 2 * ((v[E] + v[W]) + (v[N] + v[S]) - 4 * v[C]) + (cx * cy > 0 ? xy : -xy);
    return;
  }
  constexpr int wa = FORM == FORM_ISO ? 4 : 1, wb = FORM == FORM_ISO ? 10 : 1;
  const int64_t dx = (v[NE] - v[NW]) + (v[SE] - v[SW]) + wa * (v[E] - v[W]);
  const int64_t dy = (v[NE] - v[SE]) + (v[NW] - v[SW]) + wa * (v[N] - v[S]);
  const int64_t xx = (v[NE] + v[NW] - 2 * v[N]) + (v[SE] + v[SW] - 2 * v[S]) + wb * (v[E] + v[W] - 2 * v[C]);
  const int64_t yy = (v[NE] + v[SE] - 2 * v[E]) + (v[NW] + v[SW] - 2 * v[W]) + wb * (v[N] + v[S] - 2 * v[C]);
  d1 = (cx > 0 ? dx : (cx < 0 ? -dx : 0)) + (cy > 0 ? dy : (cy < 0 ? -dy : 0));
  if (q <= 4) {
    d2 = cx ? xx : yy;
  } else {
    const int64_t xy = (v[NE] + v[SW]) - (v[NW] + v[SE]);
    constexpr int kx = FORM == FORM_ISO ? 1 : 2, kd = FORM == FORM_ISO ? 6 : 3;
    d2 = kx * (xx + yy) + (cx * cy > 0 ? kd * xy : -kd * xy);
  }
}

__host__ __device__ constexpr int form_taps(int form) {
  return form == FORM_LINE ? sch::TAPS_LINE : (form == FORM_CENTRAL ? sch::TAPS_AXIS3 : sch::TAPS_FULL);
}

// 256 threads: warp w loads population w + 1 of the tile, then takes the columns
// w, w + 8, ... below TX (its lanes the 32 rows).
template <int FORM, int KIND, int TX>
__global__ void __launch_bounds__(256, KIND == K_RR ? 3 : 4)
    k_step_scheme_fixed(const double* __restrict__ src, double* __restrict__ dst, int nx, int ny, int ld, int ytiles,
                        SchemeFx sc, sch::Stencil st, HybridArgs a) {
  chain_begin();
  constexpr int ROWS = 34;
  __shared__ int64_t sm[8][TX + 2][ROWS];
  __shared__ int tile_bad;
  const int x0 = (blockIdx.x / ytiles) * TX, y0 = (blockIdx.x % ytiles) * 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) tile_bad = 0;
  __syncthreads();
  {
    bool bad = false;
    const double* f = src + (size_t)(warp + 1) * ld * nx;
    // every load first, then the conversions (their rare out-of-line path would
    // otherwise put one memory latency after the other)
    auto load = [&](int c, int r) {
      const int gx = x0 - 1 + c, gy = y0 - 1 + r;
      if (gx > nx || gy > ny) return 0.0;  // past the last cell's neighbours
      return ld_chain(f + (size_t)(gx < 0 ? nx - 1 : (gx == nx ? 0 : gx)) * ld +
                   (gy < 0 ? ny - 1 : (gy == ny ? 0 : gy)));
    };
    auto convert = [&](double d) {
      return warp < 4 ? hy::to_fixed_nonneg<1020>(d, bad) : hy::to_fixed_nonneg<1019>(d, bad);
    };
    constexpr int EX = (2 * (TX + 2) + 31) / 32;  // rows 32 and 33, two per column
    double d[TX + 2], e[EX];
#pragma unroll
    for (int c = 0; c < TX + 2; c++) d[c] = load(c, lane);
#pragma unroll
    for (int i = 0; i < EX; i++) e[i] = lane + 32 * i < 2 * (TX + 2) ? load((lane >> 1) + 16 * i, 32 + (lane & 1)) : 0.0;
#pragma unroll
    for (int c = 0; c < TX + 2; c++) sm[warp][c][lane] = convert(d[c]);
#pragma unroll
    for (int i = 0; i < EX; i++)
      if (lane + 32 * i < 2 * (TX + 2)) sm[warp][(lane >> 1) + 16 * i][32 + (lane & 1)] = convert(e[i]);
    if (bad) tile_bad = 1;
  }
  __syncthreads();
  const int y = y0 + lane;
  if (y >= ny) return;
  const size_t P = (size_t)ld * nx;
#pragma unroll 1
  for (int c = warp; c < TX && x0 + c < nx; c += 8) {
    const int x = x0 + c;
    const size_t o = (size_t)x * ld + y;
    bool bad = tile_bad;
    int64_t F[9], Z[9];
    if (!bad) {
      F[0] = hy::to_fixed_nonneg<1022>(ld_chain(src + o), bad);
      Z[0] = hy::shl(F[0], 2);
#pragma unroll
      for (int q = 1; q < 9; q++) {
        int64_t v[9], d1, d2;
#pragma unroll
        for (int k = 0; k < 9; k++) v[k] = sm[q - 1][c + 1 + sch::ex(k)][lane + 1 + sch::ey(k)];
        scheme_differences<FORM>(v, q, d1, d2);
        constexpr int S = form_shift(FORM);
        const int64_t d = hy::mulh64(hy::shl(d2, S), q < 5 ? sc.a2s : sc.a2d) -
                          hy::mulh64(hy::shl(d1, S), q < 5 ? sc.a1s : sc.a1d);
        Z[q] = hy::shl(v[sch::C], 2) + d;
        F[q] = hy::round_shr(Z[q], 2);
        bad |= (uint32_t)((uint64_t)F[q] >> 32) >= (1u << (q < 5 ? 25 : 24));
      }
      int64_t Y[9];
      if (KIND == K_TRT) hy::trt_brackets(F, a.trt, Y, bad);
      else if (KIND == K_RR) hy::rr_brackets<false>(F, a.rr, a.rr1, Y, bad);
      else hy::bgk_brackets<false>(F, a.bgk1, Y, bad);
#pragma unroll
      for (int q = 0; q < 9; q++) {
        const int k = q == 0 ? 4 : (q > 4 ? 1 : (KIND == K_TRT ? 2 : 4));
        Z[q] += k * hy::mulh64(Y[q], sc.c);
        bad |= Z[q] <= 0;
      }
    }
    if (bad) {
      scheme_fallback_cell<form_taps(FORM), KIND>(src, dst, x, y, nx, ny, ld, st, a.ref, a.report);
      continue;
    }
#pragma unroll
    for (int q = 0; q < 9; q++) dst[q * P + o] = hy::pos_fixed_to_double<61>(Z[q]);
  }
}

// The plugin step (sim/sim.F90:404-505 + :568-624) in the hybrid arithmetic:
// shifted binary64 populations h = f - w in the x-fastest layout, collide at
// the cell, push along c_q.  Out-of-range cells take the shifted binary64
// operator of the FMA plugin kernel (out of line), BGK cells of tiny h finer units.
template <int KIND>
__device__ __noinline__ void push_fallback_cell(const double* __restrict__ src, double* __restrict__ dst, int x,
                                                int y, int nx, int ny, int ld, const HybridArgs& a) {
  double f[9];
#pragma unroll
  for (int q = 0; q < 9; q++) f[q] = ld_chain(src + XFast::off(x, y, q, nx, ny, ld));
  const bool fixed = KIND == K_BGK && hy::bgk_rest(f, a.bgk1);
  if (!fixed) collide_shift<KIND, double>(f, a.ref);
#pragma unroll
  for (int q = 0; q < 9; q++) dst[XFast::off(wrap_add(x, cx_of(q), nx), wrap_add(y, cy_of(q), ny), q, nx, ny, ld)] = f[q];
  if (!fixed && a.report) g_hybrid_range_flag = 1;
}

template <typename I, int KIND>
__global__ void __launch_bounds__(kBlock, hybrid_min_blocks(KIND)) k_push_hybrid(const double* __restrict__ src,
                                                                                double* __restrict__ dst, int nx,
                                                                                int ny, int ld, Rows rows,
                                                                                HybridArgs a) {
  chain_begin();
  int x, y;
  flat_cell(rows, y, x);
  if (y >= ny) return;
  const I L = (I)ld, P = (I)ld * (I)ny;
  const I o = (I)y * L + (I)x;
  double f[9];
#pragma unroll
  for (int q = 0; q < 9; q++) f[q] = ld_chain(src + ((I)q * P + o));
  bool bad = false;
  if (KIND == K_TRT) hy::trt_fma<true>(f, a.trt, bad);
  else if (KIND == K_RR) hy::rr_fma<true>(f, a.rr, a.rr1, bad);
  else hy::bgk_fma<true>(f, a.bgk1, bad);
  if (bad) {
    push_fallback_cell<KIND>(src, dst, x, y, nx, ny, ld, a);
    return;
  }
  const I xm = (I)wrap_m(x, nx), xp = (I)wrap_p(x, nx), x0 = (I)x;
  const I rm = (I)wrap_m(y, ny) * L, rp = (I)wrap_p(y, ny) * L, r0 = (I)y * L;
  // push: f_q goes to (x + cx_q, y + cy_q)
  dst[r0 + x0] = f[0];
  dst[P + r0 + xp] = f[1];
  dst[2 * P + rp + x0] = f[2];
  dst[3 * P + r0 + xm] = f[3];
  dst[4 * P + rm + x0] = f[4];
  dst[5 * P + rp + xp] = f[5];
  dst[6 * P + rp + xm] = f[6];
  dst[7 * P + rm + xm] = f[7];
  dst[8 * P + rm + xp] = f[8];
}

// Cells up to which the last operations take the branch-free form (hy::finish): a
// grid of so few warps waits for one warp's chain of instructions, which that form
// shortens; with more warps its 130 further instructions per cell, and the cells
// that change binade, cost more.  us per step of a Taylor-Green flow, RR / BGK / TRT,
// with and without: 64^2 2.23 / 1.97 / 2.09 and 2.58 / 2.33 / 2.45, 128^2 2.44 / 2.19 /
// 2.31 and 2.71 / 2.45 / 2.58, 192^2 3.23 / 2.98 / 2.97 and 3.09 / 2.83 / 2.88.
constexpr long long kQuickCells = 1 << 14;

template <int KIND>
cudaError_t launch_hybrid(const Sweep& s, const HybridArgs& a) {
  if ((unsigned long long)s.ld * (unsigned long long)s.nx * 9ull >= (1ull << 32))
    return step_cells<k_step_hybrid<size_t, KIND, false>>(s, s.ny, s.nx, true, true, a);
  if ((long long)s.nx * s.ny > kQuickCells || !hy::finish_takes(a.ref.omega))
    return step_cells<k_step_hybrid<uint32_t, KIND, false>>(s, s.ny, s.nx, true, true, a);
  // rows that fill their blocks: the same cells, 0.1 us (of 2) sooner
  const bool flat = s.ny % block_for((long long)s.nx * s.ny, true) != 0;
  return step_cells<k_step_hybrid<uint32_t, KIND, true>>(s, s.ny, s.nx, true, flat, a);
}

template <int KIND>
cudaError_t launch_push(const Sweep& s, const HybridArgs& a) {
  if ((unsigned long long)s.ld * (unsigned long long)s.ny * 9ull < (1ull << 32))
    return step_cells<k_push_hybrid<uint32_t, KIND>>(s, s.nx, s.ny, true, true, a);
  return step_cells<k_push_hybrid<size_t, KIND>>(s, s.nx, s.ny, true, true, a);
}

}  // namespace

hy::BgkParams hybrid_bgk_params(double omega) {
  const double w[3] = {W0, WS, WD};
  return hy::bgk_fma_params(omega, w);
}

// Constants of the one-FMA TRT from the launch's binary64 parameters
// (lambda_e = omega, lambda_d as the reference forms it).
hy::TrtFmaParams hybrid_trt_params(const CollParams& cp) {
  const double w[3] = {W0, WS, WD};
  return hy::trt_fma_params(cp.omega, cp.lambda_d, w);
}

namespace {
HybridArgs hybrid_args(const CollParams& cp, bool report) {
  HybridArgs a;
  a.bgk1 = hybrid_bgk_params(cp.omega);
  a.rr1 = hybrid_bgk_params(1.0);
  a.trt = hybrid_trt_params(cp);
  a.rr = hy::rr_fma_params(cp.omega);
  a.ref = cp;
  a.report = report;
  return a;
}
}  // namespace

cudaError_t step_pull_fixed(int kind, const Sweep& s, const CollParams& cp, bool report) {
  if (kind != K_BGK && kind != K_TRT && kind != K_RR) return cudaErrorNotSupported;
  const HybridArgs a = hybrid_args(cp, report);
  if (kind == K_RR) return launch_hybrid<K_RR>(s, a);
  if (takes_ahead(kind, s)) return kind == K_TRT ? launch_ahead<K_TRT>(s, a) : launch_ahead<K_BGK>(s, a);
  return kind == K_TRT ? launch_hybrid<K_TRT>(s, a) : launch_hybrid<K_BGK>(s, a);
}

cudaError_t step_push_fixed(int kind, const Sweep& s, const CollParams& cp, bool report) {
  if (kind != K_BGK && kind != K_TRT && kind != K_RR) return cudaErrorNotSupported;
  const HybridArgs a = hybrid_args(cp, report);
  return kind == K_TRT ? launch_push<K_TRT>(s, a) : (kind == K_RR ? launch_push<K_RR>(s, a) : launch_push<K_BGK>(s, a));
}

namespace {
// The fixed-point constants of a scheme, or false where it keeps the stencil
// form (see k_step_scheme_fixed).
bool scheme_fixed_constants(int scheme, int kind, double dt, double omega, int& form, SchemeFx& c) {
  if (!hy::finish_takes(omega)) return false;
  double a1s, a2s, a1d, a2d;
  switch (scheme) {
    case sch::SOFONEA:
      form = FORM_LINE;
      a1s = 0.5 * dt, a2s = 0.5 * dt * dt;
      a1d = dt * 0.35355339059327373, a2d = 0.25 * dt * dt;
      break;
    case sch::FVM:
    case sch::FDM:
      form = FORM_CENTRAL;
      a1s = a1d = 0.5 * dt, a2s = 0.5 * dt * dt, a2d = 0.25 * dt * dt;
      break;
    case sch::FDM_ISO:
      form = FORM_ISO;
      a1s = a1d = dt / 12.0, a2s = a2d = dt * dt / 24.0;
      break;
    case sch::FDM_WLS:
      form = FORM_WLS;
      a1s = a1d = dt / 6.0, a2s = dt * dt / 6.0, a2d = dt * dt / 12.0;
      break;
    default: return false;
  }
  const int s = form_shift(form);
  const double lim = ldexp(1.0, s - 4);
  if (!(a1s < lim && a2s < lim && a1d < lim && a2d < lim)) return false;
  c.a1s = llrint(ldexp(a1s, 66 - s));
  c.a2s = llrint(ldexp(a2s, 66 - s));
  c.a1d = llrint(ldexp(a1d, 66 - s));
  c.a2d = llrint(ldexp(a2d, 66 - s));
  c.c = llrint(ldexp((kind == K_RR ? 1.0 : omega) / 36.0, 66));
  return true;
}

// Tile columns of k_step_scheme_fixed: four for grids whose wider tiles would not
// give every SM a CTA, 16 (two cells per thread, the smaller halo) where every SM
// gets several.  BGK, central FDM, us per step with 2 / 4 / 8 / 16 columns: 64^2 3.2 / 3.3 /
// 4.4 / -, 128^2 4.0 / 3.3 / 4.3 / -, 180^2 6.2 / 5.2 / 5.9 / -, 256^2 - / 6.4 / 6.1 / 7.7,
// 512^2 - / 18.5 / 16.9 / 19.6, 1000^2 - / 70.8 / 64.3 / 66.5; 6, 10, 12 and 14 columns lie
// between or above, and so do 3 and 5 CTAs per SM.
int scheme_tile(const Sweep& s) {
  const long long cells = (long long)s.nx * s.ny;
  return cells > (1 << 20) ? 16 : (cells > 40000 ? 8 : 4);
}

template <int FORM, int TX>
void launch_scheme_fixed(int kind, const Sweep& s, const SchemeFx& c, const sch::Stencil& st, const HybridArgs& a) {
  const double* src = static_cast<const double*>(s.src);
  double* dst = static_cast<double*>(s.dst);
  const int yt = (s.ny + 31) / 32;
  const unsigned nb = (unsigned)((long long)yt * ((s.nx + TX - 1) / TX));
  if (kind == K_TRT) chained(k_step_scheme_fixed<FORM, K_TRT, TX>, nb, 256, s.stream)(src, dst, s.nx, s.ny, s.ld, yt, c, st, a);
  else if (kind == K_RR) chained(k_step_scheme_fixed<FORM, K_RR, TX>, nb, 256, s.stream)(src, dst, s.nx, s.ny, s.ld, yt, c, st, a);
  else chained(k_step_scheme_fixed<FORM, K_BGK, TX>, nb, 256, s.stream)(src, dst, s.nx, s.ny, s.ld, yt, c, st, a);
}
// The stencil form, rows in blocks by the grid's size and an even share for each SM: chained in
// blocks of 256, an SM could get two shares (304 x 256 TRT, Gaussian-weighted: 20.1 us per step, 14.9 with
// launches apart and 14.1 now; 300 x 257 BGK 25.9 and 16.6, 128 x 130 6.3 and 6.6, 1024^2 164.2 and 164.3).
template <int TAPS, int KIND>
cudaError_t launch_scheme_stencil(const Sweep& s, const sch::Stencil& st, const HybridArgs& a) {
  constexpr auto kernel = k_step_scheme_hybrid<TAPS, KIND>;
  Spread w;
  if (cudaError_t e = spread_cells(s.ny, s.nx, true, false, resident_threads<kernel>(), &w)) return e;
  chained(kernel, w, s.stream)(static_cast<const double*>(s.src), static_cast<double*>(s.dst), s.nx, s.ny, s.ld,
                               w.rows.tiles, st, a);
  return cudaGetLastError();
}
}  // namespace

cudaError_t step_scheme_fixed(int scheme, int kind, const Sweep& s, double dt, const CollParams& cp, bool report) {
  if (kind != K_BGK && kind != K_TRT && kind != K_RR) return cudaErrorNotSupported;
  if (scheme < sch::FVM || scheme > sch::FDM_WLS_G2) return cudaErrorInvalidValue;
  const sch::Stencil st = sch::stencil_coefficients(scheme, dt);
  const HybridArgs a = hybrid_args(cp, report);
  int form;
  SchemeFx c;
  if (scheme_fixed_constants(scheme, kind, dt, cp.omega, form, c)) {
    const int tx = scheme_tile(s);
#define PLBM_SCH_FX(F)                                             \
  if (tx == 16) launch_scheme_fixed<F, 16>(kind, s, c, st, a);     \
  else if (tx == 8) launch_scheme_fixed<F, 8>(kind, s, c, st, a);  \
  else launch_scheme_fixed<F, 4>(kind, s, c, st, a)
    switch (form) {
      case FORM_LINE: PLBM_SCH_FX(FORM_LINE); break;
      case FORM_CENTRAL: PLBM_SCH_FX(FORM_CENTRAL); break;
      case FORM_ISO: PLBM_SCH_FX(FORM_ISO); break;
      default: PLBM_SCH_FX(FORM_WLS); break;
    }
#undef PLBM_SCH_FX
    return cudaGetLastError();
  }
#define PLBM_SCH_HY(T)                                                        \
  switch (kind) {                                                             \
    case K_BGK: return launch_scheme_stencil<T, K_BGK>(s, st, a);             \
    case K_TRT: return launch_scheme_stencil<T, K_TRT>(s, st, a);             \
    default: return launch_scheme_stencil<T, K_RR>(s, st, a);                 \
  }
  switch (sch::taps_of(scheme)) {
    case sch::TAPS_LINE: PLBM_SCH_HY(sch::TAPS_LINE)
    case sch::TAPS_AXIS3: PLBM_SCH_HY(sch::TAPS_AXIS3)
    default: PLBM_SCH_HY(sch::TAPS_FULL)
  }
#undef PLBM_SCH_HY
}

cudaError_t hybrid_range_flag(int* flag, int reset) {
  cudaError_t e = cudaMemcpyFromSymbol(flag, g_hybrid_range_flag, sizeof(int));
  if (e == cudaSuccess && reset) {
    const int z = 0;
    e = cudaMemcpyToSymbol(g_hybrid_range_flag, &z, sizeof(int));
  }
  return e;
}

}  // namespace plbm
