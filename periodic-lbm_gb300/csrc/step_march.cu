// step_march.cu -- several time steps of a deviation-storage lattice in one pass
// over memory.
//
// A single step moves 72 B (binary32) or 36 B (binary16) per cell and runs at
// the memory's rate; its arithmetic takes a fifth of that time.  Here a warp
// marches along x over a strip of 64 rows, two per lane, and carries T steps at
// once: in iteration x it pulls column x and takes it through step 1, column
// x - 1 through step 2 and column x - 2 through step 3, and stores the last.
// What a step needs from the neighbouring columns of the step before stays in
// registers: populations moving in +x for two columns, resting in x for one,
// moving in -x none; the shift by one row within the strip is one shuffle of half
// a pair.  No shared memory and no barrier: the warps are independent.  Each step
// loses one row at either end of the strip, so that, in whole lanes, 60 of its 64 rows are
// stored for T <= 2 and 56 for T = 3, and the T - 1 columns before and after a segment of
// columns are computed twice.
// Binary16 values are rounded to storage between the steps, so that the result has
// the bits of T single steps.
//
// 4096 x 3000, us per step, single / marched: binary32 130 / 55 (the memory moves 24 B
// per cell and step at 5.1 TB/s; issue 55 %, 12 warps per SM at 140 registers),
// compensated binary32 169 / 136 (the packed binary32 pipe), binary16 78 / 57.  Two
// columns are loaded ahead: without, the loads' latency left issue at 39 % (65 us);
// four CTAs per SM instead of three spill (71 us).
#include <atomic>

#include "coll_df64.cuh"
#include "f32x2.cuh"
#include "plbm_launch.h"

namespace plbm {
namespace {

constexpr int kMarchWarps = 4;  // warps (strips) per CTA
// Lanes whose rows are lost at either end of a strip (one row per step), and the
// rows stored.
__host__ __device__ constexpr int march_edge(int steps) { return (steps + 1) / 2; }
__host__ __device__ constexpr int march_rows(int steps) { return 64 - 4 * march_edge(steps); }

// Storage of a pair of rows.  A load leaves its data as it comes (Raw), so that
// nothing waits for it before the next column is due.
struct MarchF32 {
  typedef float elem;
  typedef f32x2 Raw;
  static constexpr bool sc = false;
  __device__ __forceinline__ static Raw load2(const float* p) {
    f32x2 r;
    asm volatile("ld.global.b64 %0, [%1];" : "=l"(r.v) : "l"(p));
    return r;
  }
  __device__ __forceinline__ static Raw load1(const float* p, const float* q) { return pack2(ld_chain(p), ld_chain(q)); }
  __device__ __forceinline__ static f32x2 value(Raw r) { return r; }
  __device__ __forceinline__ static void store2(float* p, f32x2 v) { *reinterpret_cast<unsigned long long*>(p) = v.v; }
  __device__ __forceinline__ static void store1(float* p, float v) { *p = v; }
  __device__ __forceinline__ static f32x2 rounded(f32x2 v) { return v; }
};
struct MarchF16 {
  typedef __half elem;
  typedef __half2 Raw;
  static constexpr bool sc = true;
  __device__ __forceinline__ static Raw load2(const __half* p) { return ld_chain(reinterpret_cast<const __half2*>(p)); }
  __device__ __forceinline__ static Raw load1(const __half* p, const __half* q) {
    return __halves2half2(ld_chain(p), ld_chain(q));
  }
  __device__ __forceinline__ static f32x2 value(Raw r) {
    const float2 f = __half22float2(r);
    return pack2(f.x, f.y);
  }
  __device__ __forceinline__ static void store2(__half* p, f32x2 v) {
    *reinterpret_cast<__half2*>(p) = __floats2half2_rn(lo2(v), hi2(v));
  }
  __device__ __forceinline__ static void store1(__half* p, float v) { *p = __float2half_rn(v); }
  __device__ __forceinline__ static f32x2 rounded(f32x2 v) {
    const float2 f = __half22float2(__floats2half2_rn(lo2(v), hi2(v)));
    return pack2(f.x, f.y);
  }
};

// Collisions.
template <class S>
struct MarchBgk {
  typedef float Params;  // omega
  __device__ __forceinline__ static void collide(f32x2 (&h)[9], Params omega) {
    if constexpr (S::sc) bgk_f16(h, omega);
    else bgk_dev(h, omega);
  }
};

struct MarchComp {
  typedef df::DevParams Params;
  __device__ __forceinline__ static void collide(f32x2 (&h)[9], const Params& p) { df::bgk_dev_comp(h, p); }
};

// Row r - 1 (up) or r + 1 (down) of a strip whose lane holds rows (2l, 2l + 1).
__device__ __forceinline__ f32x2 row_above(f32x2 v) {
  return pack2(__shfl_up_sync(0xffffffffu, hi2(v), 1), lo2(v));
}
__device__ __forceinline__ f32x2 row_below(f32x2 v) {
  return pack2(hi2(v), __shfl_down_sync(0xffffffffu, lo2(v), 1));
}

// What one step keeps of the columns before: populations resting in x (0, 2, 4) of
// the last one, moving in +x (1, 5, 8) of the last two.
struct Delay {
  f32x2 rest[3], plus0[3], plus1[3];
};

template <class S, class C, int T>
__global__ void __launch_bounds__(32 * kMarchWarps, 3)
    k_march(const typename S::elem* __restrict__ src, typename S::elem* __restrict__ dst, int nx, int ny, int ld,
            int seg, typename C::Params p) {
  chain_begin();
  typedef typename S::elem E;
  const int strip = blockIdx.x * kMarchWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (strip * march_rows(T) >= ny) return;
  const int r0 = strip * march_rows(T) - 2 * march_edge(T) + 2 * lane;  // this lane's rows r0, r0 + 1
  auto wrap = [ny](int r) { return (unsigned)(r < 0 ? r + ny : (r >= ny ? r - ny : r)); };
  const unsigned ra = wrap(r0), rb = wrap(r0 + 1);
  // pairs load as one access unless the strip wraps at an odd row
  const bool pairs = __all_sync(0xffffffffu, rb == ra + 1 && (ra & 1u) == 0);
  const bool store = lane >= march_edge(T) && lane < 32 - march_edge(T) && r0 < ny;
  const bool store_both = r0 + 1 < ny;
  const size_t P = (size_t)ld * nx;
  const int x0 = blockIdx.y * seg, x1 = min(x0 + seg, nx);
  Delay d[T > 1 ? T - 1 : 1];
  const f32x2 zero = pack2(0.0f, 0.0f);
#pragma unroll
  for (int t = 0; t < T - 1; t++)
#pragma unroll
    for (int i = 0; i < 3; i++) d[t].rest[i] = d[t].plus0[i] = d[t].plus1[i] = zero;
  // Column x of the source as the first step pulls it, before the shift in y.
  typename S::Raw buf[2][9];
  auto load_column = [&](typename S::Raw (&n)[9], int xc) {
    const int xm = xc == 0 ? nx - 1 : xc - 1, xp = xc + 1 == nx ? 0 : xc + 1;
#pragma unroll
    for (int q = 0; q < 9; q++) {
      const E* c = src + (size_t)(cx_of(q) > 0 ? xm : (cx_of(q) < 0 ? xp : xc)) * ld + q * P;
      n[q] = pairs ? S::load2(c + ra) : S::load1(c + ra, c + rb);
    }
  };
  auto pull_rows = [](f32x2 (&h)[9]) {
    h[2] = row_above(h[2]), h[5] = row_above(h[5]), h[6] = row_above(h[6]);
    h[4] = row_below(h[4]), h[7] = row_below(h[7]), h[8] = row_below(h[8]);
  };
  const int first = x0 - (T - 1), last = x1 + T - 2;
  int xl = first < 0 ? first + nx : first;  // the next column to load
  auto advance = [&](typename S::Raw (&n)[9], int x) {
    f32x2 h[9];
#pragma unroll
    for (int q = 0; q < 9; q++) h[q] = S::value(n[q]);
    if (x + 2 <= last) {
      load_column(n, xl);
      xl = xl + 1 == nx ? 0 : xl + 1;
    }
    pull_rows(h);
    C::collide(h, p);
#pragma unroll
    for (int t = 0; t < T - 1; t++) {
      // column x - t is through step t + 1; pull column x - t - 1 for step t + 2
      f32x2 g[9];
#pragma unroll
      for (int q = 0; q < 9; q++) h[q] = S::rounded(h[q]);
      g[0] = d[t].rest[0], g[2] = d[t].rest[1], g[4] = d[t].rest[2];
      g[1] = d[t].plus1[0], g[5] = d[t].plus1[1], g[8] = d[t].plus1[2];
      g[3] = h[3], g[6] = h[6], g[7] = h[7];
#pragma unroll
      for (int i = 0; i < 3; i++) d[t].plus1[i] = d[t].plus0[i];
      d[t].rest[0] = h[0], d[t].rest[1] = h[2], d[t].rest[2] = h[4];
      d[t].plus0[0] = h[1], d[t].plus0[1] = h[5], d[t].plus0[2] = h[8];
      pull_rows(g);
      C::collide(g, p);
#pragma unroll
      for (int q = 0; q < 9; q++) h[q] = g[q];
    }
    const int xo = x - (T - 1);
    if (xo >= x0 && xo < x1 && store) {
      E* o = dst + (size_t)xo * ld + r0;
      if (store_both) {
#pragma unroll
        for (int q = 0; q < 9; q++) S::store2(o + q * P, h[q]);
      } else {
#pragma unroll
        for (int q = 0; q < 9; q++) S::store1(o + q * P, lo2(h[q]));
      }
    }
  };
#pragma unroll
  for (int i = 0; i < 2; i++) {
    load_column(buf[i], xl);
    xl = xl + 1 == nx ? 0 : xl + 1;
  }
#pragma unroll 1
  for (int x = first; x <= last; x += 2) {  // an odd count takes one column more, not stored
    advance(buf[0], x);
    advance(buf[1], x + 1);
  }
}

template <class S, class C, int T>
cudaError_t launch_march(const Sweep& s, const typename C::Params& p) {
  static std::atomic<int> capacity[64];  // resident CTAs on the device, by device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int cap = dev < 64 ? capacity[dev].load(std::memory_order_relaxed) : 0;
  if (cap == 0) {
    int per_sm = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_march<S, C, T>, 32 * kMarchWarps, 0);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    cap = per_sm * sms;
    if (dev < 64) capacity[dev].store(cap, std::memory_order_relaxed);
  }
  const int strips = (s.ny + march_rows(T) - 1) / march_rows(T);
  const int gx = (strips + kMarchWarps - 1) / kMarchWarps;
  // One wave of CTAs, in segments of at least 16 columns; on grids long enough
  // for segments of 160 columns all the same, up to four waves, which even out the
  // strips at the grid's edge (8192^2, 1 / 2 / 4 waves: binary32 215 / 218 / 220 GLUPS,
  // binary16 224 / 232 / 240; 2048^2 binary32 186 / 174 / 166).  Binary16 with an odd ny,
  // whose edge strips load row by row, from 32 columns on (1 / 2 / 3 / 4 waves: 3001 x 2999
  // 180 / 194 / 196 / 195, 2999 x 5001 178 / 199 / 203 / 206, 5121^2 178 / 205 / 215 / 217, but 1500 x
  // 1401 157 / 135, 700 x 2999 165 / 154).  Binary32 with an odd ny is no different from
  // an even one (3001 x 2999 226 / 218 / 212, compensated 88.6 / 88.0 / 85.6, 1500 x 1401 185 /
  // 140 and 80 / 69).
  int segs = cap / gx;
  if (segs > s.nx / 16) segs = s.nx / 16;
  if (segs < 1) segs = 1;
  int waves = s.nx / ((S::sc && s.ny % 2 != 0 ? 32 : 160) * segs);
  if (waves > 4) waves = 4;
  if (waves > 1) segs = segs * waves < s.nx / 16 ? segs * waves : s.nx / 16;
  const int seg = (s.nx + segs - 1) / segs;
  segs = (s.nx + seg - 1) / seg;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)gx, (unsigned)segs);
  cfg.blockDim = dim3(32 * kMarchWarps);
  cfg.stream = s.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  typedef typename S::elem E;
  return cudaLaunchKernelEx(&cfg, k_march<S, C, T>, static_cast<const E*>(s.src), static_cast<E*>(s.dst), s.nx, s.ny,
                            s.ld, seg, p);
}

}  // namespace

// Grids whose passes gain (the last two figures: single steps / marched, GLUPS).
// binary32 from 2^20 cells (1024^2 120 / 131, 1448^2 91 / 171, 2048^2 94 / 190, 4096 x
// 3000 95 / 209, 8192 x 130 91 / 115; 724^2 97 / 75), compensated from 2^21 (1448^2
// 65 / 62, 2048^2 70 / 79, 4096 x 3000 73 / 84, 8192^2 75 / 97), binary16 from 1.25
// 2^20 with the CTAs' strips at least three quarters used (1024^2 136 / 120, 1200^2 140 /
// 163, 2048^2 153 / 187, 8192^2 166 / 235, 8192 x 256 150 / 125).
bool march_applies(int storage, bool comp, int kind, int nx, int ny) {
  if (kind != K_BGK || nx < 64 || ny < 128 || (comp && storage != ST_F32DEV)) return false;
  const long long cells = (long long)nx * ny;
  if (storage == ST_F32DEV) return cells >= (comp ? 1 << 21 : 1 << 20);
  const int strips = (ny + march_rows(3) - 1) / march_rows(3), ctas = (strips + kMarchWarps - 1) / kMarchWarps;
  return cells >= (5 << 18) && strips >= 3 * ctas;
}

// A pass of k steps swaps the buffers once, k single steps k times: threes keep the
// parity, twos come in pairs of passes.  The plain collisions are bound by memory
// and take three steps at a time; the compensated one, bound by arithmetic, loses
// fewer rows with two (4096 x 3000: 136 us per step in twos, 157 in threes) and takes
// up to two threes where that leaves one single step at the end.
MarchPlan march_plan(bool comp, int nsteps) {
  if (!comp) {
    const int threes = nsteps > 1 ? (nsteps - 1) / 3 : 0;
    return {threes, 0};
  }
  const int r = nsteps > 1 ? (nsteps - 1) % 4 : 0;
  const int threes = r == 3 ? 1 : (r == 2 && nsteps >= 7 ? 2 : 0);
  return {threes, nsteps > 1 ? (nsteps - 1 - 3 * threes) / 4 * 2 : 0};
}

cudaError_t march_dev(int storage, bool comp, int steps, const Sweep& s, double omega) {
  if (comp)
    return steps == 2 ? launch_march<MarchF32, MarchComp, 2>(s, df::dev_params(omega))
                      : launch_march<MarchF32, MarchComp, 3>(s, df::dev_params(omega));
  if (storage == ST_F32DEV) return launch_march<MarchF32, MarchBgk<MarchF32>, 3>(s, (float)omega);
  return launch_march<MarchF16, MarchBgk<MarchF16>, 3>(s, (float)omega);
}

}  // namespace plbm
