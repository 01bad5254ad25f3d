// batched.cu -- many independent periodic D2Q9 grids of uneven sizes and
// relaxation times advanced together.
//
// Layout: every grid keeps the reference layout f(ld,nx,0:8) (ld = pad16(ny))
// with two lattices A and B, all grids packed into one device allocation.
// Work unit: a tile of `threads` consecutive cells of a strip of one grid's rows
// (y fastest), the strips cut by the schedule's ty.  The tiles of all grids are
// numbered 0..T-1, the BGK grids' first; a table holds each tile's grid and first
// cell.  Persistent CTA b takes tiles b, b + nCTA, ...; the per-step launch gives
// each tile its own CTA.  (Tiles of ty rows by threads / ty columns left 28 % of
// their threads past the edges of 48 grids of 32 to 512 cells a side.)
//
// Two launch modes, both capturable in a CUDA graph:
//   * persistent: ONE cooperative launch runs all steps; the CTAs meet at a
//     grid-wide barrier between steps.  Every wait on the barrier is bounded:
//     after kSpinLimit polls the CTA records a timeout in the control block and
//     the kernel returns, so a lost CTA cannot hang the GPU.
//   * per-step: ordinary launches, one per collision kind and step (the graph
//     then holds those nodes); with 128-thread CTAs each kind runs a kernel
//     compiled for it alone.
//
// Deviation-storage lattice loads of the persistent kernel use ld.global.cg (L2
// only): a lattice written in step s by other SMs is read in step s+1.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "../../include/plbm_gpu.h"
#include "plbm_batched.h"
#include "plbm_launch.h"

namespace plbm {
namespace {

constexpr unsigned kSpinLimit = 1u << 24;  // polls of the barrier word (~seconds)

struct alignas(16) Ctrl {
  unsigned count;     // CTAs arrived at the current barrier
  unsigned gen;       // barrier generation
  int error;          // 0 ok, 1 barrier timeout
  int where;          // step at which the timeout happened
};

// Population load: ld.global.cg (L2 only) inside the persistent kernel, an
// ordinary load in the per-step kernels.
template <bool CG, typename E>
__device__ __forceinline__ E load_pop(const E* p) {
  if constexpr (CG) return __ldcg(p);
  else return ld_chain(p);
}

// One binary64 cell outside the hybrid range: pull, the binary64 operator,
// store.  Out of line so that the hot path's registers and code are not
// shaped by this rarely taken path.  gp points at the grid's table entry.
template <bool CG>
__device__ __noinline__ void fallback_cell(const double* __restrict__ src, double* __restrict__ dst, int x, int y,
                                           const BatchGrid* __restrict__ gp) {
  const int nx = gp->nx, ny = gp->ny, ld = gp->ld;
  double f[9];
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const int sx = wrap_add(x, -cx_of(q), nx), sy = wrap_add(y, -cy_of(q), ny);
    f[q] = load_pop<CG>(src + YFast::off(sx, sy, q, nx, ny, ld));
  }
  if (gp->kind == K_TRT) collide_ref<K_TRT>(f, gp->p);
  else collide_ref<K_BGK>(f, gp->p);
#pragma unroll
  for (int q = 0; q < 9; q++) dst[YFast::off(x, y, q, nx, ny, ld)] = f[q];
}

// The cell of this thread in tile t, one of `threads` consecutive cells of a strip of
// rows (y fastest; see plbm_batched.h).
struct Cell {
  const BatchGrid* gp;
  int x, y;  // x >= nx: past the strip's last cell
};
__device__ __forceinline__ Cell cell_of(const BatchGrid* __restrict__ grids, const BatchTile* __restrict__ tiles, int t) {
  const int4 a = __ldg(reinterpret_cast<const int4*>(tiles + t));
  const unsigned h = (unsigned)a.z >> 16, j = ((unsigned)a.z & 0xffffu) + threadIdx.x;
  const unsigned c = (j * (unsigned)a.w) >> kTileDivShift;  // j / h
  return {grids + __ldg(&tiles[t].grid), a.x + (int)c, a.y + (int)(j - c * h)};
}

// Offsets of the nine populations that stream into a cell.
// I: index type inside one grid's lattice pair (32-bit when every grid's pair has
// fewer than 2^32 elements).
template <typename I>
struct PullOff {
  I q[9];
  __device__ __forceinline__ PullOff(int x, int y, int nx, int ny, int ld) {
    const I L = (I)ld, P = L * (I)nx;
    const I c0 = (I)x * L, cm = (I)wrap_m(x, nx) * L, cp = (I)wrap_p(x, nx) * L;
    const I y0 = (I)y, ym = (I)wrap_m(y, ny), yp = (I)wrap_p(y, ny);
    q[0] = c0 + y0;
    q[1] = P + cm + y0;
    q[2] = 2 * P + c0 + ym;
    q[3] = 3 * P + cp + y0;
    q[4] = 4 * P + c0 + yp;
    q[5] = 5 * P + cm + ym;
    q[6] = 6 * P + cp + ym;
    q[7] = 7 * P + cp + yp;
    q[8] = 8 * P + cm + yp;
  }
};
template <typename E>
__device__ __forceinline__ E* lattice_of(const BatchGrid* gp, int which, E* base) {
  const long long lat = 9LL * __ldg(&gp->ld) * __ldg(&gp->nx);
  return base + __ldg(&gp->off) + (which ? lat : 0);
}

// Collide and store one cell.  KIND: K_BGK or K_TRT, or (deviation storage) -1 for
// the grid's own, read at run time.  Binary64 grids take the fixed-point
// collisions of hybrid.cuh in either arithmetic (their error is no larger than
// the binary64 operator's).  The grid's relaxation constants are read where they
// are used (through the read-only path) rather than held in registers.
template <class S, bool CG, typename I, int KIND>
__device__ __forceinline__ void collide_cell(typename S::real (&f)[9], const Cell& c, int parity,
                                             typename S::elem* __restrict__ base) {
  const BatchGrid* gp = c.gp;
  typename S::elem* dst = lattice_of(gp, !parity, base);
  if constexpr (S::ddf) {
    if (KIND == K_TRT || (KIND < 0 && __ldg(&gp->kind) == K_TRT)) collide_shift<K_TRT, typename S::real>(f, gp->p);
    else collide_shift<K_BGK, typename S::real>(f, gp->p);
  } else {
    bool bad = false;
    if constexpr (KIND == K_TRT) hy::trt_fma(f, gp->ht, bad);
    else hy::bgk_fma(f, gp->hp, bad);
    if (bad) {  // outside the fixed point's range: the binary64 operator on the same inputs
      fallback_cell<CG>(lattice_of(gp, parity, base), dst, c.x, c.y, gp);
      return;
    }
  }
  const I L = (I)__ldg(&gp->ld), P = L * (I)__ldg(&gp->nx), o = (I)c.x * L + (I)c.y;
#pragma unroll
  for (int q = 0; q < 9; q++) S::store(dst, (size_t)((I)q * P + o), f[q]);
}

// One tile for one step.
template <class S, bool CG, typename I, int KIND>
__device__ __forceinline__ void do_tile(const BatchGrid* __restrict__ grids, const BatchTile* __restrict__ tiles, int t,
                                        int parity, typename S::elem* __restrict__ base) {
  const Cell c = cell_of(grids, tiles, t);
  if (c.x >= __ldg(&c.gp->nx)) return;
  const typename S::elem* src = lattice_of(c.gp, parity, base);
  typename S::elem e[9];
  {
    const PullOff<I> off(c.x, c.y, __ldg(&c.gp->nx), __ldg(&c.gp->ny), __ldg(&c.gp->ld));
#pragma unroll
    for (int q = 0; q < 9; q++) e[q] = load_pop<CG>(src + off.q[q]);
  }
  typename S::real f[9];
#pragma unroll
  for (int q = 0; q < 9; q++) f[q] = (typename S::real)e[q];
  collide_cell<S, CG, I, KIND>(f, c, parity, base);
}

// Grid-wide barrier with a bounded wait.  Returns false when the wait ran out
// (then Ctrl::error is set and every CTA leaves the kernel).
__device__ __forceinline__ bool barrier(Ctrl* ctrl, int step) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    volatile unsigned* vgen = &ctrl->gen;
    const unsigned gen = *vgen;
    __threadfence();
    const unsigned arrived = atomicAdd(&ctrl->count, 1u);
    if (arrived == gridDim.x - 1) {
      ctrl->count = 0;
      __threadfence();
      atomicAdd(&ctrl->gen, 1u);
    } else {
      unsigned n = 0;
      while (*vgen == gen) {
        if (++n > kSpinLimit || *(volatile int*)&ctrl->error) {
          atomicExch(&ctrl->error, 1);
          atomicExch(&ctrl->where, step);
          ok = 0;
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// CTAs per SM the kernels are compiled for: binary64 1024 resident threads (64
// registers), deviation storage 1536 (40; uncapped the persistent kernel takes
// 52 and runs 48 grids at 0.062 ms per step instead of 0.057).
template <class S>
constexpr int batch_min_blocks(int max_threads) {
  return (S::ddf ? 1536 : 1024) / max_threads;
}

// The persistent binary64 kernel at 256 threads: three CTAs (80 registers, 16 bytes spilled) hide
// the copies as well as four (64, 84 bytes spilled), and fewer meet at the barrier: 512
// grids 1.117 -> 1.091 ms per step, 8 grids 17.6 -> 16.6 us; two CTAs 1.162 and 15.3.
template <class S>
constexpr int persistent_min_blocks(int max_threads) {
  return !S::ddf && max_threads == 256 ? 3 : batch_min_blocks<S>(max_threads);
}

// A binary64 tile as the persistent kernel keeps it in shared memory: the tile, its
// grid's sizes and the relaxation constants (a CTA has the same tiles in every step;
// read from global memory for each tile, they put three dependent L2 latencies
// before its loads and several before its collision).
struct alignas(16) OwnTile {
  int x0, y0;
  unsigned r0_h, div;
  int nx, ny, ld, grid;
  long long off;  // of the lattice pair
  union {
    hy::BgkParams hp;
    hy::TrtFmaParams ht;
  };
};
constexpr int kOwnTiles = 32;  // CTAs with more read them in turns

__device__ __forceinline__ void own_tile(OwnTile& o, const BatchGrid* __restrict__ grids,
                                         const BatchTile* __restrict__ tiles, int t, int nt_bgk) {
  const BatchTile b = tiles[t];
  const BatchGrid* g = grids + b.grid;
  o.x0 = b.x0, o.y0 = b.y0, o.r0_h = b.r0_h, o.div = b.div;
  o.nx = g->nx, o.ny = g->ny, o.ld = g->ld, o.grid = b.grid, o.off = g->off;
  if (t < nt_bgk) o.hp = g->hp;
  else o.ht = g->ht;
}

__device__ __forceinline__ void own_cell(const OwnTile& o, int& x, int& y) {
  const unsigned h = o.r0_h >> 16, j = (o.r0_h & 0xffffu) + threadIdx.x;
  const unsigned c = (j * o.div) >> kTileDivShift;  // j / h
  x = o.x0 + (int)c;
  y = o.y0 + (int)(j - c * h);
}

// This thread's nine populations of a tile into a stage of shared memory.
template <typename I>
__device__ __forceinline__ void copy_tile(const OwnTile& o, int parity, const double* base, double* stage) {
  int x, y;
  own_cell(o, x, y);
  if (x < o.nx) {
    const double* src = base + o.off + (parity ? 9LL * o.ld * o.nx : 0);
    const PullOff<I> off(x, y, o.nx, o.ny, o.ld);
    const unsigned s0 = (unsigned)__cvta_generic_to_shared(stage + threadIdx.x);
#pragma unroll
    for (int q = 0; q < 9; q++)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s0 + q * 8u * blockDim.x), "l"(src + off.q[q])
                   : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Binary64 tiles [i, last) of a CTA's table (the copies end at n), of one kind: the BGK
// grids' and the TRT grids' tiles in a loop each (with the kind read per tile the
// kernel took 114 registers).  Each thread copies its own nine populations of the next
// tile into shared memory (cp.async) while it collides the present ones.  The copies
// go through L1: the fence of the grid barrier before them discards what an earlier
// step left there.
template <typename I, int KIND>
__device__ __forceinline__ void sweep_ahead(const BatchGrid* __restrict__ grids, const OwnTile* own, int& i, int last,
                                            int n, int parity, int& stage, double* sm, double* base) {
  for (; i < last; i++) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    double f[9];
    const double* mine = sm + stage * 9 * blockDim.x + threadIdx.x;
#pragma unroll
    for (int q = 0; q < 9; q++) f[q] = mine[q * blockDim.x];
    stage ^= 1;
    if (i + 1 < n) copy_tile<I>(own[i + 1], parity, base, sm + stage * 9 * blockDim.x);
    const OwnTile& o = own[i];
    int x, y;
    own_cell(o, x, y);
    if (x >= o.nx) continue;
    bool bad = false;
    if constexpr (KIND == K_TRT) hy::trt_fma(f, o.ht, bad);
    else hy::bgk_fma(f, o.hp, bad);
    const long long lat = 9LL * o.ld * o.nx;
    double* pair = base + o.off;
    double* dst = pair + (parity ? 0 : lat);
    if (bad) {  // outside the fixed point's range: the binary64 operator on the same inputs
      fallback_cell<true>(pair + (parity ? lat : 0), dst, x, y, grids + o.grid);
      continue;
    }
    const I P = (I)o.ld * (I)o.nx;
    dst += (I)x * (I)o.ld + (I)y;
#pragma unroll
    for (int q = 0; q < 9; q++) dst[(I)q * P] = f[q];
  }
}

// All steps of a run.  Tile t belongs to CTA t mod gridDim.x.  Binary64: see
// sweep_ahead.  Deviation storage reads the kind per tile: both collisions fit in the
// registers of one (0.0566 ms per step of 48 grids, 4.0 M cells; 0.0571 in two loops).
//
// 48 grids of 32 to 512 cells a side, 1.42 M cells, us per step: tiles of ty by
// threads / ty cells with loads for each 70; tiles of consecutive cells, columns copied
// ahead 62; the tiles' table and constants in shared memory 53; three CTAs per SM 49.  A quarter
// of it is the barrier and the memory's latency after it.  Waiting for chunks of
// whole grids instead (each of which depends on itself alone) lost more to every
// further release and acquire, 4 us each, than it gained: 2 chunks 53, 4 chunks 61.
// 512 grids, 39 M cells: 1.94 -> 1.09 ms per step.
template <class S, typename I, int MAXT>
__global__ void __launch_bounds__(MAXT, persistent_min_blocks<S>(MAXT))
    k_batch_persistent(const BatchGrid* __restrict__ grids, const BatchTile* __restrict__ tiles, int nt_bgk, int ntiles,
                       int nsteps, int parity0, typename S::elem* base, Ctrl* ctrl) {
  // own tiles below tile t
  auto own_below = [](int t) { return t > (int)blockIdx.x ? (t - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0; };
  const int count = own_below(ntiles), nb = own_below(nt_bgk);
  int stage = 0;
  for (int s = 0; s < nsteps; s++) {
    const int parity = (parity0 + s) & 1;
    if constexpr (S::ddf) {
      for (int t = blockIdx.x; t < ntiles; t += gridDim.x) do_tile<S, true, I, -1>(grids, tiles, t, parity, base);
    } else {
      extern __shared__ double sm[];  // 2 x 9 x threads
      __shared__ OwnTile own[kOwnTiles];
      for (int i0 = 0; i0 < count; i0 += kOwnTiles) {
        const int n = min(kOwnTiles, count - i0);
        if (s == 0 || count > kOwnTiles) {
          __syncthreads();
          if ((int)threadIdx.x < n)
            own_tile(own[threadIdx.x], grids, tiles, blockIdx.x + (i0 + threadIdx.x) * gridDim.x, nt_bgk);
          __syncthreads();
        }
        int i = 0;
        copy_tile<I>(own[0], parity, base, sm + stage * 9 * blockDim.x);
        sweep_ahead<I, K_BGK>(grids, own, i, max(0, min(nb - i0, n)), n, parity, stage, sm, base);
        sweep_ahead<I, K_TRT>(grids, own, i, n, n, parity, stage, sm, base);
      }
    }
    if (s + 1 < nsteps && !barrier(ctrl, s)) return;
  }
}

// Per-step launch over the tiles of one collision kind (tile t0 + blockIdx.x),
// compiled for that kind alone: the binary64 BGK tiles take 64 registers and
// the TRT tiles 72.  One kernel for both kinds needed far more registers than
// either (97 for the earlier forms, 80 under a cap with spills, 20.9k MLUPS on
// the 512-grid batch against 24.5k split by kind; 33.7k with tiles of consecutive
// cells and the present collisions).
template <class S, typename I, int KIND, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) k_batch_kind(const BatchGrid* __restrict__ grids,
                                                          const BatchTile* __restrict__ tiles, int t0, int parity,
                                                          typename S::elem* base) {
  chain_begin();
  do_tile<S, false, I, KIND>(grids, tiles, t0 + (int)blockIdx.x, parity, base);
}

// Per-step launch over all tiles, for deviation storage in CTAs other than 128
// threads (48 grids, 256 threads: 0.0645 ms per step, 0.070 as a launch per
// kind).
template <class S, typename I>
__global__ void __launch_bounds__(kBatchMaxThreads) k_batch_step(const BatchGrid* __restrict__ grids,
                                                                const BatchTile* __restrict__ tiles, int parity,
                                                                typename S::elem* base) {
  chain_begin();
  do_tile<S, false, I, -1>(grids, tiles, (int)blockIdx.x, parity, base);
}

template <class S, typename I, int MAXT>
cudaError_t launch_kinds(const BatchLaunch& L, int parity) {
  typedef typename S::elem E;
  E* base = static_cast<E*>(L.base);
  const int ntrt = L.ntiles - L.nt_bgk;
  constexpr int bgk_blocks = MAXT == 128 ? 8 : batch_min_blocks<S>(MAXT);
  constexpr int trt_blocks = MAXT == 128 ? 7 : batch_min_blocks<S>(MAXT);
  if (L.nt_bgk > 0)
    chained(k_batch_kind<S, I, K_BGK, MAXT, bgk_blocks>, L.nt_bgk, L.threads, L.stream)(L.grids, L.tiles, 0, parity, base);
  if (ntrt > 0)
    chained(k_batch_kind<S, I, K_TRT, MAXT, trt_blocks>, ntrt, L.threads, L.stream)(L.grids, L.tiles, L.nt_bgk, parity, base);
  return cudaGetLastError();
}

// Dynamic shared memory of the persistent kernel.
template <class S>
int persistent_smem(int threads) {
  return S::ddf ? 0 : 2 * 9 * 8 * threads;
}

template <class S, typename I>
cudaError_t launch_batch(const BatchLaunch& L, int nsteps, int parity0) {
  typedef typename S::elem E;
  E* base = static_cast<E*>(L.base);
  if (L.persistent) {
    Ctrl* ctrl = static_cast<Ctrl*>(L.ctrl);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(L.ctas);
    cfg.blockDim = dim3(L.threads);
    cfg.stream = L.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto kernel = !S::ddf && L.threads <= 256 ? k_batch_persistent<S, I, 256> : k_batch_persistent<S, I, kBatchMaxThreads>;
    cfg.dynamicSmemBytes = persistent_smem<S>(L.threads);
    return cudaLaunchKernelEx(&cfg, kernel, L.grids, L.tiles, L.nt_bgk, L.ntiles, nsteps, parity0,
                              base, ctrl);
  }
  // one tile per CTA
  for (int s = 0; s < nsteps; s++) {
    const int parity = (parity0 + s) & 1;
    cudaError_t e;
    if (L.threads <= 128 && (!S::ddf || L.threads == 128)) {
      e = launch_kinds<S, I, 128>(L, parity);
    } else if constexpr (S::ddf) {
      chained(k_batch_step<S, I>, L.ntiles, L.threads, L.stream)(L.grids, L.tiles, parity, base);
      e = cudaGetLastError();
    } else {
      e = L.threads <= 256 ? launch_kinds<S, I, 256>(L, parity) : launch_kinds<S, I, kBatchMaxThreads>(L, parity);
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <class S>
cudaError_t launch_batch_i(const BatchLaunch& L, int nsteps, int parity0) {
  if (L.small_index) return launch_batch<S, uint32_t>(L, nsteps, parity0);
  return launch_batch<S, size_t>(L, nsteps, parity0);
}

}  // namespace

size_t batch_ctrl_bytes() { return sizeof(Ctrl); }

namespace {
template <class S, typename I>
cudaError_t persistent_ctas(int threads, int* per_sm) {
  auto kernel = !S::ddf && threads <= 256 ? k_batch_persistent<S, I, 256> : k_batch_persistent<S, I, kBatchMaxThreads>;
  // With its static tables the kernel for more than 256 threads passes 48 KB, from 320
  // threads on.  The limit belongs to the kernel, which every batch shares: the most that
  // any schedule asks for, whichever schedule this is.
  if (!S::ddf && threads > 256)
    if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             persistent_smem<S>(kBatchMaxThreads)))
      return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kernel, threads, persistent_smem<S>(threads));
}
}  // namespace

cudaError_t batch_max_ctas(int storage, int threads, int small_index, int* per_sm) {
  if (storage == ST_F64)
    return small_index ? persistent_ctas<StoreF64, uint32_t>(threads, per_sm)
                       : persistent_ctas<StoreF64, size_t>(threads, per_sm);
  return small_index ? persistent_ctas<StoreF32Dev, uint32_t>(threads, per_sm)
                     : persistent_ctas<StoreF32Dev, size_t>(threads, per_sm);
}

cudaError_t batch_run(int storage, const BatchLaunch& L, int nsteps, int parity0) {
  if (nsteps <= 0) return cudaSuccess;
  if (L.threads <= 0 || L.threads > kBatchMaxThreads || (L.threads & 31)) return cudaErrorInvalidConfiguration;
  if (storage == ST_F64) return launch_batch_i<StoreF64>(L, nsteps, parity0);
  if (storage == ST_F32DEV) return launch_batch_i<StoreF32Dev>(L, nsteps, parity0);
  return cudaErrorNotSupported;
}

cudaError_t batch_arm_stall(void* ctrl, cudaStream_t st) {
  // arrival count far above any CTA count: the first barrier never completes
  // and every CTA's wait runs out (kSpinLimit polls)
  static const Ctrl stalled = {0x80000000u, 0u, 0, 0};
  return cudaMemcpyAsync(ctrl, &stalled, sizeof stalled, cudaMemcpyHostToDevice, st);
}

cudaError_t batch_read_ctrl(const void* ctrl, int* error, int* where, cudaStream_t st) {
  Ctrl h;
  cudaError_t e = cudaMemcpyAsync(&h, ctrl, sizeof h, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  *error = h.error;
  *where = h.where;
  return cudaSuccess;
}

}  // namespace plbm
