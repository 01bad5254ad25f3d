// plbm_launch.h -- internal launcher interface shared by the translation units
// of libplbmgpu.so.  Not part of the public C ABI.
#pragma once
#include <algorithm>
#include <atomic>
#include <cuda_runtime.h>
#include <stddef.h>
#include "plbm_device.cuh"

namespace plbm {

// One lattice sweep: nx, ny, ld and the two lattices.
struct Sweep {
  int nx, ny, ld;
  const void* src;
  void* dst;
  cudaStream_t stream;
};

// Threads per block of the per-cell kernels.
constexpr int kBlock = 256;
// Blocks of the binary64 field reductions (152 SMs x 8); each writes one
// partial triple (the staging of plbm_velocity_l2_error_noalloc holds them).
constexpr int kReduceBlocks = 1216;

// Threads per block for a fused step of `cells` threads (cells, or pairs of
// cells).  Small CTAs spread a small grid evenly: with kernels chained, the CTAs
// of the next step take the slots this one leaves, and 256-thread CTAs then end up
// 3 on some SMs and 1 on others (256^2 RR, 256 / 128 / 64 threads: 5.5 / 5.4 / 5.45 us
// per step; 320^2 BGK 6.1 / 5.2 / 5.3, 2048^2 RR 149 / 143 / 143; binary32 deviation
// storage 320^2 2.9 / 2.6 / 2.1, 512^2 3.7 / 3.8 / 5.0).  A grid with less than that per
// SM takes the smallest multiple of 32 that covers it with one CTA per SM: each
// SM's binary64 pipe retires about 2 FMAs per cycle, so the strict kernel of a 64^2
// grid in 16 CTAs of 256 threads spent ~4.5 us per step in its collision.
int block_for(long long cells, bool binary64);

// Cells in flat order, rows one after the other: thread t of block b has cell
// b blockDim + t, and no thread lies past a row's end.  (A row in blocks of its own left
// 17 % of the threads of a 641 x 500 plugin grid without a cell.)
struct Rows {
  unsigned n;  // cells of a row
  unsigned m;  // floor(2^32 / n); 0: blocks of one row each
  unsigned tiles;  // blocks of a row (m == 0)
};
// A launch over such cells.  smem: shared memory that nothing uses, which limits the
// CTAs an SM holds to its even share of the grid, where an SM holds that share but not
// two.  Chained launches otherwise fill the rest of every SM with the next step's first
// CTAs and give its last ones to whichever SM ends early, which then takes twice the
// others' time (us per step, without flat cells and limit / with flat cells / with both:
// 300^2 BGK 5.1 / 5.1 / 4.1, 256^2 RR 5.3 / 5.3 / 4.2, 1000 x 65 BGK 4.9 / 3.6 / 3.7,
// 641 x 500 plugin BGK 11.1 / 10.0 / 10.0, 300^2 plugin RR 45.9 / 45.9 / 29.6).  The same limit
// on grids of two waves and more: 400^2 BGK 5.6 -> 6.3, not taken.  A kernel of another stream
// that needs shared memory or more warps than the limit leaves waits for the limited CTAs: a
// 300^2 BGK grid beside a 2048^2 binary32 one, 25.3 us per pair of steps without the limit
// and 31.6 with it; two 300^2 BGK grids 5.8 and 4.8, 256^2 RR beside 128^2 BGK 5.4 and 4.8.
struct Spread {
  unsigned blocks;
  int threads, smem;
  Rows rows;
};
// flat: rows cut into blocks of their own otherwise, and with 2^32 cells or more.
// resident: threads of the kernel that an SM's registers hold; 0: no limit.
cudaError_t spread_cells(int nfast, int nslow, bool binary64, bool flat, int resident, Spread* out);
// Whether rows cut into blocks of their own leave at most 1/32 of the threads without a
// cell.
bool rows_fit(int nfast, int nslow, bool binary64);

// Launches of a time loop's kernels, chained by programmatic dependent launch:
// the next kernel's CTAs are placed while this kernel still runs, and each waits
// (chain_begin, the first statement of every such kernel) until the kernels
// before it have completed and their writes are visible.  A dependent launch on
// one stream otherwise leaves the GPU idle for about 4 us (2 us inside a CUDA
// graph): 64^2 BGK steps issued one call at a time 5.2 -> 2.7 us each, in a captured
// loop 2.8 -> 2.45; 2048^2 binary32 47.3 -> 44.8, binary16 30.9 -> 28.3.
// A kernel lets its successor be placed only after its own wait, so at most two
// kernels of a chain are on the GPU, the second one waiting; no kernel's reads
// can be left in an SM's L1 by the time its buffer is overwritten and read again.
// The lattices are read with ld_chain, not through the read-only path, whose data
// may not change during a kernel's residence.
#ifdef __CUDACC__
__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
}
template <typename... P>
struct Chained {
  void (*kernel)(P...);
  unsigned blocks;
  int threads;
  cudaStream_t stream;
  int smem;
  // The launch error is returned, and kept for cudaGetLastError.
  template <typename... A>
  cudaError_t operator()(const A&... args) const {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = stream;
    cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
  }
};
template <typename... P>
Chained<P...> chained(void (*kernel)(P...), unsigned blocks, int threads, cudaStream_t stream, int smem = 0) {
  return {kernel, blocks, threads, stream, smem};
}
template <typename... P>
Chained<P...> chained(void (*kernel)(P...), const Spread& w, cudaStream_t stream) {
  return {kernel, w.blocks, w.threads, stream, w.smem};
}

// Threads of kernel K that an SM's registers hold.
template <auto K>
int resident_threads() {
  static std::atomic<int> threads{0};  // 0 until first asked
  int n = threads.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, K) != cudaSuccess || a.numRegs < 1) return 2048;
    // 16,384 registers for each of the four schedulers, a warp's in multiples of 256
    n = std::min(16, 16384 / (32 * ((a.numRegs + 7) / 8 * 8))) * 4 * 32;
    threads.store(n, std::memory_order_relaxed);
  }
  return n;
}

// binary32 deviation-storage BGK: the packed operators (bgk_dev, bgk_dev_comp) on grids of at
// least 2^20 cells, the smallest that a pass of several steps is taken on, in single steps too,
// and the former ones (coll_bgk_shift, bgk_dev_comp_one) below.  The line is not one of speed:
// small grids' moments are read in binary64, and keep every bit they had; the packed operator
// errs less (velocities 3e-7 against 3e-6 after the same steps) and rounds otherwise.  binary16
// has one operator at every size: its stores are 2^-11 of h apart, so that another rounding
// before them shows (compensated, one cell per thread against pairs: 2048^2 59.4 and 57.2 us
// per step, 3001 x 2999 123.6 and 127.5).
inline bool packed_bgk(int nx, int ny) { return (long long)nx * ny >= 1 << 20; }

// Deviation storage takes flat cells but on grids larger than the L2 cache whose rows fit
// their blocks and not their 128-byte lines: warps that straddle lines cost there
// (binary32 RR 3001 x 2999 97.8 us per step in rows, 102.2 flat; 1000^2 10.6 and 10.0).
inline bool dev_flat(int nfast, int nslow) {
  return (long long)nfast * nslow <= (1 << 20) || nfast % 32 == 0 || !rows_fit(nfast, nslow, false);
}

// Kernel K(src, dst, nx, ny, ld, rows, p), a thread per cell of nslow rows of nfast.
template <auto K, typename P>
cudaError_t step_cells(const Sweep& s, int nfast, int nslow, bool binary64, bool flat, const P& p) {
  Spread w;
  if (cudaError_t e = spread_cells(nfast, nslow, binary64, flat, resident_threads<K>(), &w)) return e;
  chained(K, w, s.stream)(s.src, s.dst, s.nx, s.ny, s.ld, w.rows, p);
  return cudaGetLastError();
}

// The row and the place in it of this thread's cell; row >= its count: none.
__device__ __forceinline__ void flat_cell(const Rows& r, int& row, int& place) {
  if (r.m == 0) {
    const unsigned s = blockIdx.x / r.tiles, f = (blockIdx.x - s * r.tiles) * blockDim.x + threadIdx.x;
    row = f < r.n ? (int)s : 0x7fffffff;
    place = (int)f;
    return;
  }
  const unsigned j = blockIdx.x * blockDim.x;
  unsigned s = __umulhi(j, r.m);  // j / n or one less
  unsigned f = j - s * r.n + threadIdx.x;
  while (f >= r.n) f -= r.n, s++;
  row = (int)s;
  place = (int)f;
}
#endif

// The binary64 reference kernels exist twice, once compiled with FMA
// contraction (namespace fma) and once without (namespace strict).
#define PLBM_DECLARE_F64(NS)                                                              \
  namespace NS {                                                                          \
  /* fused lbm_stream + collide_* (src/periodic_lbm.f90:15-29), YFast layout */            \
  cudaError_t step_pull_f64(int kind, const Sweep& s, const CollParams& p);               \
  /* lbm_stream alone (src/periodic_lbm.f90:45-127) */                                   \
  cudaError_t stream_f64(const Sweep& s);                                                 \
  /* collide_* alone, in place on s.dst (s.src ignored) */                                \
  cudaError_t collide_f64(int kind, const Sweep& s, const CollParams& p);                 \
  /* plugin step: shifted binary64 collide + push (sim/sim.F90:404-505), XFast */          \
  cudaError_t step_push_shift_f64(int kind, const Sweep& s, const CollParams& p);         \
  /* perform_triple_step fused: also stores the pre-collision populations to pre */       \
  cudaError_t step_pull_pre_f64(int kind, const Sweep& s, void* pre, const CollParams& p); \
  /* grid%streaming => stream_fvm_bardow (1), stream_fdm_bardow (2, 3 iso,    */          \
  /* 4 least squares), stream_fdm_sofonea (5): src/fvm_bardow.F90:393-886     */          \
  cudaError_t stream_scheme_f64(int scheme, const Sweep& s, double dt);                   \
  }
PLBM_DECLARE_F64(fma)
PLBM_DECLARE_F64(strict)
#undef PLBM_DECLARE_F64
namespace fma {
// a finite-volume / finite-difference scheme in stencil form fused with
// collide_bgk_improved (ld == ny)
cudaError_t step_scheme_f64(int scheme, const Sweep& s, double dt, const CollParams& p);
}

// binary64 storage, fixed-point arithmetic (hybrid.cuh), YFast pull, BGK, TRT
// and RR: the step of PLBM_MATH_HYBRID (report: a cell out of range sets the
// range flag) and of PLBM_MATH_FMA.
cudaError_t step_pull_fixed(int kind, const Sweep& s, const CollParams& p, bool report);
// The plugin step (shifted binary64, x-fastest, collide then push) in the same
// arithmetic (BGK, TRT, RR).
cudaError_t step_push_fixed(int kind, const Sweep& s, const CollParams& p, bool report);
// A finite-volume / finite-difference streaming scheme fused with the
// fixed-point collision (BGK, TRT, RR).
cudaError_t step_scheme_fixed(int scheme, int kind, const Sweep& s, double dt, const CollParams& p, bool report);
cudaError_t hybrid_range_flag(int* flag, int reset);
// The PLBM_MATH_FMA step: the fixed point for BGK, TRT and RR, the binary64
// kernel for the improved BGK.
inline cudaError_t step_pull_f64(int kind, const Sweep& s, const CollParams& p) {
  return kind == K_BGKI ? fma::step_pull_f64(kind, s, p) : step_pull_fixed(kind, s, p, false);
}

// Deviation storage (storage = 1 float, 2 half), binary32 arithmetic.
cudaError_t step_pull_dev(int storage, int kind, const Sweep& s, const CollParams& p);
// Two or three steps of collide_bgk in one pass over memory (step_march.cu), bit for
// bit those of step_pull_dev or (comp, binary32) of step_pull_dev_hi in compensated
// arithmetic.  march_applies says for which grids, march_plan how many passes of
// three and of two steps to take of nsteps; the rest are single steps, at least one.
bool march_applies(int storage, bool comp, int kind, int nx, int ny);
struct MarchPlan {
  int threes, twos;
};
MarchPlan march_plan(bool comp, int nsteps);
cudaError_t march_dev(int storage, bool comp, int steps, const Sweep& s, double omega);
cudaError_t stream_dev(int storage, const Sweep& s);
cudaError_t collide_dev(int storage, int kind, const Sweep& s, const CollParams& p);
cudaError_t step_push_dev(int storage, int kind, const Sweep& s, const CollParams& p);
// Deviation storage with the collision in binary64 (math 1, BGK/TRT/RR),
// compensated binary32 (math 2, BGK) or double-float (math 3, BGK)
// arithmetic; step_df64.cu.
cudaError_t step_pull_dev_hi(int storage, int math, int kind, const Sweep& s, const CollParams& p);

// Field kernels (fields.cu).  layout: 0 = YFast (src/), 1 = XFast (sim/).
// storage 0 = binary64 f (unshifted), 3 = binary64 shifted, 1/2 = deviation.
enum { ST_F64 = 0, ST_F32DEV = 1, ST_F16DEV = 2, ST_F64SHIFT = 3 };
// Moments of one lattice into (fast,slow) arrays; reference order of
// update_macros (YFast, unshifted) or lbm_macros (shifted).  exact (binary64
// storages 0 and 3): correctly rounded from the exact integer moments instead
// (exact_fields.cuh), the arithmetic of grids in hybrid mode.
cudaError_t macros(int storage, int layout, int nx, int ny, int ld, const void* f, double* rho,
                   double* ux, double* uy, cudaStream_t st, bool exact = false);
// Equilibrium from (fast,slow) rho/ux/uy arrays into a lattice.
//   storage 0: equilibrium() of src/fvm_bardow.F90:99-126;
//   storage 3/1/2: shifted equilibrium of sim/sim.F90:353-401 with rho = 1 + p/cs^2
//   when from_pressure != 0.
// exact (storages 0 and 3): the integer form of exact_fields.cuh.
cudaError_t equilibrium(int storage, int layout, int nx, int ny, int ld, const double* rho,
                        const double* ux, const double* uy, int from_pressure, void* f,
                        cudaStream_t st, bool exact = false);
// The same over the slow lines [slow0, slow1) only (x columns of the YFast
// layout): a slab of the grid, for pipelining with host transfers.  The
// field pointers still address the whole (fast, slow) arrays.
cudaError_t macros_range(int storage, int layout, int nx, int ny, int ld, const void* f, double* rho,
                         double* ux, double* uy, int slow0, int slow1, cudaStream_t st, bool exact = false);
cudaError_t equilibrium_range(int storage, int layout, int nx, int ny, int ld, const double* rho,
                              const double* ux, const double* uy, int from_pressure, void* f, int slow0,
                              int slow1, cudaStream_t st, bool exact = false);
// n doubles from src to dst (device addresses; either may be a mapped host
// array), by a kernel: 16-byte accesses when both are 16-byte aligned.
cudaError_t copy_doubles(const double* src, double* dst, size_t n, cudaStream_t st);
// binary64 f (YFast) <-> deviation storage conversion: h = f - w_i.
cudaError_t f64_to_dev(int storage, int nx, int ny, int ld, const double* f, void* h, cudaStream_t st);
cudaError_t dev_to_f64(int storage, int nx, int ny, int ld, const void* h, double* f, cudaStream_t st);
// Vorticity on (ny,nx) device arrays.
cudaError_t vorticity(int order, int nx, int ny, const double* ux, const double* uy, double* w,
                      cudaStream_t st);
// Per-block binary64 partial sums of 0.5*rho*|u|^2 and of |u-ua|^2, |ua|^2
// over the moments of a lattice; partial has room for reduce_blocks() triples.
int reduce_blocks(int nx, int ny);
cudaError_t energy_error_partials(int storage, int layout, int nx, int ny, int ld, const void* f,
                                  const double* uxa, const double* uya, double* partial,
                                  cudaStream_t st);

}  // namespace plbm
