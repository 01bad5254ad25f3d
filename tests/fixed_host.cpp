// Host build of single operations of periodic-lbm_gb300/csrc (hybrid.cuh, fixed.cuh,
// df64.cuh) for test_fixed_host.py.
#include <stdint.h>
#include "hybrid.cuh"
using namespace plbm;

extern "C" double fx_to_double(int64_t T, int exact) {
  return exact ? hy::fixed_to_double_tr<hy::kScale, true>(T) : hy::fixed_to_double_tr(T);
}
