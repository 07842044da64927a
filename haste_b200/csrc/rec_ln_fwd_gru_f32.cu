// Instantiates the persistent LayerNormGRU fwd recurrence kernels for f32 storage
// (one translation unit per combination so that they compile in parallel).
#include "rec_ln_grid.cuh"

namespace hb {
namespace rec {
int run_lngru_cl_fwd_f32(const LnFwdParams& p, cudaStream_t s) { return run_ln_cl_fwd<3, 2, float>(p, s); }
int run_lngru_grid_fwd_f32(const LnFwdParams& p, const LnGridGeometry& g, int wide, cudaStream_t s) {
  return run_ln_grid_fwd<3, 2, float>(p, g, wide, s);
}
}  // namespace rec
}  // namespace hb
