// Instantiates the persistent LayerNormLSTM fwd recurrence kernels for bf16 storage
// (one translation unit per combination so that they compile in parallel).
#include "rec_ln_grid.cuh"

namespace hb {
namespace rec {
int run_ln_cl_fwd_bf16(const LnFwdParams& p, cudaStream_t s) { return run_ln_cl_fwd<4, 1, __nv_bfloat16>(p, s); }
int run_ln_grid_fwd_bf16(const LnFwdParams& p, const LnGridGeometry& g, int wide, cudaStream_t s) {
  return run_ln_grid_fwd<4, 1, __nv_bfloat16>(p, g, wide, s);
}
}  // namespace rec
}  // namespace hb
