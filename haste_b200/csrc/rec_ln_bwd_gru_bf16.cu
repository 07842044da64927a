// Instantiates the persistent LayerNormGRU bwd recurrence kernels for bf16 storage
// (one translation unit per combination so that they compile in parallel).
#include "rec_ln_grid.cuh"

namespace hb {
namespace rec {
int run_lngru_cl_bwd_bf16(const LnBwdParams& p, float* db_part, int* row_groups, cudaStream_t s) {
  return run_ln_cl_bwd<3, 1, __nv_bfloat16>(p, db_part, row_groups, s);
}
int run_lngru_grid_bwd_bf16(const LnBwdParams& p, float* db_part, const LnGridGeometry& g, int wide, cudaStream_t s) {
  return run_ln_grid_bwd<3, 1, __nv_bfloat16>(p, db_part, g, wide, s);
}
}  // namespace rec
}  // namespace hb
