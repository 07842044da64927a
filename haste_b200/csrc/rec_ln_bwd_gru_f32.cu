// Instantiates the persistent LayerNormGRU bwd recurrence kernels for f32 storage
// (one translation unit per combination so that they compile in parallel).
#include "rec_ln_cluster.cuh"

namespace hb {
namespace rec {
int run_lngru_bwd_f32(LnBwdParams& p, const Geometry& g, cudaStream_t s) { return run_ln_bwd<3, 2, float>(p, g, s); }
int run_lngru_cl_bwd_f32(const LnBwdParams& p, float* db_part, int* row_groups, cudaStream_t s) {
  return run_ln_cl_bwd<3, 2, float>(p, db_part, row_groups, s);
}
}  // namespace rec
}  // namespace hb
