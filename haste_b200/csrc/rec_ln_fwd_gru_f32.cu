// Instantiates the persistent LayerNormGRU fwd recurrence kernels for f32 storage
// (one translation unit per combination so that they compile in parallel).
#include "rec_ln_cluster.cuh"

namespace hb {
namespace rec {
int run_lngru_fwd_f32(LnFwdParams& p, const Geometry& g, cudaStream_t s) { return run_ln_fwd<3, 2, float>(p, g, s); }
int run_lngru_cl_fwd_f32(const LnFwdParams& p, cudaStream_t s) { return run_ln_cl_fwd<3, 2, float>(p, s); }
}  // namespace rec
}  // namespace hb
