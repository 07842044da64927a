// Instantiates the grid recurrence, gru fwd, for every storage type.
#include "rec_grid_launch.cuh"

namespace hb {
namespace rec {
int run_gl_fwd_gru(int dtype, ChainParams& p, const GlGeometry& g, cudaStream_t s) {
  if (dtype == HASTE_B200_F16) return gl_fwd<3, 2, __half>(p, g, s);
  if (dtype == HASTE_B200_F32) return gl_fwd<3, 2, float>(p, g, s);
  return gl_fwd<3, 1, __nv_bfloat16>(p, g, s);
}
}  // namespace rec
}  // namespace hb
