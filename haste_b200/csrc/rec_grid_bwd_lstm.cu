// Instantiates the grid recurrence, lstm bwd, for every storage type.
#include "rec_grid_launch.cuh"

namespace hb {
namespace rec {
int run_gl_bwd_lstm(int dtype, ChainParams& p, const GlGeometry& g, cudaStream_t s) {
  if (dtype == HASTE_B200_F32) return gl_bwd<4, 2, float>(p, g, s);
  return gl_bwd<4, 1, __nv_bfloat16>(p, g, s);
}
}  // namespace rec
}  // namespace hb
