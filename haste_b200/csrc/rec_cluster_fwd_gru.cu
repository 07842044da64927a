// Instantiates the cluster recurrence, gru fwd, for every storage type.
#include "rec_cluster_launch.cuh"

namespace hb {
namespace rec {
int run_cl_fwd_gru(int dtype, ChainParams& p, int most, int* row_groups, cudaStream_t s) {
  if (dtype == HASTE_B200_F16) return cl_fwd<3, 2, __half>(p, most, row_groups, s);
  if (dtype == HASTE_B200_F32) return cl_fwd<3, 2, float>(p, most, row_groups, s);
  return cl_fwd<3, 1, __nv_bfloat16>(p, most, row_groups, s);
}
}  // namespace rec
}  // namespace hb
