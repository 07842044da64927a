// hb::gemm dispatcher: tcgen05/TMA kernel when the operands qualify, CUDA cores otherwise.
#include "cells.cuh"

namespace hb {

int gemm_sm100(const GemmDesc& g, cudaStream_t stream);     // gemm_sm100.cu
int gemm_simt_few(const GemmDesc& g, cudaStream_t stream);  // gemm_simt.cu

// Fewer than 32 rows stay on fp32 FMAs unless they are bf16: bf16 planes are less.  Relative error
// and time at 16 x 2048 x 512: FMAs 4.0e-7, two planes 4.5e-6 and 19 us, three planes 1.2e-6.
static bool few_rows(const GemmDesc& g) {
  return g.dtype != HASTE_B200_BF16 && g.M < 32 && (long long)g.M * g.N * g.K >= (1LL << 21);
}

int gemm(const GemmDesc& g, cudaStream_t stream) {
  const int path = gemm_path();
  if (path != HASTE_B200_GEMM_SIMT) {
    const int st_ = gemm_sm100(g, stream);
    if (st_ != HASTE_B200_ERR_UNSUPPORTED) return st_;
    // forced, or operands that exist as planes only: report rather than fall through
    if (!g.a || !g.b || path == HASTE_B200_GEMM_TCGEN05 || path == HASTE_B200_GEMM_TCGEN05_SINGLE) return st_;
  }
  return path == HASTE_B200_GEMM_AUTO && few_rows(g) ? gemm_simt_few(g, stream) : gemm_simt(g, stream);
}

int split_once(const void* src, long long rows, int width, bool wanted, GradPlanes* planes, long long* ld, bool* have,
               cudaStream_t s) {
  if (!wanted) return HASTE_B200_OK;
  const long long pad = (width + 7) & ~7LL;
  const size_t pe = Arena::pad((size_t)rows * pad * 2) / 2;  // elements per plane
  planes->p = static_cast<__nv_bfloat16*>(workspace(s, 2 * pe * 2 + 256, /*slot=*/3));
  if (!planes->p) return HASTE_B200_OK;
  planes->stride = (long long)pe;
  *ld = pad;
  *have = true;
  return gemm_split_planes(static_cast<const float*>(src), width, (int)rows, width, planes->p, pad, planes->stride, s);
}

}  // namespace hb
