// Launch side of the grid recurrence kernels (rec_grid_kernels.cuh): template dispatch shared by
// the instantiation files.
#pragma once

#include "rec_cluster_launch.cuh"
#include "rec_grid_kernels.cuh"

namespace hb {
namespace rec {

constexpr int kGlMaxSmem = 226 * 1024;

struct GlGeometry {
  int NMT, nHS, nRG, CH, KS16;  // KS16: 16-unit tiles of the hidden dimension
};

// One CTA per SM, all resident (cooperative launch).  `attr_set`: per kernel and device.
template <typename P>
int gl_launch(void (*kernel)(P), P& p, int grid, size_t smem, std::atomic<int>* attr_set,
                     cudaStream_t s) {
  int dev = 0;
  HB_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kChainMaxDevices || smem > (size_t)kGlMaxSmem || grid > sm_count())
    return HASTE_B200_ERR_UNSUPPORTED;
  if (!attr_set[dev].load(std::memory_order_acquire)) {
    // The register split assumes 128 registers per thread at launch: less, and a product warp
    // would wait for registers that nobody frees.
    cudaFuncAttributes fa;
    int per_sm = 0;
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess || fa.numRegs != 128 ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGlMaxSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, GL_THREADS, kGlMaxSmem) != cudaSuccess ||
        per_sm < 1) {
      cudaGetLastError();
      return HASTE_B200_ERR_UNSUPPORTED;
    }
    attr_set[dev].store(1, std::memory_order_release);
  }
  void* args[] = {&p};
  const cudaError_t e = cudaLaunchCooperativeKernel((const void*)kernel, dim3(grid), dim3(GL_THREADS), args, smem, s);
  if (e != cudaSuccess) {
    set_last_error("cooperative launch failed: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return HASTE_B200_ERR_CUDA;
  }
  count_launch(1);
  return HASTE_B200_OK;
}

template <int G, int NMT, int KSW, int SPLIT, typename T>
int gl_fwd_go(ChainParams& p, const GlGeometry& g, cudaStream_t s) {
  static std::atomic<int> set[kChainMaxDevices];
  const size_t slot = (size_t)GL_WARPS * NMT * 512 + 16;
  const size_t rest = (size_t)g.CH * 2 * NMT * 128 + (size_t)GL_WARPS * IoBytes<T>::WARP +
                      (gl_lo_in_smem<NMT, KSW, SPLIT>() ? (size_t)GL_WARPS * NMT * KSW * 512 : 0);
  // two slots per chain where they fit, else as many as do
  const int fit = rest >= (size_t)kGlMaxSmem ? 0 : (int)(((size_t)kGlMaxSmem - rest) / slot);
  p.ring = min(2 * g.CH, fit);
  p.throttle = p.ring < 2 * g.CH;
  if (p.ring < 2) return HASTE_B200_ERR_UNSUPPORTED;
  return gl_launch(gl_fwd_kernel<G, NMT, KSW, SPLIT, T>, p, g.nHS * g.nRG, p.ring * slot + rest, set, s);
}

template <int G, int SPLIT, typename T>
int gl_fwd(ChainParams& p, const GlGeometry& g, cudaStream_t s) {
  const int ksw = ceil_div(g.KS16, GL_WARPS);
#define HB_GL(nmt, k) \
  if (g.NMT == nmt && ksw <= k) return gl_fwd_go<G, nmt, k, SPLIT, T>(p, g, s);
  HB_GL(4, 2) HB_GL(4, 4) HB_GL(4, 6) HB_GL(4, 8)
  if constexpr (SPLIT == 2) { HB_GL(2, 6) HB_GL(2, 8) }
#undef HB_GL
  return HASTE_B200_ERR_UNSUPPORTED;
}

template <int G, int NMT, int TPW, int SPLIT, typename T>
int gl_bwd_go(ChainParams& p, const GlGeometry& g, cudaStream_t s) {
  static std::atomic<int> set[kChainMaxDevices];
  constexpr int KSB = (G * NMT + 3) / 4, SP = 4 / NMT;
  const size_t smem = (size_t)GL_GRING * KSB * 512 + (gl_lo_in_smem<NMT, TPW, SPLIT>() ? (size_t)GL_WARPS * TPW * KSB * 512 : 0) + (size_t)4 * SP * NMT * 128 + (size_t)g.CH * 3 * NMT * 128 +
                      (2 * GL_GRING + 2) * 8 + (size_t)GL_WARPS * IoBytes<T>::WARP;
  return gl_launch(gl_bwd_kernel<G, NMT, TPW, SPLIT, T>, p, g.nHS * g.nRG, smem, set, s);
}

template <int G, int SPLIT, typename T>
int gl_bwd(ChainParams& p, const GlGeometry& g, cudaStream_t s) {
  const int tpw = ceil_div(g.KS16, GL_WARPS);
#define HB_GL(nmt, k) \
  if (g.NMT == nmt && tpw <= k) return gl_bwd_go<G, nmt, k, SPLIT, T>(p, g, s);
  HB_GL(4, 2) HB_GL(4, 4) HB_GL(4, 6) HB_GL(4, 8)
  if constexpr (SPLIT == 2) { HB_GL(2, 6) HB_GL(2, 8) }
#undef HB_GL
  return HASTE_B200_ERR_UNSUPPORTED;
}

int run_gl_fwd_lstm(int dtype, ChainParams& p, const GlGeometry& g, cudaStream_t s);
int run_gl_fwd_gru(int dtype, ChainParams& p, const GlGeometry& g, cudaStream_t s);
int run_gl_bwd_lstm(int dtype, ChainParams& p, const GlGeometry& g, cudaStream_t s);
int run_gl_bwd_gru(int dtype, ChainParams& p, const GlGeometry& g, cudaStream_t s);

}  // namespace rec
}  // namespace hb
