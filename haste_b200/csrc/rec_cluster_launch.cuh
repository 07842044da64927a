// Launch side of the cluster recurrence kernels (rec_cluster_kernels.cuh): tiling choice and the
// template dispatch shared by the instantiation files.
#pragma once

#include <atomic>

#include "rec_cluster_kernels.cuh"

namespace hb {
namespace rec {

struct ClGeometry {
  int NW, CS, K16;  // stage warps (unit quads) per CTA, CTAs per cluster, 16-unit tiles in use
};

// 16 units per CTA up to H = 256 (one quad per tensor-core sub-partition); from there to 320 five
// quads keep the cluster at 16 CTAs - the largest there is - and R in registers.
// Backward with bf16 storage - half the weights, a third of the MMAs - 32 units per CTA reach 512.
// (In the other places that would fit, halving the cluster that way loses to the doubled work per
// sub-partition: H = 256, 32 rows 1.05 -> 1.30 us per step forward, 0.97 -> 1.21 backward, and
// forward at 512 units 1.65 -> 2.09 against the grid.)
inline bool cl_geometry(int H, bool wide_bwd, ClGeometry* g) {
  if (wide_bwd && H > 256 && H <= 512) {
    g->NW = 8;
    g->CS = ceil_div(H, 32);
  } else if (H <= 256) {
    g->NW = 4;
    g->CS = ceil_div(H, 16);
  } else if (H <= 320) {
    g->NW = 5;
    g->CS = 16;
  } else {
    return false;
  }
  g->K16 = g->CS * g->NW / 4;
  return true;
}

constexpr int kChainMaxDevices = 64;
constexpr int kClMaxChains = 6;

// Launches `kernel` over ceil(N / 8) chains in clusters of CTAS CTAs.  The number of chains a CTA
// carries is the smallest that lets all clusters be resident at once (further clusters would
// queue behind whole passes); more than `most` (below kClMaxChains) is not taken.  `smem_chain` / `smem_fixed`: dynamic shared memory per chain and
// besides.  `slots`: resident clusters per (device, cluster size), asked once.
template <typename P>
int cl_launch(void (*kernel)(P), P& p, int threads, size_t smem_chain, size_t smem_fixed,
                     std::atomic<int> (*slots)[17], int most, int* row_groups, cudaStream_t s) {
  int dev = 0;
  HB_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kChainMaxDevices) return HASTE_B200_ERR_UNSUPPORTED;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.CTAS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  constexpr int kMostSmem = 227 * 1024;
  int mc = slots[dev][p.CTAS].load(std::memory_order_acquire);
  if (mc == 0) {
    mc = -1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem - 64) == cudaSuccess &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
      cfg.gridDim = dim3(p.CTAS * 64);
      cfg.dynamicSmemBytes = smem_fixed + 2 * smem_chain;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0) mc = n;
    }
    cudaGetLastError();
    slots[dev][p.CTAS].store(mc, std::memory_order_release);
  }
  if (mc < 0) return HASTE_B200_ERR_UNSUPPORTED;
  const int budget = sm_budget();
  if (budget > 0 && budget < sm_count()) mc = max(1, (int)((long long)mc * budget / sm_count()));
  const int tiles = ceil_div(p.N, 8);
  if (most < kClMaxChains && ceil_div(tiles, mc) > most) return HASTE_B200_ERR_UNSUPPORTED;
  p.CH = min(kClMaxChains, ceil_div(tiles, mc));
  *row_groups = ceil_div(tiles, p.CH);
  cfg.gridDim = dim3(p.CTAS * *row_groups);
  cfg.dynamicSmemBytes = smem_fixed + (size_t)p.CH * smem_chain;
  HB_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, p));
  count_launch(1);
  return HASTE_B200_OK;
}

template <int G, int NW, int KS, int SPLIT, typename T>
int cl_fwd_go(ChainParams& p, int most, int* row_groups, cudaStream_t s) {
  static std::atomic<int> slots[kChainMaxDevices][17];
  const size_t chain = (size_t)2 * p.K16 * 512 + (size_t)2 * NW * 32 * 4;
  return cl_launch(cl_fwd_kernel<G, NW, KS, SPLIT, T>, p, NW * 32, chain, (size_t)NW * IoBytes<T>::WARP, slots,
                   most, row_groups, s);
}

template <int G, int SPLIT, typename T>
int cl_fwd(ChainParams& p, int most, int* row_groups, cudaStream_t s) {
  ClGeometry g;
  if (!cl_geometry(p.H, false, &g)) return HASTE_B200_ERR_UNSUPPORTED;
  p.CTAS = g.CS;
  p.K16 = g.K16;
  if (g.NW == 5) return cl_fwd_go<G, 5, 20, SPLIT, T>(p, most, row_groups, s);
  if (g.K16 <= 4) return cl_fwd_go<G, 4, 4, SPLIT, T>(p, most, row_groups, s);
  if (g.K16 <= 8) return cl_fwd_go<G, 4, 8, SPLIT, T>(p, most, row_groups, s);
  if (g.K16 <= 12) return cl_fwd_go<G, 4, 12, SPLIT, T>(p, most, row_groups, s);
  return cl_fwd_go<G, 4, 16, SPLIT, T>(p, most, row_groups, s);
}

template <int G, int NW, int TPW, int SPLIT, typename T>
int cl_bwd_go(ChainParams& p, int most, int* row_groups, cudaStream_t s) {
  static std::atomic<int> slots[kChainMaxDevices][17];
  const size_t chain = (size_t)2 * p.CTAS * NW * 128 + (size_t)3 * NW * 32 * 4;
  const size_t fixed = (size_t)2 * ((G * NW + 3) / 4) * 512 + (size_t)NW * IoBytes<T>::WARP;
  return cl_launch(cl_bwd_kernel<G, NW, TPW, SPLIT, T>, p, NW * 32, chain, fixed, slots, most, row_groups, s);
}

template <int G, int SPLIT, typename T>
int cl_bwd(ChainParams& p, int most, int* row_groups, cudaStream_t s) {
  ClGeometry g;
  if (!cl_geometry(p.H, SPLIT == 1, &g)) return HASTE_B200_ERR_UNSUPPORTED;
  p.CTAS = g.CS;
  p.K16 = g.K16;
  if constexpr (SPLIT == 1) {
    if (g.NW == 8 && g.CS <= 12) return cl_bwd_go<G, 8, 3, SPLIT, T>(p, most, row_groups, s);
    if (g.NW == 8) return cl_bwd_go<G, 8, 4, SPLIT, T>(p, most, row_groups, s);
  }
  if (g.NW == 5) return cl_bwd_go<G, 5, 4, SPLIT, T>(p, most, row_groups, s);
  if (g.K16 <= 4) return cl_bwd_go<G, 4, 1, SPLIT, T>(p, most, row_groups, s);
  if (g.K16 <= 8) return cl_bwd_go<G, 4, 2, SPLIT, T>(p, most, row_groups, s);
  if (g.K16 <= 12) return cl_bwd_go<G, 4, 3, SPLIT, T>(p, most, row_groups, s);
  return cl_bwd_go<G, 4, 4, SPLIT, T>(p, most, row_groups, s);
}

// One translation unit per cell and direction.
int run_cl_fwd_lstm(int dtype, ChainParams& p, int most, int* row_groups, cudaStream_t s);
int run_cl_fwd_gru(int dtype, ChainParams& p, int most, int* row_groups, cudaStream_t s);
int run_cl_bwd_lstm(int dtype, ChainParams& p, int most, int* row_groups, cudaStream_t s);
int run_cl_bwd_gru(int dtype, ChainParams& p, int most, int* row_groups, cudaStream_t s);

}  // namespace rec
}  // namespace hb
