// Shared parts of the LayerNormLSTM / LayerNormGRU recurrences (rec_ln_cluster.cuh, rec_ln_grid.cuh),
// sm_100a: kernel parameters, exchange words, gate functions.
//
// A normalisation runs over a whole row (all G*H gate columns of h.R, all H units of c') while a CTA holds
// some of those columns, so row statistics are built in two levels: inside the CTA, then one pair per
// row and CTA, exchanged as tagged words and combined in a fixed order by every CTA.  Forward: (mean,
// M2) pairs combined with Chan's formula (no E[x^2]-mean^2 cancellation); backward: the two row sums
// of the LayerNorm gradient.  All LayerNorm inputs stay in fp32 between the stages of a step (with
// bf16 storage too: a value is rounded only when it is saved for the backward pass).
//
// Math and saved tensors follow the reference (lib/layer_norm_lstm_forward_gpu.cu.cc:26-109,
// 191-273; lib/layer_norm_lstm_backward_gpu.cu.cc:27-118,207-252; LayerNorm gradient
// lib/layer_norm_backward_gpu.cu.cc:44-91).  One deliberate difference: the reference's
// LayerNorm gradient carries a term proportional to sum(x - mean), which is zero in exact
// arithmetic; it is left out here.
#pragma once

#include "recurrent_common.cuh"

namespace hb {
namespace rec {

struct LnFwdParams {
  int T, N, H, training, has_zoneout;
  float zoneout_prob;
  const void* R;        // [H, 4H]
  const void* b;        // LSTM: b [4H];  GRU: bx [3H]
  const void* b2;       // GRU: br [3H]
  const void* Wx;       // LN(x.W) [T,N,G*H] (LSTM: aliases v)
  const void* gamma_Rh; // [G*H]
  const void* gamma_h;  // [H]
  const void* beta_h;   // [H]
  void* v;              // LSTM: act_Wx_norm [T,N,4H], LN(x.W) in, gate activations out
                        // GRU: cache [T,N,4H] = (z, r, g, LN(h.R)_g + br_g), may be null in inference
  void* act_Rh;         // [T,N,G*H] pre-norm h.R (saved)
  void* cache_Rh;       // [T,N,2]
  void* act_c_norm;     // [T,N,H]
  void* cache_c;        // [T,N,2]
  void* h;              // [T+1,N,H]
  void* c;              // [T+1,N,H] un-normalised cell state
  const void* mask;
  uint32_t* xbuf;       // grid: tagged h words
  uint32_t* sbuf;       // grid: tagged statistic pairs
  Sync sync;
};

struct LnBwdParams {
  int T, N, H, has_zoneout, r_transposed;
  const void* R;
  const void* gamma_Rh;
  const void* gamma_h;
  const void* c;          // LSTM [T+1,N,H]
  const void* h;          // GRU [T+1,N,H]
  void* dp;               // GRU out [T,N,3H]: gradient w.r.t. LN(x.W)+bx
  void* dq;               // GRU out [T,N,3H]: gradient w.r.t. LN(h.R)+br
  void* v;                // LSTM: act_Wx_norm, gate activations in, gate gradients out.
                          // GRU: cache [T,N,4H] in (untouched)
  void* act_Rh;           // pre-norm h.R in, d(h.R) out
  const void* cache_Rh;
  void* act_c_norm;       // LN(c') in (left untouched)
  const void* cache_c;
  const void* dh_new;
  const void* dc_new;
  const void* mask;
  float* dh_carry;        // [N,H] in/out
  float* dc_carry;        // [N,H] in/out
  float* dgRh_part;       // [rows][G*H] partial sums of dgamma_Rh, a row per row group (or half of one)
  float* dgh_part;        // [rows][H]
  float* dbh_part;        // [rows][H]
  uint32_t* exch;         // tagged partial dh [2][nBS][dst CTA][src CTA][rows][16]
  uint32_t* sbuf;         // [2 stats][2 parity][nBS][rows][nHS][2]
  Sync sync;
};

// Statistics, partial gradients and (with fp32 storage) h travel as tagged fp32 words
// (fword_* of recurrent_common.cuh): LayerNorm amplifies a relative error of the exchanged
// value roughly tenfold, so the 17 bits of the (hi, lo) bf16 pair are not enough here.
// h words: tagged fp32 with fp32 storage, the (hi, lo) bf16 pair with bf16 storage.
template <int SPLIT> __device__ __forceinline__ uint32_t hword_encode(float x, uint32_t tag) {
  return SPLIT == 2 ? fword_encode(x, tag) : xword_encode(x, tag);
}
// Gate functions of the LayerNorm cells.  With fp32 storage the accurate expf and tanhf: three
// normalisations per step amplify a relative error of 1e-6 (the ex2.approx-based fast forms) a
// hundredfold over a few dozen steps.  (1 - 2 / (1 + e^2x) with an accurate expf loses the small
// arguments' last bits: 20 steps of 64 rows, H = 512, relative error of h against fp64 6.8e-7, with tanhf
// 6.4e-7.)  bf16 storage keeps the fast forms (its bar is 2e-2).
template <int SPLIT> __device__ __forceinline__ float ln_sigmoid(float x) {
  return SPLIT == 2 ? 1.0f / (1.0f + expf(-x)) : sigmoid_fast(x);
}
template <int SPLIT> __device__ __forceinline__ float ln_tanh(float x) {
  if (SPLIT != 2) return tanh_fast(x);
  return tanhf(x);
}

// x = p[0] + p[1] + p[2], each the bf16 rounding of what the previous ones left.
__device__ __forceinline__ void split3_bf16(float x, float (&p)[3]) {
  p[0] = __bfloat162float(__float2bfloat16_rn(x));
  const float r1 = x - p[0];
  p[1] = __bfloat162float(__float2bfloat16_rn(r1));
  p[2] = __bfloat162float(__float2bfloat16_rn(r1 - p[1]));
}

// How the rows are shared out over the grid (rec_ln_grid.cuh): slices of 16 units x row groups, CH chains of
// eight rows per CTA.
struct LnGridGeometry {
  int nHS, nRG, CH;
};

// Clusters (rec_ln_cluster.cuh): HASTE_B200_ERR_UNSUPPORTED beyond 320 units.  Grid: up to 512 units, bf16
// storage 1024.  db_part and the partial sums of the gains: a row per row group (clusters) or two.
int run_ln_cl_fwd_f32(const LnFwdParams& p, cudaStream_t s);
int run_ln_cl_bwd_f32(const LnBwdParams& p, float* db_part, int* row_groups, cudaStream_t s);
int run_ln_grid_fwd_f32(const LnFwdParams& p, const LnGridGeometry& g, int wide, cudaStream_t s);
int run_ln_grid_bwd_f32(const LnBwdParams& p, float* db_part, const LnGridGeometry& g, int wide, cudaStream_t s);
int run_ln_cl_fwd_bf16(const LnFwdParams& p, cudaStream_t s);
int run_ln_cl_bwd_bf16(const LnBwdParams& p, float* db_part, int* row_groups, cudaStream_t s);
int run_ln_grid_fwd_bf16(const LnFwdParams& p, const LnGridGeometry& g, int wide, cudaStream_t s);
int run_ln_grid_bwd_bf16(const LnBwdParams& p, float* db_part, const LnGridGeometry& g, int wide, cudaStream_t s);
int run_lngru_cl_fwd_f32(const LnFwdParams& p, cudaStream_t s);
int run_lngru_cl_bwd_f32(const LnBwdParams& p, float* db_part, int* row_groups, cudaStream_t s);
int run_lngru_grid_fwd_f32(const LnFwdParams& p, const LnGridGeometry& g, int wide, cudaStream_t s);
int run_lngru_grid_bwd_f32(const LnBwdParams& p, float* db_part, const LnGridGeometry& g, int wide, cudaStream_t s);
int run_lngru_cl_fwd_bf16(const LnFwdParams& p, cudaStream_t s);
int run_lngru_cl_bwd_bf16(const LnBwdParams& p, float* db_part, int* row_groups, cudaStream_t s);
int run_lngru_grid_fwd_bf16(const LnFwdParams& p, const LnGridGeometry& g, int wide, cudaStream_t s);
int run_lngru_grid_bwd_bf16(const LnBwdParams& p, float* db_part, const LnGridGeometry& g, int wide, cudaStream_t s);

}  // namespace rec
}  // namespace hb
