// Argument blocks and driver entry points of the six cells (internal C++ layer
// directly under the C ABI of include/haste_b200.h; field meanings are documented
// there).
#pragma once

#include "common.cuh"
#include "util.cuh"

namespace hb {

struct LstmFwd {
  int dtype, training, T, N, C, H;
  const void *W, *R, *b, *x;
  void *h, *c, *v, *tmp_Rh;
  float zoneout_prob;
  const void* zoneout_mask;
  // Single-step form (T == 1, the reference's Iterate): new state goes to separate [N,H]
  // buffers instead of slot 1 of h / c.
  void *h_out = nullptr, *c_out = nullptr;
};
struct LstmBwd {
  int dtype, transposed_inputs, T, N, C, H;
  const void *W, *R, *b, *x, *h, *c, *dh_new, *dc_new;
  void *dx, *dW, *dR, *db, *dh, *dc, *v;
  const void* zoneout_mask;
  // Single-step form (T == 1): h, c, dh_new, dc_new are the step's own [N,H] buffers and
  // c_new is the cell state the forward step produced.
  int iterate = 0;
  const void* c_new = nullptr;
};
struct GruFwd {
  int dtype, training, T, N, C, H;
  const void *W, *R, *bx, *br, *x;
  void *h, *v, *tmp_Wx, *tmp_Rh;
  float zoneout_prob;
  const void* zoneout_mask;
  void* h_out = nullptr;  // single-step form (T == 1): new state, [N,H]
};
struct GruBwd {
  int dtype, transposed_inputs, T, N, C, H;
  const void *W, *R, *bx, *br, *x, *h, *v, *dh_new;
  void *dx, *dW, *dR, *dbx, *dbr, *dh, *dp, *dq;
  const void* zoneout_mask;
  int iterate = 0;  // single-step form (T == 1): dh_new is the step's own [N,H] buffer
};
struct IndrnnFwd {
  int dtype, training, T, N, C, H;
  const void *W, *u, *b, *x;
  void *h, *workspace;
  float zoneout_prob;
  const void* zoneout_mask;
  // LayerNorm variant only (gamma == nullptr selects the plain cell)
  const void* gamma;
  void *act_Wx, *cache_Wx;
};
struct IndrnnBwd {
  int dtype, transposed_inputs, T, N, C, H;
  const void *W, *u, *b, *x, *h, *dh_new;
  void *dx, *dW, *du, *db, *dh, *workspace;
  const void* zoneout_mask;
  const void* gamma;
  void* dgamma;
  const void *act_Wx, *cache_Wx;
};
struct LnLstmFwd {
  int dtype, training, T, N, C, H;
  const void *W, *R, *b, *gamma_Wx, *gamma_Rh, *gamma_h, *beta_h, *x;
  void *h, *c, *act_Wx, *act_Wx_norm, *cache_Wx, *act_Rh, *cache_Rh, *act_c_norm, *cache_c,
      *tmp_Rh;
  float zoneout_prob;
  const void* zoneout_mask;
};
struct LnLstmBwd {
  int dtype, transposed_inputs, T, N, C, H;
  const void *W, *R, *b, *gamma_Wx, *gamma_Rh, *gamma_h, *beta_h, *x, *h, *c, *dh_new, *dc_new;
  void *dx, *dW, *dR, *db, *dgamma_Wx, *dgamma_Rh, *dgamma_h, *dbeta_h, *dh, *dc, *act_Wx, *act_Wx_norm;
  const void* cache_Wx;
  void* act_Rh;
  const void* cache_Rh;
  void* act_c_norm;
  const void* cache_c;
  const void* zoneout_mask;
};
struct LnGruFwd {
  int dtype, training, T, N, C, H;
  const void *W, *R, *bx, *br, *gamma_Wx, *gamma_Rh, *x;
  void *h, *v, *act_Wx, *cache_Wx, *tmp_Wx_norm, *act_Rh, *cache_Rh, *tmp_Rh_norm;
  float zoneout_prob;
  const void* zoneout_mask;
};
struct LnGruBwd {
  int dtype, transposed_inputs, T, N, C, H;
  const void *W, *R, *bx, *br, *gamma_Wx, *gamma_Rh, *x, *h, *v, *dh_new;
  void *dx, *dW, *dR, *dbx, *dbr, *dgamma_Wx, *dgamma_Rh, *dh, *dp, *dq;
  const void *act_Wx, *cache_Wx;
  void* act_Rh;  // overwritten with d(h.R)
  const void* cache_Rh;
  const void* zoneout_mask;
};

int lstm_forward(const LstmFwd& a, cudaStream_t s);
int lstm_backward(const LstmBwd& a, cudaStream_t s);
int gru_forward(const GruFwd& a, cudaStream_t s);
int gru_backward(const GruBwd& a, cudaStream_t s);
int indrnn_forward(const IndrnnFwd& a, cudaStream_t s);
int indrnn_backward(const IndrnnBwd& a, cudaStream_t s);
int layer_norm_lstm_forward(const LnLstmFwd& a, cudaStream_t s);
int layer_norm_lstm_backward(const LnLstmBwd& a, cudaStream_t s);
int layer_norm_gru_forward(const LnGruFwd& a, cudaStream_t s);
int layer_norm_gru_backward(const LnGruBwd& a, cudaStream_t s);

// single-step (Iterate) forward in one launch (iterate_fused.cu); UNSUPPORTED: take the general path
int lstm_forward_step_fused(const LstmFwd& a, cudaStream_t s);
int gru_forward_step_fused(const GruFwd& a, cudaStream_t s);
// Optional bf16 (hi, lo) planes of the gate gradients, written by the persistent backward
// kernels in fp32 mode (p: dv / dp, p2: dq; lo plane `stride` elements after hi).
struct GradPlanes {
  __nv_bfloat16* p = nullptr;
  __nv_bfloat16* p2 = nullptr;
  long long stride = 0;
};
// Persistent implementations of the recurrences.  Each returns HASTE_B200_ERR_UNSUPPORTED
// (without touching any buffer) when the shape is not its own, in which case the caller goes on to
// the next one, at last to its step-wise path.
// Chain recurrences (rec_chain_host.cu): on a thread-block cluster or the whole grid, H up to
// 1024.  Forward: the input projection is already in a.v (LSTM) / a.tmp_Wx (GRU).  Backward:
// complete - dh and dc are read and written in place (dc_new may be null), the bias gradients
// added.  `few`: leave batches to the tensor-core recurrence where that is faster.
int lstm_forward_chain(const LstmFwd& a, bool few, cudaStream_t s);
int lstm_backward_chain(const LstmBwd& a, const GradPlanes& planes, bool few, cudaStream_t s);
int gru_forward_chain(const GruFwd& a, bool few, cudaStream_t s);
int gru_backward_chain(const GruBwd& a, const GradPlanes& planes, bool few, cudaStream_t s);
// Tensor-core recurrence for bf16 batches of about a hundred rows and more (rec_tc.cu).  The
// backward kernel carries dh in an fp32 [N,H] buffer and does not sum the bias gradients.
bool lstm_tc_takes(int dtype, int N, int H, bool fwd);
int lstm_forward_tc(const LstmFwd& a, float* c_carry, cudaStream_t s);
int lstm_backward_tc(const LstmBwd& a, float* dh_carry, float* dc_carry, cudaStream_t s);
int gru_forward_tc(const GruFwd& a, cudaStream_t s);
int gru_backward_tc(const GruBwd& a, float* dh_carry, cudaStream_t s);
// LayerNorm cells (recurrent_host.cu): forward expects LN(x.W) in a.act_Wx_norm / a.tmp_Wx_norm; backward is
// complete - fp32 carries read and written in place, bias and LayerNorm gradients of h.R and c added or
// assigned - and leaves d(h.R) in a.act_Rh.
int layer_norm_lstm_forward_persistent(const LnLstmFwd& a, cudaStream_t s);
int layer_norm_lstm_backward_persistent(const LnLstmBwd& a, float* dh_carry, float* dc_carry, cudaStream_t s);
int layer_norm_gru_forward_persistent(const LnGruFwd& a, cudaStream_t s);
int layer_norm_gru_backward_persistent(const LnGruBwd& a, float* dh_carry, cudaStream_t s);

// Exchange-only probe (recurrent_host.cu): device microseconds per step of the forward
// recurrence's hand-off alone, for the tiling (N, H) would get.
int exchange_probe(int N, int H, int steps, float* us_per_step, cudaStream_t s);

// Per-step contraction (M = batch rows).  Small products are launch-bound and stay on the
// CUDA-core kernel; from 2^26 multiply-adds up the tensor-core kernel pays for its set-up
// (operand split and tensor maps) even with a partly empty 128-row tile.
inline bool tensor_core_step(long long M, long long N, long long K) { return M >= 32 && M * N * K >= (1LL << 26); }
inline int gemm_small(const GemmDesc& g, cudaStream_t s) {
  return tensor_core_step(g.M, g.N, g.K) ? gemm(g, s) : gemm_simt(g, s);
}
// fp32 LSTM / GRU layers of 512 to 1024 units whose step product would be fp32 FMAs if the grid
// recurrence did not take it, with two planes: their input projection is made exact (six products), so
// that the outputs as a whole are no less exact than by that path.  Relative error against fp64, step
// by step / grid / grid with this: LSTM, T = 100, 16 rows, H = 640 h 4.6e-6 / 5.2e-6 / 2.4e-6, dx 5.3 /
// 6.0 / 5.3, dR 5.4 / 6.6 / 4.6; 31 rows, H = 1024 4.6 / 5.1 / 2.4.  (The bias gradient, a sum over all
// rows and steps, keeps the planes of R: 2.0 / 3.6 / 3.2.)  1 to 3 % of a pass, 6 % of GRU inference.
inline int wide_few_rows(int dtype, int N, int GH, int H) {
  return dtype == HASTE_B200_F32 && H > 512 && H <= 1024 && !tensor_core_step(N, GH, H);
}

// fp32 [rows, width] -> planes for several contractions, in the scratch the recurrence kernels would
// have written them to; *have stays false if `wanted` is or the scratch cannot be had.
int split_once(const void* src, long long rows, int width, bool wanted, GradPlanes* planes, long long* ld, bool* have,
               cudaStream_t s);

// Knobs of the process (set through the C ABI); the budget also of a thread, in front of it.
int recurrence_path();
int sm_budget();  // 0: the whole GPU; else the SMs one recurrence launch may occupy
int gemm_path();
// This thread: backward passes assign parameter gradients, dh and dc instead of adding to them.
bool assign_gradients();

}  // namespace hb
