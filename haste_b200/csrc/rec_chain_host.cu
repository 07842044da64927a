// Host side of the chain recurrences: what the kernels of rec_cluster_kernels.cuh and
// rec_grid_kernels.cuh read and write, and which of the two takes a shape.
#include <initializer_list>

#include "rec_grid_launch.cuh"

namespace hb {

using namespace rec;

namespace {

// Whole-quad accesses: every row of every array starts on a multiple of four elements.
bool aligned(std::initializer_list<const void*> ptrs, int H, int dtype) {
  uintptr_t a = 0;
  for (const void* q : ptrs) a |= reinterpret_cast<uintptr_t>(q);
  return H % 4 == 0 && a % (4 * dtype_size(dtype)) == 0;
}

// Grid tiling: NMT quads of hidden units per CTA such that its slice of R fits on chip, as
// many row groups as there are SMs for, the rest of the rows as chains - at most `most` of them: a
// chain adds 0.7 .. 2 us to a step (H = 512 .. 1024), which the step-wise path (about 20 us plus the
// product) undercuts from a dozen on, and before that the tensor-core recurrence of bf16 layers (rec_tc.cu), whose
// step hardly depends on the rows.  us per step forward / backward, chains / tensor cores.  GRU H = 1024: five chains
// 5.7 / 8.4 and 6.8 / 7.8, six 6.8 / 8.9 and 6.8 / 7.9; H = 512: six 5.7 / 6.0 and 5.5 / 6.9.  LSTM H = 1024: six
// 7.1 / 8.8 and 8.3 / 8.7, seven 8.3 / 10.7 and 8.3 / 8.9, eight 9.4 / 11.6 and 8.4 / 9.0; H = 768: seven 7.3 / 10.8 and
// 8.0 / 11.2; H = 512: eight 7.2 / 8.0 and 6.9 / 7.2 on half of the GPU, 6.9 / 8.1 and 7.1 / 7.7 on all of it.  Backward the
// chains keep more than their time says: they sum the bias gradients before these are rounded to bf16 (GRU 90 rows
// H = 1000, relative to fp64: 2.6e-3, summed from the rounded gradients 2.85e-3).
constexpr int kGridChains = 12;
constexpr int kGruChainsBeforeTc = 6, kLstmChainsBeforeTcFwd = 7, kLstmChainsBeforeTcBwd = 8;

// fp32 and fp16 storage beyond 512 units: two quads per CTA keep both planes of R in registers, four put the
// second plane into shared memory and so take half the CTAs per row group.  Half the CTAs read (backward:
// add up) each state, and twice the row groups share the chains; but a chain's product takes twice as long, so
// the chains must be enough to fill that time (LSTM fp32, us per step, two quads / four: forward H = 1024 24
// rows, three chains 3.2 / 3.8, 32 rows, four 4.2 / 3.8, 64 rows 8.2 / 7.0, H = 768 64 rows 7.3 / 4.5; backward
// H = 1024 16 rows 3.8 / 4.0, 24 rows 5.9 / 4.9, 32 rows 6.4 / 5.0, 64 rows 12.8 / 8.8, 90 rows 24.4 / 12.3).
constexpr int kFourQuadsFwd = 4, kFourQuadsBwd = 3;

bool gl_geometry(int dtype, int N, int H, bool bwd, int most, GlGeometry* g) {
  g->KS16 = ceil_div(H, 16);
  const int ks = ceil_div(g->KS16, GL_WARPS);
  if (ks > 8) return false;
  const int tiles = ceil_div(N, 8), sms = sm_count(), budget = sm_budget();
  const bool wide = dtype != HASTE_B200_BF16 && ks > 4;
  auto within = [&](int use, GlGeometry* g) {
    if (use < g->KS16) return false;  // (four quads take the fewest CTAs: one per 16 units)
    for (int nmt : {2, 4}) {
      if (nmt == 2 && !wide) continue;
      g->NMT = nmt;
      g->nHS = ceil_div(H, 4 * nmt);
      if (use < g->nHS) continue;
      g->nRG = min(tiles, use / g->nHS);
      g->CH = ceil_div(tiles, g->nRG);
      g->nRG = ceil_div(tiles, g->CH);
      if (nmt == 2 && g->CH >= (bwd ? kFourQuadsBwd : kFourQuadsFwd)) continue;
      if (g->CH <= most) return true;
    }
    return false;
  };
  // Under an SM budget (two directions side by side) first within it; if that takes too many chains, the whole
  // GPU for one direction after the other is ahead: of the step-wise path (bf16 LSTM, two directions of 139
  // rows, H = 696: 18 chains within the budget, 6 without), and for wide fp32 layers, where half of the GPU holds one
  // row group and all of it two or three, also of twice and three times the chains (budget_pays).
  if (budget >= g->KS16 && budget <= sms) {
    GlGeometry whole = *g;
    if (within(budget, g)) {
      if (wide && within(sms, &whole) && !budget_pays(bwd, budget, g->CH, whole.CH)) *g = whole;
      return true;
    }
    if (most < kGridChains) return false;  // the tensor-core recurrence comes next, within the budget too
  }
  return within(sms, g);
}

// How many chains per CTA the cluster kernels may take before the grid kernels do better (us per
// step, fp32 LSTM, cluster / grid).  Up to 192 units clusters are small enough that there are
// always enough of them (H = 192, 128 rows: 1.4 / 2.2 forward).  At 256 units a cluster is 16 CTAs
// and only seven are resident one CTA per SM: 32 rows 1.15 / 1.5 forward, 1.2 / 2.0 backward, but
// 128 rows 2.8 / 1.8 and 3.0 / 2.4.  Five quads per CTA (to 320 units) pay in the backward pass
// only: 2.0 / 1.7 and 1.8 / 2.2 at 19 rows.  Eight (bf16, backward, to 512 units): one chain 1.47 / 1.96
// at H = 384 and 1.58 / 2.41 at H = 512 (48 and 56 rows), two chains 2.87 / 2.31 and 3.0 / 2.4.
int cluster_chains(const ClGeometry& g, bool bwd) {
  if (g.NW == 8) return 1;
  if (g.NW == 5) return bwd ? 1 : 0;
  return g.CS <= 12 ? kClMaxChains : 1;
}

// Zeroed scratch: abort flag, then `words` exchange words, then `floats` that need no zeroing.
int gl_scratch(ChainParams* p, size_t words, size_t floats, float** extra, cudaStream_t s) {
  const size_t head = 256, bytes = head + Arena::pad(words * 4);
  char* base = static_cast<char*>(workspace(s, bytes + Arena::pad(floats * 4), /*slot=*/2));
  if (!base) return HASTE_B200_ERR_CUDA;
  HB_CUDA_OK(cudaMemsetAsync(base, 0, bytes, s));
  p->sync.abort_flag = reinterpret_cast<int*>(base);
  p->xbuf = reinterpret_cast<uint32_t*>(base + head);
  if (extra) *extra = reinterpret_cast<float*>(base + bytes);
  return HASTE_B200_OK;
}

typedef int (*ClRun)(int, ChainParams&, int, int*, cudaStream_t);
typedef int (*GlRun)(int, ChainParams&, const GlGeometry&, cudaStream_t);

int run_fwd(ChainParams& p, int dtype, int grid_most, ClRun cl, GlRun gl, cudaStream_t s) {
  p.sync.err = device_error_word();
  HB_REQUIRE(p.sync.err, "error word");
  ClGeometry cg;
  if (cl_geometry(p.H, false, &cg)) {
    int groups = 0;
    const int st_ = cl(dtype, p, cluster_chains(cg, false), &groups, s);
    if (st_ != HASTE_B200_ERR_UNSUPPORTED) return st_;
  }
  GlGeometry g;
  if (!gl_geometry(dtype, p.N, p.H, false, grid_most, &g)) return HASTE_B200_ERR_UNSUPPORTED;
  p.CTAS = g.nHS; p.CH = g.CH; p.K16 = g.KS16;
  HB_TRY(gl_scratch(&p, (size_t)2 * ceil_div(p.N, 8) * g.KS16 * 128, 0, nullptr, s));
  return gl(dtype, p, g, s);
}

int run_bwd(ChainParams& p, int dtype, int grid_most, int gates, void* db, void* db2, ClRun cl, GlRun gl,
            cudaStream_t s) {
  p.sync.err = device_error_word();
  p.zero_init = assign_gradients();
  HB_REQUIRE(p.sync.err, "error word");
  const int tiles = ceil_div(p.N, 8);
  ClGeometry cg;
  if (cl_geometry(p.H, dtype == HASTE_B200_BF16, &cg)) {
    p.db_part = static_cast<float*>(workspace(s, (size_t)tiles * 4 * p.H * sizeof(float), /*slot=*/2));
    if (!p.db_part) return HASTE_B200_ERR_CUDA;
    int groups = 0;
    const int st_ = cl(dtype, p, cluster_chains(cg, true), &groups, s);
    if (st_ == HASTE_B200_OK) return bias_grad_finish(gates, p.db_part, groups, p.H, dtype, db, db2, !p.zero_init, s);
    if (st_ != HASTE_B200_ERR_UNSUPPORTED) return st_;
  }
  GlGeometry g;
  if (!gl_geometry(dtype, p.N, p.H, true, grid_most, &g)) return HASTE_B200_ERR_UNSUPPORTED;
  p.CTAS = g.nHS; p.CH = g.CH; p.K16 = ceil_div(g.nHS * g.NMT, 4);
  HB_TRY(gl_scratch(&p, (size_t)2 * tiles * g.nHS * g.nHS * g.NMT * 32, (size_t)g.nRG * 8 * p.H, &p.db_part, s));
  HB_TRY(gl(dtype, p, g, s));
  return bias_grad_finish(gates, p.db_part, 2 * g.nRG, p.H, dtype, db, db2, !p.zero_init, s);
}

// Rows the tensor-core GRU recurrence would take (rec_tc.cu).
bool tc_waits(int dtype, int N, int H) {
  return dtype == HASTE_B200_BF16 && N >= 64 && H % 8 == 0 && recurrence_path() != HASTE_B200_PATH_NO_TENSOR_CORE;
}

}  // namespace

int lstm_forward_chain(const LstmFwd& a, bool few, cudaStream_t s) {
  if (recurrence_path() == HASTE_B200_PATH_STEPWISE) return HASTE_B200_ERR_UNSUPPORTED;
  ChainParams p{};
  p.T = a.T; p.N = a.N; p.H = a.H;
  p.training = a.training; p.has_zoneout = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  p.zoneout_prob = a.zoneout_prob;
  p.R = a.R; p.b = a.b; p.gin = a.v; p.gout = a.training ? a.v : nullptr; p.mask = a.zoneout_mask;
  p.h = a.h; p.c = a.c;
  p.wide = aligned({a.v, a.h, a.c, a.zoneout_mask}, a.H, a.dtype);
  const int most = few && lstm_tc_takes(a.dtype, a.N, a.H, true) ? kLstmChainsBeforeTcFwd : kGridChains;
  return run_fwd(p, a.dtype, most, run_cl_fwd_lstm, run_gl_fwd_lstm, s);
}

int gru_forward_chain(const GruFwd& a, bool few, cudaStream_t s) {
  if (recurrence_path() == HASTE_B200_PATH_STEPWISE) return HASTE_B200_ERR_UNSUPPORTED;
  ChainParams p{};
  p.T = a.T; p.N = a.N; p.H = a.H;
  p.training = a.training; p.has_zoneout = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  p.zoneout_prob = a.zoneout_prob;
  p.R = a.R; p.b = a.bx; p.b2 = a.br; p.gin = a.tmp_Wx; p.gout = a.training ? a.v : nullptr;
  p.mask = a.zoneout_mask; p.h = a.h;
  p.wide = aligned({a.tmp_Wx, a.v, a.h, a.zoneout_mask}, a.H, a.dtype);
  return run_fwd(p, a.dtype, few && tc_waits(a.dtype, a.N, a.H) ? kGruChainsBeforeTc : kGridChains,
                 run_cl_fwd_gru, run_gl_fwd_gru, s);
}

int lstm_backward_chain(const LstmBwd& a, const GradPlanes& planes, bool few, cudaStream_t s) {
  if (recurrence_path() == HASTE_B200_PATH_STEPWISE) return HASTE_B200_ERR_UNSUPPORTED;
  ChainParams p{};
  p.T = a.T; p.N = a.N; p.H = a.H;
  p.has_zoneout = a.zoneout_mask ? 1 : 0; p.r_transposed = a.transposed_inputs;
  p.R = a.R; p.gin = a.v; p.dv = a.v; p.c = const_cast<void*>(a.c); p.dh_new = a.dh_new; p.dc_new = a.dc_new;
  p.mask = a.zoneout_mask; p.dh = a.dh; p.dc = a.dc;
  p.gpl = planes.p; p.gpl_stride = planes.stride;
  p.wide = aligned({a.v, a.c, a.dh_new, a.dc_new, a.zoneout_mask}, a.H, a.dtype);
  const int most = few && lstm_tc_takes(a.dtype, a.N, a.H, false) ? kLstmChainsBeforeTcBwd : kGridChains;
  return run_bwd(p, a.dtype, most, 4, a.db, nullptr, run_cl_bwd_lstm, run_gl_bwd_lstm, s);
}

int gru_backward_chain(const GruBwd& a, const GradPlanes& planes, bool few, cudaStream_t s) {
  if (recurrence_path() == HASTE_B200_PATH_STEPWISE) return HASTE_B200_ERR_UNSUPPORTED;
  ChainParams p{};
  p.T = a.T; p.N = a.N; p.H = a.H;
  p.has_zoneout = a.zoneout_mask ? 1 : 0; p.r_transposed = a.transposed_inputs;
  p.R = a.R; p.gin = a.v; p.dp = a.dp; p.dq = a.dq; p.h = const_cast<void*>(a.h); p.dh_new = a.dh_new;
  p.mask = a.zoneout_mask; p.dh = a.dh;
  p.gpl = planes.p; p.gpl2 = planes.p2; p.gpl_stride = planes.stride;
  p.wide = aligned({a.v, a.dp, a.dq, a.h, a.dh_new, a.zoneout_mask}, a.H, a.dtype);
  return run_bwd(p, a.dtype, few && tc_waits(a.dtype, a.N, a.H) ? kGruChainsBeforeTc : kGridChains,
                 3, a.dbx, a.dbr, run_cl_bwd_gru, run_gl_bwd_gru, s);
}

}  // namespace hb
