// Host side of the LayerNorm recurrence kernels (rec_ln_cluster.cuh, rec_ln_grid.cuh) - tiling choice,
// exchange-buffer scratch and the entry points the cell drivers call - and the exchange probe.
#include <initializer_list>

#include "rec_ln_common.cuh"

namespace hb {
namespace rec {


namespace {

// The grid kernels' tiling: as many row groups as the SMs have room for, one CTA per SM, the rest of the rows
// as chains.  Under an SM budget (two directions side by side) within it first, where that pays (budget_pays).
constexpr int kLnGridChains = 8;

bool ln_grid_geometry(int dtype, int N, int H, bool bwd, LnGridGeometry* g) {
  // R's slice must fit the registers: two planes with fp32 storage, one with bf16
  if (H > (dtype == HASTE_B200_BF16 ? 1024 : 512)) return false;
  g->nHS = ceil_div(H, 16);
  const int tiles = ceil_div(N, 8), sms = sm_count(), budget = sm_budget();
  auto within = [&](int use, LnGridGeometry* g) {
    if (use < g->nHS) return false;
    g->nRG = min(tiles, use / g->nHS);
    g->CH = ceil_div(tiles, g->nRG);
    g->nRG = ceil_div(tiles, g->CH);
    return g->CH <= kLnGridChains;
  };
  LnGridGeometry whole = *g;
  const bool fits = within(sms, &whole);
  if (budget <= sms && within(budget, g) && (!fits || budget_pays(bwd, budget, g->CH, whole.CH))) return true;
  *g = whole;
  return fits;
}
// Whole-quad accesses: every row of every array starts on a multiple of four elements.
int wide_rows(std::initializer_list<const void*> ptrs, int H, int dtype) {
  uintptr_t a = 0;
  for (const void* q : ptrs) a |= reinterpret_cast<uintptr_t>(q);
  return H % 4 == 0 && a % (4 * dtype_size(dtype)) == 0;
}

// Zeroed scratch: abort flag followed by `words` exchange words; then `floats` that need no zeroing.
int make_scratch(size_t words, Sync* sync, uint32_t** xwords, cudaStream_t s, size_t floats = 0) {
  Arena ws;
  const size_t bytes = Arena::pad(4096) + Arena::pad(words * 4);
  HB_TRY(make_arena(&ws, s, bytes + floats * 4 + 512, /*slot=*/2));
  int* flag = ws.take<int>(1024);
  uint32_t* x = ws.take<uint32_t>(words + floats);
  HB_REQUIRE(flag && x, "scratch arena");
  HB_CUDA_OK(cudaMemsetAsync(flag, 0, bytes, s));
  sync->abort_flag = flag;
  sync->err = device_error_word();
  HB_REQUIRE(sync->err, "error word");
  *xwords = x;
  return HASTE_B200_OK;
}

}  // namespace
}  // namespace rec

// ---- exchange-only probe ---------------------------------------------------------------
// The hand-off of the forward recurrence with everything else taken out: per step every CTA
// publishes its 16 x 16 tagged words and every warp waits for its K range of all rows, then
// the CTA meets at its barrier.  No contraction, no gate math, no activation traffic.  Its
// time per step is the part of a recurrence step that no amount of arithmetic tuning removes
// (store -> L2 -> polling load, plus the CTA barrier); benchmarks quote it beside the measured
// step time.  No reference counterpart.
namespace rec {
namespace {

template <int KSW>
__global__ void __launch_bounds__(THREADS, 1)
exchange_probe_kernel(int T, int N, int Hx, int nHS, uint32_t* xbuf, Sync sync) {
  constexpr int KW = KSW * 16, CPR = KW / 4, CPL = 16 * CPR / 32;
  __shared__ int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hs = blockIdx.x % nHS, bs = blockIdx.x / nHS;
  const int nl = tid >> 4, ul = tid & 15;
  const int u0 = hs * U, n0 = bs * 16;
  if (tid == 0) s_abort = 0;
  __syncthreads();
  float carry = 0.f;
  for (int t = 0; t < T; ++t) {
    const uint32_t tag = (((uint32_t)t >> 1) & 1u) ^ 1u;
    const int n = n0 + nl;
    if (n < N && u0 + ul < Hx)
      publish_u32(xbuf + (size_t)(t & 1) * N * Hx + (size_t)n * Hx + u0 + ul,
                  xword_encode(carry * 0.5f + 0.25f, tag));
    const uint32_t wtag = tag << 30;
    const uint32_t* xsrc = xbuf + (size_t)(t & 1) * N * Hx;
    uint4 w[CPL];
    const long long t0 = clock64();
    unsigned int spins = 0;
    bool alive = true;
    for (;;) {
#pragma unroll
      for (int i = 0; i < CPL; ++i) {
        const int e = lane + i * 32;
        const int r = e / CPR, k = warp * KW + (e % CPR) * 4;
        if (n0 + r < N && k < Hx) w[i] = ld_relaxed_u32x4(xsrc + (size_t)(n0 + r) * Hx + k);
        else w[i] = make_uint4(wtag, wtag, wtag, wtag);
      }
      uint32_t bad = 0;
#pragma unroll
      for (int i = 0; i < CPL; ++i)
        bad |= (w[i].x ^ wtag) | (w[i].y ^ wtag) | (w[i].z ^ wtag) | (w[i].w ^ wtag);
      if (__all_sync(0xffffffffu, (bad & 0x40000000u) == 0)) break;
      if ((++spins & 63u) == 0) {
        bool stop = *reinterpret_cast<volatile int*>(sync.abort_flag) != 0;
        if (!stop && clock64() - t0 > SPIN_LIMIT_CYCLES) {
          raise_abort(sync, &s_abort, 46, blockIdx.x, t);
          stop = true;
        }
        if (__any_sync(0xffffffffu, stop)) { alive = false; break; }
      }
    }
    if (!alive) *reinterpret_cast<volatile int*>(&s_abort) = 1;
    carry = xword_value(w[0].x);  // the next word depends on a received one, as h does
    if (__syncthreads_or(*reinterpret_cast<volatile int*>(&s_abort))) break;
  }
}

}  // namespace
}  // namespace rec

// Runs the probe for `steps` steps with the tiling the recurrence would use for (N, H) and
// returns the device time per step in microseconds.
int exchange_probe(int N, int H, int steps, float* us_per_step, cudaStream_t s) {
  using namespace rec;
  HB_REQUIRE(N > 0 && H > 0 && steps > 0 && us_per_step, "arguments");
  const int nHS = ceil_div(H, U), nBS = ceil_div(N, 16);
  HB_REQUIRE((long long)nHS * nBS <= sm_count(), "does not fit one CTA per SM");
  const int Hx = nHS * U;
  const int ksw = ceil_div(nHS, WARPS);
  HB_REQUIRE(ksw <= 8, "H too large for the probe");
  Sync sync;
  uint32_t* xbuf = nullptr;
  HB_TRY(make_scratch((size_t)2 * N * Hx, &sync, &xbuf, s));
  cudaEvent_t e0, e1;
  HB_CUDA_OK(cudaEventCreate(&e0));
  HB_CUDA_OK(cudaEventCreate(&e1));
  int T = steps, Nn = N, Hxx = Hx, nhs = nHS;
  void* args[] = {&T, &Nn, &Hxx, &nhs, &xbuf, &sync};
  const void* fn = ksw <= 1   ? (const void*)exchange_probe_kernel<1>
                   : ksw <= 2 ? (const void*)exchange_probe_kernel<2>
                   : ksw <= 4 ? (const void*)exchange_probe_kernel<4>
                              : (const void*)exchange_probe_kernel<8>;
  HB_CUDA_OK(cudaEventRecord(e0, s));
  cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(nHS * nBS), dim3(THREADS), args, 0, s);
  if (e != cudaSuccess) {
    set_last_error("cooperative launch failed: %s", cudaGetErrorString(e));
    cudaGetLastError();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return HASTE_B200_ERR_CUDA;
  }
  count_launch(1);
  HB_CUDA_OK(cudaEventRecord(e1, s));
  HB_CUDA_OK(cudaEventSynchronize(e1));
  float ms = 0.f;
  HB_CUDA_OK(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *us_per_step = ms * 1e3f / steps;
  return HASTE_B200_OK;
}

using namespace rec;

namespace {

typedef int (*ClFwd)(const LnFwdParams&, cudaStream_t);
typedef int (*GridFwd)(const LnFwdParams&, const LnGridGeometry&, int, cudaStream_t);
typedef int (*ClBwd)(const LnBwdParams&, float*, int*, cudaStream_t);
typedef int (*GridBwd)(const LnBwdParams&, float*, const LnGridGeometry&, int, cudaStream_t);

// The cluster kernels where they take the shape, else the grid kernels.
int run_forward(LnFwdParams& p, int dtype, int wide, ClFwd cluster, GridFwd grid, cudaStream_t s) {
  if (recurrence_path() == HASTE_B200_PATH_STEPWISE) return HASTE_B200_ERR_UNSUPPORTED;
  p.sync.err = device_error_word();
  HB_REQUIRE(p.sync.err, "error word");
  const int cl = cluster(p, s);
  if (cl != HASTE_B200_ERR_UNSUPPORTED) return cl;
  LnGridGeometry g;
  if (!ln_grid_geometry(dtype, p.N, p.H, false, &g)) return HASTE_B200_ERR_UNSUPPORTED;
  const size_t tiles = ceil_div(p.N, 8), xwords = 2 * tiles * g.nHS * 128, swords = 4 * tiles * g.nHS * 16;
  HB_TRY(make_scratch(xwords + swords, &p.sync, &p.xbuf, s));
  p.sbuf = p.xbuf + xwords;
  return grid(p, g, wide, s);
}
// Sums of the row groups' partial parameter gradients, into the caller's tensors: bias (as
// bias_grad_finish), gains of h.R and, LSTM, gain and offset of the cell state.
struct LnGrads {
  void *db, *db2, *dgRh, *dgh, *dbh;
};
template <typename T>
__global__ void ln_grad_finish(int G, const float* db_part, const float* dgRh_part, const float* dgh_part,
                               const float* dbh_part, int rows, int H, LnGrads out, int accumulate) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  const float* part = nullptr;
  int width = 0;
  T *d = nullptr, *d2 = nullptr;
  if (j < 4 * H) {
    part = db_part; width = 4 * H;
    if (G == 4 || j < 3 * H) d = static_cast<T*>(out.db) + j;
    if (G == 3 && (j < 2 * H || j >= 3 * H)) d2 = static_cast<T*>(out.db2) + (j < 2 * H ? j : j - H);
  } else if ((j -= 4 * H) < G * H) {
    part = dgRh_part; width = G * H;
    d = static_cast<T*>(out.dgRh) + j;
  } else if (G == 4 && (j -= G * H) < 2 * H) {
    part = j < H ? dgh_part : dbh_part; width = H;
    d = static_cast<T*>(j < H ? out.dgh : out.dbh);
    j = j < H ? j : j - H;
    d += j;
  } else {
    return;
  }
  float s = 0.f;
  for (int r = 0; r < rows; ++r) s += part[(long long)r * width + j];
  if (d) st(d, accumulate ? s + ld(d) : s);
  if (d2) st(d2, accumulate ? s + ld(d2) : s);
}

int run_backward(LnBwdParams& p, int gates, int dtype, int wide, const LnGrads& out, ClBwd cluster, GridBwd grid,
                 cudaStream_t s) {
  if (recurrence_path() == HASTE_B200_PATH_STEPWISE) return HASTE_B200_ERR_UNSUPPORTED;
  p.sync.err = device_error_word();
  HB_REQUIRE(p.sync.err, "error word");
  const int H = p.H;
  const size_t tiles = ceil_div(p.N, 8);
  // partial parameter gradients: rows x (gains of h.R, gain and offset of c, gates)
  float* db_part = nullptr;
  auto partials = [&](float* part, size_t rows) {
    p.dgRh_part = part;
    p.dgh_part = part + rows * 4 * H;
    p.dbh_part = part + rows * 5 * H;
    db_part = part + rows * 6 * H;
  };
  int rows = 0, st_ = HASTE_B200_ERR_UNSUPPORTED;
  if (H <= 320) {
    float* part = static_cast<float*>(workspace(s, tiles * 10 * H * sizeof(float), /*slot=*/2));
    if (!part) return HASTE_B200_ERR_CUDA;
    partials(part, tiles);
    st_ = cluster(p, db_part, &rows, s);
  }
  if (st_ == HASTE_B200_ERR_UNSUPPORTED) {
    LnGridGeometry g;
    if (!ln_grid_geometry(dtype, p.N, H, true, &g)) return HASTE_B200_ERR_UNSUPPORTED;
    rows = 2 * g.nRG;
    const size_t xwords = 2 * tiles * g.nHS * g.nHS * 128, swords = 4 * tiles * g.nHS * 16;
    HB_TRY(make_scratch(xwords + swords, &p.sync, &p.exch, s, (size_t)rows * 10 * H));
    p.sbuf = p.exch + xwords;
    partials(reinterpret_cast<float*>(p.sbuf + swords), rows);
    st_ = grid(p, db_part, g, wide, s);
  }
  if (st_ != HASTE_B200_OK) return st_;
  const int blocks = ceil_div((gates == 4 ? 10LL : 7LL) * H, 128), add = assign_gradients() ? 0 : 1;
  if (dtype == HASTE_B200_F32)
    ln_grad_finish<float><<<blocks, 128, 0, s>>>(gates, db_part, p.dgRh_part, p.dgh_part, p.dbh_part, rows, H, out, add);
  else
    ln_grad_finish<__nv_bfloat16><<<blocks, 128, 0, s>>>(gates, db_part, p.dgRh_part, p.dgh_part, p.dbh_part, rows, H,
                                                         out, add);
  HB_LAUNCH_OK();
  count_launch(1);
  return HASTE_B200_OK;
}

}  // namespace

// ---- LayerNormLSTM: LN(x.W) is already in a.act_Wx_norm ---------------------------------
int layer_norm_lstm_forward_persistent(const LnLstmFwd& a, cudaStream_t s) {
  const bool zo = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  LnFwdParams p{a.T, a.N, a.H, a.training, zo ? 1 : 0, a.zoneout_prob, a.R, a.b, nullptr, a.act_Wx_norm, a.gamma_Rh,
                a.gamma_h, a.beta_h, a.act_Wx_norm, a.act_Rh, a.cache_Rh, a.act_c_norm, a.cache_c, a.h, a.c,
                a.zoneout_mask, nullptr, nullptr, Sync{}};
  const int wide = wide_rows({a.act_Wx_norm, a.act_Rh, a.act_c_norm, a.h, a.c, a.zoneout_mask}, a.H, a.dtype);
  return a.dtype == HASTE_B200_F32 ? run_forward(p, a.dtype, wide, run_ln_cl_fwd_f32, run_ln_grid_fwd_f32, s)
                                   : run_forward(p, a.dtype, wide, run_ln_cl_fwd_bf16, run_ln_grid_fwd_bf16, s);
}

// dh and dc come back complete, and the bias and LayerNorm gradients of h.R and c go into the caller's
// tensors (added or assigned).
int layer_norm_lstm_backward_persistent(const LnLstmBwd& a, float* dh_carry, float* dc_carry, cudaStream_t s) {
  LnBwdParams p{a.T, a.N, a.H, a.zoneout_mask ? 1 : 0, a.transposed_inputs, a.R, a.gamma_Rh, a.gamma_h, a.c, nullptr,
                nullptr, nullptr, a.act_Wx_norm, a.act_Rh, a.cache_Rh, a.act_c_norm, a.cache_c, a.dh_new, a.dc_new,
                a.zoneout_mask, dh_carry, dc_carry, nullptr, nullptr, nullptr, nullptr, nullptr, Sync{}};
  const LnGrads out{a.db, nullptr, a.dgamma_Rh, a.dgamma_h, a.dbeta_h};
  const int wide = wide_rows({a.act_Wx_norm, a.act_Rh, a.act_c_norm, a.c, a.dh_new, a.dc_new, a.zoneout_mask}, a.H, a.dtype);
  return a.dtype == HASTE_B200_F32 ? run_backward(p, 4, a.dtype, wide, out, run_ln_cl_bwd_f32, run_ln_grid_bwd_f32, s)
                                   : run_backward(p, 4, a.dtype, wide, out, run_ln_cl_bwd_bf16, run_ln_grid_bwd_bf16, s);
}

// ---- LayerNormGRU (the G = 3 instantiations): LN(x.W) is already in a.tmp_Wx_norm --------
int layer_norm_gru_forward_persistent(const LnGruFwd& a, cudaStream_t s) {
  const bool zo = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  LnFwdParams p{a.T, a.N, a.H, a.training, zo ? 1 : 0, a.zoneout_prob, a.R, a.bx, a.br, a.tmp_Wx_norm, a.gamma_Rh,
                nullptr, nullptr, a.v, a.act_Rh, a.cache_Rh, nullptr, nullptr, a.h, nullptr, a.zoneout_mask, nullptr,
                nullptr, Sync{}};
  const int wide = wide_rows({a.tmp_Wx_norm, a.v, a.act_Rh, a.h, a.zoneout_mask}, a.H, a.dtype);
  return a.dtype == HASTE_B200_F32 ? run_forward(p, a.dtype, wide, run_lngru_cl_fwd_f32, run_lngru_grid_fwd_f32, s)
                                   : run_forward(p, a.dtype, wide, run_lngru_cl_fwd_bf16, run_lngru_grid_fwd_bf16, s);
}

// a.act_Rh is overwritten with d(h.R); a.dp / a.dq receive the gradients w.r.t. the normalised projections
// (+ biases).
int layer_norm_gru_backward_persistent(const LnGruBwd& a, float* dh_carry, cudaStream_t s) {
  LnBwdParams p{a.T, a.N, a.H, a.zoneout_mask ? 1 : 0, a.transposed_inputs, a.R, a.gamma_Rh, nullptr, nullptr, a.h,
                a.dp, a.dq, const_cast<void*>(a.v), a.act_Rh, a.cache_Rh, nullptr, nullptr, a.dh_new, nullptr,
                a.zoneout_mask, dh_carry, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, Sync{}};
  const LnGrads out{a.dbx, a.dbr, a.dgamma_Rh, nullptr, nullptr};
  const int wide = wide_rows({a.v, a.act_Rh, a.h, a.dp, a.dq, a.dh_new, a.zoneout_mask}, a.H, a.dtype);
  return a.dtype == HASTE_B200_F32
             ? run_backward(p, 3, a.dtype, wide, out, run_lngru_cl_bwd_f32, run_lngru_grid_bwd_f32, s)
             : run_backward(p, 3, a.dtype, wide, out, run_lngru_cl_bwd_bf16, run_lngru_grid_bwd_bf16, s);
}

}  // namespace hb
