// Host side of the LayerNorm recurrence kernels (recurrent_ln_kernels.cuh) - tiling choice,
// exchange-buffer scratch and the entry points the cell drivers call - and the exchange probe.
#include <cstdio>
#include <cstdlib>

#include "recurrent_ln_kernels.cuh"

namespace hb {
namespace rec {


namespace {

constexpr int MAX_MT = 4;

// Picks the batch tiling: as many CTAs as fit on the GPU at once (one CTA per SM).
bool pick_geometry(int N, int H, Geometry* g) {
  const int nHS = ceil_div(H, U);
  const int sms = sm_count();
  for (int mt = 1; mt <= MAX_MT; ++mt) {
    const int nBS = ceil_div(N, 16 * mt);
    if ((long long)nHS * nBS <= sms) {
      g->nHS = nHS; g->nBS = nBS; g->MT = mt;
      return true;
    }
  }
  return false;
}

bool supported(int dtype, int N, int H, Geometry* g) {
  if (recurrence_path() == HASTE_B200_PATH_STEPWISE) return false;
  // R slice must fit the register file (two bf16 planes for fp32 and fp16 storage, one for bf16)
  if (dtype != HASTE_B200_BF16 && H > 512) return false;
  if (dtype == HASTE_B200_BF16 && H > 1024) return false;
  return pick_geometry(N, H, g);
}

// Timing-experiment builds only (-DHASTE_B200_TIMING_EXPERIMENTS): the environment variable
// HASTE_B200_TIMING_EXPERIMENT=<bits> switches parts of the persistent kernels off to attribute
// step time to them; results of such a run are wrong by construction and the library says so
// on stderr.  The shipped library reads no environment variable and compiles the switches out.
int debug_skip() {
#ifdef HASTE_B200_TIMING_EXPERIMENTS
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("HASTE_B200_TIMING_EXPERIMENT");
    v = e ? atoi(e) : 0;
    if (v != 0)
      fprintf(stderr, "haste_b200: HASTE_B200_TIMING_EXPERIMENT=%d - parts of the recurrence "
                      "kernels are switched off, results are wrong\n", v);
  }
  return v;
#else
  return 0;
#endif
}

// Zeroed scratch: abort flag followed by `words` exchange words.
int make_scratch(size_t words, Sync* sync, uint32_t** xwords, cudaStream_t s) {
  Arena ws;
  const size_t bytes = Arena::pad(4096) + Arena::pad(words * 4);
  HB_TRY(make_arena(&ws, s, bytes + 512, /*slot=*/2));
  int* flag = ws.take<int>(1024);
  uint32_t* x = ws.take<uint32_t>(words);
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

// The cluster kernels (rec_ln_cluster.cuh), where they take the shape.
int cluster_forward(LnFwdParams& p, int (*run)(const LnFwdParams&, cudaStream_t), cudaStream_t s) {
  if (recurrence_path() == HASTE_B200_PATH_STEPWISE) return HASTE_B200_ERR_UNSUPPORTED;
  p.sync.err = device_error_word();
  HB_REQUIRE(p.sync.err, "error word");
  return run(p, s);
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

int cluster_backward(LnBwdParams& p, int gates, int dtype, const LnGrads& out,
                     int (*run)(const LnBwdParams&, float*, int*, cudaStream_t), cudaStream_t s) {
  if (recurrence_path() == HASTE_B200_PATH_STEPWISE || p.H > 320) return HASTE_B200_ERR_UNSUPPORTED;
  p.sync.err = device_error_word();
  HB_REQUIRE(p.sync.err, "error word");
  const int H = p.H;
  const size_t tiles = ceil_div(p.N, 8);
  float* part = static_cast<float*>(workspace(s, tiles * 10 * H * sizeof(float), /*slot=*/2));
  if (!part) return HASTE_B200_ERR_CUDA;
  float* db_part = part + tiles * 6 * H;
  p.dgRh_part = part;
  p.dgh_part = part + tiles * 4 * H;
  p.dbh_part = part + tiles * 5 * H;
  int rows = 0;
  HB_TRY(run(p, db_part, &rows, s));
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

// ---- LayerNormLSTM (recurrent_ln_kernels.cuh) ------------------------------------------
// Forward: LN(x.W) is already in a.act_Wx_norm.  Four source slices per thread in the
// statistic exchange limit the kernels to 64 hidden slices, which `supported` guarantees.
int layer_norm_lstm_forward_persistent(const LnLstmFwd& a, cudaStream_t s) {
  const bool zo = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  LnFwdParams p{a.T, a.N, a.H, 0, 0, 0, a.training, zo ? 1 : 0, a.zoneout_prob, a.R, a.b,
                nullptr, a.act_Wx_norm, a.gamma_Rh, a.gamma_h, a.beta_h, a.act_Wx_norm, a.act_Rh, a.cache_Rh,
                a.act_c_norm, a.cache_c, a.h, a.c, a.zoneout_mask, nullptr, nullptr, Sync{}, debug_skip()};
  const int cl = cluster_forward(p, a.dtype == HASTE_B200_F32 ? run_ln_cl_fwd_f32 : run_ln_cl_fwd_bf16, s);
  if (cl != HASTE_B200_ERR_UNSUPPORTED) return cl;
  Geometry g;
  if (!supported(a.dtype, a.N, a.H, &g) || g.nHS > 64) return HASTE_B200_ERR_UNSUPPORTED;
  p.Hx = (a.H + 3) & ~3;
  p.nHS = g.nHS;
  p.MT = g.MT;
  const size_t xwords = (size_t)2 * a.N * p.Hx;
  const size_t swords = (size_t)2 * 2 * g.nBS * g.MT * 16 * g.nHS * 2;
  HB_TRY(make_scratch(xwords + swords + 64, &p.sync, &p.xbuf, s));
  p.sbuf = p.xbuf + ((xwords + 63) & ~size_t(63));
  return a.dtype == HASTE_B200_F32 ? run_ln_fwd_f32(p, g, s) : run_ln_fwd_bf16(p, g, s);
}

namespace {
LnBwdParams ln_lstm_params(const LnLstmBwd& a, float* dh_carry, float* dc_carry, const GradPlanes& planes) {
  return LnBwdParams{a.T, a.N, a.H, 0, 0, a.zoneout_mask ? 1 : 0, a.transposed_inputs, a.R,
                     a.gamma_Rh, a.gamma_h, a.c, nullptr, nullptr, nullptr, a.act_Wx_norm, a.act_Rh,
                     a.cache_Rh, a.act_c_norm,
                     a.cache_c, a.dh_new, a.dc_new, a.zoneout_mask, dh_carry, dc_carry, nullptr, nullptr, nullptr,
                     nullptr, nullptr, Sync{}, planes.p, planes.p2, planes.stride, debug_skip()};
}
}  // namespace

// The cluster kernels, up to 320 units: dh and dc come back complete, and the bias and LayerNorm
// gradients of h.R and c go into the caller's tensors (added or assigned).
int layer_norm_lstm_backward_cluster(const LnLstmBwd& a, float* dh_carry, float* dc_carry, cudaStream_t s) {
  LnBwdParams p = ln_lstm_params(a, dh_carry, dc_carry, GradPlanes{});
  return cluster_backward(p, 4, a.dtype, LnGrads{a.db, nullptr, a.dgamma_Rh, a.dgamma_h, a.dbeta_h},
                          a.dtype == HASTE_B200_F32 ? run_ln_cl_bwd_f32 : run_ln_cl_bwd_bf16, s);
}

// Backward.  `acc` holds fp32 accumulators [dgamma_Rh 4H | dgamma_h H | dbeta_h H] that the
// per-row-group partial sums of the kernel are added into (fixed order).  As for the plain
// LSTM, the recurrent contribution of step 0 to dh is added here by one small contraction.
int layer_norm_lstm_backward_persistent(const LnLstmBwd& a, float* dh_carry, float* dc_carry,
                                        float* acc, const GradPlanes& planes, cudaStream_t s) {
  const int H = a.H;
  LnBwdParams p = ln_lstm_params(a, dh_carry, dc_carry, planes);
  Geometry g;
  if (!supported(a.dtype, a.N, a.H, &g) || g.nHS > 64) return HASTE_B200_ERR_UNSUPPORTED;
  p.nHS = g.nHS;
  p.MT = g.MT;
  const size_t ewords = ((size_t)2 * g.nBS * g.nHS * g.nHS * g.MT * 16 * U + 63) & ~size_t(63);
  const size_t swords = ((size_t)2 * 2 * g.nBS * g.MT * 16 * g.nHS * 2 + 63) & ~size_t(63);
  const int prow = g.nBS * 16;
  const size_t pwords = (size_t)prow * 6 * H;
  const size_t cwords = colsum_scratch_floats(prow, 4 * H);
  HB_TRY(make_scratch(ewords + swords + pwords + cwords + 64, &p.sync, &p.exch, s));
  p.sbuf = p.exch + ewords;
  float* part = reinterpret_cast<float*>(p.sbuf + swords);
  float* cs = part + pwords;
  p.dgRh_part = part;
  p.dgh_part = part + (size_t)prow * 4 * H;
  p.dbh_part = part + (size_t)prow * 5 * H;
  int st_ = a.dtype == HASTE_B200_F32 ? run_ln_bwd_f32(p, g, s) : run_ln_bwd_bf16(p, g, s);
  if (st_ != HASTE_B200_OK) return st_;
  HB_TRY(colsum(HASTE_B200_F32, part, 4LL * H, prow, 4 * H, HASTE_B200_F32, acc, 1, cs, s));
  HB_TRY(colsum(HASTE_B200_F32, part + (size_t)prow * 4 * H, H, prow, H, HASTE_B200_F32,
                acc + 4 * H, 1, cs, s));
  HB_TRY(colsum(HASTE_B200_F32, part + (size_t)prow * 5 * H, H, prow, H, HASTE_B200_F32,
                acc + 5 * H, 1, cs, s));
  GemmDesc gd{a.dtype, HASTE_B200_F32, a.N, H, 4 * H, a.act_Rh, 4LL * H, 1, a.R,
              a.transposed_inputs ? H : 1, a.transposed_inputs ? 1 : 4LL * H, dh_carry, H, 1};
  gd.precise = 1;
  // (once per pass, not once per step: the CUDA-core kernel would take 92 us for 45 rows, H = 296)
  return gemm(gd, s);
}

// ---- LayerNormGRU (the G = 3 instantiation of the same kernels) ---------------------------
// Forward: LN(x.W) is already in a.tmp_Wx_norm.
int layer_norm_gru_forward_persistent(const LnGruFwd& a, cudaStream_t s) {
  const bool zo = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  LnFwdParams p{a.T, a.N, a.H, 0, 0, 0, a.training, zo ? 1 : 0, a.zoneout_prob, a.R, a.bx,
                a.br, a.tmp_Wx_norm, a.gamma_Rh, nullptr, nullptr, a.v, a.act_Rh, a.cache_Rh,
                nullptr, nullptr, a.h, nullptr, a.zoneout_mask, nullptr, nullptr, Sync{}};
  const int cl = cluster_forward(p, a.dtype == HASTE_B200_F32 ? run_lngru_cl_fwd_f32 : run_lngru_cl_fwd_bf16, s);
  if (cl != HASTE_B200_ERR_UNSUPPORTED) return cl;
  Geometry g;
  if (!supported(a.dtype, a.N, a.H, &g) || g.nHS > 64) return HASTE_B200_ERR_UNSUPPORTED;
  p.Hx = (a.H + 3) & ~3;
  p.nHS = g.nHS;
  p.MT = g.MT;
  const size_t xwords = (size_t)2 * a.N * p.Hx;
  const size_t swords = (size_t)2 * 2 * g.nBS * g.MT * 16 * g.nHS * 2;
  HB_TRY(make_scratch(xwords + swords + 64, &p.sync, &p.xbuf, s));
  p.sbuf = p.xbuf + ((xwords + 63) & ~size_t(63));
  return a.dtype == HASTE_B200_F32 ? run_lngru_fwd_f32(p, g, s) : run_lngru_fwd_bf16(p, g, s);
}

namespace {
LnBwdParams ln_gru_params(const LnGruBwd& a, float* dh_carry, const GradPlanes& planes) {
  return LnBwdParams{a.T, a.N, a.H, 0, 0, a.zoneout_mask ? 1 : 0, a.transposed_inputs, a.R,
                     a.gamma_Rh, nullptr, nullptr, a.h, a.dp, a.dq, const_cast<void*>(a.v), a.act_Rh,
                     a.cache_Rh, nullptr, nullptr, a.dh_new, nullptr, a.zoneout_mask, dh_carry, nullptr,
                     nullptr, nullptr, nullptr, nullptr, nullptr, Sync{}, planes.p, planes.p2, planes.stride};
}
}  // namespace

int layer_norm_gru_backward_cluster(const LnGruBwd& a, float* dh_carry, cudaStream_t s) {
  LnBwdParams p = ln_gru_params(a, dh_carry, GradPlanes{});
  return cluster_backward(p, 3, a.dtype, LnGrads{a.dbx, a.dbr, a.dgamma_Rh, nullptr, nullptr},
                          a.dtype == HASTE_B200_F32 ? run_lngru_cl_bwd_f32 : run_lngru_cl_bwd_bf16, s);
}

// Backward.  `acc` is the fp32 accumulator [3H] for dgamma_Rh.  a.act_Rh is overwritten with
// d(h.R); a.dp / a.dq receive the gradients w.r.t. the normalised projections (+ biases).
int layer_norm_gru_backward_persistent(const LnGruBwd& a, float* dh_carry, float* acc,
                                       const GradPlanes& planes, cudaStream_t s) {
  const int H = a.H;
  LnBwdParams p = ln_gru_params(a, dh_carry, planes);
  Geometry g;
  if (!supported(a.dtype, a.N, a.H, &g) || g.nHS > 64) return HASTE_B200_ERR_UNSUPPORTED;
  p.nHS = g.nHS;
  p.MT = g.MT;
  const size_t ewords = ((size_t)2 * g.nBS * g.nHS * g.nHS * g.MT * 16 * U + 63) & ~size_t(63);
  const size_t swords = ((size_t)2 * 2 * g.nBS * g.MT * 16 * g.nHS * 2 + 63) & ~size_t(63);
  const int prow = g.nBS * 16;
  const size_t pwords = (size_t)prow * 3 * H;
  const size_t cwords = colsum_scratch_floats(prow, 3 * H);
  HB_TRY(make_scratch(ewords + swords + pwords + cwords + 64, &p.sync, &p.exch, s));
  p.sbuf = p.exch + ewords;
  float* part = reinterpret_cast<float*>(p.sbuf + swords);
  float* cs = part + pwords;
  p.dgRh_part = part;
  int st_ = a.dtype == HASTE_B200_F32 ? run_lngru_bwd_f32(p, g, s) : run_lngru_bwd_bf16(p, g, s);
  if (st_ != HASTE_B200_OK) return st_;
  HB_TRY(colsum(HASTE_B200_F32, part, 3LL * H, prow, 3 * H, HASTE_B200_F32, acc, 1, cs, s));
  GemmDesc gd{a.dtype, HASTE_B200_F32, a.N, H, 3 * H, a.act_Rh, 3LL * H, 1, a.R,
              a.transposed_inputs ? H : 1, a.transposed_inputs ? 1 : 3LL * H, dh_carry, H, 1};
  gd.precise = 1;
  // (once per pass, not once per step: the CUDA-core kernel would take 92 us for 45 rows, H = 296)
  return gemm(gd, s);
}

}  // namespace hb
