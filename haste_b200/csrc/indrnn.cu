// IndRNN and LayerNormIndRNN: h_t = tanh(Wx_t + u * h_{t-1} + b), with zoneout.
//
// The recurrence is elementwise, so one thread owns one (batch, unit) pair for
// all T steps and the kernels are pure HBM streams; loads that do not depend on
// the carried state are issued several steps ahead.  The parameter gradients
// du/db are per-thread sums reduced over the batch by a deterministic column sum.
// Math follows lib/indrnn_forward_gpu.cu.cc:25-63 and
// lib/indrnn_backward_gpu.cu.cc:25-74 (LayerNorm variant:
// lib/layer_norm_indrnn_{forward,backward}_gpu.cu.cc).
#include "cells.cuh"

namespace hb {
namespace {

constexpr int AHEAD = 8;  // steps whose inputs are loaded together

// Piped: a group's loads are issued before the group in front of it is computed.  With few (batch,
// unit) pairs the GPU has too little in flight to hide a group's latency behind other threads, and
// the scan took T / 8 latencies; with many, the registers cost more threads than that wins (ScanShape).
template <typename T, bool Training, bool Zoneout, bool Piped>
__global__ void __launch_bounds__(128) indrnn_scan_fwd(int T_, long long NH, int H, const T* __restrict__ Wx,
                                const T* __restrict__ u, const T* __restrict__ b,
                                T* __restrict__ h, float zoneout_prob,
                                const T* __restrict__ mask) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= NH) return;
  const int j = (int)(idx % H);
  const float uj = ld(u + j), bj = ld(b + j);
  float hp = ld(h + idx);
  float wx[AHEAD], m[AHEAD];
  auto load = [&](int t0, float (&x)[AHEAD], float (&z)[AHEAD]) {
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      const int t = t0 + k;
      x[k] = (t < T_) ? ld(Wx + t * NH + idx) : 0.f;
      z[k] = (Zoneout && Training && t < T_) ? ld(mask + t * NH + idx) : 0.f;
    }
  };
  if (Piped) load(0, wx, m);
  for (int t0 = 0; t0 < T_; t0 += AHEAD) {
    float wn[AHEAD], mn[AHEAD];
    if (Piped) load(t0 + AHEAD, wn, mn);
    else load(t0, wx, m);
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      const int t = t0 + k;
      if (t < T_) {
        float hn = tanhf(wx[k] + uj * hp + bj);
        if (Zoneout) hn = zoneout<Training>(hn, hp, zoneout_prob, m[k]);
        st(h + (t + 1) * NH + idx, hn);
        hp = hn;  // the carried state stays fp32 whatever the storage type
      }
    }
    if (Piped) {
#pragma unroll
      for (int k = 0; k < AHEAD; ++k) {
        wx[k] = wn[k];
        m[k] = mn[k];
      }
    }
  }
}

// Planes: dk is written as two bf16 planes (hi, lo; `dk_planes`, the lo plane `plane_stride`
// elements later) - the form the two contractions that read it take their fp32 operands in, so
// that neither splits it again.  dk_out: null if nothing reads the fp32 values.
template <typename T, bool Zoneout, bool Planes, bool Piped>
__global__ void __launch_bounds__(128) indrnn_scan_bwd(int T_, long long NH, int H, const T* __restrict__ u,
                                const T* __restrict__ h, const T* __restrict__ dh_new,
                                float* __restrict__ du_part, float* __restrict__ db_part,
                                float* __restrict__ dh_carry, T* __restrict__ dk_out,
                                const T* __restrict__ mask,
                                __nv_bfloat16* __restrict__ dk_planes, long long plane_stride) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= NH) return;
  const int j = (int)(idx % H);
  const float uj = ld(u + j);
  float carry = dh_carry[idx];
  float du = 0.f, db = 0.f;
  float hn = ld(h + (long long)T_ * NH + idx);  // h after the step at hand
  float hv[AHEAD], dn[AHEAD], m[AHEAD];
  auto load = [&](int t0, float (&hp)[AHEAD], float (&d)[AHEAD], float (&z)[AHEAD]) {
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      const int t = t0 - k;
      const bool ok = t >= 0;
      hp[k] = ok ? ld(h + t * NH + idx) : 0.f;
      d[k] = ok ? ld(dh_new + (t + 1) * NH + idx) : 0.f;
      z[k] = (Zoneout && ok) ? ld(mask + t * NH + idx) : 0.f;
    }
  };
  if (Piped) load(T_ - 1, hv, dn, m);
  for (int t0 = T_ - 1; t0 >= 0; t0 -= AHEAD) {
    float hx[AHEAD], dx[AHEAD], mx[AHEAD];
    if (Piped) load(t0 - AHEAD, hx, dx, mx);
    else load(t0, hv, dn, m);
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) {
      const int t = t0 - k;
      if (t >= 0) {
        float dh_total = dn[k] + carry;
        float keep = 0.f;
        if (Zoneout) {
          keep = (1.0f - m[k]) * dh_total;
          dh_total = m[k] * dh_total;
        }
        const float dk = d_tanh(hn) * dh_total;
        if (!Planes || dk_out) st(dk_out + t * NH + idx, dk);
        if (Planes) {
          const __nv_bfloat16 hi = __float2bfloat16_rn(dk);
          dk_planes[t * NH + idx] = hi;
          dk_planes[plane_stride + t * NH + idx] = __float2bfloat16_rn(dk - __bfloat162float(hi));
        }
        carry = keep + uj * dk;
        du += hv[k] * dk;
        db += dk;
        hn = hv[k];
      }
    }
    if (Piped) {
#pragma unroll
      for (int k = 0; k < AHEAD; ++k) {
        hv[k] = hx[k];
        dn[k] = dx[k];
        m[k] = mx[k];
      }
    }
  }
  dh_carry[idx] = carry;
  du_part[idx] = du;
  db_part[idx] = db;
}

// The piped form runs while the pairs fit in a quarter of the 2048 threads that an SM holds.  400 steps
// with zoneout, us forward / backward, plain -> piped: 8 192 pairs 51 / 45 -> 41 / 41; 32 768 72 / 72 ->
// 56 / 60; 75 776, where the line lies on 148 SMs, 88 / 94 -> 78 / 87; 98 304 99 / 111 -> 93 / 123.
// (Blocks of 32 threads, to spread few pairs over more SMs, measured the same as 128 everywhere.)
struct ScanShape {
  int blocks, threads = 128;
  bool piped;
  explicit ScanShape(long long NH) : blocks(ceil_div(NH, 128)), piped(NH <= 512LL * sm_count()) {}
};

template <typename T, bool Piped>
int scan_fwd_p(const IndrnnFwd& a, const void* Wx, const ScanShape& sc, cudaStream_t s) {
  const long long NH = (long long)a.N * a.H;
  const T* mask = (const T*)a.zoneout_mask;
  const bool zo = a.zoneout_prob != 0.0f && mask != nullptr;
#define HB_ARGS a.T, NH, a.H, (const T*)Wx, (const T*)a.u, (const T*)a.b, (T*)a.h, \
                a.zoneout_prob, zo ? mask : nullptr
  if (a.training) {
    if (zo) indrnn_scan_fwd<T, true, true, Piped><<<sc.blocks, sc.threads, 0, s>>>(HB_ARGS);
    else    indrnn_scan_fwd<T, true, false, Piped><<<sc.blocks, sc.threads, 0, s>>>(HB_ARGS);
  } else {
    if (zo) indrnn_scan_fwd<T, false, true, Piped><<<sc.blocks, sc.threads, 0, s>>>(HB_ARGS);
    else    indrnn_scan_fwd<T, false, false, Piped><<<sc.blocks, sc.threads, 0, s>>>(HB_ARGS);
  }
#undef HB_ARGS
  HB_LAUNCH_OK();
  count_launch(1);
  return HASTE_B200_OK;
}
template <typename T>
int scan_fwd(const IndrnnFwd& a, const void* Wx, cudaStream_t s) {
  const ScanShape sc((long long)a.N * a.H);
  return sc.piped ? scan_fwd_p<T, true>(a, Wx, sc, s) : scan_fwd_p<T, false>(a, Wx, sc, s);
}

template <typename T, bool Piped>
int scan_bwd_p(const IndrnnBwd& a, float* du_part, float* db_part, float* dh_carry, void* dk,
               __nv_bfloat16* planes, long long plane_stride, const ScanShape& sc, cudaStream_t s) {
  const long long NH = (long long)a.N * a.H;
#define HB_ARGS a.T, NH, a.H, (const T*)a.u, (const T*)a.h, (const T*)a.dh_new, du_part, db_part, \
                dh_carry, (T*)dk, (const T*)a.zoneout_mask, planes, plane_stride
  if (planes) {
    if (a.zoneout_mask) indrnn_scan_bwd<T, true, true, Piped><<<sc.blocks, sc.threads, 0, s>>>(HB_ARGS);
    else                indrnn_scan_bwd<T, false, true, Piped><<<sc.blocks, sc.threads, 0, s>>>(HB_ARGS);
  } else {
    if (a.zoneout_mask) indrnn_scan_bwd<T, true, false, Piped><<<sc.blocks, sc.threads, 0, s>>>(HB_ARGS);
    else                indrnn_scan_bwd<T, false, false, Piped><<<sc.blocks, sc.threads, 0, s>>>(HB_ARGS);
  }
#undef HB_ARGS
  HB_LAUNCH_OK();
  count_launch(1);
  return HASTE_B200_OK;
}
template <typename T>
int scan_bwd(const IndrnnBwd& a, float* du_part, float* db_part, float* dh_carry, void* dk,
             __nv_bfloat16* planes, long long plane_stride, cudaStream_t s) {
  const ScanShape sc((long long)a.N * a.H);
  return sc.piped ? scan_bwd_p<T, true>(a, du_part, db_part, dh_carry, dk, planes, plane_stride, sc, s)
                  : scan_bwd_p<T, false>(a, du_part, db_part, dh_carry, dk, planes, plane_stride, sc, s);
}

}  // namespace

int indrnn_forward(const IndrnnFwd& a, cudaStream_t s) {
  HB_REQUIRE(a.dtype == HASTE_B200_F32 || a.dtype == HASTE_B200_BF16, "dtype");
  HB_REQUIRE(a.T >= 0 && a.N > 0 && a.C > 0 && a.H > 0, "T,N,C,H");
  HB_REQUIRE(a.W && a.u && a.b && a.h && a.workspace, "null pointer");
  HB_REQUIRE(!a.gamma || (a.act_Wx && a.cache_Wx), "act_Wx/cache_Wx required with gamma");
  if (a.T == 0) return HASTE_B200_OK;
  HB_REQUIRE(a.x, "x is null");
  const long long TN = (long long)a.T * a.N;
  HB_REQUIRE(TN < (1LL << 31), "T*N too large");
  void* proj = a.gamma ? a.act_Wx : a.workspace;
  GemmDesc g{a.dtype, a.dtype, (int)TN, a.H, a.C, a.x, a.C, 1, a.W, a.H, 1, proj, a.H, 0};
  // The projection feeds a recurrence whose gain u * (1 - h^2) is close to one for u near 1:
  // an error of x.W is carried along the whole sequence and on through the layers of a stack
  // (measured: two-plane products leave 1.6e-4 on the output of six layers, three planes
  // 1.5e-5), so the forward projection always uses the fp32-accurate product.
  g.precise = 1;
  {
    ProfScope p(PH_PROJ, s);
    HB_TRY(gemm(g, s));
  }
  if (a.gamma) {
    ProfScope p(PH_OTHER, s);
    HB_TRY(layer_norm_forward(a.dtype, (int)TN, a.H, a.gamma, nullptr, a.act_Wx, a.workspace,
                              a.cache_Wx, s));
  }
  ProfScope p(PH_REC_FWD, s);
  if (a.dtype == HASTE_B200_F32) return scan_fwd<float>(a, a.workspace, s);
  return scan_fwd<__nv_bfloat16>(a, a.workspace, s);
}

int indrnn_backward(const IndrnnBwd& a, cudaStream_t s) {
  HB_REQUIRE(a.dtype == HASTE_B200_F32 || a.dtype == HASTE_B200_BF16, "dtype");
  HB_REQUIRE(a.T >= 0 && a.N > 0 && a.C > 0 && a.H > 0, "T,N,C,H");
  HB_REQUIRE(a.W && a.u && a.h && a.dh_new && a.dW && a.du && a.db && a.dh && a.workspace,
             "null pointer");
  HB_REQUIRE(!a.gamma || (a.dgamma && a.act_Wx && a.cache_Wx), "LayerNorm buffers");
  const int N = a.N, H = a.H, C = a.C;
  const long long TN = (long long)a.T * N;
  HB_REQUIRE(TN < (1LL << 31), "T*N too large");
  if (a.T == 0) return HASTE_B200_OK;
  HB_REQUIRE(a.x, "x is null");
  const int add = assign_gradients() ? 0 : 1;
  const size_t NH = (size_t)N * H;
  const size_t csf = colsum_scratch_floats(N, H);
  const size_t lnf = a.gamma ? layer_norm_backward_scratch_floats((int)TN, H) : 0;
  Arena ws;
  HB_TRY(make_arena(&ws, s, 3 * Arena::pad(NH * 4) + Arena::pad(csf * 4) + Arena::pad(lnf * 4) + 1024));
  float* dh_carry = ws.take<float>(NH);
  float* du_part = ws.take<float>(NH);
  float* db_part = ws.take<float>(NH);
  float* cs = ws.take<float>(csf);
  float* lns = ws.take<float>(lnf);
  HB_REQUIRE(dh_carry && du_part && db_part && cs && (lns || !lnf), "scratch arena");
  if (add) HB_TRY(to_float(a.dtype, a.dh, dh_carry, NH, s));
  else HB_CUDA_OK(cudaMemsetAsync(dh_carry, 0, NH * 4, s));
  // fp32: dk = d/d(x.W) is read by both contractions below as two bf16 planes.  Without
  // LayerNorm the scan writes them next to the fp32 values; with LayerNorm its backward pass
  // does.  (Grow-only library scratch; without it the contractions split for themselves.)
  __nv_bfloat16* planes = nullptr;
  long long plane_stride = 0;
  if (a.dtype == HASTE_B200_F32 && (H % 8) == 0) {
    const size_t pe = Arena::pad((size_t)TN * H * 2) / 2;  // elements per plane
    planes = static_cast<__nv_bfloat16*>(workspace(s, 2 * pe * 2 + 256, /*slot=*/3));
    plane_stride = (long long)pe;
  }
  const bool tr = a.transposed_inputs != 0;
  // dW[C,H] = x^T . dk   (assigned, as in the reference)
  GemmDesc gw{a.dtype, a.dtype, C, H, (int)TN, a.x, tr ? TN : 1, tr ? 1 : C, a.workspace, H, 1,
              a.dW, H, 0};
  // the backward contractions feed no recurrence: the three-product form is enough also for
  // the LayerNorm variant (six products measured the same 2.6e-5 on a six-layer stack)
  if (planes) { gw.b_pl = planes; gw.b_pl_ld = H; gw.b_pl_stride = plane_stride; }
  GemmDesc gx{a.dtype, a.dtype, (int)TN, C, H, a.workspace, H, 1, a.W, tr ? C : 1, tr ? 1 : H,
              a.dx, C, 0};
  if (planes) { gx.a_pl = planes; gx.a_pl_ld = H; gx.a_pl_stride = plane_stride; }
  // The fp32 values then go nowhere, unless LayerNorm works on them or a contraction is one for
  // the CUDA cores: a fifth of the scan's traffic.
  void* dk = a.workspace;
  if (planes && !a.gamma && gemm_reads_planes(gw) && (!a.dx || gemm_reads_planes(gx))) {
    dk = nullptr;
    gw.b = nullptr;
    gx.a = nullptr;
  }
  {
    ProfScope p(PH_REC_BWD, s);
    __nv_bfloat16* sp = a.gamma ? nullptr : planes;
    if (a.dtype == HASTE_B200_F32) HB_TRY(scan_bwd<float>(a, du_part, db_part, dh_carry, dk, sp, plane_stride, s));
    else HB_TRY(scan_bwd<__nv_bfloat16>(a, du_part, db_part, dh_carry, dk, nullptr, 0, s));
  }
  HB_TRY(from_float(a.dtype, dh_carry, a.dh, NH, s));
  HB_TRY(colsum(HASTE_B200_F32, du_part, H, N, H, a.dtype, a.du, add, cs, s));
  HB_TRY(colsum(HASTE_B200_F32, db_part, H, N, H, a.dtype, a.db, add, cs, s));
  if (a.gamma) {
    ProfScope p(PH_OTHER, s);
    if (!add) HB_CUDA_OK(cudaMemsetAsync(a.dgamma, 0, (size_t)H * dtype_size(a.dtype), s));
    // workspace holds dk = d/d(LN(x.W)); turn it into d/d(x.W) in place.
    HB_TRY(layer_norm_backward(a.dtype, (int)TN, H, a.gamma, a.act_Wx, a.workspace, a.workspace,
                               a.dtype, a.dgamma, nullptr, a.cache_Wx, lns, s, planes,
                               plane_stride));
  }
  {
    ProfScope p(PH_WGRAD, s);
    HB_TRY(gemm(gw, s));
  }
  if (!a.dx) return HASTE_B200_OK;
  {
    ProfScope p(PH_DGRAD, s);
    HB_TRY(gemm(gx, s));
  }
  return HASTE_B200_OK;
}

}  // namespace hb
