// LayerNormLSTM / LayerNormGRU recurrences on thread-block clusters, sm_100a: up to 320 units.
//
// A LayerNorm step is a chain of hand-offs: besides the new state, the row statistics of h.R (and,
// LSTM, of the cell state) have to meet from all columns before any of them can go on.  Through L2
// (rec_ln_grid.cuh) each takes 0.7 us from store to load; here the layer's row group lives in
// one cluster - 16 or 20 hidden units per CTA, R in registers, chains of eight rows, as in
// rec_cluster_kernels.cuh, whose layouts and tagged words these kernels use - and a hand-off is a
// store into the peers' shared memory.  The statistics of a CTA's warps meet in its own
// shared memory first, so that a peer receives one 64-byte line (8 rows x 2 words) per CTA: a
// remote store is paid per line.
//
// The stages of a step run over all chains of the CTA in turn (product of every chain, then the
// normalised gates of every chain, ...), so that one chain's hand-off is under way while the others
// compute; what a chain carries from stage to stage waits in shared memory.
//
// Arithmetic: fp32 storage multiplies three bf16 planes per
// operand (all products down to 2^-16 of the largest, smallest terms in accumulators of their own)
// and exchanges fp32 words; statistics are (mean, M2) pairs combined by Chan's formula forward and
// plain sums backward.  Waits are bounded; a warp that gives up says so at the next barrier of its
// CTA, where all four leave, and the peers run into their own limits.
#pragma once

#include <atomic>

#include "rec_cluster_launch.cuh"
#include "rec_ln_common.cuh"

namespace hb {
namespace rec {

struct LnClFwd : LnFwdParams {
  int CTAS, CH;
};
struct LnClBwd : LnBwdParams {
  int CTAS, CH;
  float* db_part;  // [row groups][4][H] sums of the gate gradients (GRU: z, r, g of dp, g of dq)
};

constexpr int LC_FWD_STASH = 9, LC_BWD_STASH = 16;  // floats per thread and chain

__device__ __forceinline__ uint2 lc_poll2(uint32_t a) {
  uint2 v;
  asm volatile("ld.relaxed.cluster.shared::cta.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void lc_store2(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.relaxed.cluster.shared::cluster.v2.u32 [%0], {%1,%2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ uint4 lc_lds4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}

// Two values -> the same pair in one, two or three bf16 planes.
template <int PL>
__device__ __forceinline__ void pair_planes(float a, float b, uint32_t (&p)[PL]) {
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    p[i] = pack_bf16(a, b);
    if (i + 1 < PL) {
      a -= __uint_as_float(p[i] << 16);
      b -= __uint_as_float(p[i] & 0xFFFF0000u);
    }
  }
}
// A fragment planes of rows half 0 / 1, four consecutive k each (as pack_weights)
template <int PL>
__device__ __forceinline__ void fragment_planes(const float (&x)[2][4], uint32_t (&f)[PL][4]) {
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    uint32_t p[PL];
    pair_planes<PL>(x[a & 1][(a >> 1) * 2], x[a & 1][(a >> 1) * 2 + 1], p);
#pragma unroll
    for (int i = 0; i < PL; ++i) f[i][a] = p[i];
  }
}
// acc[0] += a0 b0; acc[1] += terms of 2^-8; acc[2] += terms of 2^-16
template <int PL>
__device__ __forceinline__ void plane_mma(float (&acc)[PL][4], const uint32_t (&a)[PL][4], const uint32_t (&b0)[PL],
                                          const uint32_t (&b1)[PL]) {
  if constexpr (PL == 3) {
    mma_bf16(acc[2], a[2], b0[0], b1[0]);
    mma_bf16(acc[1], a[1], b0[0], b1[0]);
    mma_bf16(acc[0], a[0], b0[0], b1[0]);
    mma_bf16(acc[2], a[1], b0[1], b1[1]);
    mma_bf16(acc[1], a[0], b0[1], b1[1]);
    mma_bf16(acc[2], a[0], b0[2], b1[2]);
  } else {
    mma_bf16(acc[0], a[0], b0[0], b1[0]);
  }
}
template <int PL>
__device__ __forceinline__ float plane_sum(const float (&a)[PL][4], int j) {
  float s = a[PL - 1][j];
  if (PL == 3) s += a[PL == 3 ? 1 : 0][j];
  if (PL > 1) s += a[0][j];
  return s;
}

// The exchange of row statistics: buffers of the CTA ([stat][parity][chain][source][row] pairs of
// tagged words) and the meeting place of its warps ([stat][parity][warp][row]).
template <int NW>
struct Stats {
  uint32_t buf, dst, SB;  // own buffers; this lane's place in its destination's; bytes per buffer
  float2* part;
  int CS, CH;
  bool sends;

  __device__ __forceinline__ uint32_t area(int stat, int par, int ch) const {
    return (uint32_t)((stat * 2 + par) * CH + ch) * SB;
  }
  __device__ __forceinline__ float2* meet(int stat, int par) const { return part + (stat * 2 + par) * NW * 8; }
  // Pairs of this lane's quarter of the sources for `row`; zeros beyond the cluster.
  __device__ __forceinline__ bool collect(int stat, int par, int ch, int row, int quarter, uint32_t tag, float (&a)[4],
                                          float (&b)[4], const Sync& sync, volatile int* s_abort, int code) const {
    const uint32_t src = buf + area(stat, par, ch) + (uint32_t)(quarter * 4) * 64 + row * 8;
    uint2 y[4];
    long long t0 = 0;
    unsigned int spins = 0;
    bool ok = true;
    for (;;) {
      uint32_t bad = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        y[k] = make_uint2(tag, tag);
        if (quarter * 4 + k < CS) y[k] = lc_poll2(src + k * 64);
        bad |= (y[k].x ^ tag) | (y[k].y ^ tag);
      }
      if (__all_sync(0xffffffffu, (bad & 1u) == 0)) break;
      if (__any_sync(0xffffffffu, !may_spin(spins, t0, sync, s_abort, code))) { ok = false; break; }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[k] = fword_value(y[k].x);
      b[k] = fword_value(y[k].y);
    }
    return ok;
  }
};

// ---------------------------------------------------------------------------------------
template <int G, int NW, int KS, int SPLIT, typename T>
__global__ void __launch_bounds__(NW * 32, 1) ln_cl_fwd_kernel(const __grid_constant__ LnClFwd p) {
  constexpr int PL = SPLIT == 2 ? 3 : 1, U = 4 * NW, THREADS_ = NW * 32;
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int CS = p.CTAS, my = (int)cl_rank(), rg = blockIdx.x / CS;
  const int H = p.H, N = p.N, u0 = my * U, tile0 = rg * p.CH, ch_n = min(p.CH, ((N + 7) >> 3) - tile0);
  const long long NH = (long long)N * H;
  const int KSR = CS * NW / 4, rot = my * NW / 4;  // k-steps of 16 units; the first to arrive
  const uint32_t XB = (uint32_t)KSR * 512;  // one buffer of h words
  const uint32_t xb = smem_u32(smem);      // [CH][2][XB]
  Stats<NW> st_;
  st_.SB = (uint32_t)CS * 64;
  st_.CS = CS;
  st_.CH = p.CH;
  const size_t stats_at = (size_t)p.CH * 2 * XB, pl_at = stats_at + (size_t)4 * p.CH * st_.SB;
  st_.buf = xb + (uint32_t)stats_at;
  const uint32_t pl3 = xb + (uint32_t)pl_at + (uint32_t)(w * KS) * 512 + lane * 16;  // third plane of R
  uint8_t* after = smem + pl_at + (PL == 3 ? (size_t)NW * KS * 512 : 0);
  st_.part = reinterpret_cast<float2*>(after);
  float* carry = reinterpret_cast<float*>(after + 4 * NW * 8 * 8);  // [CH][h, c][threads]
  float* stash = carry + p.CH * 2 * THREADS_;                        // [CH][LC_FWD_STASH][threads]
  __shared__ int s_abort_;
  volatile int* s_abort = &s_abort_;

  if (tid == 0) *s_abort = 0;
  for (size_t i = tid; i < pl_at / 16; i += THREADS_)
    reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  {
    const T* h0 = reinterpret_cast<const T*>(p.h);
    const int units = CS * U;
    for (int i = tid; i < ch_n * 8 * units; i += THREADS_) {
      const int r = i / units, k = i - r * units, n = tile0 * 8 + r, Q = k >> 2;
      const float x = (n < N && k < H) ? ld(h0 + (long long)n * H + k) : 0.f;
      *reinterpret_cast<uint32_t*>(smem + (size_t)(r >> 3) * 2 * XB + (Q >> 2) * 512 + quad_piece(Q & 3, r & 7) +
                                   (k & 3) * 4) = hword_encode<SPLIT>(x, 1u);
    }
  }

  // ---- weights, in the order of arrival (slot s: k-step rot - s)
  const int gq = lane >> 2, q = lane & 3;
  uint32_t wf[SPLIT][KS][4];
#pragma unroll
  for (int s = 0; s < KS; ++s) {
    int ks = rot - s;
    if (ks < 0) ks += KSR;
    const int unit = u0 + 4 * w + (gq >> 1), ga = gq & 1, k = (ks * 4 + q) * 4;
    float x[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool ok = s < KSR && unit < H && k + i < H;
      const T* r = reinterpret_cast<const T*>(p.R) + (long long)(k + i) * G * H + unit;
      x[0][i] = ok ? ld(r + (long long)ga * H) : 0.f;
      x[1][i] = (ok && ga + 2 < G) ? ld(r + (long long)(ga + 2) * H) : 0.f;
    }
    uint32_t f[PL][4];
    fragment_planes<PL>(x, f);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      wf[0][s][a] = f[0][a];
      if (SPLIT == 2) wf[SPLIT - 1][s][a] = f[PL > 1 ? 1 : 0][a];
    }
    if (PL == 3)
      *reinterpret_cast<uint4*>(smem + (pl3 - xb) + s * 512) =
          make_uint4(f[PL - 1][0], f[PL - 1][1], f[PL - 1][2], f[PL - 1][3]);
  }
  // ---- the gate stage: unit 4w + lane/8, row 2(lane & 3) + ((lane >> 2) & 1)
  const int ul = lane >> 3, row = 2 * q + (gq & 1);
  const bool odd = gq & 1;
  const int unit = u0 + 4 * w + ul;
  const bool uok = unit < H;
  T *hb = reinterpret_cast<T*>(p.h), *cb = reinterpret_cast<T*>(p.c), *vb = reinterpret_cast<T*>(p.v);
  T *rhb = reinterpret_cast<T*>(p.act_Rh), *cnb = reinterpret_cast<T*>(p.act_c_norm);
  T *cache1 = reinterpret_cast<T*>(p.cache_Rh), *cache3 = reinterpret_cast<T*>(p.cache_c);
  const T *wx = reinterpret_cast<const T*>(p.Wx), *mask = reinterpret_cast<const T*>(p.mask);
  float bias[G], bias2[G], g1[G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    bias[g] = uok ? ld(reinterpret_cast<const T*>(p.b) + g * H + unit) : 0.f;
    bias2[g] = (G == 3 && uok) ? ld(reinterpret_cast<const T*>(p.b2) + g * H + unit) : 0.f;
    g1[g] = uok ? ld(reinterpret_cast<const T*>(p.gamma_Rh) + g * H + unit) : 0.f;
  }
  const float gh = (G == 4 && uok) ? ld(reinterpret_cast<const T*>(p.gamma_h) + unit) : 0.f;
  const float bh = (G == 4 && uok) ? ld(reinterpret_cast<const T*>(p.beta_h) + unit) : 0.f;
  for (int ch = 0; ch < ch_n; ++ch) {
    const int n = (tile0 + ch) * 8 + row;
    const bool ok = n < N && uok;
    carry[(ch * 2 + 0) * THREADS_ + tid] = ok ? ld(hb + (long long)n * H + unit) : 0.f;
    carry[(ch * 2 + 1) * THREADS_ + tid] = (G == 4 && ok) ? ld(cb + (long long)n * H + unit) : 0.f;
  }
  // ---- how many values lie behind a mean: of a warp, of a CTA (per gate), and of the row
  const float units_w = (float)max(0, min(4, H - (u0 + 4 * w)));
  const float rec_w = units_w > 0.f ? 1.0f / units_w : 0.f;
  float units_v[NW], units_s[4];  // of the CTA's warps; of this lane's quarter of the CTAs
#pragma unroll
  for (int k = 0; k < NW; ++k) units_v[k] = (float)max(0, min(4, H - (u0 + 4 * k)));
#pragma unroll
  for (int k = 0; k < 4; ++k) units_s[k] = ul * 4 + k < CS ? (float)max(0, min(U, H - (ul * 4 + k) * U)) : 0.f;
  const float rec_c = 1.0f / (float)max(1, min(U, H - u0)), rec_H = 1.0f / (float)H;
  // ---- destinations: lines of h to peers my + ul, my + ul + 4, ...; statistics to peer 4w + ul
  uint32_t dst[4];
  {
    const int Q = my * NW + w;
    const uint32_t off = (Q >> 2) * 512 + quad_piece(Q & 3, row);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      int d = my + ul + 4 * i;
      if (d >= CS) d -= CS;
      if (d >= CS) d -= CS;
      dst[i] = ul + 4 * i < CS ? cl_mapa(xb + off, (uint32_t)d) : 0u;
    }
    st_.sends = w * 4 + ul < CS;
    st_.dst = st_.sends ? cl_mapa(st_.buf + my * 64 + (lane & 7) * 8, (uint32_t)(w * 4 + ul)) : 0u;
  }
  __syncthreads();
  cl_sync();

  bool alive = true, stop = false;
  int turn[2] = {0, 0};  // parity of the warps' meeting place, per statistic
  // A row's pair for the columns of this lane (NV values v[0 .. NV)): warp, CTA, then on its way
  // to every peer.  One CTA barrier.
  auto publish = [&](int stat, int t, int ch, const float* v, int nv, bool ok, uint32_t tag) {
    const float inv = rec_w / (float)nv;
    float s = 0.f;
    for (int g = 0; g < nv; ++g) s += v[g];
    s = ok ? s : 0.f;
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    const float m = s * inv;
    float d = 0.f;
    for (int g = 0; g < nv; ++g) d += (v[g] - m) * (v[g] - m);
    d = ok ? d : 0.f;
    d += __shfl_xor_sync(0xffffffffu, d, 8);
    d += __shfl_xor_sync(0xffffffffu, d, 16);
    float2* at = st_.meet(stat, turn[stat]);
    turn[stat] ^= 1;
    if (ul == 0) at[w * 8 + row] = make_float2(m, d);
    stop = stage_barrier_or<NW>(!alive);
    if (stop) return;
    float2 y[NW];
    float mc = 0.f;
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      y[k] = at[k * 8 + (lane & 7)];
      mc += units_v[k] * y[k].x;
    }
    mc *= rec_c;
    float m2 = 0.f;
#pragma unroll
    for (int k = 0; k < NW; ++k) m2 += y[k].y + units_v[k] * (float)nv * (y[k].x - mc) * (y[k].x - mc);
    if (st_.sends) lc_store2(st_.dst + st_.area(stat, t & 1, ch), fword_encode(mc, tag), fword_encode(m2, tag));
  };
  auto collect = [&](int stat, int t, int ch, int nv, uint32_t tag, float& mean, float& inv, int code) {
    float a[4], b[4];
    if (!st_.collect(stat, t & 1, ch, row, ul, tag, a, b, p.sync, s_abort, code)) alive = false;
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) s += units_s[k] * a[k];
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    mean = s * rec_H;
    float m2 = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) m2 += units_s[k] > 0.f ? b[k] + units_s[k] * (float)nv * (a[k] - mean) * (a[k] - mean) : 0.f;
    m2 += __shfl_xor_sync(0xffffffffu, m2, 8);
    m2 += __shfl_xor_sync(0xffffffffu, m2, 16);
    inv = rsqrtf(m2 * rec_H / (float)nv + kLnEps);
  };
  // inputs of a (step, chain), fetched one ahead
  float nx[G + 1];
  auto fetch_inputs = [&](int t, int ch) {
    const int n = (tile0 + ch) * 8 + row;
    const bool ok = t < p.T && n < N && uok;
    const long long e = (long long)t * N + n;
#pragma unroll
    for (int g = 0; g < G; ++g) nx[g] = ok ? ld(wx + (e * G + g) * H + unit) : 0.f;
    nx[G] = (ok && p.has_zoneout && p.training) ? ld(mask + e * H + unit) : 0.f;
  };
  fetch_inputs(0, 0);
  const uint32_t lsrc = quad_piece(q, gq);
  constexpr uint32_t TAGBIT = SPLIT == 2 ? 1u : 0x40000000u;
  for (int t = 0; t < p.T && !stop; ++t) {
    const uint32_t rt = (((uint32_t)t >> 1) & 1u) ^ 1u;            // tag of h_t and of this step's statistics
    const uint32_t rtag = SPLIT == 2 ? rt : rt << 30;
    const uint32_t wtag = (((uint32_t)(t + 1) >> 1) & 1u) ^ 1u;    // of h_{t+1}
    // ---- stage A: h.R, its statistics
    for (int ch = 0; ch < ch_n; ++ch) {
      float* sh = stash + (size_t)ch * LC_FWD_STASH * THREADS_ + tid;
#pragma unroll
      for (int g = 0; g <= G; ++g) sh[(4 + g) * THREADS_] = nx[g];
      fetch_inputs(ch + 1 < ch_n ? t : t + 1, ch + 1 < ch_n ? ch + 1 : 0);
      float acc[2][PL][4];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < PL; ++b) acc[a][b][0] = acc[a][b][1] = acc[a][b][2] = acc[a][b][3] = 0.f;
      const uint32_t src = xb + (uint32_t)ch * 2 * XB + (t & 1) * XB + lsrc;
      uint4 x[2][4];
      auto fetch = [&](int b0, uint4 (&y)[4]) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          int ks = rot - (b0 + k);
          if (ks < 0) ks += KSR;
          if (b0 + k < KS - 3 || b0 + k < KSR) y[k] = cl_poll(src + (uint32_t)ks * 512);
          else y[k] = make_uint4(rtag, rtag, rtag, rtag);
        }
      };
      fetch(0, x[0]);
      long long t0 = 0;
      unsigned int spins = 0;
#pragma unroll
      for (int b0 = 0; b0 < KS; b0 += 4) {
        uint4(&y)[4] = x[(b0 >> 2) & 1];
        while (alive) {
          uint32_t bad = 0;
#pragma unroll
          for (int k = 0; k < 4; ++k) bad |= stale4(y[k], rtag);
          if (__all_sync(0xffffffffu, (bad & TAGBIT) == 0)) break;
          if (__any_sync(0xffffffffu, !may_spin(spins, t0, p.sync, s_abort, 63))) { alive = false; break; }
          fetch(b0, y);
        }
        if (b0 + 4 < KS) fetch(b0 + 4, x[((b0 >> 2) + 1) & 1]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint32_t a[PL][4], b_0[PL], b_1[PL];
          if constexpr (SPLIT == 2) {
            pair_planes<PL>(fword_value(y[k].x), fword_value(y[k].y), b_0);
            pair_planes<PL>(fword_value(y[k].z), fword_value(y[k].w), b_1);
            const uint4 third = lc_lds4(pl3 + (b0 + k) * 512);
            a[PL - 1][0] = third.x; a[PL - 1][1] = third.y; a[PL - 1][2] = third.z; a[PL - 1][3] = third.w;
          } else {
            b_0[0] = __byte_perm(y[k].x, y[k].y, 0x5410);
            b_1[0] = __byte_perm(y[k].z, y[k].w, 0x5410);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            a[0][i] = wf[0][b0 + k][i];
            if (SPLIT == 2) a[PL > 1 ? 1 : 0][i] = wf[SPLIT - 1][b0 + k][i];
          }
          plane_mma<PL>(acc[k & 1], a, b_0, b_1);
        }
      }
      float d[4], rh[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) d[j] = plane_sum<PL>(acc[0], j) + plane_sum<PL>(acc[1], j);
      swap_gates(d, odd, rh);
      const int n = (tile0 + ch) * 8 + row;
      const bool ok = n < N && uok;
      publish(0, t, ch, rh, G, ok, rt);
      if (stop) break;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        sh[g * THREADS_] = rh[g];
        if (ok) st(rhb + (((long long)t * N + n) * G + g) * H + unit, rh[g]);
      }
    }
    if (stop) break;
    // ---- stage B (LSTM): gates and the new cell state, its statistics
    if constexpr (G == 4) {
      for (int ch = 0; ch < ch_n; ++ch) {
        float* sh = stash + (size_t)ch * LC_FWD_STASH * THREADS_ + tid;
        const int n = (tile0 + ch) * 8 + row;
        const bool ok = n < N && uok;
        float mean1, inv1;
        collect(0, t, ch, G, rt, mean1, inv1, 64);
        float pre[4];
#pragma unroll
        for (int g = 0; g < 4; ++g)
          pre[g] = (sh[g * THREADS_] - mean1) * inv1 * g1[g % G] + sh[(4 + g) * THREADS_] + bias[g % G];
        const float i = ln_sigmoid<SPLIT>(pre[0]), gg = ln_tanh<SPLIT>(pre[1]), f = ln_sigmoid<SPLIT>(pre[2]),
                    o = ln_sigmoid<SPLIT>(pre[3]);
        float c_new[1] = {f * carry[(ch * 2 + 1) * THREADS_ + tid] + i * gg};
        publish(1, t, ch, c_new, 1, ok, rt);
        if (stop) break;
        sh[0] = o;
        sh[THREADS_] = c_new[0];
        if (ok) {
          st(cb + (long long)(t + 1) * NH + (long long)n * H + unit, c_new[0]);
          if (p.training) {
            T* vt = vb + ((long long)t * N + n) * 4 * H + unit;
            st(vt, i); st(vt + H, gg); st(vt + 2 * H, f); st(vt + 3 * H, o);
          }
        }
        if (my == 0 && w == 0 && ul == 0 && n < N) {
          st(cache1 + ((long long)t * N + n) * 2, mean1);
          st(cache1 + ((long long)t * N + n) * 2 + 1, inv1);
        }
      }
      if (stop) break;
    }
    // ---- last stage: the new state, on its way to every peer
    for (int ch = 0; ch < ch_n; ++ch) {
      float* sh = stash + (size_t)ch * LC_FWD_STASH * THREADS_ + tid;
      float* cy = carry + (size_t)ch * 2 * THREADS_ + tid;
      const int n = (tile0 + ch) * 8 + row;
      const bool ok = n < N && uok;
      float mean, inv;
      collect(G == 4 ? 1 : 0, t, ch, G == 4 ? 1 : G, rt, mean, inv, 65);
      const float hp = cy[0], m = sh[(4 + G) * THREADS_];
      float h_new, c_norm = 0.f, z = 0.f, r = 0.f, gg = 0.f, qg = 0.f;
      if (G == 4) {
        c_norm = (sh[THREADS_] - mean) * inv * gh + bh;
        h_new = sh[0] * ln_tanh<SPLIT>(c_norm);
      } else {
        float rn[3];
#pragma unroll
        for (int g = 0; g < 3; ++g) rn[g] = (sh[g * THREADS_] - mean) * inv * g1[g] + bias2[g];
        z = ln_sigmoid<SPLIT>(sh[4 * THREADS_] + bias[0] + rn[0]);
        r = ln_sigmoid<SPLIT>(sh[5 * THREADS_] + bias[1] + rn[1]);
        qg = rn[2];
        gg = ln_tanh<SPLIT>(sh[6 * THREADS_] + bias[2] + r * qg);
        h_new = z * hp + (1.0f - z) * gg;
      }
      if (p.has_zoneout)
        h_new = p.training ? zoneout<true>(h_new, hp, p.zoneout_prob, m) : zoneout<false>(h_new, hp, p.zoneout_prob, m);
      h_new = ok ? round_to_storage<T>(h_new) : 0.f;
      if (t + 1 < p.T) {
        const uint32_t word = hword_encode<SPLIT>(h_new, wtag);
        const uint32_t a1 = __shfl_xor_sync(0xffffffffu, word, 8);
        const uint32_t a2 = __shfl_xor_sync(0xffffffffu, word, 16);
        const uint32_t a3 = __shfl_xor_sync(0xffffffffu, word, 24);
        const bool o1 = ul & 1, o2 = ul & 2;
        const uint32_t e0 = o1 ? a1 : word, e1 = o1 ? word : a1, f0 = o1 ? a3 : a2, f1 = o1 ? a2 : a3;
        const uint32_t off = (uint32_t)ch * 2 * XB + ((t + 1) & 1) * XB;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (ul + 4 * i < CS)
            cl_store(dst[i] + off, o2 ? f0 : e0, o2 ? f1 : e1, o2 ? e0 : f0, o2 ? e1 : f1);
      }
      cy[0] = h_new;
      if (G == 4) cy[THREADS_] = sh[THREADS_];
      if (ok) {
        const long long e = (long long)t * N + n;
        st(hb + NH + e * H + unit, h_new);
        if (G == 4) {
          st(cnb + e * H + unit, c_norm);
        } else if (p.training && vb) {
          T* vt = vb + e * 4 * H + unit;
          st(vt, z); st(vt + H, r); st(vt + 2 * H, gg); st(vt + 3 * H, qg);
        }
      }
      if (my == 0 && w == 0 && ul == 0 && n < N) {
        T* cc = (G == 4 ? cache3 : cache1) + ((long long)t * N + n) * 2;
        st(cc, mean);
        st(cc + 1, inv);
      }
    }
  }
  __syncthreads();
  cl_sync();  // nobody leaves while a peer may still store into its shared memory
}

// ---------------------------------------------------------------------------------------
template <int G, int NW, int TPW, int SPLIT, typename T>
__global__ void __launch_bounds__(NW * 32, 1) ln_cl_bwd_kernel(const __grid_constant__ LnClBwd p) {
  constexpr int PL = SPLIT == 2 ? 3 : 1, U = 4 * NW, THREADS_ = NW * 32;
  constexpr int KSB = (G * NW + 3) / 4;  // k-steps: G * NW unit quads of own gate columns
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int CS = p.CTAS, my = (int)cl_rank(), rg = blockIdx.x / CS;
  const int H = p.H, N = p.N, u0 = my * U, tile0 = rg * p.CH, ch_n = min(p.CH, ((N + 7) >> 3) - tile0);
  const long long NH = (long long)N * H;
  const uint32_t XB = (uint32_t)CS * NW * 128;  // one exchange buffer: [source][own quad][128]
  const uint32_t xb = smem_u32(smem);              // [CH][2][XB]
  Stats<NW> st_;
  st_.SB = (uint32_t)CS * 64;
  st_.CS = CS;
  st_.CH = p.CH;
  const size_t stats_at = (size_t)p.CH * 2 * XB, g_at = stats_at + (size_t)4 * p.CH * st_.SB;
  st_.buf = xb + (uint32_t)stats_at;
  uint8_t* gsm = smem + g_at;                     // d(h.R), B operand: [2][KSB][512]
  uint8_t* gsm3 = gsm + 2 * KSB * 512;            // its third plane: [2][KSB][256]
  const size_t pl_at = g_at + 2 * KSB * 512 + (PL == 3 ? 2 * KSB * 256 : 0);
  const uint32_t pl3 = xb + (uint32_t)pl_at + (uint32_t)(w * TPW * KSB) * 512 + lane * 16;
  uint8_t* after = smem + pl_at + (PL == 3 ? (size_t)NW * TPW * KSB * 512 : 0);
  st_.part = reinterpret_cast<float2*>(after);
  float* carry = reinterpret_cast<float*>(after + 4 * NW * 8 * 8);  // [CH][dh, dc, c][threads]
  float* stash = carry + p.CH * 3 * THREADS_;                        // [CH][LC_BWD_STASH][threads]
  __shared__ int s_abort_;
  volatile int* s_abort = &s_abort_;
  if (tid == 0) *s_abort = 0;
  for (size_t i = tid; i < pl_at / 16; i += THREADS_)
    reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);

  // ---- weights: slot i of warp w is output tile (w + NW i + my NW / 4) mod MTR (see cl_bwd_kernel)
  const int gq = lane >> 2, q = lane & 3, MTR = CS * NW / 4;
  uint32_t wf[SPLIT][TPW][KSB][4];
  uint32_t dst[TPW];
#pragma unroll
  for (int i = 0; i < TPW; ++i) {
    const int Lt = w + NW * i;
    int tile = Lt + my * NW / 4;
    while (tile >= MTR) tile -= MTR;
    const int Q = tile * 4 + (gq >> 1), d = Q / NW, qw = Q - d * NW;
    const bool live = Lt < MTR;
    dst[i] = live ? cl_mapa(xb + (uint32_t)(my * NW + qw) * 128 + ((gq & 1) * 4 + q) * 16, (uint32_t)d) : 0u;
#pragma unroll
    for (int kk = 0; kk < KSB; ++kk) {
      const int lq = kk * 4 + q, gate = lq / NW, j = Q * 4 + (gq & 1), k = u0 + 4 * (lq - gate * NW);
      const T* R = reinterpret_cast<const T*>(p.R);
      float x[2][4];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool ok = live && gate < G && j + 2 * hf < H && k + e < H;
          const long long col = (long long)gate * H + k + e;
          x[hf][e] = ok ? ld(p.r_transposed ? R + col * H + j + 2 * hf : R + (long long)(j + 2 * hf) * G * H + col) : 0.f;
        }
      uint32_t f[PL][4];
      fragment_planes<PL>(x, f);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        wf[0][i][kk][a] = f[0][a];
        if (SPLIT == 2) wf[SPLIT - 1][i][kk][a] = f[PL > 1 ? 1 : 0][a];
      }
      if (PL == 3)
        *reinterpret_cast<uint4*>(smem + (pl3 - xb) + (i * KSB + kk) * 512) =
            make_uint4(f[PL - 1][0], f[PL - 1][1], f[PL - 1][2], f[PL - 1][3]);
    }
  }
  // ---- ownership (see cl_bwd_kernel): piece c8 of the quad's line, word sub of it
  const int sub = lane >> 3, c8 = lane & 7;
  const int row = 2 * (c8 & 3) + (sub & 1), ul = (c8 >> 2) + 2 * (sub >> 1);
  const int unit = u0 + 4 * w + ul;
  const bool uok = unit < H, second = (c8 & 4) != 0;
  T *vb = reinterpret_cast<T*>(p.v), *rhb = reinterpret_cast<T*>(p.act_Rh);
  T *dpb = reinterpret_cast<T*>(p.dp), *dqb = reinterpret_cast<T*>(p.dq);
  const T *cb = reinterpret_cast<const T*>(p.c), *hb = reinterpret_cast<const T*>(p.h);
  const T* cnb = reinterpret_cast<const T*>(p.act_c_norm);
  const T *cache1 = reinterpret_cast<const T*>(p.cache_Rh), *cache3 = reinterpret_cast<const T*>(p.cache_c);
  const T *dhn = reinterpret_cast<const T*>(p.dh_new), *dcn = reinterpret_cast<const T*>(p.dc_new);
  const T* mask = reinterpret_cast<const T*>(p.mask);
  float g1[G];
#pragma unroll
  for (int g = 0; g < G; ++g) g1[g] = uok ? ld(reinterpret_cast<const T*>(p.gamma_Rh) + g * H + unit) : 0.f;
  const float gh = (G == 4 && uok) ? ld(reinterpret_cast<const T*>(p.gamma_h) + unit) : 0.f;
  const float inv_H = 1.0f / (float)H, inv_GH = 1.0f / (float)(G * H);
  for (int ch = 0; ch < ch_n; ++ch) {
    const int n = (tile0 + ch) * 8 + row;
    const bool ok = n < N && uok;
    const long long o = (long long)n * H + unit;
    float* cy = carry + (size_t)ch * 3 * THREADS_ + tid;
    cy[0] = ok ? p.dh_carry[o] : 0.f;
    cy[THREADS_] = (G == 4 && ok) ? p.dc_carry[o] : 0.f;
    cy[2 * THREADS_] = (G == 4 && ok) ? ld(cb + (long long)p.T * NH + o) : 0.f;
  }
  st_.sends = w * 4 + (lane >> 3) < CS;
  st_.dst = st_.sends ? cl_mapa(st_.buf + my * 64 + (lane & 7) * 8, (uint32_t)(w * 4 + (lane >> 3))) : 0u;
  float acc_b[4] = {0.f, 0.f, 0.f, 0.f}, acc_g1[G], acc_gh = 0.f, acc_bh = 0.f;
#pragma unroll
  for (int g = 0; g < G; ++g) acc_g1[g] = 0.f;
  __syncthreads();
  cl_sync();

  bool alive = true, stop = false;
  int turn[2] = {0, 0}, gpar = 0;
  // Sums of a row's pair (x, y) over this CTA, on their way to every peer.  One CTA barrier.
  auto publish = [&](int stat, int ti, int ch, float x, float y, uint32_t tag) {
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    y += __shfl_xor_sync(0xffffffffu, y, 4);
    x += __shfl_xor_sync(0xffffffffu, x, 16);
    y += __shfl_xor_sync(0xffffffffu, y, 16);
    float2* at = st_.meet(stat, turn[stat]);
    turn[stat] ^= 1;
    if (ul == 0) at[w * 8 + row] = make_float2(x, y);
    stop = stage_barrier_or<NW>(!alive);
    if (stop) return;
    float sx = 0.f, sy = 0.f;
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      const float2 v = at[k * 8 + (lane & 7)];
      sx += v.x;
      sy += v.y;
    }
    if (st_.sends) lc_store2(st_.dst + st_.area(stat, ti & 1, ch), fword_encode(sx, tag), fword_encode(sy, tag));
  };
  auto collect = [&](int stat, int ti, int ch, uint32_t tag, float& x, float& y, int code) {
    float a[4], b[4];
    if (!st_.collect(stat, ti & 1, ch, row, ul, tag, a, b, p.sync, s_abort, code)) alive = false;
#pragma unroll
    for (int k = 0; k < 4; ++k)  // beyond the cluster the words are the bare tag: a value of zero
      if (ul * 4 + k >= CS) a[k] = b[k] = 0.f;
    x = (a[0] + a[1]) + (a[2] + a[3]);
    y = (b[0] + b[1]) + (b[2] + b[3]);
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    y += __shfl_xor_sync(0xffffffffu, y, 4);
    x += __shfl_xor_sync(0xffffffffu, x, 16);
    y += __shfl_xor_sync(0xffffffffu, y, 16);
  };
  // The recurrent part of dh published at production step s (see cl_bwd_kernel).
  auto gather = [&](int ch, int s, float& dh_c) {
    const uint32_t want = (((uint32_t)s >> 1) & 1u) ^ 1u;
    const uint32_t src = xb + (uint32_t)ch * 2 * XB + (s & 1) * XB + (uint32_t)(w * 128 + c8 * 16);
    uint4 y[TPW];
    long long t0 = 0;
    unsigned int spins = 0;
    for (;;) {
      uint32_t bad = 0;
#pragma unroll
      for (int k = 0; k < TPW; ++k) {
        const int j = sub * TPW + k;
        y[k] = make_uint4(want, want, want, want);
        if (j < CS) y[k] = cl_poll(src + (uint32_t)(j * NW) * 128);
        bad |= stale4(y[k], want);
      }
      if (__all_sync(0xffffffffu, (bad & 1u) == 0)) break;
      if (__any_sync(0xffffffffu, !may_spin(spins, t0, p.sync, s_abort, 66))) { alive = false; break; }
    }
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < TPW; ++k) {
      s4[0] += fword_value(y[k].x); s4[1] += fword_value(y[k].y);
      s4[2] += fword_value(y[k].z); s4[3] += fword_value(y[k].w);
    }
    dh_c += gather_reduce(s4, sub);
  };
  // inputs of a (step, chain), fetched one ahead: gates 4, h.R G, dh_new, mask, then LSTM dc_new, c
  // before, LN(c), GRU h before; statistics of h.R, LSTM those of c
  constexpr int NI = 4 + G + 2 + (G == 4 ? 3 : 1) + (G == 4 ? 4 : 2);
  constexpr int I_RH = 4, I_DH = 4 + G, I_M = I_DH + 1, I_S = I_M + 1, I_C1 = I_S + (G == 4 ? 3 : 1);
  float nx[NI];
  auto fetch_inputs = [&](int ti, int ch) {
    const int n = (tile0 + ch) * 8 + row, t = p.T - 1 - ti;
    const bool rok = t >= 0 && n < N, ok = rok && uok;
    const long long e = (long long)t * N + n;
#pragma unroll
    for (int i = 0; i < NI; ++i) nx[i] = 0.f;
    nx[I_M] = 1.f;
    if (ok) {
#pragma unroll
      for (int g = 0; g < 4; ++g) nx[g] = ld(vb + (e * 4 + g) * H + unit);
#pragma unroll
      for (int g = 0; g < G; ++g) nx[I_RH + g] = ld(rhb + (e * G + g) * H + unit);
      nx[I_DH] = ld(dhn + NH + e * H + unit);
      if (p.has_zoneout) nx[I_M] = ld(mask + e * H + unit);
      if (G == 4) {
        if (dcn) nx[I_S] = ld(dcn + NH + e * H + unit);
        nx[I_S + (G == 4 ? 1 : 0)] = ld(cb + e * H + unit);
        nx[I_S + (G == 4 ? 2 : 0)] = ld(cnb + e * H + unit);
      } else {
        nx[I_S] = ld(hb + e * H + unit);
      }
    }
    if (rok) {
      nx[I_C1] = ld(cache1 + e * 2);
      nx[I_C1 + 1] = ld(cache1 + e * 2 + 1);
      if (G == 4) {
        nx[NI - 2] = ld(cache3 + e * 2);
        nx[NI - 1] = ld(cache3 + e * 2 + 1);
      }
    }
  };
  // stash: 0..G-1 gate gradients, 4..4+G-1 h.R - mean, 8 its 1/sigma; LSTM before stage B: 9 dc
  // arriving, 10 c before, 11 c - mean, 12 its 1/sigma, 13 gamma_h d(LN c), 0..2 gates i, g, f, 3 d_o
  fetch_inputs(0, 0);
  for (int ti = 0; ti < p.T && !stop; ++ti) {
    const int t = p.T - 1 - ti;
    const uint32_t tag = (((uint32_t)ti >> 1) & 1u) ^ 1u;
    // the rest of LayerNorm(h.R): row sums of the gate gradients
    auto norm_sums = [&](const float (&dg)[G], const float (&cx)[G], float inv1, bool ok, int ch) {
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float db = g1[g] * dg[g];
        if (ok) {
          s1 += cx[g] * db;
          s2 += db;
          acc_g1[g] += cx[g] * inv1 * dg[g];
        }
      }
      publish(0, ti, ch, s1, s2, tag);
    };
    // ---- stage A
    for (int ch = 0; ch < ch_n; ++ch) {
      float* sh = stash + (size_t)ch * LC_BWD_STASH * THREADS_ + tid;
      float* cy = carry + (size_t)ch * 3 * THREADS_ + tid;
      float in[NI];
#pragma unroll
      for (int i = 0; i < NI; ++i) in[i] = nx[i];
      fetch_inputs(ch + 1 < ch_n ? ti : ti + 1, ch + 1 < ch_n ? ch + 1 : 0);
      const int n = (tile0 + ch) * 8 + row;
      const bool ok = n < N && uok;
      float dh_c = cy[0];
      if (ti > 0) gather(ch, ti - 1, dh_c);
      float dh_total = in[I_DH] + dh_c, keep = 0.f;
      if (p.has_zoneout) {
        keep = (1.0f - in[I_M]) * dh_total;
        dh_total = in[I_M] * dh_total;
      }
      float cx[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        cx[g] = in[I_RH + g] - in[I_C1];
        sh[(4 + g) * THREADS_] = cx[g];
      }
      sh[8 * THREADS_] = in[I_C1 + 1];
      if constexpr (G == 4) {
        const float o = in[3], inv3 = in[NI - 1];
        const float cx3 = ok ? cy[2 * THREADS_] - in[NI - 2] : 0.f;
        const float c_tanh = ln_tanh<SPLIT>(in[I_S + 2]);
        const float d_norm = ok ? d_tanh(c_tanh) * (o * dh_total) : 0.f;  // gradient w.r.t. LayerNorm(c')
        acc_gh += cx3 * inv3 * d_norm;
        acc_bh += d_norm;
        const float db3 = gh * d_norm;
        cy[0] = ok ? keep : 0.f;
        sh[0] = in[0]; sh[THREADS_] = in[1]; sh[2 * THREADS_] = in[2];
        sh[3 * THREADS_] = d_sigmoid(o) * (c_tanh * dh_total);
        sh[9 * THREADS_] = in[I_S]; sh[10 * THREADS_] = in[I_S + 1];
        sh[11 * THREADS_] = cx3; sh[12 * THREADS_] = inv3; sh[13 * THREADS_] = db3;
        publish(1, ti, ch, cx3 * db3, db3, tag);
        if (stop) break;
      } else {
        const float z = in[0], r = in[1], gg = in[2], qg = in[3];
        const float dp_g = d_tanh(gg) * ((1.0f - z) * dh_total);
        float dg[G];
        dg[0] = ok ? d_sigmoid(z) * ((in[I_S] - gg) * dh_total) : 0.f;
        dg[1] = ok ? d_sigmoid(r) * (dp_g * qg) : 0.f;
        dg[2] = ok ? dp_g * r : 0.f;
        cy[0] = ok ? keep + z * dh_total : 0.f;
        norm_sums(dg, cx, in[I_C1 + 1], ok, ch);
        if (stop) break;
#pragma unroll
        for (int g = 0; g < G; ++g) sh[g * THREADS_] = dg[g];
        if (ok) {
          const long long w0 = ((long long)t * N + n) * 3 * H + unit;
          st(dpb + w0, dg[0]); st(dpb + w0 + H, dg[1]); st(dpb + w0 + 2 * H, dp_g);
          st(dqb + w0, dg[0]); st(dqb + w0 + H, dg[1]); st(dqb + w0 + 2 * H, dg[2]);
          acc_b[0] += dg[0]; acc_b[1] += dg[1]; acc_b[2] += dp_g; acc_b[3] += dg[2];
        }
      }
    }
    if (stop) break;
    // ---- stage B (LSTM): the cell state's LayerNorm, the gate gradients
    if constexpr (G == 4) {
      for (int ch = 0; ch < ch_n; ++ch) {
        float* sh = stash + (size_t)ch * LC_BWD_STASH * THREADS_ + tid;
        float* cy = carry + (size_t)ch * 3 * THREADS_ + tid;
        const int n = (tile0 + ch) * 8 + row;
        const bool ok = n < N && uok;
        float S1, S2;
        collect(1, ti, ch, tag, S1, S2, 67);
        const float r = sh[12 * THREADS_];
        const float dsigma = -0.5f * S1 * r * r * r, dmu = -S2 * r;
        const float dcl = 2.0f * sh[11 * THREADS_] * dsigma * inv_H + r * sh[13 * THREADS_] + dmu * inv_H;
        const float i = sh[0], gg = sh[THREADS_], f = sh[2 * THREADS_], cprev = sh[10 * THREADS_];
        const float dc_total = ok ? sh[9 * THREADS_] + cy[THREADS_] + dcl : 0.f;
        float dg[G], cx[G];
        dg[0] = d_sigmoid(i) * (gg * dc_total);
        dg[1] = d_tanh(gg) * (i * dc_total);
        dg[2] = d_sigmoid(f) * (cprev * dc_total);
        dg[G - 1] = ok ? sh[3 * THREADS_] : 0.f;
        cy[THREADS_] = f * dc_total;
        cy[2 * THREADS_] = cprev;
#pragma unroll
        for (int g = 0; g < G; ++g) cx[g] = sh[(4 + g) * THREADS_];
        norm_sums(dg, cx, sh[8 * THREADS_], ok, ch);
        if (stop) break;
#pragma unroll
        for (int g = 0; g < G; ++g) {
          sh[g * THREADS_] = dg[g];
          acc_b[g] += dg[g];
          if (ok) st(vb + (((long long)t * N + n) * 4 + g) * H + unit, dg[g]);
        }
      }
      if (stop) break;
    }
    // ---- stage C: d(h.R), and what it makes of dh for every unit
    for (int ch = 0; ch < ch_n; ++ch) {
      float* sh = stash + (size_t)ch * LC_BWD_STASH * THREADS_ + tid;
      const int n = (tile0 + ch) * 8 + row;
      const bool ok = n < N && uok;
      float S1, S2;
      collect(0, ti, ch, tag, S1, S2, 68);
      const float r = sh[8 * THREADS_];
      const float dsigma = -0.5f * S1 * r * r * r, dmu = -S2 * r;
      uint8_t *gb = gsm + gpar * KSB * 512, *gb3 = gsm3 + gpar * KSB * 256;
      gpar ^= 1;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const float x = ok ? 2.0f * sh[(4 + g) * THREADS_] * dsigma * inv_GH + r * (g1[g] * sh[g * THREADS_]) +
                                 dmu * inv_GH
                           : 0.f;
        if (ok) st(rhb + (((long long)t * N + n) * G + g) * H + unit, x);
        // operand: (gate, quad w), the even unit of a pair writes the high halves (and the third
        // plane), the odd one the middle ones
        float pl[3] = {x, 0.f, 0.f};
        if (PL == 3) split3_bf16(x, pl);
        const uint32_t own = pack_bf16(pl[0], pl[1]);
        const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 4);
        const int lq = g * NW + w;
        *reinterpret_cast<uint32_t*>(gb + (lq >> 2) * 512 + quad_piece(lq & 3, row) + (second ? 8 : 0) + (sub >> 1) * 4) =
            second ? __byte_perm(other, own, 0x7632) : __byte_perm(own, other, 0x5410);
        if (PL == 3) {
          const float third = __shfl_xor_sync(0xffffffffu, pl[2], 4);
          if (!second) *reinterpret_cast<uint32_t*>(gb3 + lq * 64 + row * 8 + (sub >> 1) * 4) = pack_bf16(pl[2], third);
        }
      }
      stop = stage_barrier_or<NW>(!alive);
      if (stop) break;
      const uint32_t off = (uint32_t)ch * 2 * XB + (ti & 1) * XB;
      uint32_t b0[KSB][PL], b1[KSB][PL];
#pragma unroll
      for (int kk = 0; kk < KSB; ++kk) {
        const uint4 y = *reinterpret_cast<const uint4*>(gb + kk * 512 + quad_piece(q, gq));
        b0[kk][0] = y.x;
        b1[kk][0] = y.y;
        if constexpr (PL == 3) {
          const uint2 y3 = *reinterpret_cast<const uint2*>(gb3 + kk * 256 + q * 64 + gq * 8);
          b0[kk][1] = y.z; b1[kk][1] = y.w;
          b0[kk][2] = y3.x; b1[kk][2] = y3.y;
        }
      }
#pragma unroll
      for (int i = 0; i < TPW; ++i) {
        float acc[PL][4];
#pragma unroll
        for (int e = 0; e < PL; ++e) acc[e][0] = acc[e][1] = acc[e][2] = acc[e][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < KSB; ++kk) {
          uint32_t a[PL][4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            a[0][e] = wf[0][i][kk][e];
            if (SPLIT == 2) a[PL > 1 ? 1 : 0][e] = wf[SPLIT - 1][i][kk][e];
          }
          if (PL == 3) {
            const uint4 third = lc_lds4(pl3 + (i * KSB + kk) * 512);
            a[PL - 1][0] = third.x; a[PL - 1][1] = third.y; a[PL - 1][2] = third.z; a[PL - 1][3] = third.w;
          }
          plane_mma<PL>(acc, a, b0[kk], b1[kk]);
        }
        if (dst[i])
          cl_store(dst[i] + off, fword_encode(plane_sum<PL>(acc, 0), tag), fword_encode(plane_sum<PL>(acc, 1), tag),
                   fword_encode(plane_sum<PL>(acc, 2), tag), fword_encode(plane_sum<PL>(acc, 3), tag));
      }
    }
  }
  // ---- what is left of dh: the recurrent part of step 0, then the carries go out
  for (int ch = 0; ch < ch_n && alive && !stop; ++ch) {
    const int n = (tile0 + ch) * 8 + row;
    float* cy = carry + (size_t)ch * 3 * THREADS_ + tid;
    float dh_c = cy[0];
    gather(ch, p.T - 1, dh_c);
    if (alive && n < N && uok) {
      p.dh_carry[(long long)n * H + unit] = dh_c;
      if (G == 4) p.dc_carry[(long long)n * H + unit] = cy[THREADS_];
    }
  }
  // ---- parameter gradients of this row group: sums over the eight rows
  auto rows = [&](float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v + __shfl_xor_sync(0xffffffffu, v, 8);
  };
  const bool first = row == 0 && uok;
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const float s = rows(acc_b[g]);
    if (first) p.db_part[((size_t)rg * 4 + g) * H + unit] = s;
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const float s = rows(acc_g1[g]);
    if (first) p.dgRh_part[((size_t)rg * G + g) * H + unit] = s;
  }
  if (G == 4) {
    const float s = rows(acc_gh), b = rows(acc_bh);
    if (first) {
      p.dgh_part[(size_t)rg * H + unit] = s;
      p.dbh_part[(size_t)rg * H + unit] = b;
    }
  }
  __syncthreads();
  cl_sync();
}

// ---------------------------------------------------------------------------------------
// Host side.  Sixteen CTAs of 16 units (four warps) reach 256, of 20 units (five warps) 320; these only
// while the chains of a CTA stay few, as seven such clusters are resident and the fifth warp shares a
// sub-partition (LSTM fp32, us per step, these / the grid kernels: one chain, 45 rows H = 296 5.1 / 11.7
// forward, 4.4 / 11.9 backward; two chains, 64 rows H = 320 9.7 / 8.0 and 8.2 / 11.7).
constexpr int kLnClMost = 320, kLnWideFwdChains = 1, kLnWideBwdChains = 2;
// `row_groups` receives the number of partial rows in db_part and the others.
template <int G, int NW, int KS, int SPLIT, typename T>
int ln_cl_fwd_go(LnClFwd& p, int most, cudaStream_t s) {
  static std::atomic<int> slots[kChainMaxDevices][17];
  const size_t chain = (size_t)2 * (p.CTAS * NW / 4) * 512 + (size_t)4 * p.CTAS * 64 +
                       (size_t)(2 + LC_FWD_STASH) * NW * 32 * 4;
  const size_t fixed = (SPLIT == 2 ? (size_t)NW * KS * 512 : 0) + 4 * NW * 8 * 8;
  int groups = 0;
  return cl_launch(ln_cl_fwd_kernel<G, NW, KS, SPLIT, T>, p, NW * 32, chain, fixed, slots, most, &groups, s);
}
template <int G, int SPLIT, typename T>
int run_ln_cl_fwd(const LnFwdParams& q, cudaStream_t s) {
  if (q.H > kLnClMost) return HASTE_B200_ERR_UNSUPPORTED;
  LnClFwd p;
  static_cast<LnFwdParams&>(p) = q;
  p.CTAS = q.H > 256 ? 16 : ceil_div(q.H, 16);
  if (q.H > 256) return ln_cl_fwd_go<G, 5, 20, SPLIT, T>(p, kLnWideFwdChains, s);
  if (p.CTAS <= 4) return ln_cl_fwd_go<G, 4, 4, SPLIT, T>(p, kClMaxChains, s);
  if (p.CTAS <= 8) return ln_cl_fwd_go<G, 4, 8, SPLIT, T>(p, kClMaxChains, s);
  if (p.CTAS <= 12) return ln_cl_fwd_go<G, 4, 12, SPLIT, T>(p, kClMaxChains, s);
  return ln_cl_fwd_go<G, 4, 16, SPLIT, T>(p, kClMaxChains, s);
}

template <int G, int NW, int TPW, int SPLIT, typename T>
int ln_cl_bwd_go(LnClBwd& p, int most, int* row_groups, cudaStream_t s) {
  constexpr int KSB = (G * NW + 3) / 4;
  static std::atomic<int> slots[kChainMaxDevices][17];
  const size_t chain = (size_t)2 * p.CTAS * NW * 128 + (size_t)4 * p.CTAS * 64 +
                       (size_t)(3 + LC_BWD_STASH) * NW * 32 * 4;
  const size_t fixed = (size_t)2 * KSB * 512 + (SPLIT == 2 ? (size_t)2 * KSB * 256 + (size_t)NW * TPW * KSB * 512 : 0) +
                       4 * NW * 8 * 8;
  return cl_launch(ln_cl_bwd_kernel<G, NW, TPW, SPLIT, T>, p, NW * 32, chain, fixed, slots, most, row_groups, s);
}
template <int G, int SPLIT, typename T>
int run_ln_cl_bwd(const LnBwdParams& q, float* db_part, int* row_groups, cudaStream_t s) {
  if (q.H > kLnClMost) return HASTE_B200_ERR_UNSUPPORTED;
  LnClBwd p;
  static_cast<LnBwdParams&>(p) = q;
  p.CTAS = q.H > 256 ? 16 : ceil_div(q.H, 16);
  p.db_part = db_part;
  if (q.H > 256) return ln_cl_bwd_go<G, 5, 4, SPLIT, T>(p, kLnWideBwdChains, row_groups, s);
  if (p.CTAS <= 4) return ln_cl_bwd_go<G, 4, 1, SPLIT, T>(p, kClMaxChains, row_groups, s);
  if (p.CTAS <= 8) return ln_cl_bwd_go<G, 4, 2, SPLIT, T>(p, kClMaxChains, row_groups, s);
  if (p.CTAS <= 12) return ln_cl_bwd_go<G, 4, 3, SPLIT, T>(p, kClMaxChains, row_groups, s);
  return ln_cl_bwd_go<G, 4, 4, SPLIT, T>(p, kClMaxChains, row_groups, s);
}

}  // namespace rec
}  // namespace hb
