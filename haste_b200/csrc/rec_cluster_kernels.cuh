// Persistent LSTM / GRU recurrence on thread-block clusters, sm_100a: hidden sizes up to 320.
//
// What bounds a recurrence step is a serial chain - product, gate math, hand-off of the new state
// to every CTA that needs it - so a step costs the latency of that chain, not its arithmetic.
// Here one cluster of CS = ceil(H / (4 NW)) CTAs holds the whole recurrent matrix in registers
// and the hand-off is a store into the peers' shared memory:
//
// * A CTA owns U = 4 NW hidden units (all gates) and carries CH chains of eight batch rows
//   through each step.
// * Forward: warp w computes 16 gate columns (4 gates of units 4w..4w+3) over all of K, so a
//   quad of lanes ends up with every gate of its (unit, row) after one shuffle: no partial
//   tiles, no CTA barrier in the step.
// * Backward: the CTA turns its gate gradients into partial dh for every unit; the owner adds
//   the CS partials in a fixed order.  One barrier per step (the gate gradients meet in shared
//   memory as the B operand).
// * Exchanged words carry their own readiness (a tag that flips whenever a buffer is reused), as
//   in recurrent_common.cuh; here the consumer polls its own shared memory.
// * What a remote store costs is counted in 128-byte lines, not bytes: an exchange alone was
//   measured at 470 cycles + 11.5 cycles per line sent and received by a CTA (CS = 4 / 8 / 16:
//   667 / 899 / 1326 cycles), against 1280 / 1640 / 1640 cycles through L2.  Lines are therefore
//   whole - 8 rows x 4 units x 4 bytes, the 16-byte pieces rotated so that the fragment loads
//   stay free of bank conflicts - and every CTA starts with another destination, so that a
//   consumer can multiply what has arrived while the rest is on its way.
//
// Every wait is bounded; a warp that gives up reports through the error word, its peers run into
// their own limits, and all CTAs of the cluster meet at the final cluster barrier.
#pragma once

#include "rec_chain.cuh"

namespace hb {
namespace rec {

__device__ __forceinline__ uint32_t cl_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cl_mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A peer's store becomes visible word by word; the tags of all four words are checked.
__device__ __forceinline__ uint4 cl_poll(uint32_t a) {
  uint4 v;
  asm volatile("ld.relaxed.cluster.shared::cta.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(a)
               : "memory");
  return v;
}
__device__ __forceinline__ void cl_store(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.relaxed.cluster.shared::cluster.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z),
               "r"(w)
               : "memory");
}
// Barrier of the NW stage warps; true in every thread if `flag` was in any.
template <int NW>
__device__ __forceinline__ bool stage_barrier_or(bool flag) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)flag), "n"(NW * 32)
      : "memory");
  return r != 0;
}

template <int G, int NW, int KS, int SPLIT, typename T>
__global__ void __launch_bounds__(NW * 32, 1) cl_fwd_kernel(const __grid_constant__ ChainParams p) {
  constexpr int U = 4 * NW;
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int CS = p.CTAS, KSR = p.K16, my = (int)cl_rank(), rg = blockIdx.x / CS;
  const int H = p.H, N = p.N, u0 = my * U, tile0 = rg * p.CH, ch_n = min(p.CH, ((N + 7) >> 3) - tile0);
  const uint32_t XB = (uint32_t)KSR * 512;  // bytes of one exchange buffer
  const uint32_t xb = smem_u32(smem);       // [CH][2][KSR][512]
  float* carry = reinterpret_cast<float*>(smem + (size_t)p.CH * 2 * XB);  // [CH][h, c][NW * 32]
  uint8_t* io = reinterpret_cast<uint8_t*>(carry + p.CH * 2 * NW * 32) + w * IoBytes<T>::WARP;
  __shared__ int s_abort_;
  volatile int* s_abort = &s_abort_;

  // ---- exchange buffers: buffer 0 holds h_0 (tag 1), buffer 1 is empty (tag 0)
  if (tid == 0) *s_abort = 0;
  for (uint32_t i = tid; i < (uint32_t)p.CH * 2 * XB / 16; i += NW * 32)
    reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  {
    const T* h0 = reinterpret_cast<const T*>(p.h);
    const int units = CS * U;
    for (int i = tid; i < ch_n * 8 * units; i += NW * 32) {
      const int r = i / units, k = i - r * units, n = tile0 * 8 + r, Q = k >> 2;
      const float x = (n < N && k < H) ? ld(h0 + (long long)n * H + k) : 0.f;
      *reinterpret_cast<uint32_t*>(smem + (size_t)(r >> 3) * 2 * XB + (Q >> 2) * 512 + quad_piece(Q & 3, r & 7) +
                                   (k & 3) * 4) = xword_encode(x, 1u);
    }
  }

  // ---- weights: slot s of a warp is k-step (rot - s) mod KSR, the order in which it arrives
  const int gq = lane >> 2, q = lane & 3, rot = my * NW / 4;
  uint32_t wf[SPLIT][KS][4];
#pragma unroll
  for (int s = 0; s < KS; ++s) {
    int ks = rot - s;
    if (ks < 0) ks += KSR;
    fwd_weights<G, SPLIT, T>(p, u0 + 4 * w + (gq >> 1), gq & 1, (ks * 4 + q) * 4, s < KSR, wf[0][s], wf[SPLIT - 1][s]);
  }
  // ---- ownership of the gate stage: unit 4w + lane/8, row 2(lane & 3) + ((lane >> 2) & 1)
  const int ul = lane >> 3, row = 2 * q + (gq & 1);
  const bool odd = gq & 1;
  const int unit = u0 + 4 * w + ul;
  float bias[4];
  load_bias<G, T>(p, unit, bias);
  for (int ch = 0; ch < ch_n; ++ch) {
    const int n = (tile0 + ch) * 8 + row;
    const bool ok = n < N && unit < H;
    carry[(ch * 2 + 0) * NW * 32 + tid] = ok ? ld(reinterpret_cast<const T*>(p.h) + (long long)n * H + unit) : 0.f;
    carry[(ch * 2 + 1) * NW * 32 + tid] =
        (G == 4 && ok) ? ld(reinterpret_cast<const T*>(p.c) + (long long)n * H + unit) : 0.f;
  }
  // ---- destinations of this lane's lines: peers my + ul, my + ul + 4, ...
  constexpr int ND = 4;  // up to 16 peers
  uint32_t dst[ND];
  {
    const int Q = my * NW + w;
    const uint32_t off = (Q >> 2) * 512 + quad_piece(Q & 3, row);
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      int d = my + ul + 4 * i;
      if (d >= CS) d -= CS;
      if (d >= CS) d -= CS;
      dst[i] = ul + 4 * i < CS ? cl_mapa(xb + off, (uint32_t)d) : 0u;
    }
  }
  __syncthreads();
  cl_sync();  // every CTA's buffers are ready before anything is stored into them

  bool alive = true;
  const uint32_t lsrc = quad_piece(q, gq);
  WarpInputs<T, G, false> inputs;
  inputs.init(p, io, lane, u0 + 4 * w, G * H, 0);
#pragma unroll
  for (int i = 0; i < IO_RING - 1; ++i) inputs.fetch(p, lane, tile0, ch_n, 0, 1);
  for (int t = 0; t < p.T && alive; ++t) {
    const uint32_t rtag = ((((uint32_t)t >> 1) & 1u) ^ 1u) << 30;       // of h_t
    const uint32_t wtag = (((uint32_t)(t + 1) >> 1) & 1u) ^ 1u;         // of h_{t+1}
    for (int ch = 0; ch < ch_n; ++ch) {
      // ---- inputs of this step
      const int n0 = (tile0 + ch) * 8;
      float wv[G], m = 0.f;
      fwd_inputs<T, G>(p, inputs.take(p, io, lane, tile0, ch_n, 0, 1), t, n0 + row, unit, row, ul, wv, m);
      // ---- the product: batches of four k-steps, the next batch's loads under this one's MMAs
      float acc[2][3][4];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) acc[a][b][0] = acc[a][b][1] = acc[a][b][2] = acc[a][b][3] = 0.f;
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
        for (;;) {
          uint32_t bad = 0;
#pragma unroll
          for (int k = 0; k < 4; ++k) bad |= stale4(y[k], rtag);
          if (__all_sync(0xffffffffu, (bad & 0x40000000u) == 0)) break;
          if (__any_sync(0xffffffffu, !may_spin(spins, t0, p.sync, s_abort, 61))) { alive = false; break; }
          fetch(b0, y);
        }
        if (b0 + 4 < KS) fetch(b0 + 4, x[((b0 >> 2) + 1) & 1]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint32_t bh[2], bl[2];
          unpack_words<SPLIT>(y[k], bh, bl);
          mma_bf16(acc[k & 1][0], wf[0][b0 + k], bh[0], bh[1]);
          if (SPLIT == 2) {
            mma_bf16(acc[k & 1][1], wf[0][b0 + k], bl[0], bl[1]);
            mma_bf16(acc[k & 1][2], wf[SPLIT - 1][b0 + k], bh[0], bh[1]);
          }
        }
      }
      if (!alive) break;
      float d[4], rh[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        d[j] = SPLIT == 2 ? (acc[0][0][j] + acc[1][0][j]) +
                                ((acc[0][1][j] + acc[1][1][j]) + (acc[0][2][j] + acc[1][2][j]))
                          : acc[0][0][j] + acc[1][0][j];
      swap_gates(d, odd, rh);
      float* cy = carry + (size_t)ch * 2 * NW * 32 + tid;
      const float hp = cy[0], cp = G == 4 ? cy[NW * 32] : 0.f;
      float gate[4], h_new, c_new;
      cell_fwd<G>(rh, wv, bias, hp, cp, gate, h_new, c_new);
      if (p.has_zoneout)
        h_new = p.training ? zoneout<true>(h_new, hp, p.zoneout_prob, m)
                           : zoneout<false>(h_new, hp, p.zoneout_prob, m);
      h_new = (n0 + row < N && unit < H) ? round_to_storage<T>(h_new) : 0.f;
      if (t + 1 < p.T) {
        // ---- publish: the four units of a row meet in every lane of their group, each lane
        // serves a quarter of the peers with 16-byte stores (a warp's store fills whole lines)
        const uint32_t word = xword_encode(h_new, wtag);
        const uint32_t a1 = __shfl_xor_sync(0xffffffffu, word, 8);
        const uint32_t a2 = __shfl_xor_sync(0xffffffffu, word, 16);
        const uint32_t a3 = __shfl_xor_sync(0xffffffffu, word, 24);
        const bool o1 = ul & 1, o2 = ul & 2;
        const uint32_t e0 = o1 ? a1 : word, e1 = o1 ? word : a1, f0 = o1 ? a3 : a2, f1 = o1 ? a2 : a3;
        const uint32_t off = (uint32_t)ch * 2 * XB + ((t + 1) & 1) * XB;
#pragma unroll
        for (int i = 0; i < ND; ++i)
          if (ul + 4 * i < CS)
            cl_store(dst[i] + off, o2 ? f0 : e0, o2 ? f1 : e1, o2 ? e0 : f0, o2 ? e1 : f1);
      }
      cy[0] = h_new;
      if (G == 4) cy[NW * 32] = c_new;
      fwd_outputs<T, G>(p, io + IO_RING * IoBytes<T>::SLOT, lane, t, n0, u0 + 4 * w, row, ul, h_new, c_new, gate);
    }
  }
  __syncthreads();
  cl_sync();  // nobody leaves while a peer may still store into its shared memory
}

template <int G, int NW, int TPW, int SPLIT, typename T>
__global__ void __launch_bounds__(NW * 32, 1) cl_bwd_kernel(const __grid_constant__ ChainParams p) {
  constexpr int U = 4 * NW;
  constexpr int KSB = (G * NW + 3) / 4;  // k-steps: G * NW unit quads of own gate columns
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int CS = p.CTAS, MTR = p.K16, my = (int)cl_rank(), rg = blockIdx.x / CS;
  const int H = p.H, N = p.N, u0 = my * U, tile0 = rg * p.CH, ch_n = min(p.CH, ((N + 7) >> 3) - tile0);
  const uint32_t XB = (uint32_t)CS * NW * 128;  // one exchange buffer: [source][own quad][128]
  const uint32_t xb = smem_u32(smem);           // [CH][2][XB]
  uint8_t* gsm = smem + (size_t)p.CH * 2 * XB;  // gate gradients, B operand: [2][KSB][512]
  float* carry = reinterpret_cast<float*>(gsm + 2 * KSB * 512);  // [CH][dh, dc, c][NW * 32]
  uint8_t* io = reinterpret_cast<uint8_t*>(carry + p.CH * 3 * NW * 32) + w * IoBytes<T>::WARP;
  __shared__ int s_abort_;
  volatile int* s_abort = &s_abort_;
  if (tid == 0) *s_abort = 0;
  for (uint32_t i = tid; i < ((uint32_t)p.CH * 2 * XB + 2 * KSB * 512) / 16; i += NW * 32)
    reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);

  // ---- weights: slot i of warp w is output tile (w + NW i + rot) mod MTR; tile row m is unit
  // m & 1 (+ 2 for m >= 8) of unit quad (m & 7) / 2
  const int gq = lane >> 2, q = lane & 3, rot = my * NW / 4;
  uint32_t wf[SPLIT][TPW][KSB][4];
  uint32_t dst[TPW];
#pragma unroll
  for (int i = 0; i < TPW; ++i) {
    const int Lt = w + NW * i;
    int tile = Lt + rot;
    while (tile >= MTR) tile -= MTR;
    const int Q = tile * 4 + (gq >> 1), d = Q / NW, qw = Q - d * NW;
    const bool live = Lt < MTR;
    dst[i] = (live && d < CS)
                 ? cl_mapa(xb + (uint32_t)(my * NW + qw) * 128 + ((gq & 1) * 4 + q) * 16, (uint32_t)d) : 0u;
#pragma unroll
    for (int kk = 0; kk < KSB; ++kk) {
      const int lq = kk * 4 + q, gate = lq / NW, wq = lq - gate * NW;
      bwd_weights<G, SPLIT, T>(p, Q * 4 + (gq & 1), gate, u0 + 4 * wq, live, wf[0][i][kk], wf[SPLIT - 1][i][kk]);
    }
  }
  // ---- ownership: piece c8 = lane & 7 of the quad's line (unit bit c8 >> 2, rows 2(c8 & 3), +1);
  // word sub = lane >> 3 of it (second unit pair for sub >= 2, second row for odd sub)
  const int sub = lane >> 3, c8 = lane & 7;
  const int row = 2 * (c8 & 3) + (sub & 1), ul = (c8 >> 2) + 2 * (sub >> 1);
  const int unit = u0 + 4 * w + ul;
  for (int ch = 0; ch < ch_n; ++ch) {
    const int n = (tile0 + ch) * 8 + row;
    const bool ok = n < N && unit < H;
    const long long o = (long long)n * H + unit;
    float* cy = carry + (size_t)ch * 3 * NW * 32 + tid;
    const bool given = ok && !p.zero_init;
    cy[0] = given ? ld(reinterpret_cast<const T*>(p.dh) + o) : 0.f;
    cy[NW * 32] = (G == 4 && given) ? ld(reinterpret_cast<const T*>(p.dc) + o) : 0.f;
    cy[2 * NW * 32] = (G == 4 && ok) ? ld(reinterpret_cast<const T*>(p.c) + (long long)p.T * N * H + o) : 0.f;
  }
  float acc_b[4] = {0.f, 0.f, 0.f, 0.f};
  bool alive = true;
  __syncthreads();
  cl_sync();

  // Adds the recurrent part of dh published at production step s: lane group `sub` sums its
  // quarter of the sources, the four groups meet in shuffles, the lane keeps its own word.
  auto gather = [&](int ch, int s, float& dh_c) {
    const uint32_t want = (((uint32_t)s >> 1) & 1u) ^ 1u;
    const uint32_t src = xb + (uint32_t)ch * 2 * XB + (s & 1) * XB + (uint32_t)(w * 128 + c8 * 16);
    uint4 y[TPW];  // (TPW = ceil(CS / 4), the sources per lane)
    long long t0 = 0;
    unsigned int spins = 0;
    for (;;) {
      uint32_t bad = 0;
#pragma unroll
      for (int k = 0; k < TPW; ++k) {
        const int j = sub * TPW + k;
        if (j < CS) y[k] = cl_poll(src + (uint32_t)(j * NW) * 128);
        else y[k] = make_uint4(want, want, want, want);
      }
#pragma unroll
      for (int k = 0; k < TPW; ++k) bad |= stale4(y[k], want);
      if (__all_sync(0xffffffffu, (bad & 1u) == 0)) break;
      if (__any_sync(0xffffffffu, !may_spin(spins, t0, p.sync, s_abort, 62))) { alive = false; break; }
    }
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < TPW; ++k) {
      s4[0] += fword_value(y[k].x); s4[1] += fword_value(y[k].y);
      s4[2] += fword_value(y[k].z); s4[3] += fword_value(y[k].w);
    }
    dh_c += gather_reduce(s4, sub);
  };

  const bool zo = p.has_zoneout != 0, second = (c8 & 4) != 0;
  int gpar = 0;
  WarpInputs<T, 4, true> inputs;
  inputs.init(p, io, lane, u0 + 4 * w, 4 * H, 0);
#pragma unroll
  for (int i = 0; i < IO_RING - 1; ++i) inputs.fetch(p, lane, tile0, ch_n, 0, 1);
  for (int ti = 0; ti < p.T && alive; ++ti) {
    for (int ch = 0; ch < ch_n; ++ch) {
      const int n0 = (tile0 + ch) * 8, t = p.T - 1 - ti;
      const bool ok = n0 + row < N && unit < H;
      float gv[4], dhv, prev, m, dcv;
      bwd_inputs<T, G>(p, inputs.take(p, io, lane, tile0, ch_n, 0, 1), t, n0 + row, unit, row, ul, gv, dhv, prev, m,
                       dcv);
      float* cy = carry + (size_t)ch * 3 * NW * 32 + tid;
      float dh_c = cy[0], dc_c = G == 4 ? cy[NW * 32] : 0.f;
      const float cnew = G == 4 ? cy[2 * NW * 32] : 0.f;
      if (ti > 0) gather(ch, ti - 1, dh_c);
      float dg[4];
      cell_bwd<G>(gv, prev, cnew, dhv + dh_c, dcv, zo, m, dh_c, dc_c, dg);
      if (!ok) dg[0] = dg[1] = dg[2] = dg[3] = dh_c = dc_c = 0.f;
      uint8_t* gb = gsm + gpar * KSB * 512;
      store_gate_operand<G, NW>(gb, dg, w, row, sub, second);
      // (the gate gradients are double-buffered: one barrier per step and chain)
      if (stage_barrier_or<NW>(!alive)) { alive = false; break; }
      gpar ^= 1;
      // ---- partial dh of every unit
      uint4 y[KSB];
#pragma unroll
      for (int kk = 0; kk < KSB; ++kk) y[kk] = *reinterpret_cast<const uint4*>(gb + kk * 512 + quad_piece(q, gq));
      const uint32_t tag = (((uint32_t)ti >> 1) & 1u) ^ 1u;
      const uint32_t off = (uint32_t)ch * 2 * XB + (ti & 1) * XB;
#pragma unroll
      for (int i0 = 0; i0 < TPW; i0 += 2) {
        float acc[2][2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) acc[i][e][0] = acc[i][e][1] = acc[i][e][2] = acc[i][e][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < KSB; ++kk) {
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (i0 + i < TPW) mma_bf16(acc[i][0], wf[0][(i0 + i) % TPW][kk], y[kk].x, y[kk].y);
          if (SPLIT == 2) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
              if (i0 + i < TPW) mma_bf16(acc[i][1], wf[0][(i0 + i) % TPW][kk], y[kk].z, y[kk].w);
#pragma unroll
            for (int i = 0; i < 2; ++i)
              if (i0 + i < TPW) mma_bf16(acc[i][1], wf[SPLIT - 1][(i0 + i) % TPW][kk], y[kk].x, y[kk].y);
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (i0 + i < TPW && dst[(i0 + i) % TPW])
            cl_store(dst[(i0 + i) % TPW] + off, fword_encode(acc[i][0][0] + acc[i][1][0], tag),
                     fword_encode(acc[i][0][1] + acc[i][1][1], tag), fword_encode(acc[i][0][2] + acc[i][1][2], tag),
                     fword_encode(acc[i][0][3] + acc[i][1][3], tag));
      }
      // ---- off the chain: carries, bias sums, outputs
      cy[0] = dh_c;
      if (G == 4) {
        cy[NW * 32] = dc_c;
        cy[2 * NW * 32] = prev;
      }
#pragma unroll
      for (int g = 0; g < 4; ++g) acc_b[g] += dg[g];
      bwd_outputs<T, G>(p, io + IO_RING * IoBytes<T>::SLOT, lane, t, n0, u0 + 4 * w, row, ul, dg);
    }
  }
  // ---- what is left of dh: the recurrent part of step 0, then the carries go out
  for (int ch = 0; ch < ch_n && alive; ++ch) {
    const int n = (tile0 + ch) * 8 + row;
    float* cy = carry + (size_t)ch * 3 * NW * 32 + tid;
    float dh_c = cy[0];
    gather(ch, p.T - 1, dh_c);
    if (alive && n < N && unit < H) {
      st(reinterpret_cast<T*>(p.dh) + (long long)n * H + unit, dh_c);
      if (G == 4) st(reinterpret_cast<T*>(p.dc) + (long long)n * H + unit, cy[NW * 32]);
    }
  }
  // ---- bias gradients of this row group: sum over the eight rows
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    float s = acc_b[g];
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    if (unit < H && row == 0) p.db_part[(size_t)rg * 4 * H + (size_t)g * H + unit] = s;
  }
  __syncthreads();
  cl_sync();
}

}  // namespace rec
}  // namespace hb
