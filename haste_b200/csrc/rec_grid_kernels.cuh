// Persistent LSTM / GRU recurrence over the whole grid, sm_100a: the sizes that do not fit one
// thread-block cluster (rec_cluster_kernels.cuh) - hidden sizes up to 1024, or many batch rows.
//
// Same arithmetic as the cluster kernels - weights as the A operand of mma.m16n8k16 in registers
// for the whole pass, the batch in chains of eight rows - with the hand-off through L2:
//
// * Grid = (hidden slices of U = 4 NMT units) x (row groups), one CTA of sixteen warps per SM,
//   cooperative launch.  R is read from HBM once per pass.
// * An exchange through L2 takes 1100 cycles from the publishing store to the polling load that
//   sees it, about as long as everything else in a step.  A CTA carries its rows as CH
//   independent chains of eight: while one chain's words travel, the others are worked on, by
//   warps of different roles:
//     forward   8 product warps (K split over them; a warp polls the words of its own K range -
//               16-byte loads that are the B fragments already - and leaves a partial tile in a
//               shared-memory ring) and 8 finishing warps (add the partials, apply the cell,
//               publish);
//     backward  8 gather warps (add the partial dh in a fixed order, apply the cell's gradient,
//               put the gate gradients into a ring as the B operand) and 8 product warps (multiply
//               them against their share of the output units, publish).
//   The second kind takes a chain's latency (about 1700 cycles) rather than its arithmetic, so it
//   comes in groups that take the chains in turn.  setmaxnreg moves registers to the product
//   warps, which hold R.
// * Words carry their own readiness as in recurrent_common.cuh.
#pragma once

#include "rec_chain.cuh"

namespace hb {
namespace rec {

constexpr int GL_WARPS = 8;               // product warps
constexpr int GL_THREADS = 2 * GL_WARPS * 32;  // + 8 finishing / gather warps
constexpr int GL_GRING = 4;               // backward: gate-gradient tiles in flight
// Register split: 512 threads x 128 at launch = 256 x (P + F).
constexpr int GL_FWD_P = 192, GL_FWD_F = 64, GL_BWD_P = 176, GL_BWD_F = 80;
static_assert(GL_FWD_P + GL_FWD_F == 256 && GL_BWD_P + GL_BWD_F == 256,
              "the split must be what the block was launched with");

// Layers beyond 512 units of fp32 or fp16 storage, 16 units per CTA: R's second plane lies in shared memory
// (128 KB at 1024 units) because both do not fit the registers.
template <int NMT, int TILES, int SPLIT>
constexpr bool gl_lo_in_smem() { return SPLIT == 2 && NMT == 4 && TILES > 4; }

template <int N>
__device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

__device__ __forceinline__ void gl_publish(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void gl_publish4(uint32_t* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}

// Exchange words, forward: [2][row tiles][K16][128] (a 128-byte line per quad of units).
template <int G, int NMT, int KSW, int SPLIT, typename T>
__global__ void __launch_bounds__(GL_THREADS, 1) gl_fwd_kernel(const __grid_constant__ ChainParams p) {
  constexpr int U = 4 * NMT, GROUPS = GL_WARPS / NMT;
  constexpr int PART = GL_WARPS * NMT * 32;
  constexpr bool LO = gl_lo_in_smem<NMT, KSW, SPLIT>();
  constexpr int RP = LO ? 1 : SPLIT;  // planes of R in registers
  extern __shared__ __align__(16) uint8_t smem[];
  float4* part = reinterpret_cast<float4*>(smem);                                // [ring][warp][NMT][lane]
  uint4* lo = reinterpret_cast<uint4*>(part + p.ring * PART);                    // LO: [warp][NMT][KSW][lane]
  float* carry = reinterpret_cast<float*>(lo + (LO ? PART * KSW : 0));           // [CH][h, c][NMT * 32]
  uint64_t* barp = reinterpret_cast<uint64_t*>(carry + p.CH * 2 * NMT * 32);     // full[ring], empty[ring]
  const uint32_t pbar = smem_u32(barp);
  uint8_t* io_base = reinterpret_cast<uint8_t*>(barp + 2 * p.ring);              // per finishing warp
  __shared__ int s_abort_;
  volatile int* s_abort = &s_abort_;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, q = lane & 3;
  const int hs = blockIdx.x % p.CTAS, rg = blockIdx.x / p.CTAS;
  const int H = p.H, N = p.N, u0 = hs * U, tile0 = rg * p.CH, tiles = (N + 7) >> 3;
  const int ch_n = min(p.CH, tiles - tile0);
  if (tid == 0) {
    *s_abort = 0;
    for (int i = 0; i < p.ring; ++i) {
      mb_init(pbar + 8 * i, GL_WARPS);         // full: every warp's partial is written
      mb_init(pbar + 8 * (p.ring + i), NMT);   // empty: the finishing warps have read it
    }
  }
  __syncthreads();
  int slot = 0;
  uint32_t phase = 0;
  auto next_slot = [&]() {
    if (++slot == p.ring) { slot = 0; phase ^= 1u; }
  };

  if (w < GL_WARPS) {
    // ------------------------------------------------------------------ product warps
    reg_inc<GL_FWD_P>();
    uint32_t wf[RP][NMT][KSW][4];
    lo += w * NMT * KSW * 32 + lane;  // this lane's
#pragma unroll
    for (int mt = 0; mt < NMT; ++mt)
#pragma unroll
      for (int s = 0; s < KSW; ++s)
      {
        uint32_t l[4];
        fwd_weights<G, SPLIT, T>(p, u0 + 4 * mt + (gq >> 1), gq & 1, ((w * KSW + s) * 4 + q) * 4, true, wf[0][mt][s], l);
        if (LO) lo[(mt * KSW + s) * 32] = make_uint4(l[0], l[1], l[2], l[3]);
        else if (SPLIT == 2) {
#pragma unroll
          for (int a = 0; a < 4; ++a) wf[RP - 1][mt][s][a] = l[a];
        }
      }
    // words of h_t for the rows of one chain, this warp's K range.  Quads and rows that do not
    // exist count as ready.
    const int kq = w * KSW * 4 + q;  // first quad of this lane
    const uint32_t* src0 = p.xbuf + ((size_t)tile0 * p.K16 + w * KSW) * 128 + q * 32 + gq * 4;
    const uint32_t xtile = (uint32_t)p.K16 * 128, xpar = (uint32_t)tiles * xtile;
    const int nrow = N - tile0 * 8 - gq;  // chain ch has this lane's row if ch * 8 < nrow
    auto fetch = [&](uint32_t par, uint32_t wt, int ch, uint4 (&y)[KSW]) {
      const uint32_t* src = src0 + par * xpar + (uint32_t)ch * xtile;
      const bool rok = ch * 8 < nrow;
#pragma unroll
      for (int s = 0; s < KSW; ++s)
        y[s] = (rok && kq + s * 4 < p.CTAS * NMT) ? ld_relaxed_u32x4(src + s * 128) : make_uint4(wt, wt, wt, wt);
    };
    auto tag_of = [](int t) { return ((((uint32_t)t >> 1) & 1u) ^ 1u) << 30; };
    uint4 y[KSW];
    // (a warp beyond the end of K waits for no words, so only the ring holds it back)
    const bool throttle = p.throttle || w * KSW * 4 >= p.CTAS * NMT;
    bool alive = true;
    for (int t = 0; t < p.T && alive; ++t) {
      const uint32_t wt = tag_of(t);
      for (int ch = 0; ch < ch_n; ++ch) {
        fetch(t & 1, wt, ch, y);
        long long t0 = 0;
        unsigned int spins = 0;
        for (;;) {
          uint32_t bad = 0;
#pragma unroll
          for (int s = 0; s < KSW; ++s) bad |= stale4(y[s], wt);
          if (__all_sync(0xffffffffu, (bad & 0x40000000u) == 0)) break;
          if (__any_sync(0xffffffffu, !may_spin(spins, t0, p.sync, s_abort, 63))) { alive = false; break; }
          fetch(t & 1, wt, ch, y);
        }
        if (!alive) break;
        float acc[NMT][4];
#pragma unroll
        for (int mt = 0; mt < NMT; ++mt) acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.f;
#pragma unroll
        for (int s = 0; s < KSW; ++s) {
          uint32_t bh[2], bl[2];
          unpack_words<SPLIT>(y[s], bh, bl);
#pragma unroll
          for (int mt = 0; mt < NMT; ++mt) mma_bf16(acc[mt], wf[0][mt][s], bh[0], bh[1]);
          if (SPLIT == 2) {
#pragma unroll
            for (int mt = 0; mt < NMT; ++mt) mma_bf16(acc[mt], wf[0][mt][s], bl[0], bl[1]);
#pragma unroll
            for (int mt = 0; mt < NMT; ++mt) {
              if (LO) mma_bf16(acc[mt], lo[(mt * KSW + s) * 32], bh[0], bh[1]);
              else mma_bf16(acc[mt], wf[RP - 1][mt][s], bh[0], bh[1]);
            }
          }
        }
        // partial tile into the ring.  (A ring of two slots per chain needs no look at `empty`:
        // a slot comes round after a step, and h of that step took the partial before it.)
        if (throttle &&
            !mb_wait_warp(pbar + 8 * (p.ring + slot), phase ^ 1u, p.sync, s_abort, 64)) { alive = false; break; }
        float4* pw = part + slot * PART + w * NMT * 32 + lane;
#pragma unroll
        for (int mt = 0; mt < NMT; ++mt) pw[mt * 32] = make_float4(acc[mt][0], acc[mt][1], acc[mt][2], acc[mt][3]);
        __syncwarp();
        if (lane == 0) mb_arrive(pbar + 8 * slot);
        next_slot();
      }
    }
  } else {
    // ------------------------------------------------------------------ finishing warps
    // warp f finishes tile f % NMT of every GROUPS-th chain
    reg_dec<GL_FWD_F>();
    const int f = w - GL_WARPS, grp = f / NMT, mtf = f % NMT;
    const int ul = lane >> 3, row = 2 * q + (gq & 1);
    const bool odd = gq & 1;
    const int unit = u0 + 4 * mtf + ul;
    const int Q = hs * NMT + mtf;
    uint32_t* xdst = p.xbuf + (size_t)(Q >> 2) * 128 + (Q & 3) * 32 + row * 4 + ul;
    const size_t xtile = (size_t)p.K16 * 128;
    float bias[4];
    load_bias<G, T>(p, unit, bias);
    for (int ch = grp; ch < ch_n; ch += GROUPS) {
      const int n = (tile0 + ch) * 8 + row;
      const bool ok = n < N && unit < H;
      float* cy = carry + (size_t)ch * 2 * NMT * 32 + mtf * 32 + lane;
      const float h0 = ok ? ld(reinterpret_cast<const T*>(p.h) + (long long)n * H + unit) : 0.f;
      if (n < N) gl_publish(xdst + (size_t)(tile0 + ch) * xtile, xword_encode(h0, 1u));
      cy[0] = h0;
      cy[NMT * 32] = (G == 4 && ok) ? ld(reinterpret_cast<const T*>(p.c) + (long long)n * H + unit) : 0.f;
    }
    uint8_t* io = io_base + f * IoBytes<T>::WARP;
    WarpInputs<T, G, false> inputs;
    inputs.init(p, io, lane, u0 + 4 * mtf, G * H, grp);
    if (grp < ch_n) {
#pragma unroll
      for (int i = 0; i < IO_RING - 1; ++i) inputs.fetch(p, lane, tile0, ch_n, grp, GROUPS);
    }
    bool alive = true;
    for (int t = 0; t < p.T && alive; ++t) {
      const uint32_t wtag = (((uint32_t)(t + 1) >> 1) & 1u) ^ 1u;  // of h_{t+1}
      for (int ch = 0; ch < ch_n; ++ch, next_slot()) {
        if (GROUPS > 1 && ch % GROUPS != grp) continue;
        const int tile = tile0 + ch, n = tile * 8 + row;
        float wv[G], m = 0.f;
        fwd_inputs<T, G>(p, inputs.take(p, io, lane, tile0, ch_n, grp, GROUPS), t, n, unit, row, ul, wv, m);
        float* cy = carry + (size_t)ch * 2 * NMT * 32 + mtf * 32 + lane;
        const float hp = cy[0], cp = G == 4 ? cy[NMT * 32] : 0.f;
        if (!mb_wait_warp(pbar + 8 * slot, phase, p.sync, s_abort, 65)) { alive = false; break; }
        const float4* pr = part + slot * PART + mtf * 32 + lane;
        float4 v[GL_WARPS];
#pragma unroll
        for (int k = 0; k < GL_WARPS; ++k) v[k] = pr[k * NMT * 32];
        float d[4], rh[4];
        d[0] = ((v[0].x + v[1].x) + (v[2].x + v[3].x)) + ((v[4].x + v[5].x) + (v[6].x + v[7].x));
        d[1] = ((v[0].y + v[1].y) + (v[2].y + v[3].y)) + ((v[4].y + v[5].y) + (v[6].y + v[7].y));
        d[2] = ((v[0].z + v[1].z) + (v[2].z + v[3].z)) + ((v[4].z + v[5].z) + (v[6].z + v[7].z));
        d[3] = ((v[0].w + v[1].w) + (v[2].w + v[3].w)) + ((v[4].w + v[5].w) + (v[6].w + v[7].w));
        swap_gates(d, odd, rh);
        float gate[4], h_new, c_new;
        cell_fwd<G>(rh, wv, bias, hp, cp, gate, h_new, c_new);
        if (p.has_zoneout)
          h_new = p.training ? zoneout<true>(h_new, hp, p.zoneout_prob, m)
                             : zoneout<false>(h_new, hp, p.zoneout_prob, m);
        h_new = unit < H ? round_to_storage<T>(h_new) : 0.f;
        if (t + 1 < p.T && n < N) gl_publish(xdst + ((size_t)((t + 1) & 1) * tiles + tile) * xtile, xword_encode(h_new, wtag));
        // ---- off the chain
        cy[0] = h_new;
        if (G == 4) cy[NMT * 32] = c_new;
        if (lane == 0) mb_arrive(pbar + 8 * (p.ring + slot));
        fwd_outputs<T, G>(p, io + IO_RING * IoBytes<T>::SLOT, lane, t, tile * 8, u0 + 4 * mtf, row, ul, h_new, c_new,
                          gate);
      }
    }
  }
}

// Exchange words, backward: [2][row tiles][destination CTA][source CTA][NMT][32].
template <int G, int NMT, int TPW, int SPLIT, typename T>
__global__ void __launch_bounds__(GL_THREADS, 1) gl_bwd_kernel(const __grid_constant__ ChainParams p) {
  constexpr int U = 4 * NMT;
  constexpr int KSB = (G * NMT + 3) / 4;  // k-steps of the CTA's own gate columns
  constexpr int SP = 4 / NMT;             // parts the sources of a gather are split into
  constexpr bool LO = gl_lo_in_smem<NMT, TPW, SPLIT>();
  constexpr int RP = LO ? 1 : SPLIT;
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t* gsm = smem;                                                    // [ring][KSB][512]
  uint4* lo = reinterpret_cast<uint4*>(gsm + GL_GRING * KSB * 512);       // LO: [warp][TPW][KSB][lane]
  float* red = reinterpret_cast<float*>(lo + (LO ? GL_WARPS * TPW * KSB * 32 : 0));  // [2 groups][2][SP][NMT * 32]
  float* carry = red + 4 * SP * NMT * 32;                                 // [CH][dh, dc, c][NMT * 32]
  uint64_t* barp = reinterpret_cast<uint64_t*>(carry + p.CH * 3 * NMT * 32);
  const uint32_t gbar = smem_u32(barp);                                   // full, empty, parts met (a group each)
  uint8_t* io_base = reinterpret_cast<uint8_t*>(barp + 2 * GL_GRING + 2); // per gather warp
  __shared__ int s_abort_;
  volatile int* s_abort = &s_abort_;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, q = lane & 3;
  const int nHS = p.CTAS, hs = blockIdx.x % nHS, rg = blockIdx.x / nHS;
  const int H = p.H, N = p.N, u0 = hs * U, tile0 = rg * p.CH, tiles = (N + 7) >> 3;
  const int ch_n = min(p.CH, tiles - tile0);
  if (tid == 0) {
    *s_abort = 0;
    for (int i = 0; i < GL_GRING; ++i) {
      mb_init(gbar + 8 * i, NMT);
      mb_init(gbar + 8 * (GL_GRING + i), GL_WARPS);
    }
    mb_init(gbar + 8 * (2 * GL_GRING), 4);
    mb_init(gbar + 8 * (2 * GL_GRING + 1), 4);
  }
  for (int i = tid; i < GL_GRING * KSB * 512 / 16; i += GL_THREADS)
    reinterpret_cast<uint4*>(gsm)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const size_t line = (size_t)NMT * 32;
  RingPos<GL_GRING> gp;

  if (w < GL_WARPS) {
    // ------------------------------------------------------------------ product warps
    // output tiles w, w + 8, ... (rotated by the CTA's index, so that the CTAs store to different
    // destinations at a time); tile row m is unit m & 1 (+ 2 for m >= 8) of quad (m & 7) / 2
    reg_inc<GL_BWD_P>();
    const int rot = hs % p.K16;
    uint32_t wf[RP][TPW][KSB][4];
    lo += w * TPW * KSB * 32 + lane;
    uint32_t doff[TPW];  // word offset of this lane's piece, ~0: nothing to store
#pragma unroll
    for (int i = 0; i < TPW; ++i) {
      const int Lt = w + GL_WARPS * i;
      const bool live = Lt < p.K16;
      const int tile = Lt + rot < p.K16 ? Lt + rot : Lt + rot - p.K16;
      const int Q = tile * 4 + (gq >> 1), d = Q / NMT, qw = Q - d * NMT;
      doff[i] = live && d < nHS ? (uint32_t)(((d * nHS + hs) * NMT + qw) * 32 + ((gq & 1) * 4 + q) * 4) : ~0u;
#pragma unroll
      for (int kk = 0; kk < KSB; ++kk) {
        const int lq = kk * 4 + q, gate = lq / NMT, wq = lq - gate * NMT;
        uint32_t l[4];
        bwd_weights<G, SPLIT, T>(p, Q * 4 + (gq & 1), gate, u0 + 4 * wq, live, wf[0][i][kk], l);
        if (LO) lo[(i * KSB + kk) * 32] = make_uint4(l[0], l[1], l[2], l[3]);
        else if (SPLIT == 2) {
#pragma unroll
          for (int a = 0; a < 4; ++a) wf[RP - 1][i][kk][a] = l[a];
        }
      }
    }
    bool alive = true;
    for (int ti = 0; ti < p.T && alive; ++ti) {
      const uint32_t tag = (((uint32_t)ti >> 1) & 1u) ^ 1u;
      for (int ch = 0; ch < ch_n; ++ch, gp.next()) {
        const int tile = tile0 + ch;
        if (!mb_wait_warp(gbar + 8 * gp.slot, gp.phase, p.sync, s_abort, 68)) { alive = false; break; }
        uint4 y[KSB];
        const uint8_t* gb = gsm + gp.slot * KSB * 512;
#pragma unroll
        for (int kk = 0; kk < KSB; ++kk) y[kk] = *reinterpret_cast<const uint4*>(gb + kk * 512 + quad_piece(q, gq));
        uint32_t* dst = p.xbuf + ((size_t)(ti & 1) * tiles + tile) * nHS * nHS * line;
        const bool send = tile * 8 + 2 * q < N;  // at least one of the piece's two rows exists
#pragma unroll
        for (int i0 = 0; i0 < TPW; i0 += 4) {
          float acc[4][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll
          for (int kk = 0; kk < KSB; ++kk) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (i0 + i < TPW) mma_bf16(acc[i], wf[0][(i0 + i) % TPW][kk], y[kk].x, y[kk].y);
            if (SPLIT == 2) {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (i0 + i < TPW) mma_bf16(acc[i], wf[0][(i0 + i) % TPW][kk], y[kk].z, y[kk].w);
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (i0 + i < TPW) {
                  if (LO) mma_bf16(acc[i], lo[((i0 + i) * KSB + kk) * 32], y[kk].x, y[kk].y);
                  else mma_bf16(acc[i], wf[RP - 1][(i0 + i) % TPW][kk], y[kk].x, y[kk].y);
                }
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (i0 + i < TPW && send && doff[(i0 + i) % TPW] != ~0u)
              gl_publish4(dst + doff[(i0 + i) % TPW], fword_encode(acc[i][0], tag), fword_encode(acc[i][1], tag),
                          fword_encode(acc[i][2], tag), fword_encode(acc[i][3], tag));
        }
        if (lane == 0) mb_arrive(gbar + 8 * (GL_GRING + gp.slot));
      }
    }
  } else {
    // ------------------------------------------------------------------ gather and gate stage
    // two groups of four warps take the chains in turn; warp = (quad, part of the sources), lanes as
    // in the cluster kernel
    reg_dec<GL_BWD_F>();
    const int f = w - GL_WARPS, grp = f >> 2, quad = (f & 3) % NMT, prt = (f & 3) / NMT;
    const bool leader = prt == 0;
    const int sub = lane >> 3, c8 = lane & 7;
    const int row = 2 * (c8 & 3) + (sub & 1), ul = (c8 >> 2) + 2 * (sub >> 1);
    const int unit = u0 + 4 * quad + ul;
    const bool zo = p.has_zoneout != 0, second = (c8 & 4) != 0;
    const int NPS = (nHS + 4 * SP - 1) / (4 * SP);  // sources per lane
    const int j0 = (prt * 4 + sub) * NPS, nj = max(0, min(NPS, nHS - j0));
    if (leader)
      for (int ch = grp; ch < ch_n; ch += 2) {
        const int n = (tile0 + ch) * 8 + row;
        const bool ok = n < N && unit < H;
        const long long o = (long long)n * H + unit;
        float* cy = carry + (size_t)ch * 3 * NMT * 32 + quad * 32 + lane;
        const bool given = ok && !p.zero_init;
        cy[0] = given ? ld(reinterpret_cast<const T*>(p.dh) + o) : 0.f;
        cy[NMT * 32] = (G == 4 && given) ? ld(reinterpret_cast<const T*>(p.dc) + o) : 0.f;
        cy[2 * NMT * 32] = (G == 4 && ok) ? ld(reinterpret_cast<const T*>(p.c) + (long long)p.T * N * H + o) : 0.f;
      }
    float acc_b[4] = {0.f, 0.f, 0.f, 0.f};
    bool alive = true;
    uint32_t rpar = 0;
    const uint32_t* src0 = p.xbuf + ((size_t)hs * nHS + j0) * line + quad * 32 + c8 * 4;
    const size_t tile_words = (size_t)nHS * nHS * line;
    // eight sources of one chain's partials of production step s, b .. b+7
    auto fetch = [&](int ch, int s, int b, uint4 (&y)[8]) {
      const uint32_t want = (((uint32_t)s >> 1) & 1u) ^ 1u;
      const uint32_t* src = src0 + ((size_t)(s & 1) * tiles + tile0 + ch) * tile_words + (size_t)b * line;
      const bool need = (tile0 + ch) * 8 + 2 * (c8 & 3) < N;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        y[k] = (need && b + k < nj) ? ld_relaxed_u32x4(src + (size_t)k * line) : make_uint4(want, want, want, want);
    };
    auto gather = [&](int ch, int s, float& dh_c) {
      uint4 y[8];
      const uint32_t want = (((uint32_t)s >> 1) & 1u) ^ 1u;
      float s4[4] = {0.f, 0.f, 0.f, 0.f};
      for (int b = 0; b < NPS && alive; b += 8) {
        fetch(ch, s, b, y);
        long long t0 = 0;
        unsigned int spins = 0;
        for (;;) {
          uint32_t bad = 0;
#pragma unroll
          for (int k = 0; k < 8; ++k) bad |= stale4(y[k], want);
          if (__all_sync(0xffffffffu, (bad & 1u) == 0)) break;
          if (__any_sync(0xffffffffu, !may_spin(spins, t0, p.sync, s_abort, 66))) { alive = false; break; }
          fetch(ch, s, b, y);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          s4[0] += fword_value(y[k].x); s4[1] += fword_value(y[k].y);
          s4[2] += fword_value(y[k].z); s4[3] += fword_value(y[k].w);
        }
      }
      float v = gather_reduce(s4, sub);
      if (SP > 1) {  // the parts meet in shared memory (double-buffered)
        float* rd = red + (grp * 2 + (int)rpar) * SP * NMT * 32 + quad * 32 + lane;
        rd[prt * NMT * 32] = v;
        __syncwarp();
        if (lane == 0) mb_arrive(gbar + 8 * (2 * GL_GRING + grp));
        if (!mb_wait_warp(gbar + 8 * (2 * GL_GRING + grp), rpar, p.sync, s_abort, 69)) alive = false;
        rpar ^= 1u;
        v = 0.f;
#pragma unroll
        for (int k = 0; k < SP; ++k) v += rd[k * NMT * 32];
      }
      dh_c += v;
    };

    uint8_t* io = io_base + f * IoBytes<T>::WARP;
    WarpInputs<T, 4, true> inputs;
    inputs.init(p, io, lane, u0 + 4 * quad, 4 * H, grp);
    if (leader && grp < ch_n) {
#pragma unroll
      for (int i = 0; i < IO_RING - 1; ++i) inputs.fetch(p, lane, tile0, ch_n, grp, 2);
    }
    for (int ti = 0; ti < p.T && alive; ++ti) {
      for (int ch = 0; ch < ch_n; ++ch, gp.next()) {
        if ((ch & 1) != grp) continue;
        const int n0 = (tile0 + ch) * 8, t = p.T - 1 - ti;
        const bool ok = n0 + row < N && unit < H;
        float gv[4], dcv = 0.f, m = 1.f, dhv = 0.f, prev = 0.f, cnew = 0.f, dh_c = 0.f, dc_c = 0.f;
        float* cy = carry + (size_t)ch * 3 * NMT * 32 + quad * 32 + lane;
        if (leader) {
          bwd_inputs<T, G>(p, inputs.take(p, io, lane, tile0, ch_n, grp, 2), t, n0 + row, unit, row, ul, gv, dhv, prev,
                           m, dcv);
          dh_c = cy[0];
          if (G == 4) { dc_c = cy[NMT * 32]; cnew = cy[2 * NMT * 32]; }
        }
        if (ti > 0) {
          gather(ch, ti - 1, dh_c);
          if (!alive) break;
        }
        if (leader) {
          float dg[4];
          cell_bwd<G>(gv, prev, cnew, dhv + dh_c, dcv, zo, m, dh_c, dc_c, dg);
          if (!ok) dg[0] = dg[1] = dg[2] = dg[3] = dh_c = dc_c = 0.f;
          if (!mb_wait_warp(gbar + 8 * (GL_GRING + gp.slot), gp.phase ^ 1u, p.sync, s_abort, 67)) { alive = false; break; }
          store_gate_operand<G, NMT>(gsm + gp.slot * KSB * 512, dg, quad, row, sub, second);
          __syncwarp();
          if (lane == 0) mb_arrive(gbar + 8 * gp.slot);
          // ---- off the chain
          cy[0] = dh_c;
          if (G == 4) { cy[NMT * 32] = dc_c; cy[2 * NMT * 32] = prev; }
#pragma unroll
          for (int g = 0; g < 4; ++g) acc_b[g] += dg[g];
          bwd_outputs<T, G>(p, io + IO_RING * IoBytes<T>::SLOT, lane, t, n0, u0 + 4 * quad, row, ul, dg);
        }
      }
    }
    // ---- what is left of dh: the recurrent part of step 0, then the carries go out
    for (int ch = grp; ch < ch_n && alive; ch += 2) {
      const int n = (tile0 + ch) * 8 + row;
      float* cy = carry + (size_t)ch * 3 * NMT * 32 + quad * 32 + lane;
      float dh_c = leader ? cy[0] : 0.f;
      gather(ch, p.T - 1, dh_c);
      if (alive && leader && n < N && unit < H) {
        st(reinterpret_cast<T*>(p.dh) + (long long)n * H + unit, dh_c);
        if (G == 4) st(reinterpret_cast<T*>(p.dc) + (long long)n * H + unit, cy[NMT * 32]);
      }
    }
    // ---- bias gradients of this row group: over the eight rows (a row of partials per group)
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      float s = acc_b[g];
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 8);
      if (leader && row == 0 && unit < H)
        p.db_part[((size_t)rg * 2 + grp) * 4 * H + (size_t)g * H + unit] = s;
    }
  }
}

}  // namespace rec
}  // namespace hb
