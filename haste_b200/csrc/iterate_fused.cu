// One time step of LSTM / GRU in ONE launch: x.W + h.R, biases, gate functions, state update
// and zoneout fused, for single-step calls of the layers and for the reference's per-step Iterate
// API (lib/haste/lstm.h:73-86, lib/haste/gru.h:72-84; lib/lstm_forward_gpu.cu.cc:141-208,
// lib/gru_forward_gpu.cu.cc:160-212), which the reference runs as two cuBLAS calls and a
// pointwise kernel.
//
// A step is bound by latency and by reading W and R, once each and mostly out of L2.  So every SM
// takes a share: a CTA owns 64 bytes of each gate's columns (16 fp32 or 32 bf16 hidden units), and
// a cluster of up to eight CTAs splits K = C + H among itself, which makes 128 or so CTAs from 64
// to 1024 units; their partial sums meet through distributed shared memory, where the same launch
// applies the cell.  Sixteen warps are four accumulator slots (the LSTM's gates; z, r, x.W_g and
// h.R_g of the GRU, whose reset gate multiplies the last) times shares of K.
//   * Up to four rows: fp32 FMAs on weights that go straight from wide loads to registers.
//   * More rows: mma.sync, the weights' tile as the 16-row operand and batch rows as the 8-column
//     one, in pieces of 128 values of k staged through shared memory.  bf16 storage is exact there;
//     fp32 operands are split into three bf16 planes (24 bits) and all products down to 2^-24 of
//     the largest are added, so that fp32 storage loses nothing to the FMA form.
// Kernel time, one CTA per four units and no split of K -> this (LSTM, C = H): fp32 1 row H = 512
// 9.0 -> 5.1 us, 1 row H = 1024 22.1 -> 8.2, 32 rows H = 512 13.0 -> 10.1, 64 rows 20.8 -> 15.5; FMAs for
// 64 rows measured 24.  Beyond the old limit the general path took several launches: bf16 GRU
// 32 rows C = 256 H = 1024 16.7 -> 10.5 us, 64 rows C = 1024 21 -> 18.7, fp32 LSTM 64 rows 50 -> 43.5.  What
// is left above reading W and R once (1 .. 4 us) is the launch and the chain of latencies: stage,
// product, meeting of the cluster.
#include <algorithm>

#include <cooperative_groups.h>

#include "cells.cuh"

namespace hb {
namespace {

namespace cg = cooperative_groups;

constexpr int IT_THREADS = 512;
constexpr int IT_MAXN = 64;               // batch rows
constexpr int IT_FMA_ROWS = 4;            // up to here FMAs, beyond mma.sync
constexpr int IT_XS_BYTES = 160 * 1024;   // FMA form: staged x and h at most; longer K goes in pieces
constexpr int IT_KC = 128;                // mma form: values of k per piece
constexpr int kSlots = 4;                 // accumulators per hidden unit

struct StepParams {
  int N, C, H;
  int rows;   // N padded to what the kernel computes
  int chunk;  // FMA form: values of k staged at a time
  const void *W, *R, *b0, *b1, *x, *h_prev, *c_prev;
  void *h_out, *c_out, *v;
  int training;
  float zoneout_prob;
  const void* mask;
};

// This CTA's columns and part of K: [x0, x0 + nx) of x, then [h0, h0 + nh) of h.
struct Share {
  int KS, rank, x0, nx, h0, nh;
  __device__ Share(const StepParams& p, cg::cluster_group& cl) : KS(cl.num_blocks()), rank(cl.block_rank()) {
    x0 = (int)((long long)p.C * rank / KS);
    nx = (int)((long long)p.C * (rank + 1) / KS) - x0;
    h0 = (int)((long long)p.H * rank / KS);
    nh = (int)((long long)p.H * (rank + 1) / KS) - h0;
  }
};

// red holds the partial sums [part][slot][row][unit] of this CTA.  Adds up the parts, then the
// cluster's CTAs, and applies the cell: four lanes per (row, unit), one per slot.
template <typename T, bool GRU, int U>
__device__ __forceinline__ void finish(const StepParams& p, cg::cluster_group& cluster, const Share& sh, float* red,
                                       int parts, int u0) {
  const int N = p.N, H = p.H, tid = threadIdx.x, KS = sh.KS;
  const T* hp = static_cast<const T*>(p.h_prev);
  const T* b0 = static_cast<const T*>(p.b0);
  const T* b1 = static_cast<const T*>(p.b1);
  const T* cp = static_cast<const T*>(p.c_prev);
  const T* mask = static_cast<const T*>(p.mask);
  T* h_out = static_cast<T*>(p.h_out);
  T* c_out = static_cast<T*>(p.c_out);
  T* v = static_cast<T*>(p.v);
  __syncthreads();
  if (parts > 1) {
    const int used = kSlots * p.rows * U;
    for (int i = tid; i < used; i += IT_THREADS) {
      float a = red[i];
      for (int k = 1; k < parts; ++k) a += red[i + k * used];
      red[i] = a;
    }
  }
  cluster.sync();
  for (int i = sh.rank * IT_THREADS + tid; i < N * U * 4; i += KS * IT_THREADS) {  // whole warps: U * 4 is
    const int sl = i & 3, uu = (i >> 2) % U, row = i / (4 * U), jj = u0 + uu;
    const bool in = jj < H;
    const long long o0 = (long long)row * H + jj;
    float bias = 0.f, hprev = 0.f, cprev = 0.f, m = 0.f;
    if (in) {
      if (GRU) bias = sl < 2 ? ld(b0 + jj + sl * H) + ld(b1 + jj + sl * H) : ld((sl == 2 ? b0 : b1) + jj + 2 * H);
      else bias = ld(b0 + jj + sl * H);
      hprev = ld(hp + o0);
      if (!GRU) cprev = ld(cp + o0);
      if (mask && p.training) m = ld(mask + o0);
    }
    float sum = bias;
    for (int c = 0; c < KS; ++c)
      sum += *cluster.map_shared_rank(red + ((size_t)sl * p.rows + row) * U + uu, c);
    float g;
    if (GRU) g = sl < 2 ? sigmoidf_(sum) : sum;
    else g = sl == 1 ? tanhf(sum) : sigmoidf_(sum);
    const float g1 = __shfl_down_sync(0xffffffffu, g, 1), g2 = __shfl_down_sync(0xffffffffu, g, 2),
                g3 = __shfl_down_sync(0xffffffffu, g, 3);
    const bool cache = p.training && v;
    if (!GRU && cache && in) st(v + (long long)row * 4 * H + jj + (long long)sl * H, g);
    if (!in || sl != 0) continue;
    float h_new;
    if (GRU) {
      const float z = g, r = g1, q_g = g3, gv = tanhf(g2 + r * q_g);
      if (cache) {
        const long long v0 = (long long)row * 4 * H + jj;
        st(v + v0, z);
        st(v + v0 + H, r);
        st(v + v0 + 2 * H, gv);
        st(v + v0 + 3 * H, q_g);
      }
      h_new = z * hprev + (1.0f - z) * gv;
    } else {
      const float c_new = g2 * cprev + g * g1;
      st(c_out + o0, c_new);
      h_new = g3 * tanhf(c_new);
    }
    if (mask)  // zoneout is on only with a probability and a mask (the host passes neither otherwise)
      h_new = p.training ? zoneout<true>(h_new, hprev, p.zoneout_prob, m)
                         : zoneout<false>(h_new, hprev, p.zoneout_prob, 0.f);
    st(h_out + o0, h_new);
  }
  if (KS > 1) cluster.sync();  // the partial sums stay until every CTA has read them
}

// Four consecutive weights of one row.  vec: H is a multiple of four and the rows are aligned for
// one load; otherwise element by element, `left` of them inside the row.
__device__ __forceinline__ float4 ld4(const float* q, bool vec, int left) {
  if (vec) return __ldg(reinterpret_cast<const float4*>(q));
  return make_float4(__ldg(q), left > 1 ? __ldg(q + 1) : 0.f, left > 2 ? __ldg(q + 2) : 0.f,
                     left > 3 ? __ldg(q + 3) : 0.f);
}
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* q, bool vec, int left) {
  if (vec) {
    const uint2 w = __ldg(reinterpret_cast<const uint2*>(q));
    return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xFFFF0000u),
                       __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xFFFF0000u));
  }
  return make_float4(ld(q), left > 1 ? ld(q + 1) : 0.f, left > 2 ? ld(q + 2) : 0.f, left > 3 ? ld(q + 3) : 0.f);
}

// ---------------------------------------------------------------- FMA form: RB rows (1 or 4)
template <typename T, bool GRU, int RB, bool VEC>
__global__ void __launch_bounds__(IT_THREADS, 1) step_fma_kernel(const StepParams p) {
  constexpr int LPR = 16 / sizeof(T);   // lanes per k: 64 bytes of one gate, four units a lane
  constexpr int KR = 32 / LPR;          // values of k a warp reads at a time
  constexpr int U = 4 * LPR;            // hidden units per CTA
  constexpr int G = GRU ? 3 : 4;        // gate blocks in a row of W / R
  constexpr int UNR = 8;                // loads ahead
  constexpr int PARTS = 4;              // warps per slot: parts of K
  cg::cluster_group cluster = cg::this_cluster();
  const Share sh(p, cluster);
  extern __shared__ __align__(16) float smem[];
  float* red = smem;
  float* xs = smem + PARTS * kSlots * RB * U;  // [k][row], and a line of zeros behind the last k
  const int N = p.N, C = p.C, H = p.H;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int u0 = (blockIdx.x / sh.KS) * U;
  const int slot = warp % kSlots, kp = warp / kSlots;
  const int q = lane % LPR, kr = lane / LPR, j = u0 + 4 * q;
  const T* x = static_cast<const T*>(p.x);
  const T* hp = static_cast<const T*>(p.h_prev);
  const int nx = sh.nx, K = nx + sh.nh;
  const int block = GRU && slot == 3 ? 2 : slot;
  const int k_lo = GRU && slot == 3 ? nx : 0, k_hi = GRU && slot == 2 ? nx : K;
  const T* Wj = static_cast<const T*>(p.W) + (long long)sh.x0 * G * H + (long long)block * H + j;
  const T* Rj = static_cast<const T*>(p.R) + (long long)sh.h0 * G * H + (long long)block * H + j;

  float s[4 * RB];  // [unit][row]
#pragma unroll
  for (int i = 0; i < 4 * RB; ++i) s[i] = 0.f;

  for (int c0 = 0; c0 < K; c0 += p.chunk) {
    const int n_k = min(p.chunk, K - c0);
    if (c0) __syncthreads();
    const int lo = max(k_lo - c0, 0), hi = min(k_hi - c0, n_k), first = lo + kp * KR + kr;
    float4 w[UNR];
    auto fetch = [&](int kb) {
#pragma unroll
      for (int e = 0; e < UNR; ++e) {
        const int kk = kb + e * KR * PARTS, k = c0 + kk;
        w[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kk < hi && j < H)
          w[e] = ld4(k < nx ? Wj + (long long)k * G * H : Rj + (long long)(k - nx) * G * H, VEC, H - j);
      }
    };
    fetch(first);  // on its way while x and h are staged
    for (int kk = tid; kk <= n_k; kk += IT_THREADS) {
      const int k = c0 + kk;
      float a[RB];
#pragma unroll
      for (int row = 0; row < RB; ++row) {
        a[row] = 0.f;
        if (row < N && kk < n_k)
          a[row] = k < nx ? ld(x + (long long)row * C + sh.x0 + k) : ld(hp + (long long)row * H + sh.h0 + k - nx);
      }
#pragma unroll
      for (int row = 0; row < RB; ++row) xs[kk * RB + row] = a[row];
    }
    __syncthreads();
    for (int kb = first; kb < hi; kb += UNR * KR * PARTS) {
      if (kb != first) fetch(kb);
#pragma unroll
      for (int e = 0; e < UNR; ++e) {
        int kk = kb + e * KR * PARTS;
        if (kk >= hi) kk = n_k;  // zeros, like the weights
        float a[RB];
        if constexpr (RB == 4) {
          const float4 t = *reinterpret_cast<const float4*>(xs + kk * RB);
          a[0] = t.x; a[1] = t.y; a[2] = t.z; a[3] = t.w;
        } else {
          a[0] = xs[kk];
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) {
          s[r] += a[r] * w[e].x;
          s[RB + r] += a[r] * w[e].y;
          s[2 * RB + r] += a[r] * w[e].z;
          s[3 * RB + r] += a[r] * w[e].w;
        }
      }
    }
  }

  // ---- sum over the lanes that hold other values of k: each halving hands half of the sums over
  constexpr int S0 = 4 * RB;
  int off = 0, n = S0;
#pragma unroll
  for (int m = 16; m >= LPR; m >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = (lane & m) != 0;
#pragma unroll
      for (int i = 0; i < S0 / 2; ++i) {
        if (i < n) {
          const float send = up ? s[i] : s[i + n], keep = up ? s[i + n] : s[i];
          s[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
      }
      if (up) off += n;
    } else {
      s[0] += __shfl_xor_sync(0xffffffffu, s[0], m);
    }
  }
#pragma unroll
  for (int i = 0; i < S0; ++i)
    if (i < n) red[((kp * kSlots + slot) * RB + (off + i) % RB) * U + 4 * q + (off + i) / RB] = s[i];
  finish<T, GRU, U>(p, cluster, sh, red, PARTS, u0);
}

// ---------------------------------------------------------------- mma form: 8 .. 64 rows
__device__ __forceinline__ void ldm2(uint32_t (&r)[2], const void* at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"((uint32_t)__cvta_generic_to_shared(at)));
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], const void* at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(at)));
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// NT: tiles of 8 rows.
template <typename T, bool GRU, int NT, bool VEC>
__global__ void __launch_bounds__(IT_THREADS, 1) step_mma_kernel(const StepParams p) {
  constexpr int P = sizeof(T) == 4 ? 3 : 1;     // bf16 planes of an operand
  constexpr int U = 64 / sizeof(T);             // hidden units per CTA
  constexpr int MT = U / 16, PARTS = 4 / MT;    // warps: slot x 16 units x part of a piece's k
  constexpr int G = GRU ? 3 : 4;
  constexpr int COLS = G * U, WS = COLS + 8, XS = IT_KC + 8;  // padded rows (16 bytes): no bank conflicts
  constexpr int ROWS = 8 * NT;
  constexpr int WL = IT_KC * G * 4 / IT_THREADS;              // 16-byte weight loads per thread and piece
  constexpr int XL = IT_KC * ROWS / IT_THREADS;               // elements of x / h
  constexpr int E = 16 / sizeof(T);                           // weights per load
  cg::cluster_group cluster = cg::this_cluster();
  const Share sh(p, cluster);
  extern __shared__ __align__(16) float smem[];
  float* red = smem;                                                               // [part][slot][ROWS][U]
  __nv_bfloat16* ws = reinterpret_cast<__nv_bfloat16*>(smem + PARTS * kSlots * ROWS * U);  // [plane][k][WS]
  __nv_bfloat16* xs = ws + P * IT_KC * WS;                                         // [plane][row][XS]
  const int N = p.N, C = p.C, H = p.H;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int u0 = (blockIdx.x / sh.KS) * U;
  const int slot = warp % kSlots, mt = (warp / kSlots) % MT, kp = warp / (kSlots * MT);
  const T* x = static_cast<const T*>(p.x);
  const T* hp = static_cast<const T*>(p.h_prev);
  const T* W = static_cast<const T*>(p.W);
  const T* R = static_cast<const T*>(p.R);
  // K in order: x's values padded with zeros to whole 16s, then h's
  const int nx = sh.nx, nxp = (nx + 15) / 16 * 16, K = nxp + sh.nh;
  const int block = GRU && slot == 3 ? 2 : slot;
  const int k_lo = GRU && slot == 3 ? nxp : 0, k_hi = GRU && slot == 2 ? nxp : K;

  float wr[WL][E > 4 ? 1 : 4];
  uint4 wq[WL];  // bf16: eight weights as they are
  T xr[XL];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int e = 0; e < WL; ++e) {
      const int i = tid + e * IT_THREADS, piece = i & 3, g = (i >> 2) % G, k = c0 + (i >> 2) / G;
      const int j = u0 + piece * E;
      const bool xp = k < nxp, ok = (xp ? k < nx : k < K) && j < H;
      const T* at = (xp ? W + (long long)(sh.x0 + k) * G * H : R + (long long)(sh.h0 + k - nxp) * G * H) +
                    (long long)g * H + j;
      if constexpr (E == 4) {
        const float4 t = ok ? ld4(at, VEC, H - j) : make_float4(0.f, 0.f, 0.f, 0.f);
        wr[e][0] = t.x; wr[e][1] = t.y; wr[e][2] = t.z; wr[e][3] = t.w;
      } else {
        wq[e] = make_uint4(0u, 0u, 0u, 0u);
        if (ok) {
          if (VEC) {
            wq[e] = __ldg(reinterpret_cast<const uint4*>(at));
          } else {
            const unsigned short* u = reinterpret_cast<const unsigned short*>(at);
            uint32_t half[8];
#pragma unroll
            for (int d = 0; d < 8; ++d) half[d] = j + d < H ? __ldg(u + d) : 0;
            wq[e] = make_uint4(half[0] | half[1] << 16, half[2] | half[3] << 16, half[4] | half[5] << 16,
                               half[6] | half[7] << 16);
          }
        }
      }
    }
#pragma unroll
    for (int e = 0; e < XL; ++e) {
      const int i = tid + e * IT_THREADS, row = i / IT_KC, k = c0 + i % IT_KC;
      xr[e] = T(0.f);
      if (row < N && k < K) {
        if (k < nxp) { if (k < nx) xr[e] = x[(long long)row * C + sh.x0 + k]; }
        else xr[e] = hp[(long long)row * H + sh.h0 + k - nxp];
      }
    }
  };
  auto stage = [&]() {
#pragma unroll
    for (int e = 0; e < WL; ++e) {
      const int i = tid + e * IT_THREADS, piece = i & 3, g = (i >> 2) % G, k = (i >> 2) / G;
      __nv_bfloat16* to = ws + k * WS + g * U + piece * E;
      if constexpr (E == 4) {
        float a[4] = {wr[e][0], wr[e][1], wr[e][2], wr[e][3]};
#pragma unroll
        for (int pl = 0; pl < P; ++pl) {
          const __nv_bfloat162 lo = __floats2bfloat162_rn(a[0], a[1]), hi = __floats2bfloat162_rn(a[2], a[3]);
          uint2 out;
          out.x = *reinterpret_cast<const uint32_t*>(&lo);
          out.y = *reinterpret_cast<const uint32_t*>(&hi);
          *reinterpret_cast<uint2*>(to + pl * IT_KC * WS) = out;
          a[0] -= __uint_as_float(out.x << 16); a[1] -= __uint_as_float(out.x & 0xFFFF0000u);
          a[2] -= __uint_as_float(out.y << 16); a[3] -= __uint_as_float(out.y & 0xFFFF0000u);
        }
      } else {
        *reinterpret_cast<uint4*>(to) = wq[e];
      }
    }
#pragma unroll
    for (int e = 0; e < XL; ++e) {
      const int i = tid + e * IT_THREADS, row = i / IT_KC, k = i % IT_KC;
      __nv_bfloat16* to = xs + row * XS + k;
      if constexpr (P == 1) {
        *to = xr[e];
      } else {
        float a = xr[e];
#pragma unroll
        for (int pl = 0; pl < P; ++pl) {
          const __nv_bfloat16 b = __float2bfloat16_rn(a);
          to[pl * ROWS * XS] = b;
          a -= __bfloat162float(b);
        }
      }
    }
  };

  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;

  fetch(0);
  for (int c0 = 0; c0 < K; c0 += IT_KC) {
    if (c0) __syncthreads();
    stage();
    __syncthreads();
    if (c0 + IT_KC < K) fetch(c0 + IT_KC);
#pragma unroll 1
    for (int ks = kp; ks < IT_KC / 16; ks += PARTS) {
      const int k = c0 + ks * 16;
      if (k < k_lo || k >= k_hi) continue;
      uint32_t a[P][4];  // 16 units x 16 k out of [k][unit]: matrices (k 0-7, u 0-7), (k 0-7, u 8-15), ...
#pragma unroll
      for (int pl = 0; pl < P; ++pl)
        ldm4t(a[pl], ws + pl * IT_KC * WS + (ks * 16 + (lane & 7) + (lane >> 4) * 8) * WS + block * U + mt * 16 +
                         ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        uint32_t b[P][2];
#pragma unroll
        for (int pl = 0; pl < P; ++pl)
          ldm2(b[pl], xs + pl * ROWS * XS + (n * 8 + (lane & 7)) * XS + ks * 16 + ((lane >> 3) & 1) * 8);
        if constexpr (P == 1) {
          mma(acc[n], a[0], b[0]);
        } else {  // smallest first
          mma(acc[n], a[2], b[0]);
          mma(acc[n], a[0], b[2]);
          mma(acc[n], a[1], b[1]);
          mma(acc[n], a[1], b[0]);
          mma(acc[n], a[0], b[1]);
          mma(acc[n], a[0], b[0]);
        }
      }
    }
  }
  // An infinity, or a value that bf16 rounds to one, leaves inf - inf in the lower planes where the
  // FMA form saturates the gate: a CTA that finds a sum not finite adds up its share again as that
  // form does.
  bool again = false;
  if constexpr (P > 1) {
    bool finite = true;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) finite = finite && fabsf(acc[n][i]) <= 3.402823466e38f;
    again = __syncthreads_or(!finite) != 0;
    if (again) {
      constexpr int SUMS = kSlots * ROWS * U;
      for (int i = tid; i < SUMS; i += IT_THREADS) {
        const int sl = i / (ROWS * U), row = i / U % ROWS, j = u0 + i % U, col = (GRU && sl == 3 ? 2 : sl) * H + j;
        float sum = 0.f;
        if (row < N && j < H) {
          if (!GRU || sl != 3)
            for (int k = sh.x0; k < sh.x0 + nx; ++k) sum = fmaf(x[(long long)row * C + k], W[(long long)k * G * H + col], sum);
          if (!GRU || sl != 2)
            for (int k = sh.h0; k < sh.h0 + sh.nh; ++k)
              sum = fmaf(hp[(long long)row * H + k], R[(long long)k * G * H + col], sum);
        }
        red[i] = sum;
        for (int part = 1; part < PARTS; ++part) red[part * SUMS + i] = 0.f;
      }
    }
  }
  if (!again) {
    // accumulator: units lane / 4 (+ 8), rows 2 * (lane % 4) (+ 1)
    const int unit = mt * 16 + (lane >> 2), r0 = 2 * (lane & 3);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float* to = red + ((kp * kSlots + slot) * ROWS + n * 8 + r0) * U + unit;
      to[0] = acc[n][0];
      to[U] = acc[n][1];
      to[8] = acc[n][2];
      to[U + 8] = acc[n][3];
    }
  }
  finish<T, GRU, U>(p, cluster, sh, red, PARTS, u0);
}

// ---------------------------------------------------------------- host side
typedef void (*StepKernel)(StepParams);

// Grid: 64-byte column groups x CTAs per cluster, as many of these as there are SMs for while a CTA
// keeps 32 values of k.
int launch(StepKernel k, const StepParams& p, int groups, int KS, size_t smem, cudaStream_t s) {
  if (smem > 48 * 1024)
    HB_CUDA_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(groups * KS);
  cfg.blockDim = dim3(IT_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = KS;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  HB_CUDA_OK(cudaLaunchKernelEx(&cfg, k, (StepParams)p));
  count_launch(1);
  return HASTE_B200_OK;
}

template <typename T, bool GRU, bool VEC>
int launch_step_v(StepParams& p, cudaStream_t s) {
  constexpr int U = 64 / sizeof(T), G = GRU ? 3 : 4;
  const int groups = ceil_div(p.H, U);
  int KS = 1;
  while (KS < 8 && groups * KS * 2 <= sm_count() && (p.C + p.H) / (KS * 2) >= 32) KS *= 2;
  if (p.N <= IT_FMA_ROWS) {
    p.rows = p.N == 1 ? 1 : 4;
    p.chunk = std::min(ceil_div(p.C, KS) + ceil_div(p.H, KS), IT_XS_BYTES / (p.rows * 4));
    const size_t smem = (size_t)(4 * kSlots * p.rows * U + (p.chunk + 1) * p.rows) * sizeof(float);
    return launch(p.N == 1 ? step_fma_kernel<T, GRU, 1, VEC> : step_fma_kernel<T, GRU, 4, VEC>, p, groups, KS, smem, s);
  }
  const int nt = p.N <= 8 ? 1 : (p.N <= 16 ? 2 : (p.N <= 32 ? 4 : 8));
  constexpr int P = sizeof(T) == 4 ? 3 : 1;
  p.rows = nt * 8;
  const size_t smem = (size_t)(64 / U) * kSlots * p.rows * U * sizeof(float) +
                      2 * (size_t)P * (IT_KC * (G * U + 8) + p.rows * (IT_KC + 8));
  StepKernel k = nt == 1 ? step_mma_kernel<T, GRU, 1, VEC>
                         : (nt == 2 ? step_mma_kernel<T, GRU, 2, VEC>
                                    : (nt == 4 ? step_mma_kernel<T, GRU, 4, VEC> : step_mma_kernel<T, GRU, 8, VEC>));
  return launch(k, p, groups, KS, smem, s);
}

template <typename T, bool GRU>
int launch_step_t(StepParams& p, cudaStream_t s) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p.W) | reinterpret_cast<uintptr_t>(p.R);
  return p.H % (16 / sizeof(T)) == 0 && a % 16 == 0 ? launch_step_v<T, GRU, true>(p, s)
                                                    : launch_step_v<T, GRU, false>(p, s);
}

template <bool GRU>
int launch_step(int dtype, bool training, StepParams& p, cudaStream_t s) {
  if (p.N > IT_MAXN || p.N < 1 || p.H < 1 || p.C < 1) return HASTE_B200_ERR_UNSUPPORTED;
  p.training = training;
  if (dtype == HASTE_B200_F32) return launch_step_t<float, GRU>(p, s);
  if (dtype == HASTE_B200_BF16) return launch_step_t<__nv_bfloat16, GRU>(p, s);
  return HASTE_B200_ERR_UNSUPPORTED;
}

}  // namespace

// The single-step (Iterate) forward of the LSTM in one launch.  HASTE_B200_ERR_UNSUPPORTED
// (more than 64 rows, other storage types) sends the caller to the general path.
int lstm_forward_step_fused(const LstmFwd& a, cudaStream_t s) {
  // (a new state written over the old one would race with the CTAs still reading it)
  if (a.T != 1 || !a.h_out || !a.c_out || a.h_out == a.h) return HASTE_B200_ERR_UNSUPPORTED;
  StepParams p{};
  p.N = a.N; p.C = a.C; p.H = a.H;
  p.W = a.W; p.R = a.R; p.b0 = a.b; p.b1 = nullptr; p.x = a.x; p.h_prev = a.h; p.c_prev = a.c;
  p.h_out = a.h_out; p.c_out = a.c_out; p.v = a.v;
  const bool zo = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  p.zoneout_prob = zo ? a.zoneout_prob : 0.0f;
  p.mask = zo ? a.zoneout_mask : nullptr;
  return launch_step<false>(a.dtype, a.training != 0, p, s);
}

int gru_forward_step_fused(const GruFwd& a, cudaStream_t s) {
  if (a.T != 1 || !a.h_out || a.h_out == a.h) return HASTE_B200_ERR_UNSUPPORTED;
  StepParams p{};
  p.N = a.N; p.C = a.C; p.H = a.H;
  p.W = a.W; p.R = a.R; p.b0 = a.bx; p.b1 = a.br; p.x = a.x; p.h_prev = a.h; p.c_prev = nullptr;
  p.h_out = a.h_out; p.c_out = nullptr; p.v = a.v;
  const bool zo = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  p.zoneout_prob = zo ? a.zoneout_prob : 0.0f;
  p.mask = zo ? a.zoneout_mask : nullptr;
  return launch_step<true>(a.dtype, a.training != 0, p, s);
}

}  // namespace hb
