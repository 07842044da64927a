// Tensor-core GRU and LSTM recurrences for large batches (bf16 storage), sm_100a.
//
// The chain kernels (rec_grid_kernels.cuh) take eight batch rows at a time and pay for every chain
// of a CTA.  Where they would need more than six to eight (rec_chain_host.cu) - a hundred rows of a wide
// layer, or half of that on half of the GPU - the step product is a real tile for the 5th-generation tensor
// cores, and this file runs it there:
//
//   forward   gates[rows, G*16] = h_{t-1}[rows, 0:H] . R[0:H, slice]            K = H
//   backward  dh_rec[rows, 16]  = dq_{t+1}[rows, 0:GH] . R[slice, 0:GH]^T       K = GH
//   (long K: four CTAs, a quarter of K and 64 units each - tc_geometry_for)
//
// (G = 3 for the GRU; G = 4 for the LSTM, where "dq" is the gate gradient in the cache's place.)
// A step is bound by its chain - counter, TMA, MMA issue (65 cycles each), tensor-memory read, gate
// math, publish - and, with many rows per CTA, by the stream of h or dq at 64 bytes per clock and SM.
// GRU, H = 1024, us per step forward / backward: 128 rows 6.9 / 8.0, 256 rows 7.9 / 10.4 (with one 128-row
// tile per CTA 7.9 / 11.5).  Two directions of 200 steps side by side, chain kernels -> this: GRU 90
// rows 8.2 -> 5.0 ms, LSTM 90 rows 8.1 -> 6.4, LSTM 178 rows H = 808 9.4 -> 6.9 (with all of K per CTA, below).
//
// * Grid = (H / 16 hidden slices) x (row groups), one cooperative launch per layer pass; a
//   CTA owns 16 hidden units for MT tiles of RB (64 or 128) batch rows.
// * The CTA's slice of R lives in SHARED MEMORY for the whole pass, written once in the
//   128-byte-swizzled K-major layout that tcgen05.mma reads (96 KB at H = 1024): R is read
//   from HBM once per pass.
// * The other operand is streamed every step by TMA (cp.async.bulk.tensor; every CTA fetches
//   its own copy) straight out of the tensor the step before wrote - h itself in the forward
//   pass, the gate-gradient tensor dq in the backward pass - through an mbarrier ring; nothing
//   is packed into a separate exchange buffer.
// * The accumulator lives in tensor memory (two buffers, so the tile that follows starts
//   while this one is drained); four epilogue warps read it with tcgen05.ld, one batch row
//   per thread, and do the whole gate math, zoneout and the stores for their 16 units.
// * Steps synchronise through one arrival counter per row tile: an epilogue warp that has
//   stored its part of step t adds one (release); the TMA warp of every CTA of the row group
//   waits for all of them (acquire) before it loads step t's operand.  CTAs of different row
//   groups never wait for each other, and with several tiles per CTA the wait for one tile
//   hides behind the contraction of the others.
// * The gate functions are those of rec_chain.cuh (1e-6).  One MUFU.TANH each (relative error
//   2^-11) would take 0.3 us off a forward step of the GRU, but then 0.17 % of the stored states are
//   another bf16 than the exact step gives, against 0.02 %.
// * Every wait - counter or mbarrier - is bounded; on expiry the grid's abort flag and the
//   process error word are set, all roles leave their loops, tensor memory is released and
//   the host reports HASTE_B200_ERR_TIMEOUT.
//
// Warp roles: warp 0 TMA producer (four lanes issue), warps 1..NI MMA issuers (a tcgen05.mma
// of this shape occupies its issuing thread for ~65 cycles, 2-3x its tensor-pipe time, so NI
// threads issue the k-blocks in turn, each into its own accumulator), then four epilogue warps.
// Replaces the per-step cuBLAS call + pointwise kernel of the reference
// (lib/gru_forward_gpu.cu.cc:214-308,345-363, lib/gru_backward_gpu.cu.cc:252-320) for
// bf16 batches of about a hundred rows and more; math as in lib/gru_forward_gpu.cu.cc:27-85
// and lib/gru_backward_gpu.cu.cc:26-96.
#include <atomic>

#include "rec_chain.cuh"
#include "tcgen05.cuh"

namespace hb {
namespace {

using namespace tc;
typedef __nv_bfloat16 bf16;

constexpr int UC = 16;                 // hidden units per CTA
constexpr int BK = 64;                 // K elements per TMA box / swizzle row (128 bytes)
constexpr int A_STAGE = 128 * BK * 2;  // one streamed stage: 128 rows x 128 bytes
constexpr int PL = 4;                  // lanes that issue the TMA loads (k-blocks go to them in turn)
// MMA-issuing warps (likewise).  Four, but two where a CTA has a quarter of the k-blocks: their instructions
// still hide behind the stream, and there is half as much tensor memory to read.
template <int CL> constexpr int issuers() { return CL > 1 ? 2 : 4; }
// warp 0 TMA, then the issuers, then 4 epilogue warps
template <int CL> constexpr int tc_threads() { return 32 * (1 + issuers<CL>() + 4); }
constexpr int MAX_SMEM = 227 * 1024;
constexpr int CLUSTER = 4;             // CTAs that share out a long K (backward)
constexpr int XCH = 4 * (CLUSTER - 1) * 4 * 512;  // bytes of partial dh a CTA takes: [warp][source][4 units][row][4]

struct TcParams {
  int T, N, H, nHS, MT, RB, training, has_zoneout, r_transposed;
  int stage_bytes;     // RB * 128: one stage of the ring holds one k-block of RB rows
  int ring_bytes;      // stages * stage_bytes, plus padding up to a whole 128-row tile
  float zoneout_prob;
  const bf16* R;       // forward: [H,3H]; backward: [H,3H] or R_t [3H,H]
  const bf16* bx;      // forward
  const bf16* br;
  const bf16* Wx;      // forward: x.W [T,N,3H]
  const bf16* mask;    // [T,N,H] or null
  bf16* h;             // [T+1,N,H] (backward: read only)
  bf16* v;             // [T,N,4H] gate cache (forward: out or null; backward: in)
  const bf16* dh_new;  // backward [T+1,N,H]
  bf16* dp;            // backward out [T,N,3H]
  bf16* dq;            // backward out [T,N,3H], also the streamed operand
  float* dh_carry;     // backward [N,H] fp32 in/out
  bf16* c;             // LSTM [T+1,N,H] (backward: read only)
  float* c_carry;      // LSTM [N,H] fp32: forward c, backward its gradient, in/out
  const bf16* dc_new;  // LSTM backward [T+1,N,H] or null
  unsigned int* cnt;   // [row tiles] arrival counters, zeroed before launch
  int* abort_flag;     // device-global, zeroed before launch
  int* err;            // process error word
#ifdef HASTE_B200_TIMING_EXPERIMENTS
  long long* stamps;   // [T][16] clock64 stamps of CTA 0, tile 0 (timing-experiment builds only)
#endif
};

#ifdef HASTE_B200_TIMING_EXPERIMENTS
#define HB_STAMP(p, it, mt, slot)                                            \
  do {                                                                       \
    if ((p).stamps && blockIdx.x == 0 && (mt) == 0)                          \
      (p).stamps[(size_t)(it) * 16 + (slot)] = clock64();                     \
  } while (0)
#else
#define HB_STAMP(p, it, mt, slot) do {} while (0)
#endif

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_add(unsigned int* p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t add_acq_rel_cta(uint32_t p, uint32_t v) {
  uint32_t old;
  asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ void fence_proxy_async_all() {
  asm volatile("fence.proxy.async;" ::: "memory");
}

// Waits until *c >= target.  False when the limit ran out or the grid was aborted.
__device__ __forceinline__ bool wait_count(const unsigned int* c, unsigned int target,
                                           volatile int* s_abort, const TcParams& p, int code,
                                           int d0, int d1) {
  // (polling with relaxed loads and one acquire fence at the end measured 0.2 us per step slower)
  if (ld_acquire_u32(c) >= target) return true;
  const long long t0 = clock64();
  unsigned int it = 0;
  while (ld_acquire_u32(c) < target) {
    if ((++it & 63u) == 0) {
      if (*s_abort || *reinterpret_cast<volatile int*>(p.abort_flag)) {
        *s_abort = 1;
        return false;
      }
      if (clock64() - t0 > SPIN_LIMIT_CYCLES) {
        *s_abort = 1;
        if (atomicExch(p.abort_flag, 1) == 0) {
          volatile int* e = reinterpret_cast<volatile int*>(p.err);
          e[1] = blockIdx.x; e[2] = d0; e[3] = d1; e[4] = (int)target;
          __threadfence_system();
          e[0] = code;
        }
        __threadfence_system();
        return false;
      }
    }
  }
  return true;
}

// 8 consecutive bf16 as one 16-byte load, and element u of such a group as a float
__device__ __forceinline__ uint4 ldq(const bf16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ float bfq(const uint4& q, int u) {
  const uint32_t w = (u >> 1) == 0 ? q.x : ((u >> 1) == 1 ? q.y : ((u >> 1) == 2 ? q.z : q.w));
  return (u & 1) ? __uint_as_float(w & 0xFFFF0000u) : __uint_as_float(w << 16);
}

// 8 consecutive bf16 (16 bytes, 16-byte aligned) <-> floats
__device__ __forceinline__ void ld8(const bf16* p, float (&x)[8]) {
  const uint4 a = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[2 * i] = __uint_as_float(w[i] << 16);
    x[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}
__device__ __forceinline__ void st8(bf16* p, const float (&x)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __nv_bfloat162 t2 = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
    w[i] = *reinterpret_cast<uint32_t*>(&t2);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ void ld_carry(const float* p, float (&x)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
  x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ void st_carry(float* p, const float (&x)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(x[0], x[1], x[2], x[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(x[4], x[5], x[6], x[7]);
}

// Byte offset of element (row n, k) inside one K-major, 128-byte-swizzled k-block tile
// (rows of 64 bf16 = 128 bytes; 16-byte chunk c of row n sits at chunk c ^ (n & 7)).
__device__ __forceinline__ uint32_t swz_off(int n, int kk) {
  return (uint32_t)((n >> 3) * 1024 + (n & 7) * 128 + ((((kk >> 3) ^ (n & 7)) & 7) << 4) + (kk & 7) * 2);
}

// The ring's stages belong to M lanes / issuers for good: `own` has stages own, own + M, ...  (If
// they took k-blocks in turn whatever the stage, one of them a whole ring ahead of another would
// take a phase of a stage for the one two further on, which a barrier's parity does not tell
// apart.)  From one block of `own` to its next.
template <int M>
__device__ __forceinline__ void next_block(int& stage, uint32_t& phase, int& kb, int own, int stages) {
  stage += M;
  kb += M;
  if (stage >= stages) {
    kb += stages + own - stage;
    stage = own;
    phase ^= 1u;
  }
}

// 16 bytes into another CTA's shared memory, counted on its barrier when they have arrived.
__device__ __forceinline__ void st_async_f4(uint32_t addr, uint32_t bar, float a, float b, float c, float d) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
      "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar)
      : "memory");
}

// G: gates, 3 GRU, 4 LSTM.  CL: CTAs of a cluster that share out K (backward).
template <int G, bool FWD, int CL>
__global__ void __launch_bounds__(tc_threads<CL>(), 1)
tc_recurrence_kernel(const __grid_constant__ CUtensorMap map_a, const TcParams p, const int stages) {
  constexpr int NI = issuers<CL>(), TC_THREADS = tc_threads<CL>();
  constexpr bool SPLIT = CL > 1;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
  const int H = p.H, N = p.N;
  constexpr int NB = FWD ? G * UC : CL * UC;  // columns of the step product
  const int K = FWD ? H : G * H;
  const int hs = blockIdx.x % p.nHS, rg = blockIdx.x / p.nHS;
  const int rank = hs % CL;  // in the cluster
  // this CTA's k-blocks: all or a share of them (TMA fills what lies beyond K with zeros)
  const int KBT = (K + BK - 1) / BK, KBS = (KBT + CL - 1) / CL;
  const int kb0 = SPLIT ? rank * KBS : 0, KB = SPLIT ? max(0, min(KBS, KBT - kb0)) : KBT;
  constexpr int R_TILE = NB * 128;  // bytes of the resident operand per k-block
  const uint32_t r_bytes = (uint32_t)KBS * R_TILE;
  const uint32_t ring = base + r_bytes;  // r_bytes is a multiple of 1024
  uint8_t* ring_ptr = aligned + r_bytes;
  // (a 64-row stage is read by the 128-row MMA together with the stage behind it - rows whose
  // results nobody uses - so the ring is padded by half a tile at its end)
  float4* xch = reinterpret_cast<float4*>(ring_ptr + p.ring_bytes);  // SPLIT: the other CTAs' partial dh
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring_ptr + p.ring_bytes + (SPLIT ? XCH : 0));
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (stages + s); };
  auto accf_bar = [&](int a) { return bar0 + 8u * (2 * stages + a); };
  auto acce_bar = [&](int a) { return bar0 + 8u * (2 * stages + 2 + a); };
  // SPLIT, per epilogue warp: partial dh has come; what went out has been read
  auto xfull_bar = [&](int w) { return bar0 + 8u * (2 * stages + 4 + w); };
  auto xfree_bar = [&](int w) { return bar0 + 8u * (2 * stages + 8 + w); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * stages + (SPLIT ? 12 : 4));
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t s_done = smem_u32(tmem_slot + 2);  // [2 tiles] epilogue warps that have stored
  float* s_bias = reinterpret_cast<float*>(tmem_slot + 4);  // forward: [2][48] bx, br

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int u0 = hs * UC;
  // two 64-row tiles per CTA: the second one's rows are rows 64..127 of its MMAs and belong to
  // epilogue warps of their own, so that the tiles are two chains that only share the streams
  const bool halves = p.RB == 64 && p.MT == 2;
  constexpr int ACC_COLS = NB <= 32 ? 32 : 64;   // tensor-memory columns per accumulator
  constexpr uint32_t TMEM_COLS = 2 * NI * ACC_COLS;  // two buffers x one accumulator per issuer

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(accf_bar(a), NI);
      mbar_init(acce_bar(a), halves ? 64 : 128);
    }
    for (int w = 0; SPLIT && w < 4; ++w) {
      mbar_init(xfull_bar(w), 1);
      mbar_init(xfree_bar(w), CL - 1);
    }
    *s_abort = 0;
    if (SPLIT) tmem_slot[2] = tmem_slot[3] = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // ---- streamed-operand ring: zero once, so that rows a 64-row box never writes are zeros
  for (int i = threadIdx.x; i < p.ring_bytes / 16; i += TC_THREADS)
    reinterpret_cast<uint4*>(ring_ptr)[i] = make_uint4(0u, 0u, 0u, 0u);
  // ---- resident operand: this CTA's slice of R, K-major and swizzled; zeros beyond K and beyond H
  // (H is a multiple of 8: a slice has 16 units or, the last one, 8)
  for (int i = threadIdx.x; i < (int)(r_bytes / 16); i += TC_THREADS)
    reinterpret_cast<uint4*>(aligned)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  if (FWD) {
    // B^T[n = gate*16 + u][k] = R[k][gate*H + u0 + u]
    for (int item = threadIdx.x; item < K * 2 * G; item += TC_THREADS) {
      const int k = item / (2 * G), gate = item % (2 * G) / 2, uo = item % 2 * 8;
      if (u0 + uo >= H) continue;
      float x[8];
      ld8(p.R + (size_t)k * G * H + (size_t)gate * H + u0 + uo, x);
      uint8_t* tile = aligned + (size_t)(k / BK) * R_TILE;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<bf16*>(tile + swz_off(gate * 16 + uo + u, k % BK)) = __float2bfloat16_rn(x[u]);
    }
    // (the GRU's bx, then br)
    for (int i = threadIdx.x; i < (G == 3 ? 96 : 64); i += TC_THREADS) {
      const int which = i / NB, c = i % NB, gate = c / 16, u = c % 16;
      s_bias[i] = u0 + u < H ? __bfloat162float((which ? p.br : p.bx)[gate * H + u0 + u]) : 0.f;
    }
  } else {
    // B^T[n = unit j of the cluster][k = gate column c] = R[c0 + j][c]   (R_t[c][c0 + j] when transposed)
    const int c0 = u0 - rank * UC, k0 = kb0 * BK, kn = min(K - k0, KB * BK);
    if (!p.r_transposed) {
      for (int item = threadIdx.x; item < NB * (KB * BK / 8); item += TC_THREADS) {
        const int j = item / (KB * BK / 8), c8 = (item % (KB * BK / 8)) * 8;
        if (c0 + j >= H || c8 >= kn) continue;
        const uint4 w = *reinterpret_cast<const uint4*>(p.R + (size_t)(c0 + j) * K + k0 + c8);
        uint8_t* tile = aligned + (size_t)(c8 / BK) * R_TILE;
        *reinterpret_cast<uint4*>(tile + swz_off(j, c8 % BK)) = w;  // one whole 16-byte chunk
      }
    } else {
      for (int item = threadIdx.x; item < KB * BK * (NB / 8); item += TC_THREADS) {
        const int c = item / (NB / 8), uo = item % (NB / 8) * 8;
        if (c0 + uo >= H || c >= kn) continue;
        float x[8];
        ld8(p.R + (size_t)(k0 + c) * H + c0 + uo, x);
        uint8_t* tile = aligned + (size_t)(c / BK) * R_TILE;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<bf16*>(tile + swz_off(uo + j, c % BK)) = __float2bfloat16_rn(x[j]);
      }
    }
  }
  // the tensor core reads shared memory through the async proxy
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (SPLIT) cluster_sync_all();  // the others' barriers are initialised before anything arrives on them
  const uint32_t tmem_base = *tmem_slot;

  const int tiles_total = (N + p.RB - 1) / p.RB;
  // per step: the epilogue warps of every CTA; SPLIT: the last of them
  const unsigned int arrivals = (unsigned int)p.nHS * (SPLIT ? 1u : halves ? 2u : 4u);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // PL lanes issue the k-blocks (lane l fills stages l, l + PL, ...): a cp.async.bulk.tensor
    // holds its issuing thread for about 0.1 us, which would otherwise be the rate of the whole
    // ring.
    constexpr unsigned PMASK = (1u << PL) - 1u;
    if (lane < PL) {
      int stage = lane, kb = lane;  // this lane's next stage, and its k-block counted from this tile
      uint32_t phase = 0;
      bool ok = true;
      const uint32_t box_bytes = (uint32_t)p.RB * 128u;
      for (int it = 0; it < p.T && ok; ++it) {
        if (!FWD && it == 0) continue;  // the first backward step has no recurrent part
        for (int mt = 0; mt < p.MT && ok; ++mt) {
          const int tile = rg * p.MT + mt;
          if (tile >= tiles_total) break;
          // forward step it reads h_it (published it times); backward iteration it reads the
          // dq of iteration it-1 (published it times as well)
          if (it > 0 && lane == 0)
            ok = wait_count(p.cnt + tile, arrivals * (unsigned int)it, s_abort, p, 51, it, tile);
          __syncwarp(PMASK);  // lane 0's acquire is ordered before the other lanes' loads
          HB_STAMP(p, it, mt, 0);  // the step's operand is published
          fence_proxy_async_all();
          const int trow = FWD ? it : (p.T - it);  // time slot of the streamed tensor
          const int row = trow * N + tile * p.RB;
          while (kb < KB) {
            if (!mbar_wait(empty_bar(stage), phase ^ 1u, s_abort, p.err, 52)) { ok = false; break; }
            mbar_expect_tx(full_bar(stage), box_bytes);
            tma_load_3d(ring + stage * p.stage_bytes, &map_a, full_bar(stage), (kb0 + kb) * BK, row, 0);
            next_block<PL>(stage, phase, kb, lane, stages);
          }
          kb -= KB;
          ok = __all_sync(PMASK, ok);  // all producer lanes leave together
          HB_STAMP(p, it, mt, 1);  // all TMA loads of the tile issued
        }
      }
    }
  } else if (warp <= NI) {
    // ------------------------------------------------------------------ MMA issuers
    if (lane == 0) {
      const int iss = warp - 1;  // this issuer takes what lies in stages iss, iss + NI, ...
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NB >> 3) << 17) |
                             ((uint32_t)(128 >> 4) << 24);
      int stage = iss, kb = iss;
      uint32_t phase = 0;
      uint32_t acc_phase[2] = {0, 0};
      int n_acc = 0;
      bool ok = true;
      const uint64_t a_desc0 = smem_desc(ring, 16, 1024);
      const uint64_t b_desc0 = smem_desc(base, 16, 1024);
      const uint64_t a_stage_inc = (uint64_t)(p.stage_bytes >> 4);
      for (int it = 0; it < p.T && ok; ++it) {
        if (!FWD && it == 0) continue;
        for (int mt = 0; mt < p.MT && ok; ++mt) {
          if (rg * p.MT + mt >= tiles_total) break;
          const int acc = halves ? mt : n_acc & 1;
          ++n_acc;
          if (!mbar_wait(acce_bar(acc), acc_phase[acc] ^ 1u, s_abort, p.err, 53)) { ok = false; break; }
          acc_phase[acc] ^= 1u;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (acc * NI + iss) * ACC_COLS;
          // Descriptors differ only in their 14-bit start-address field (bytes >> 4): one add
          // per MMA instead of rebuilding them.
#pragma unroll 1
          for (uint32_t more = 0; kb < KB; more = 1) {
            if (!mbar_wait(full_bar(stage), phase, s_abort, p.err, 54)) { ok = false; break; }
            tc_fence_after();
            if (kb == 0) HB_STAMP(p, it, mt, 2);  // first k-block has landed
            const uint64_t ad = a_desc0 + (uint64_t)stage * a_stage_inc - (halves && mt ? a_stage_inc : 0);
            const uint64_t bd = b_desc0 + (uint64_t)kb * (R_TILE >> 4);
            tc_mma_bf16(d_tmem, ad, bd, idesc, more);
            tc_mma_bf16(d_tmem, ad + 2, bd + 2, idesc, 1u);
            tc_mma_bf16(d_tmem, ad + 4, bd + 4, idesc, 1u);
            tc_mma_bf16(d_tmem, ad + 6, bd + 6, idesc, 1u);
            tc_commit(empty_bar(stage));
            next_block<NI>(stage, phase, kb, iss, stages);
          }
          kb -= KB;
          if (iss == 0) HB_STAMP(p, it, mt, 3);  // last MMA issued
          if (ok) tc_commit(accf_bar(acc));
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quad = warp & 3;
    const int r = (halves ? quad & 1 : quad) * 32 + lane;  // row of the tile
    uint32_t acc_phase[2] = {0, 0};
    uint32_t x_phase = 0;
    int n_acc = 0;
    bool ok = true;
    const long long NH = (long long)N * H;
    for (int it = 0; it < p.T && ok; ++it) {
      const int t = FWD ? it : (p.T - 1 - it);
      for (int mt = halves ? quad >> 1 : 0; mt < p.MT && ok; mt += halves ? 2 : 1) {
        const int tile = rg * p.MT + mt;
        if (tile >= tiles_total) break;
        const int n = tile * p.RB + r;
        const bool valid = r < p.RB && n < N;
        const bool have_acc = FWD || it > 0;
        const long long o0 = (long long)n * H + u0;
        // The 16 units are handled in two halves of 8 and the step inputs stay packed (bf16
        // pairs) until they are used, so that the live state of a thread stays within its
        // share of the register file (nine warps per CTA, seven where K is shared out).
        // ---- inputs that do not depend on the recurrence: issued before the wait below
        uint4 in0[2], in1[2], in2[2], in3[2], hp[2], mk[2], dhn[2], cn[2], dcn[2];
        float carry[2][8];  // backward: dh; LSTM forward: c
        float dc0[2][8], c_tanh[2][8];  // LSTM backward
        if (valid) {
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            const int uo = hf * 8;
            if (u0 + uo >= H) break;
            if (FWD) {
              const bf16* wx = p.Wx + ((long long)t * N + n) * G * H + u0 + uo;
              in0[hf] = ldq(wx);
              in1[hf] = ldq(wx + H);
              in2[hf] = ldq(wx + 2 * H);
              if (G == 4) in3[hf] = ldq(wx + 3 * H);
              if (G == 3 || p.has_zoneout) hp[hf] = ldq(p.h + (long long)t * NH + o0 + uo);
              if (G == 4) ld_carry(p.c_carry + o0 + uo, carry[hf]);
              if (p.has_zoneout && p.training) mk[hf] = ldq(p.mask + (long long)t * NH + o0 + uo);
            } else {
              const bf16* vt = p.v + ((long long)t * N + n) * 4 * H + u0 + uo;
              in0[hf] = ldq(vt);
              in1[hf] = ldq(vt + H);
              in2[hf] = ldq(vt + 2 * H);
              in3[hf] = ldq(vt + 3 * H);
              hp[hf] = ldq((G == 4 ? p.c : p.h) + (long long)t * NH + o0 + uo);  // before the step
              if (G == 4) cn[hf] = ldq(p.c + (long long)(t + 1) * NH + o0 + uo);
              if (G == 4 && p.dc_new) dcn[hf] = ldq(p.dc_new + (long long)(t + 1) * NH + o0 + uo);
              dhn[hf] = ldq(p.dh_new + (long long)(t + 1) * NH + o0 + uo);
              if (p.has_zoneout) mk[hf] = ldq(p.mask + (long long)t * NH + o0 + uo);
              ld_carry(p.dh_carry + o0 + uo, carry[hf]);
              if (G == 4) ld_carry(p.c_carry + o0 + uo, dc0[hf]);
            }
          }
        }
        // ---- backward: what can be done without the step product (the tanh of an LSTM's c takes 2000 cycles)
        if (!FWD && valid) {
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            if (u0 + hf * 8 >= H) break;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              carry[hf][u] += bfq(dhn[hf], u);
              if (G == 4) {
                if (p.dc_new) dc0[hf][u] += bfq(dcn[hf], u);
                c_tanh[hf][u] = rec::chain_tanh(bfq(cn[hf], u));
              }
            }
          }
        }
        // ---- wait for the step product; which issuers had a part in it (all, unless K is short)
        uint32_t have = (1u << NI) - 1u;
        if (KB < 2 * NI) {
          const int first = ((it - (FWD ? 0 : 1)) * min(p.MT, tiles_total - rg * p.MT) + mt) * KB;
          have = 0;
          for (int kb = 0; kb < KB; ++kb) have |= 1u << ((first + kb) % stages % NI);
        }
        int acc = 0;
        if (have_acc) {
          acc = halves ? mt : n_acc & 1;
          ++n_acc;
          bool got = mbar_wait(accf_bar(acc), acc_phase[acc], s_abort, p.err, 55);
          got = __all_sync(0xffffffffu, got);
          if (!got) { ok = false; break; }
          acc_phase[acc] ^= 1u;
          tc_fence_after();
          if (warp == NI + 1 && lane == 0) HB_STAMP(p, it, mt, 4);  // accumulator complete
        }
        const uint32_t taddr = tmem_base + acc * NI * ACC_COLS + ((uint32_t)(quad * 32) << 16);
        const bool takes = halves || quad * 32 < p.RB;  // some of the warp's rows are in the tile
        float rec_dh[16];  // backward: the step product
        if (!FWD && have_acc) {
          constexpr int XG = G == 4 && !SPLIT ? 2 : NI;  // accumulators in flight (registers)
          // columns of 16 units, summed over the issuers
          auto columns = [&](int col, float (&x)[16]) {
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = 0.f;
#pragma unroll
            for (int g0 = 0; g0 < NI; g0 += XG) {
              uint32_t b[XG][16];
#pragma unroll
              for (int k = 0; k < XG; ++k) {
                if (have >> (g0 + k) & 1u) {
                  tc_ld16(taddr + (g0 + k) * ACC_COLS + col, b[k]);
                } else {
#pragma unroll
                  for (int i = 0; i < 16; ++i) b[k][i] = 0u;
                }
              }
              tc_wait_ld();
#pragma unroll
              for (int k = 0; k < XG; ++k)
#pragma unroll
                for (int i = 0; i < 16; ++i) x[i] += __uint_as_float(b[k][i]);
            }
          };
          // the other CTAs' units go to them, to the warp with the same rows; then this CTA's own
          // (a second row tile's partial sums take the place of the first one's)
          if (SPLIT && takes && p.MT > 1 && !halves) {
            bool free_ = mbar_wait_cluster(xfree_bar(quad), x_phase ^ 1u, s_abort, p.err, 56);
            free_ = __all_sync(0xffffffffu, free_);
            if (!free_) { ok = false; break; }
          }
          const uint32_t xat = smem_u32(xch) + (uint32_t)(quad * (CL - 1) * 4 * 512 + lane * 16);
          if (SPLIT && takes && lane == 0) mbar_expect_tx(xfull_bar(quad), (CL - 1) * 32 * 64);
#pragma unroll 1
          for (int d = 1; takes && d < CL; ++d) {
            const uint32_t to = (uint32_t)(rank + d) % CL;
            const uint32_t at = mapa_u32(xat + (uint32_t)(CL - 1 - d) * 2048, to), bar = mapa_u32(xfull_bar(quad), to);
            float x[16];
            columns((int)to * UC, x);
#pragma unroll
            for (int c = 0; c < 4; ++c)
              st_async_f4(at + c * 512, bar, x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
          }
          columns(rank * UC, rec_dh);
          tc_fence_before();
          mbar_arrive(acce_bar(acc));  // the accumulator buffer is free
          if (warp == NI + 1 && lane == 0) HB_STAMP(p, it, mt, 5);
        }
        if (SPLIT && have_acc && takes) {
          bool got = mbar_wait_cluster(xfull_bar(quad), x_phase, s_abort, p.err, 57);
          got = __all_sync(0xffffffffu, got);
          if (!got) { ok = false; break; }
          x_phase ^= 1u;
          const float4* x = xch + quad * (CL - 1) * 4 * 32 + lane;
#pragma unroll
          for (int d = 0; d < CL - 1; ++d)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float4 v = x[(d * 4 + c) * 32];
              float* y = rec_dh + c * 4;
              y[0] += v.x; y[1] += v.y; y[2] += v.z; y[3] += v.w;
            }
          if (p.MT > 1 && !halves) {
            __syncwarp();
            if (lane < CL - 1) mbar_arrive_cluster(mapa_u32(xfree_bar(quad), (uint32_t)((rank + 1 + lane) % CL)));
          }
        }
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int uo = hf * 8;
          // this half's columns of the accumulators (one per issuer), summed
          float s0[8], s1[8], s2[8], s3[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            s0[i] = !FWD && have_acc ? rec_dh[hf * 8 + i] : 0.f;
            s1[i] = s2[i] = s3[i] = 0.f;
          }
          if (FWD) {
            // the issuers' accumulators, GRP of them per wait (all loads of a group in flight)
            constexpr int GRP = G == 4 ? 1 : 2;
#pragma unroll
            for (int g0 = 0; g0 < NI; g0 += GRP) {
              uint32_t b0[GRP][8], b1[GRP][8], b2[GRP][8], b3[GRP][8];
#pragma unroll
              for (int k = 0; k < GRP; ++k) {
                const int i2 = g0 + k;
                if (i2 < NI && (have >> i2 & 1u)) {
                  tc_ld8(taddr + i2 * ACC_COLS + uo, b0[k]);
                  tc_ld8(taddr + i2 * ACC_COLS + 16 + uo, b1[k]);
                  tc_ld8(taddr + i2 * ACC_COLS + 32 + uo, b2[k]);
                  if (G == 4) tc_ld8(taddr + i2 * ACC_COLS + 48 + uo, b3[k]);
                }
              }
              tc_wait_ld();
#pragma unroll
              for (int k = 0; k < GRP; ++k) {
                const int i2 = g0 + k;
                if (i2 < NI && (have >> i2 & 1u)) {
#pragma unroll
                  for (int i = 0; i < 8; ++i) {
                    s0[i] += __uint_as_float(b0[k][i]);
                    s1[i] += __uint_as_float(b1[k][i]);
                    s2[i] += __uint_as_float(b2[k][i]);
                    if (G == 4) s3[i] += __uint_as_float(b3[k][i]);
                  }
                }
              }
            }
            if (hf == 1) {  // both halves are in registers: the accumulator buffer is free
              tc_fence_before();
              mbar_arrive(acce_bar(acc));
              if (warp == NI + 1 && lane == 0) HB_STAMP(p, it, mt, 5);
            }
          }
          if (valid && u0 + uo < H) {
            if (FWD && G == 4) {
              float hn[8], vi[8], vg[8], vf[8], vo[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                vi[u] = rec::chain_sigmoid(bfq(in0[hf], u) + s0[u] + s_bias[uo + u]);
                vg[u] = rec::chain_tanh(bfq(in1[hf], u) + s1[u] + s_bias[16 + uo + u]);
                vf[u] = rec::chain_sigmoid(bfq(in2[hf], u) + s2[u] + s_bias[32 + uo + u]);
                vo[u] = rec::chain_sigmoid(bfq(in3[hf], u) + s3[u] + s_bias[48 + uo + u]);
                carry[hf][u] = vf[u] * carry[hf][u] + vi[u] * vg[u];
                float x = vo[u] * rec::chain_tanh(carry[hf][u]);
                if (p.has_zoneout)
                  x = p.training ? zoneout<true>(x, bfq(hp[hf], u), p.zoneout_prob, bfq(mk[hf], u))
                                 : zoneout<false>(x, bfq(hp[hf], u), p.zoneout_prob, 0.f);
                hn[u] = x;
              }
              st8(p.h + (long long)(t + 1) * NH + o0 + uo, hn);  // the next step streams it
              st8(p.c + (long long)(t + 1) * NH + o0 + uo, carry[hf]);
              st_carry(p.c_carry + o0 + uo, carry[hf]);
              if (p.training) {
                bf16* vt = p.v + ((long long)t * N + n) * 4 * H + u0 + uo;
                st8(vt, vi); st8(vt + H, vg); st8(vt + 2 * H, vf); st8(vt + 3 * H, vo);
              }
            } else if (FWD) {
              float hn[8], vz[8], vr[8], vg[8], vq[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const float hprev = bfq(hp[hf], u);
                const float z = rec::chain_sigmoid(bfq(in0[hf], u) + s0[u] + s_bias[uo + u] + s_bias[48 + uo + u]);
                const float rr = rec::chain_sigmoid(bfq(in1[hf], u) + s1[u] + s_bias[16 + uo + u] + s_bias[64 + uo + u]);
                const float qg = s2[u] + s_bias[80 + uo + u];
                const float g = rec::chain_tanh(bfq(in2[hf], u) + rr * qg + s_bias[32 + uo + u]);
                float x = z * hprev + (1.0f - z) * g;
                if (p.has_zoneout)
                  x = p.training ? zoneout<true>(x, hprev, p.zoneout_prob, bfq(mk[hf], u))
                                 : zoneout<false>(x, hprev, p.zoneout_prob, 0.f);
                hn[u] = x; vz[u] = z; vr[u] = rr; vg[u] = g; vq[u] = qg;
              }
              st8(p.h + (long long)(t + 1) * NH + o0 + uo, hn);  // the next step streams it
              if (p.training && p.v) {
                bf16* vt = p.v + ((long long)t * N + n) * 4 * H + u0 + uo;
                st8(vt, vz); st8(vt + H, vr); st8(vt + 2 * H, vg); st8(vt + 3 * H, vq);
              }
            } else if (G == 4) {
              float di[8], dg[8], df[8], d_o[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const float gv[4] = {bfq(in0[hf], u), bfq(in1[hf], u), bfq(in2[hf], u), bfq(in3[hf], u)};
                float d[4];
                rec::cell_bwd<4, true>(gv, bfq(hp[hf], u), c_tanh[hf][u], carry[hf][u] + s0[u], 0.f, p.has_zoneout != 0,
                                       p.has_zoneout ? bfq(mk[hf], u) : 1.f, carry[hf][u], dc0[hf][u], d);
                di[u] = d[0]; dg[u] = d[1]; df[u] = d[2]; d_o[u] = d[3];
              }
              bf16* vt = p.v + ((long long)t * N + n) * 4 * H + u0 + uo;  // streamed next
              st8(vt, di); st8(vt + H, dg); st8(vt + 2 * H, df); st8(vt + 3 * H, d_o);
              st_carry(p.dh_carry + o0 + uo, carry[hf]);
              st_carry(p.c_carry + o0 + uo, dc0[hf]);
            } else {
              float dpz[8], dpr[8], dpg[8], dqg[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const float z = bfq(in0[hf], u), rr = bfq(in1[hf], u), g = bfq(in2[hf], u),
                            qg = bfq(in3[hf], u);
                float dh_total = carry[hf][u] + s0[u];
                float keep = 0.f;
                if (p.has_zoneout) {
                  const float m = bfq(mk[hf], u);
                  keep = (1.0f - m) * dh_total;
                  dh_total = m * dh_total;
                }
                const float dg = (1.0f - z) * dh_total;
                const float dz = (bfq(hp[hf], u) - g) * dh_total;
                const float dp_g = d_tanh(g) * dg;
                dpz[u] = d_sigmoid(z) * dz;
                dpr[u] = d_sigmoid(rr) * (dp_g * qg);
                dpg[u] = dp_g;
                dqg[u] = dp_g * rr;
                carry[hf][u] = keep + z * dh_total;
              }
              const long long w0 = ((long long)t * N + n) * 3 * H + u0 + uo;
              st8(p.dq + w0, dpz); st8(p.dq + w0 + H, dpr); st8(p.dq + w0 + 2 * H, dqg);  // streamed next
              st8(p.dp + w0, dpz); st8(p.dp + w0 + H, dpr); st8(p.dp + w0 + 2 * H, dpg);
              st_carry(p.dh_carry + o0 + uo, carry[hf]);
            }
          }
        }
        if (warp == NI + 1 && lane == 0) HB_STAMP(p, it, mt, 6);  // gate math done, h / dq stored
        // ---- publish.  The warp barrier orders every lane's stores before lane 0's release,
        // and a release at GPU scope is cumulative: it makes visible what happened before it
        // in any thread it synchronised with, so the one red.release counts the warp's arrival
        // and publishes all 32 lanes' stores.  (A __threadfence() in front of it cost another
        // 0.5 us per step and changed nothing.)  Only lane 0 waits; the other lanes go on to
        // the next step's loads.  Rows beyond the batch store nothing but still arrive.
        // SPLIT: the tile's last warp arrives for all of them (GRU, H = 1024, 128 rows 8.4 -> 8.0 us per step;
        // forward 7.1 -> 6.7, but two tiles per CTA 8.0 -> 9.1).
        __syncwarp();
        if (lane == 0) {
          const uint32_t others = halves ? 1u : 3u;
          if (!SPLIT || (add_acq_rel_cta(s_done + 4 * (uint32_t)mt, 1u) & others) == others) red_release_add(p.cnt + tile, 1u);
        }
        if (warp == NI + 1 && lane == 0) HB_STAMP(p, it, mt, 7);  // published
      }
    }
  }

  // Drain: every role arrives here, also after a time-out, so tensor memory is released.
  tc_fence_before();
  __syncthreads();
  if (*s_abort) atomicExch(p.abort_flag, 1);
  if (SPLIT) {  // nobody leaves while another may still write to it
    if (*s_abort)  // (nor before what is under way has arrived: nobody waits for it then)
      for (const long long t0 = clock64(); clock64() - t0 < 100000;) {}
    cluster_sync_all();
  }
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(TMEM_COLS)
                 : "memory");
  }
}

// ---- host side ---------------------------------------------------------------------------
// How many clusters of the backward kernel with SPLIT the device holds at once; 0: none.
int max_tc_clusters() {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> most[kMaxDevices];  // 0: not asked yet, -1: none
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  int n = most[dev].load(std::memory_order_acquire);
  if (n == 0) {
    n = -1;
    auto kernel = tc_recurrence_kernel<3, false, CLUSTER>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count() / CLUSTER * CLUSTER);
    cfg.blockDim = dim3(tc_threads<CLUSTER>());
    cfg.dynamicSmemBytes = MAX_SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CLUSTER;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0)
      n = min(clusters, sm_count() / CLUSTER);
    cudaGetLastError();
    most[dev].store(n, std::memory_order_release);
  }
  return n > 0 ? n : 0;
}

struct TcGeometry {
  int nHS, nRG, MT, RB, stages, CL;
  size_t ring, smem;
};

// Shapes this path takes: bf16, H a multiple of 8 up to 1024 (the resident slice of R and a useful ring
// must fit shared memory), at least 64 batch rows and at most two row tiles per CTA: every CTA of a row
// group streams the group's whole h (or dq), H / 16 copies of it per step out of L2, so that a third and
// a fourth tile cost as much again, where the step-wise path's full-size contractions grow little.  GRU,
// H = 1024, us per step forward / backward, this / step by step: 128 rows 7.0 / 8.0 and 19.3 / 18.5, 256
// rows 8.0 / 10.4 and 22.6 / 18.6, 512 rows 10.2 / 16.2 and 20.5 / 22.7; 1024 rows step by step 30.4 / 30.2.
// LSTM: 256 rows 9.8 / 10.1 and 16.5 / 21.8, 512 rows 14.0 / 17.8 and 20.5 / 28.3.
// (Where the chain kernels take a batch themselves: rec_chain_host.cu.)
bool tc_geometry_of(int G, int N, int H, bool fwd, int CL, int sms, TcGeometry* g) {
  const int K = fwd ? H : G * H;
  g->CL = CL;
  const size_t r_bytes = (size_t)ceil_div(ceil_div(K, BK), CL) * (fwd ? G : CL) * UC * 128;
  const size_t fixed = 1024 /*alignment*/ + r_bytes + (CL > 1 ? XCH : 0) + 1024 /*barriers, bias*/;
  if (fixed + 2 * (size_t)A_STAGE > (size_t)MAX_SMEM) return false;
  g->nHS = ceil_div(H, UC);
  if (CL > 1) {  // whole clusters, as many as are resident at a time
    g->nHS = ceil_div(g->nHS, CLUSTER) * CLUSTER;
    sms = (int)((long long)max_tc_clusters() * sms / sm_count()) * CLUSTER;
  }
  const int groups_max = sms / g->nHS;
  if (groups_max < 1) return false;
  // 64-row tiles when that still gives one tile per CTA (more CTAs, less to stream per CTA)
  for (int rb = 64; rb <= 128; rb *= 2) {
    const int tiles = ceil_div(N, rb);
    const int mt = ceil_div(tiles, groups_max);
    // (the second 64-row tile's MMAs read 8 KB in front of their stage: there has to be as much R)
    if (rb == 64 && (mt > 2 || (mt == 2 && r_bytes < (size_t)rb * 128))) continue;
    if (mt > 2) return false;
    g->RB = rb;
    g->MT = mt;
    g->nRG = ceil_div(tiles, mt);
    // ring: as many stages of one k-block (rb rows x 128 bytes) as shared memory holds, up
    // to 16; bytes in flight are what the streaming rate of a step is made of
    const size_t stage = (size_t)rb * 128, pad = A_STAGE - stage;
    int stages = (int)(((size_t)MAX_SMEM - fixed - pad) / stage);
    if (stages > 16) stages = 16;
    if (stages < PL) return false;  // every lane owns a stage
    g->stages = stages;
    g->ring = stages * stage + pad;
    g->smem = fixed + g->ring;
    return true;
  }
  return false;
}

// Backward, K = G * H: a CTA that streams dq over all of K for its 16 units reads 128 rows at 64 bytes per clock and
// as long again into the tensor cores (65 cycles per MMA, whatever its columns).  A cluster of four shares out K
// instead: each CTA streams a quarter of it for the 64 units of all, and the partial dh - 24 KB in and out
// - travel through distributed shared memory.  That takes 1500 cycles of its own, so short K stays unsplit, and so
// does what would take more rows per CTA (clusters leave some SMs out).  us per step, all of K / a quarter: GRU
// H = 1024 128 rows 10.2 / 8.0, half of the GPU 11.9 / 9.8, 178 rows H = 808 19.2 / 13.6, 256 rows H = 640 15.0 / 15.5,
// H = 512 8.1 / 8.5; LSTM H = 1024 256 rows 19.6 / 10.1 (of that 4 from the tanh of c, now taken before the wait), 128
// rows on half of the GPU 19.3 / 9.7, H = 512 512 rows 13.1 / 9.9, H = 320 700 rows 8.0 / 9.0.
constexpr int kSplitK = 2048;

bool tc_geometry_for(int G, int N, int H, bool fwd, int sms, TcGeometry* g) {
  const bool whole = tc_geometry_of(G, N, H, fwd, 1, sms, g);
  TcGeometry split;
  if (!fwd && G * H >= kSplitK && tc_geometry_of(G, N, H, fwd, CLUSTER, sms, &split) &&
      (!whole || split.MT * split.RB <= g->MT * g->RB)) {
    *g = split;
    return true;
  }
  return whole;
}

// Under an SM budget (concurrent directions) the geometry within it, so that the two directions are
// co-resident; where that would need more than two tiles per CTA, the whole GPU.
bool tc_geometry(int G, int N, int H, bool fwd, TcGeometry* g) {
  if (H % 8 != 0 || H < 64 || H > 1024 || N < 64) return false;
  const int budget = sm_budget();
  return (budget > 0 && budget < sm_count() && tc_geometry_for(G, N, H, fwd, budget, g)) ||
         tc_geometry_for(G, N, H, fwd, sm_count(), g);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <int G, bool FWD, int CL>
int launch_tc(const CUtensorMap& map, TcParams& p, const TcGeometry& g, cudaStream_t s) {
  auto kernel = tc_recurrence_kernel<G, FWD, CL>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)g.smem);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return HASTE_B200_ERR_UNSUPPORTED;
  }
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, tc_threads<CL>(), g.smem);
  const int grid = g.nHS * g.nRG;
  if (e != cudaSuccess || per_sm * sm_count() < grid) {
    cudaGetLastError();
    return HASTE_B200_ERR_UNSUPPORTED;
  }
  int stages = g.stages;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(tc_threads<CL>());
  cfg.dynamicSmemBytes = g.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CL;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CL > 1 ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, kernel, map, static_cast<const TcParams&>(p), static_cast<const int&>(stages));
  if (e != cudaSuccess) {
    set_last_error("cooperative launch failed: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return HASTE_B200_ERR_CUDA;
  }
  count_launch(1);
  return HASTE_B200_OK;
}

#ifdef HASTE_B200_TIMING_EXPERIMENTS
long long* g_stamps = nullptr;
int g_stamp_steps = 0;
#endif

// Zeroed scratch: abort flag + one arrival counter per row tile.
int tc_scratch(int tiles, TcParams* p, cudaStream_t s) {
  const size_t bytes = Arena::pad(4096) + Arena::pad((size_t)tiles * 4);
  Arena ws;
  HB_TRY(make_arena(&ws, s, bytes + 512, /*slot=*/2));
  int* flag = ws.take<int>(1024);
  unsigned int* cnt = ws.take<unsigned int>(tiles);
  HB_REQUIRE(flag && cnt, "scratch arena");
  HB_CUDA_OK(cudaMemsetAsync(flag, 0, bytes, s));
  p->abort_flag = flag;
  p->cnt = cnt;
  p->err = device_error_word();
  HB_REQUIRE(p->err, "error word");
#ifdef HASTE_B200_TIMING_EXPERIMENTS
  if (!g_stamps) cudaMalloc(&g_stamps, (size_t)4096 * 16 * sizeof(long long));
  cudaMemsetAsync(g_stamps, 0, (size_t)4096 * 16 * sizeof(long long), s);
  p->stamps = p->T <= 4096 ? g_stamps : nullptr;
  g_stamp_steps = p->T;
#endif
  return HASTE_B200_OK;
}

}  // namespace

bool lstm_tc_takes(int dtype, int N, int H, bool fwd) {
  TcGeometry g;
  return dtype == HASTE_B200_BF16 && recurrence_path() != HASTE_B200_PATH_STEPWISE &&
         recurrence_path() != HASTE_B200_PATH_NO_TENSOR_CORE && encode_fn() &&
         tc_geometry(4, N, H, fwd, &g);
}

// Forward: x.W is already in a.tmp_Wx.  HASTE_B200_ERR_UNSUPPORTED (nothing touched) when the
// shape is not this path's.
int gru_forward_tc(const GruFwd& a, cudaStream_t s) {
  TcGeometry g;
  if (a.dtype != HASTE_B200_BF16 || recurrence_path() == HASTE_B200_PATH_STEPWISE ||
      recurrence_path() == HASTE_B200_PATH_NO_TENSOR_CORE || a.h_out ||
      !encode_fn() || !tc_geometry(3, a.N, a.H, true, &g))
    return HASTE_B200_ERR_UNSUPPORTED;
  if (!aligned16(a.R) || !aligned16(a.tmp_Wx) || !aligned16(a.h) || !aligned16(a.v) ||
      !aligned16(a.zoneout_mask) || !aligned16(a.bx) || !aligned16(a.br))
    return HASTE_B200_ERR_UNSUPPORTED;
  CUtensorMap map;
  if (!make_map(&map, a.h, a.H, (long long)(a.T + 1) * a.N, a.H, 0, 1, BK, g.RB))
    return HASTE_B200_ERR_UNSUPPORTED;
  const bool zo = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  TcParams p{};
  p.T = a.T; p.N = a.N; p.H = a.H; p.nHS = g.nHS; p.MT = g.MT; p.RB = g.RB;
  p.stage_bytes = g.RB * 128; p.ring_bytes = (int)g.ring;
  p.training = a.training; p.has_zoneout = zo ? 1 : 0; p.zoneout_prob = a.zoneout_prob;
  p.R = (const bf16*)a.R; p.bx = (const bf16*)a.bx; p.br = (const bf16*)a.br;
  p.Wx = (const bf16*)a.tmp_Wx; p.mask = (const bf16*)a.zoneout_mask;
  p.h = (bf16*)a.h; p.v = (bf16*)a.v;
  HB_TRY(tc_scratch(ceil_div(a.N, g.RB), &p, s));
  return launch_tc<3, true, 1>(map, p, g, s);
}

// Backward: dh_carry (fp32 [N,H]) holds the incoming gradient of the final state and receives
// the carry after the last processed step, without the recurrent contribution of that step
// (the caller adds dq_0 . R^T).  Bias gradients are NOT summed here.
int gru_backward_tc(const GruBwd& a, float* dh_carry, cudaStream_t s) {
  TcGeometry g;
  if (a.dtype != HASTE_B200_BF16 || recurrence_path() == HASTE_B200_PATH_STEPWISE ||
      recurrence_path() == HASTE_B200_PATH_NO_TENSOR_CORE || a.iterate ||
      !encode_fn() || !tc_geometry(3, a.N, a.H, false, &g))
    return HASTE_B200_ERR_UNSUPPORTED;
  if (!aligned16(a.R) || !aligned16(a.h) || !aligned16(a.v) || !aligned16(a.dh_new) ||
      !aligned16(a.dp) || !aligned16(a.dq) || !aligned16(a.zoneout_mask) || !aligned16(dh_carry))
    return HASTE_B200_ERR_UNSUPPORTED;
  CUtensorMap map;
  if (!make_map(&map, a.dq, 3LL * a.H, (long long)a.T * a.N, 3LL * a.H, 0, 1, BK, g.RB))
    return HASTE_B200_ERR_UNSUPPORTED;
  TcParams p{};
  p.T = a.T; p.N = a.N; p.H = a.H; p.nHS = g.nHS; p.MT = g.MT; p.RB = g.RB;
  p.stage_bytes = g.RB * 128; p.ring_bytes = (int)g.ring;
  p.has_zoneout = a.zoneout_mask ? 1 : 0; p.r_transposed = a.transposed_inputs;
  p.R = (const bf16*)a.R; p.mask = (const bf16*)a.zoneout_mask;
  p.h = (bf16*)const_cast<void*>(a.h); p.v = (bf16*)const_cast<void*>(a.v);
  p.dh_new = (const bf16*)a.dh_new; p.dp = (bf16*)a.dp; p.dq = (bf16*)a.dq;
  p.dh_carry = dh_carry;
  HB_TRY(tc_scratch(ceil_div(a.N, g.RB), &p, s));
  return g.CL > 1 ? launch_tc<3, false, CLUSTER>(map, p, g, s) : launch_tc<3, false, 1>(map, p, g, s);
}

// LSTM, in the same way: x.W is in a.v; c_carry (fp32 [N,H]) holds c_0.
int lstm_forward_tc(const LstmFwd& a, float* c_carry, cudaStream_t s) {
  TcGeometry g;
  if (!lstm_tc_takes(a.dtype, a.N, a.H, true) || !tc_geometry(4, a.N, a.H, true, &g) || !aligned16(a.R) ||
      !aligned16(a.h) || !aligned16(a.c) || !aligned16(a.v) || !aligned16(a.zoneout_mask) || !aligned16(c_carry))
    return HASTE_B200_ERR_UNSUPPORTED;
  CUtensorMap map;
  if (!make_map(&map, a.h, a.H, (long long)(a.T + 1) * a.N, a.H, 0, 1, BK, g.RB))
    return HASTE_B200_ERR_UNSUPPORTED;
  TcParams p{};
  p.T = a.T; p.N = a.N; p.H = a.H; p.nHS = g.nHS; p.MT = g.MT; p.RB = g.RB;
  p.stage_bytes = g.RB * 128; p.ring_bytes = (int)g.ring;
  p.training = a.training; p.has_zoneout = a.zoneout_prob != 0.0f && a.zoneout_mask != nullptr;
  p.zoneout_prob = a.zoneout_prob;
  p.R = (const bf16*)a.R; p.bx = (const bf16*)a.b; p.Wx = (const bf16*)a.v; p.mask = (const bf16*)a.zoneout_mask;
  p.h = (bf16*)a.h; p.c = (bf16*)a.c; p.v = (bf16*)a.v; p.c_carry = c_carry;
  HB_TRY(tc_scratch(ceil_div(a.N, g.RB), &p, s));
  return launch_tc<4, true, 1>(map, p, g, s);
}

// v: gates in, gate gradients out.  dh_carry, dc_carry as dh_carry of gru_backward_tc.
int lstm_backward_tc(const LstmBwd& a, float* dh_carry, float* dc_carry, cudaStream_t s) {
  TcGeometry g;
  if (!lstm_tc_takes(a.dtype, a.N, a.H, false) || !tc_geometry(4, a.N, a.H, false, &g) || !aligned16(a.R) ||
      !aligned16(a.c) || !aligned16(a.v) || !aligned16(a.dh_new) || !aligned16(a.dc_new) ||
      !aligned16(a.zoneout_mask) || !aligned16(dh_carry) || !aligned16(dc_carry))
    return HASTE_B200_ERR_UNSUPPORTED;
  CUtensorMap map;
  if (!make_map(&map, a.v, 4LL * a.H, (long long)a.T * a.N, 4LL * a.H, 0, 1, BK, g.RB))
    return HASTE_B200_ERR_UNSUPPORTED;
  TcParams p{};
  p.T = a.T; p.N = a.N; p.H = a.H; p.nHS = g.nHS; p.MT = g.MT; p.RB = g.RB;
  p.stage_bytes = g.RB * 128; p.ring_bytes = (int)g.ring;
  p.has_zoneout = a.zoneout_mask ? 1 : 0; p.r_transposed = a.transposed_inputs;
  p.R = (const bf16*)a.R; p.mask = (const bf16*)a.zoneout_mask;
  p.c = (bf16*)const_cast<void*>(a.c); p.v = (bf16*)a.v; p.dh_new = (const bf16*)a.dh_new;
  p.dc_new = (const bf16*)a.dc_new; p.dh_carry = dh_carry; p.c_carry = dc_carry;
  HB_TRY(tc_scratch(ceil_div(a.N, g.RB), &p, s));
  return g.CL > 1 ? launch_tc<4, false, CLUSTER>(map, p, g, s) : launch_tc<4, false, 1>(map, p, g, s);
}

#ifdef HASTE_B200_TIMING_EXPERIMENTS
// Timing-experiment builds only: the clock64 stamps the last tensor-core recurrence launch
// left (CTA 0, tile 0; eight per step), copied to host memory.
extern "C" int haste_b200_debug_read_stamps(long long* out, int max_steps) {
  if (!g_stamps) return 0;
  const int n = g_stamp_steps < max_steps ? g_stamp_steps : max_steps;
  cudaDeviceSynchronize();
  cudaMemcpy(out, g_stamps, (size_t)n * 16 * sizeof(long long), cudaMemcpyDeviceToHost);
  return n;
}
#endif

}  // namespace hb
