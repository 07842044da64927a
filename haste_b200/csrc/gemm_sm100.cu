// Dense contraction on the 5th-generation tensor cores (sm_100a):
//   TMA (cp.async.bulk.tensor, 128-byte swizzle) -> shared memory -> tcgen05.mma with
//   the fp32 accumulator in tensor memory -> tcgen05.ld epilogue.
//
//   C[M,N] (+)= sum over products p of A_p[M,K] . B_p[K,N]        (bf16 operands)
//
// * bf16 storage: one product, operands read in place.
// * fp32 storage: every operand is first split into two bf16 planes, x = hi + lo with
//   hi = bf16(x), lo = bf16(x - hi), and three products are accumulated
//   (hi.hi + hi.lo + lo.hi).  The dropped lo.lo term and the plane rounding leave a
//   relative error near 2^-17 per product, far inside the 1e-4 parity bar, at 3/16 of
//   the fp32 CUDA-core cost.
// * fp32 storage, large contractions whose error a LayerNorm or a long recurrence would amplify: two
//   fp16 planes per operand, scaled by row and column (see split_f16_kernel), three products.
// * Either operand may be K-major or MN-major (every transpose the cells need), chosen
//   from its strides; no data is ever transposed in memory.
// * Persistent kernel: one CTA per SM walks (tile, k-split) work items.  Warp 0 issues
//   TMA, warp 1 issues MMA, warps 2-5 drain the accumulator; two accumulators in tensor
//   memory let the epilogue of one tile overlap the main loop of the next.
// * Long-K, small-output contractions (the weight gradients, K = T*N) are split along K;
//   partial tiles go to scratch and a second kernel sums them in a fixed order.
// * Every wait on an mbarrier is bounded; on expiry the kernel raises an error word,
//   all roles drain and exit, tensor memory is released and the host returns
//   HASTE_B200_ERR_TIMEOUT.
//
// Replaces the cuBLAS calls of the reference (lib/blas.h:48-61 and the call sites in
// lib/*_gpu.cu.cc).
#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>

#include "cells.cuh"
#include "tcgen05.cuh"

namespace hb {
namespace {

using namespace tc;

constexpr int BM = 128, BN = 128, BK = 64;   // CTA tile; BK bf16 = one 128-byte swizzle row
constexpr int UK = 16;                       // K of one tcgen05.mma (bf16)
constexpr int TILE_BYTES = BM * BK * 2;      // one operand plane of one stage (A or B): 16 KiB
constexpr int THREADS = 192;                 // warp 0 TMA, warp 1 MMA, warps 2..5 epilogue
constexpr int NACC = 4;                      // fp32 accumulators of BN columns in tensor memory
constexpr int EPI_TILE = 32 * 32 * 4;         // shared memory of an epilogue warp
constexpr int TMEM_COLS = NACC * BN;         // (all 512 columns: one CTA per SM)

struct Params {
  int M, N, K;
  int a_mn_major, b_mn_major;  // 0: K contiguous, 1: M/N contiguous
  int tiles_m, tiles_n, splits, kb_per_split, kb_total;
  int c_is_bf16, accumulate;   // direct epilogue only; c_is_bf16: 0 fp32, 1 bf16, 2 fp16 output
  int wide;                    // C's rows take stores of four values
  void* c;
  long long ldc;
  const int* a_exp;            // fp16 planes: the result's row m, column n is to be scaled by
  const signed char* b_exp;    // 2^(a_exp[m] + b_exp[n]); null otherwise
  const int* uneven;           // fp16 planes: points to whether bf16 planes have taken their place
  float* partial;              // non-null: write fp32 partial tiles [split][M][partial_ld]
  int partial_ld;              // N rounded up to whole 32-column chunks
  int* err;
};

template <int NPROD>
struct Cfg {
  // 1 product: bf16 operands as they are.  3 products: (hi, lo) planes.  6 products:
  // (hi, mid, lo) planes, accurate to fp32 rounding (used where LayerNorm amplifies error).
  static constexpr int PLANES = NPROD == 1 ? 1 : (NPROD == 3 ? 2 : 3);
  static constexpr int STAGE_BYTES = 2 * PLANES * TILE_BYTES;
  static constexpr int STAGES = NPROD == 1 ? 6 : (NPROD == 3 ? 3 : 2);
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;  // + a tile per epilogue warp
  // fp32 storage: the tensor core adds every MMA result into the fp32 accumulator with
  // truncation, a bias of about half an ulp per accumulation that always points the same way;
  // over the few hundred accumulations of a long K it reaches 1e-5 of the result (measured:
  // 1.2e-5 at K = 1024 with six products, where the operand planes themselves are exact to
  // 2^-25).  The accumulator is therefore handed over every CHUNK k-blocks: the epilogue warps
  // add it into fp32 registers with round-to-nearest while the MMA warp continues in the
  // other accumulator.  0: one hand-over per tile (bf16 storage, where 2e-2 is the bar).
  // Four accumulators take turns, so the MMA warp runs up to three chunks ahead of the
  // epilogue; a chunk is about 1.6 us of MMA work either way.
  // (Twice these chunk lengths fails the fp32 parity test of the three-layer LayerNormLSTM stack.)
  static constexpr int CHUNK = NPROD == 1 ? 0 : (NPROD == 3 ? 4 : 2);
};

__device__ __forceinline__ float exp2_int(int e) {  // 2^e, -126 <= e <= 127
  return __uint_as_float((uint32_t)(e + 127) << 23);
}

// Planes: bf16; two of fp16; three of bf16 in the place of those, handed over as often per product.
enum { PLAIN, F16_PLANES, UNEVEN };

// The powers of two that fp16 planes leave in a tile: of this lane's row, and of the four columns that the lane
// stores of the chunk from n0 on.  (Loaded when they are used: the sums fill the registers till then.)
__device__ __forceinline__ int row_scale(const Params& p, int m0) {
  const int m = m0 + (threadIdx.x & 31);
  return m < p.M ? p.a_exp[m] : 0;
}
__device__ __forceinline__ int column_scales(const Params& p, int n0) {
  return *reinterpret_cast<const int*>(p.b_exp + n0 + (threadIdx.x & 7) * 4);
}
// Rows 0 .. rows - 1 of a 32 x 32 tile in shared memory (laid out by fill_tile) to dst, `cols` columns wide.
// `ea`, `eb`: row_scale, column_scales.  Whether C is added to is known to the code where one product is
// (bf16 64000 x 2048, K = 512 210 us, tested in the loop 220); with several, whose sums fill the registers, two kinds
// of loops spilled (fp32, the same 386 tested in the loop, 395).
enum { NEVER, SURELY, EITHER };
template <bool SCALED, int ADD, typename TC>
__device__ __forceinline__ void store_tile(const float4* tile, TC* dst, long long ld_dst, int rows, int cols, bool wide,
                                           bool adds, int ea, int eb) {
  const bool add = ADD == EITHER ? adds : ADD == SURELY;
  const int lane = threadIdx.x & 31;
  if (wide) {
    const int u = lane & 7;
    float4 fb = make_float4(1.f, 1.f, 1.f, 1.f);
    if (SCALED)
      fb = make_float4(exp2_int((signed char)eb), exp2_int((signed char)(eb >> 8)), exp2_int((signed char)(eb >> 16)),
                       exp2_int(eb >> 24));
#pragma unroll 4
    for (int i = 0; i < 8; ++i) {
      const int r = i * 4 + (lane >> 3), e = SCALED ? __shfl_sync(0xffffffffu, ea, r) : 0;
      if (r >= rows || u * 4 >= cols) continue;
      float4 x = tile[r * 8 + (u ^ (r & 7))];
      if (SCALED) {
        const float f1 = exp2_int(e >> 1), f2 = exp2_int(e - (e >> 1));
        x.x = x.x * f1 * fb.x * f2; x.y = x.y * f1 * fb.y * f2;
        x.z = x.z * f1 * fb.z * f2; x.w = x.w * f1 * fb.w * f2;
      }
      TC* to = dst + r * ld_dst + u * 4;
      if constexpr (sizeof(TC) == 4) {
        if (add) {
          const float4 c = *reinterpret_cast<const float4*>(to);
          x.x += c.x; x.y += c.y; x.z += c.z; x.w += c.w;
        }
        *reinterpret_cast<float4*>(to) = x;
      } else {
        __align__(8) TC o[4];
        if (add) {
          *reinterpret_cast<uint2*>(o) = *reinterpret_cast<const uint2*>(to);
          x.x += ld(o); x.y += ld(o + 1); x.z += ld(o + 2); x.w += ld(o + 3);
        }
        st(o, x.x); st(o + 1, x.y); st(o + 2, x.z); st(o + 3, x.w);
        *reinterpret_cast<uint2*>(to) = *reinterpret_cast<const uint2*>(o);
      }
    }
  } else {
    // column `lane`, whose power its quad's lane has
    const int e4 = SCALED ? __shfl_sync(0xffffffffu, eb, lane >> 2) : 0;
    const float fb = SCALED ? exp2_int((signed char)(e4 >> 8 * (lane & 3))) : 1.f;
    const float* at = reinterpret_cast<const float*>(tile) + (lane & 3);
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
      const int e = SCALED ? __shfl_sync(0xffffffffu, ea, r) : 0;
      if (lane >= cols) continue;
      float x = at[(r * 8 + ((lane >> 2) ^ (r & 7))) * 4];
      if (SCALED) x = x * exp2_int(e >> 1) * fb * exp2_int(e - (e >> 1));
      TC* to = dst + r * ld_dst + lane;
      st(to, add ? x + ld(to) : x);
    }
  }
}
template <typename TC>
__device__ __forceinline__ void store_tile_c(const Params& p, const float4* tile, int m0, int n0) {
  TC* dst = static_cast<TC*>(p.c) + m0 * p.ldc + n0;
  const int rows = min(32, p.M - m0), cols = min(32, p.N - n0);
  const bool wide = p.wide && (cols & 3) == 0;
  if (p.accumulate) store_tile<false, SURELY, TC>(tile, dst, p.ldc, rows, cols, wide, true, 0, 0);
  else store_tile<false, NEVER, TC>(tile, dst, p.ldc, rows, cols, wide, false, 0, 0);
}

// A warp stores 32 rows (m0 ..) x 32 columns (n0 ..) of the result; lane r holds row r.  The tile goes
// through shared memory (`buf`, 4 KB of the warp's own), because a store instruction is paid per line
// it touches: 8 lanes per row write whole 128-byte lines, four per instruction instead of 32, and
// where C's rows start anywhere a warp still writes one row at a time.  The 16-byte pieces of a row
// are rotated by the row so that both sides touch all banks.
// (Row by row from the lanes, the epilogue bounded outputs with a short K and cost the others their last
// tile; before / now: bf16 64000 x 3072, K = 512 412 / 234 us, 4096^3 112 / 97; fp32 64000 x 2048, K = 512
// 424 / 346, 256000 x 1024, K = 1024 1691 / 1475, 12321 x 750, K = 161 54 / 34, which went through a padded tile.)
// fp16 planes: row m, column n times 2^(a_exp[m] + b_exp[n]), the row's power in two halves around the
// column's, so that no step leaves the range of a float unless the result does.  (b_exp is readable up
// to whole tiles.)
// (A chunk's code stands once in a kernel, in a loop: with four copies of it for every kind of C small contractions
// waited for their instructions; with cold caches, us, rows from the lanes / four copies / this: 480 x 512, K = 64
// 8.3 / 15.4 / 8.0, 32 x 4096, K = 1024 10.4 / 13.3 / 10.9.  Except for fp16 planes on pairs, which are never small
// and also scale what they store: 128000 x 512, K = 512 with the scan 440 us in a loop, 415 without.)
__device__ __forceinline__ void fill_tile(const float* v, uint8_t* buf) {
  const int lane = threadIdx.x & 31;
  float4* tile = reinterpret_cast<float4*>(buf);
#pragma unroll
  for (int j = 0; j < 8; ++j)
    tile[lane * 8 + (j ^ (lane & 7))] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
}
template <int NPROD, int MODE>
__device__ __forceinline__ void store_chunk(const Params& p, int sp, int m0, int n0, uint8_t* buf, int ea = 0, int eb = 0) {
  if (m0 >= p.M || n0 >= p.N) return;  // the same for the whole warp
  const float4* tile = reinterpret_cast<const float4*>(buf);
  __syncwarp();
  if constexpr (NPROD == 1) {
    if (p.partial)  // rows of whole chunks
      store_tile<false, NEVER, float>(tile, p.partial + ((long long)sp * p.M + m0) * p.partial_ld + n0, p.partial_ld,
                                      min(32, p.M - m0), 32, true, false, 0, 0);
    else if (p.c_is_bf16 == 0) store_tile_c<float>(p, tile, m0, n0);
    else if (p.c_is_bf16 == 1) store_tile_c<__nv_bfloat16>(p, tile, m0, n0);
    else store_tile_c<__half>(p, tile, m0, n0);
  } else {
    const int rows = min(32, p.M - m0), cols = min(32, p.N - n0);
    const bool wide = p.wide && (cols & 3) == 0;
    const long long at = m0 * p.ldc + n0;
    if (MODE != PLAIN || p.partial || p.c_is_bf16 == 0) {  // (fp16 planes: fp32 results that are not added to)
      float* dst = p.partial ? p.partial + ((long long)sp * p.M + m0) * p.partial_ld + n0 : static_cast<float*>(p.c) + at;
      store_tile<MODE == F16_PLANES, MODE == PLAIN ? EITHER : NEVER>(tile, dst, p.partial ? p.partial_ld : p.ldc, rows,
                                                                     p.partial ? 32 : cols, p.partial || wide,
                                                                     !p.partial && p.accumulate, ea, eb);
    } else if (p.c_is_bf16 == 1) {
      store_tile<false, EITHER>(tile, static_cast<__nv_bfloat16*>(p.c) + at, p.ldc, rows, cols, wide, p.accumulate, 0, 0);
    } else {
      store_tile<false, EITHER>(tile, static_cast<__half*>(p.c) + at, p.ldc, rows, cols, wide, p.accumulate, 0, 0);
    }
  }
}

// k-blocks per hand-over of the accumulator.  fp16 planes: 24 truncated accumulations, half of the bf16 planes'
// (relative error of 16384 x 1024 x 1024 against fp64: six bf16 products 1.17e-6, these 6.2e-7, with twice the chunk
// 1.07e-6 and 2 % less time).
template <int NPROD, int MODE>
constexpr int chunk_of() { return MODE == PLAIN ? Cfg<NPROD>::CHUNK : (MODE == F16_PLANES ? 2 : 1); }

template <int NPROD, int MODE = PLAIN>
__device__ __forceinline__ void gemm_tile(const CUtensorMap& map_a, const CUtensorMap& map_b, const Params& p) {
  using C = Cfg<NPROD>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + C::STAGES * C::STAGE_BYTES);
  // barrier slots: full[STAGES], empty[STAGES], acc_full[NACC], acc_empty[NACC]
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (C::STAGES + s); };
  auto accf_bar = [&](int a) { return bar0 + 8u * (2 * C::STAGES + a); };
  auto acce_bar = [&](int a) { return bar0 + 8u * (2 * C::STAGES + NACC + a); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * C::STAGES + 2 * NACC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int chunk = chunk_of<NPROD, MODE>();

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < NACC; ++a) {
      mbar_init(accf_bar(a), 1);
      mbar_init(acce_bar(a), 128);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int total_items = p.tiles_m * p.tiles_n * p.splits;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x) {
        const int tn = item % p.tiles_n;
        const int tm = (item / p.tiles_n) % p.tiles_m;
        const int sp = item / (p.tiles_n * p.tiles_m);
        const int kb0 = sp * p.kb_per_split;
        const int kb1 = min(p.kb_total, kb0 + p.kb_per_split);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.err, 1)) { ok = false; break; }
          mbar_expect_tx(full_bar(stage), C::STAGE_BYTES);
          const uint32_t sa = base + stage * C::STAGE_BYTES;
          const uint32_t sb = sa + C::PLANES * TILE_BYTES;
          const int k0 = kb * BK, m0 = tm * BM, n0 = tn * BN;
#pragma unroll
          for (int pl = 0; pl < C::PLANES; ++pl) {
            const CUtensorMap* ma = &map_a;
            const CUtensorMap* mb = &map_b;
            const uint32_t da = sa + pl * TILE_BYTES, db = sb + pl * TILE_BYTES;
            if (p.a_mn_major) {  // two boxes of 64 (m) x 64 (k)
              tma_load_3d(da, ma, full_bar(stage), m0, k0, pl);
              tma_load_3d(da + TILE_BYTES / 2, ma, full_bar(stage), m0 + 64, k0, pl);
            } else {             // one box of 64 (k) x 128 (m)
              tma_load_3d(da, ma, full_bar(stage), k0, m0, pl);
            }
            if (p.b_mn_major) {
              tma_load_3d(db, mb, full_bar(stage), n0, k0, pl);
              tma_load_3d(db + TILE_BYTES / 2, mb, full_bar(stage), n0 + 64, k0, pl);
            } else {
              tma_load_3d(db, mb, full_bar(stage), k0, n0, pl);
            }
          }
          if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t type = MODE == F16_PLANES ? 0u : 1u;  // fp16 or bf16 operands
      const uint32_t idesc = (1u << 4) | (type << 7) | (type << 10) |
                             ((uint32_t)p.a_mn_major << 15) | ((uint32_t)p.b_mn_major << 16) |
                             ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      // K-major: 8-row groups 1024 B apart, a K step of 16 elements is 32 B along the row.
      // MN-major: 8-k-row groups 1024 B apart, 64-element MN chunks one box (8192 B) apart,
      //           a K step of 16 rows is 2048 B.
      const uint32_t a_lbo = p.a_mn_major ? TILE_BYTES / 2 : 16, a_kstep = p.a_mn_major ? 2048 : 32;
      const uint32_t b_lbo = p.b_mn_major ? TILE_BYTES / 2 : 16, b_kstep = p.b_mn_major ? 2048 : 32;
      uint32_t stage = 0, phase = 0;
      uint32_t acc_phase = 0;  // one parity bit per accumulator
      int cidx = 0;  // accumulator hand-overs so far: they alternate between the two buffers
      bool ok = true;
      for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x) {
        const int sp = item / (p.tiles_n * p.tiles_m);
        const int kb0 = sp * p.kb_per_split;
        const int kb1 = min(p.kb_total, kb0 + p.kb_per_split);
        int kb = kb0;
        while (kb < kb1 && ok) {
          const int acc = cidx % NACC;
          ++cidx;
          if (!mbar_wait(acce_bar(acc), ((acc_phase >> acc) & 1u) ^ 1u, abort_flag, p.err, 2)) { ok = false; break; }
          acc_phase ^= 1u << acc;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * BN;
          const int kend = C::CHUNK ? min(kb1, kb + chunk) : kb1;
          uint32_t first = 1;
          for (; kb < kend; ++kb) {
            if (!mbar_wait(full_bar(stage), phase, abort_flag, p.err, 3)) { ok = false; break; }
            tc_fence_after();
            const uint32_t sa = base + stage * C::STAGE_BYTES;
            const uint32_t sb = sa + C::PLANES * TILE_BYTES;
#pragma unroll
            for (int pr = 0; pr < NPROD; ++pr) {
              // plane pairs, most significant first:
              //   (0,0) (0,1) (1,0) | (1,1) (0,2) (2,0)      0 = hi, 1 = mid/lo, 2 = lo
              const int ia = pr == 2 ? 1 : (pr == 3 ? 1 : (pr == 5 ? 2 : 0));
              const int ib = pr == 1 ? 1 : (pr == 3 ? 1 : (pr == 4 ? 2 : 0));
              const uint32_t pa = sa + ia * TILE_BYTES;
              const uint32_t pb = sb + ib * TILE_BYTES;
#pragma unroll
              for (int ks = 0; ks < BK / UK; ++ks) {
                const uint64_t da = smem_desc(pa + ks * a_kstep, a_lbo, 1024);
                const uint64_t db = smem_desc(pb + ks * b_kstep, b_lbo, 1024);
                tc_mma_bf16(d_tmem, da, db, idesc, first ? 0u : 1u);
                first = 0;
              }
            }
            tc_commit(empty_bar(stage));  // frees the stage once these MMAs have read it
            if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
          }
          if (ok) tc_commit(accf_bar(acc));  // this chunk of the accumulation is complete
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quad = warp & 3;  // tensor-memory lane quadrant this warp may read
    uint8_t* tile = aligned + C::STAGES * C::STAGE_BYTES + 256 + (warp - 2) * EPI_TILE;
    uint32_t acc_phase = 0;  // one parity bit per accumulator
    int cidx = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < total_items; item += gridDim.x) {
      const int tn = item % p.tiles_n;
      const int tm = (item / p.tiles_n) % p.tiles_m;
      const int sp = item / (p.tiles_n * p.tiles_m);
      const int kb0 = sp * p.kb_per_split;
      const int kb1 = min(p.kb_total, kb0 + p.kb_per_split);
      const int nchunks = C::CHUNK ? (kb1 - kb0 + chunk - 1) / max(chunk, 1) : 1;
      const int m0 = tm * BM + quad * 32;
      const int n0 = tn * BN;
      // running sums of this thread's row of the tile (only with chunked hand-over)
      float sum[C::CHUNK ? BN : 1];
#pragma unroll
      for (int j = 0; j < (C::CHUNK ? BN : 1); ++j) sum[j] = 0.f;
      for (int c = 0; c < nchunks; ++c) {
        const int acc = cidx % NACC;
        ++cidx;
        if (ok) ok = mbar_wait(accf_bar(acc), (acc_phase >> acc) & 1u, abort_flag, p.err, 4);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        acc_phase ^= 1u << acc;
        tc_fence_after();
        const uint32_t taddr = tmem_base + acc * BN + ((uint32_t)(quad * 32) << 16);
        if (C::CHUNK) {
#pragma unroll
          for (int ch = 0; ch < BN / 32; ++ch) {
            uint32_t r[32];
            tc_ld32(taddr + ch * 32, r);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) sum[(C::CHUNK ? ch * 32 : 0) + j] += __uint_as_float(r[j]);
          }
        } else {
#pragma unroll 1
          for (int ch = 0; ch < BN / 32 && m0 < p.M && n0 + ch * 32 < p.N; ++ch) {
            uint32_t r[32];
            tc_ld32(taddr + ch * 32, r);
            tc_wait_ld();
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            __syncwarp();  // the tile before has been read
            fill_tile(v, tile);
            store_chunk<NPROD, MODE>(p, sp, m0, n0 + ch * 32, tile);
          }
        }
        tc_fence_before();
        mbar_arrive(acce_bar(acc));
      }
      if (!ok) break;
      if (C::CHUNK) {
        // Partial tiles of few rows leave from the lanes: one tile per CTA, and the four trips through shared memory, one
        // after the other, take 2 us longer than their stores (64 x 2048, K = 512 20.7 / 18.7 us, 32 x 4096, K = 1024
        // 24.9 / 22.8).
        if (MODE == PLAIN && p.partial && p.M <= 64) {
          const int m = m0 + lane;
          float* dst = p.partial + ((long long)sp * p.M + m) * p.partial_ld + n0;
#pragma unroll
          for (int j = 0; j < (C::CHUNK ? BN : 0); j += 4)
            if (m < p.M && n0 + j < p.partial_ld)
              *reinterpret_cast<float4*>(dst + j) = make_float4(sum[j], sum[j + 1], sum[j + 2], sum[j + 3]);
          continue;
        }
        const int ea = MODE == F16_PLANES ? row_scale(p, m0) : 0;
#pragma unroll 1
        for (int ch = 0; ch < BN / 32; ++ch) {
          const int eb = MODE == F16_PLANES ? column_scales(p, n0 + ch * 32) : 0;
          __syncwarp();  // the tile before has been read
#pragma unroll
          for (int c = 0; c < BN / 32; ++c)
            if (c == ch) fill_tile(sum + (C::CHUNK ? c * 32 : 0), tile);
          store_chunk<NPROD, MODE>(p, sp, m0, n0 + ch * 32, tile, ea, eb);
        }
      }
    }
  }

  // Drain: every role arrives here, also after a time-out, so tensor memory is released.
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
  }
}

template <int NPROD>
__global__ void __launch_bounds__(THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ Params p) {
  gemm_tile<NPROD>(map_a, map_b, p);
}
// fp16 planes, or the bf16 planes that have taken their place.
__global__ void __launch_bounds__(THREADS, 1)
gemm_tcgen05_f16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                        const __grid_constant__ CUtensorMap bf_a, const __grid_constant__ CUtensorMap bf_b,
                        const __grid_constant__ Params p) {
  if (*p.uneven) gemm_tile<6, UNEVEN>(bf_a, bf_b, p);
  else gemm_tile<3, F16_PLANES>(map_a, map_b, p);
}

// ---- the same contraction on CTA pairs ------------------------------------------------------
// The single-CTA kernel above runs at (shared-memory ring bytes) / (load latency): a 128 x 128
// tile needs 32 KB of operands per 64-wide k-block and product, about twice what the ring can
// have in flight per unit of tensor-pipe time.  Here two CTAs of a cluster share a 256 x 256
// tile (tcgen05.mma.cta_group::2, M = 256): each CTA loads its own 128 rows of A and its own
// 128-column half of B - the same two 16 KB boxes per plane as above - and the tensor cores of
// both SMs read both halves of B, so every loaded byte feeds twice the arithmetic.  Each CTA's
// tensor memory holds its 128 rows x 256 columns of the accumulator (two accumulators of 256
// columns).  CTA 0 of the pair issues all MMAs; its full barriers count the bytes of both
// CTAs' loads (the loads name the barrier through cta_group::2; every CTA fetches its own
// tiles), its commits arrive on the empty and accumulator-full barriers of both CTAs, and both
// CTAs' epilogue warps (eight per CTA: four lane quadrants x two column halves) arrive on its
// accumulator-empty barriers.
constexpr int PAIR_THREADS = 320;        // warp 0 TMA, warp 1 MMA / tensor memory, warps 2..9 epilogue
constexpr int PBN = 256;                 // columns of the pair's tile and of one accumulator
constexpr int PBM = 256;                 // rows of the pair's tile (128 per CTA)
constexpr int PAIR_NACC = 2;
constexpr int PAIR_EPI_WARPS = 8;

// (Ten warps put three on two of the SM's four sub-partitions, 16384 registers each, so 168
// registers per thread is the most a 320-thread CTA can have; the epilogue therefore drains the
// accumulator 16 columns at a time.)
template <int NPROD, int MODE = PLAIN>
__device__ __forceinline__ void gemm_pair(const CUtensorMap& map_a, const CUtensorMap& map_b, const Params& p) {
  using C = Cfg<NPROD>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + C::STAGES * C::STAGE_BYTES);
  // barrier slots: full[STAGES], empty[STAGES], acc_full[2], acc_empty[2]
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (C::STAGES + s); };
  auto accf_bar = [&](int a) { return bar0 + 8u * (2 * C::STAGES + a); };
  auto acce_bar = [&](int a) { return bar0 + 8u * (2 * C::STAGES + PAIR_NACC + a); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * C::STAGES + 2 * PAIR_NACC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 issues the MMAs
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  constexpr int chunk = chunk_of<NPROD, MODE>();

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(full_bar(s), 1);   // CTA 0's producer; the bytes of both CTAs' loads
      mbar_init(empty_bar(s), 1);  // one commit
    }
    for (int a = 0; a < PAIR_NACC; ++a) {
      mbar_init(accf_bar(a), 1);
      mbar_init(acce_bar(a), 2 * PAIR_EPI_WARPS);  // one arrival per epilogue warp of both CTAs
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    // collective over the pair: the same warp of both CTAs, the same shared-memory slot
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"((uint32_t)(PAIR_NACC * PBN))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int total_items = p.tiles_m * p.tiles_n * p.splits;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int item = pair; item < total_items && ok; item += npairs) {
        const int tn = item % p.tiles_n;
        const int tm = (item / p.tiles_n) % p.tiles_m;
        const int sp = item / (p.tiles_n * p.tiles_m);
        const int kb0 = sp * p.kb_per_split;
        const int kb1 = min(p.kb_total, kb0 + p.kb_per_split);
        const int m0 = tm * PBM + (int)rank * BM, n0 = tn * PBN + (int)rank * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.err, 11)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(full_bar(stage), 2 * C::STAGE_BYTES);
          const uint32_t fb = mapa_u32(full_bar(stage), 0);
          const uint32_t sa = base + stage * C::STAGE_BYTES;
          const uint32_t sb = sa + C::PLANES * TILE_BYTES;
          const int k0 = kb * BK;
#pragma unroll
          for (int pl = 0; pl < C::PLANES; ++pl) {
            const uint32_t da = sa + pl * TILE_BYTES, db = sb + pl * TILE_BYTES;
            if (p.a_mn_major) {  // two boxes of 64 (m) x 64 (k)
              tma_load_3d_pair(da, &map_a, fb, m0, k0, pl);
              tma_load_3d_pair(da + TILE_BYTES / 2, &map_a, fb, m0 + 64, k0, pl);
            } else {             // one box of 64 (k) x 128 (m)
              tma_load_3d_pair(da, &map_a, fb, k0, m0, pl);
            }
            if (p.b_mn_major) {
              tma_load_3d_pair(db, &map_b, fb, n0, k0, pl);
              tma_load_3d_pair(db + TILE_BYTES / 2, &map_b, fb, n0 + 64, k0, pl);
            } else {
              tma_load_3d_pair(db, &map_b, fb, k0, n0, pl);
            }
          }
          if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (CTA 0 only)
    if (lane == 0 && rank == 0) {
      constexpr uint32_t type = MODE == F16_PLANES ? 0u : 1u;  // fp16 or bf16 operands
      const uint32_t idesc = (1u << 4) | (type << 7) | (type << 10) |
                             ((uint32_t)p.a_mn_major << 15) | ((uint32_t)p.b_mn_major << 16) |
                             ((uint32_t)(PBN >> 3) << 17) | ((uint32_t)(PBM >> 4) << 24);
      const uint32_t a_lbo = p.a_mn_major ? TILE_BYTES / 2 : 16, a_kstep = p.a_mn_major ? 2048 : 32;
      const uint32_t b_lbo = p.b_mn_major ? TILE_BYTES / 2 : 16, b_kstep = p.b_mn_major ? 2048 : 32;
      uint32_t stage = 0, phase = 0;
      uint32_t acc_phase = 0;  // one parity bit per accumulator
      int cidx = 0;
      bool ok = true;
      for (int item = pair; item < total_items && ok; item += npairs) {
        const int sp = item / (p.tiles_n * p.tiles_m);
        const int kb0 = sp * p.kb_per_split;
        const int kb1 = min(p.kb_total, kb0 + p.kb_per_split);
        int kb = kb0;
        while (kb < kb1 && ok) {
          const int acc = cidx % PAIR_NACC;
          ++cidx;
          if (!mbar_wait_cluster(acce_bar(acc), ((acc_phase >> acc) & 1u) ^ 1u, abort_flag, p.err, 12)) { ok = false; break; }
          acc_phase ^= 1u << acc;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * PBN;
          const int kend = C::CHUNK ? min(kb1, kb + chunk) : kb1;
          uint32_t first = 1;
          for (; kb < kend; ++kb) {
            if (!mbar_wait_cluster(full_bar(stage), phase, abort_flag, p.err, 13)) { ok = false; break; }
            tc_fence_after();
            const uint32_t sa = base + stage * C::STAGE_BYTES;
            const uint32_t sb = sa + C::PLANES * TILE_BYTES;
#pragma unroll
            for (int pr = 0; pr < NPROD; ++pr) {
              const int ia = pr == 2 ? 1 : (pr == 3 ? 1 : (pr == 5 ? 2 : 0));
              const int ib = pr == 1 ? 1 : (pr == 3 ? 1 : (pr == 4 ? 2 : 0));
              const uint32_t pa = sa + ia * TILE_BYTES;
              const uint32_t pb = sb + ib * TILE_BYTES;
#pragma unroll
              for (int ks = 0; ks < BK / UK; ++ks) {
                const uint64_t da = smem_desc(pa + ks * a_kstep, a_lbo, 1024);
                const uint64_t db = smem_desc(pb + ks * b_kstep, b_lbo, 1024);
                tc_mma_bf16_pair(d_tmem, da, db, idesc, first ? 0u : 1u);
                first = 0;
              }
            }
            tc_commit_pair(empty_bar(stage), 3);  // frees the stage in both CTAs
            if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
          }
          if (ok) tc_commit_pair(accf_bar(acc), 3);  // this chunk is complete in both CTAs
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (both CTAs)
    const int quad = warp & 3;         // tensor-memory lane quadrant this warp may read
    uint8_t* tile = aligned + C::STAGES * C::STAGE_BYTES + 256 + (warp - 2) * EPI_TILE;
    const int half = (warp - 2) >> 2;  // which 128 columns of the accumulator
    uint32_t acc_phase = 0;  // one parity bit per accumulator
    int cidx = 0;
    bool ok = true;
    for (int item = pair; item < total_items; item += npairs) {
      const int tn = item % p.tiles_n;
      const int tm = (item / p.tiles_n) % p.tiles_m;
      const int sp = item / (p.tiles_n * p.tiles_m);
      const int kb0 = sp * p.kb_per_split;
      const int kb1 = min(p.kb_total, kb0 + p.kb_per_split);
      const int nchunks = C::CHUNK ? (kb1 - kb0 + chunk - 1) / max(chunk, 1) : 1;
      const int m0 = tm * PBM + (int)rank * BM + quad * 32;
      const int n0 = tn * PBN + half * BN;
      float sum[C::CHUNK ? BN : 1];
#pragma unroll
      for (int j = 0; j < (C::CHUNK ? BN : 1); ++j) sum[j] = 0.f;
      for (int c = 0; c < nchunks; ++c) {
        const int acc = cidx % PAIR_NACC;
        ++cidx;
        if (ok) ok = mbar_wait(accf_bar(acc), (acc_phase >> acc) & 1u, abort_flag, p.err, 14);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        acc_phase ^= 1u << acc;
        tc_fence_after();
        const uint32_t taddr = tmem_base + acc * PBN + half * BN + ((uint32_t)(quad * 32) << 16);
        if (C::CHUNK) {
#pragma unroll
          for (int ch = 0; ch < BN / 16; ++ch) {
            uint32_t r[16];
            tc_ld16(taddr + ch * 16, r);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[(C::CHUNK ? ch * 16 : 0) + j] += __uint_as_float(r[j]);
          }
        } else {
#pragma unroll 1
          for (int ch = 0; ch < BN / 32 && m0 < p.M && n0 + ch * 32 < p.N; ++ch) {
            uint32_t r[32];
            tc_ld32(taddr + ch * 32, r);
            tc_wait_ld();
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
            __syncwarp();  // the tile before has been read
            fill_tile(v, tile);
            store_chunk<NPROD, MODE>(p, sp, m0, n0 + ch * 32, tile);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(acce_bar(acc), 0));
      }
      if (!ok) break;
      if (C::CHUNK) {
        const int ea = MODE == F16_PLANES ? row_scale(p, m0) : 0;
#pragma unroll (MODE == F16_PLANES ? BN / 32 : 1)
        for (int ch = 0; ch < BN / 32; ++ch) {
          const int eb = MODE == F16_PLANES ? column_scales(p, n0 + ch * 32) : 0;
          __syncwarp();  // the tile before has been read
#pragma unroll
          for (int c = 0; c < BN / 32; ++c)
            if (c == ch) fill_tile(sum + (C::CHUNK ? c * 32 : 0), tile);
          store_chunk<NPROD, MODE>(p, sp, m0, n0 + ch * 32, tile, ea, eb);
        }
      }
    }
  }

  // Drain: every role of both CTAs arrives here, also after a time-out.  Neither CTA may leave
  // while the other's MMAs can still read its shared memory or signal its barriers.
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"((uint32_t)(PAIR_NACC * PBN))
                 : "memory");
  }
}

template <int NPROD>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
gemm_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         const __grid_constant__ Params p) {
  gemm_pair<NPROD>(map_a, map_b, p);
}
__global__ void __launch_bounds__(PAIR_THREADS, 1)
gemm_tcgen05_pair_f16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                             const __grid_constant__ CUtensorMap bf_a, const __grid_constant__ CUtensorMap bf_b,
                             const __grid_constant__ Params p) {
  if (*p.uneven) gemm_pair<6, UNEVEN>(bf_a, bf_b, p);
  else gemm_pair<3, F16_PLANES>(map_a, map_b, p);
}

// x -> `planes` bf16 planes (x = p0 + p1 (+ p2), each the bf16 rounding of what is left),
// same orientation as the source, leading dimension ld_dst (a multiple of 8), planes
// `plane_stride` elements apart.  One thread converts 4 consecutive elements of a row:
// a 16-byte load and one 8-byte store per plane when the source allows it.
// One launch takes up to two operands (blockIdx.y).
struct SplitJob {
  const void* src = nullptr;
  long long ld_src = 0;
  int rows = 0, cols = 0;
  __nv_bfloat16* dst = nullptr;
  long long ld_dst = 0, plane_stride = 0;
  int vec_ok = 0;
};
template <int PLANES, typename TS>
__device__ __forceinline__ void split_planes(const SplitJob& job0, const SplitJob& job1) {
  const SplitJob& job = blockIdx.y ? job1 : job0;
  const TS* __restrict__ src = static_cast<const TS*>(job.src);
  __nv_bfloat16* __restrict__ dst = job.dst;
  const long long ld_src = job.ld_src, ld_dst = job.ld_dst, plane_stride = job.plane_stride;
  const int cols = job.cols;
  const unsigned quads = (unsigned)(ld_dst / 4);
  const long long total = (long long)job.rows * quads;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = total >> 32 ? i / quads : (long long)((unsigned)i / quads);
    const int c = (int)(i - r * quads) * 4;
    float x[4] = {0.f, 0.f, 0.f, 0.f};
    const TS* sp = src + r * ld_src + c;
    if (job.vec_ok && c + 3 < cols) {
      if constexpr (sizeof(TS) == 4) {
        const float4 f = *reinterpret_cast<const float4*>(sp);
        x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
      } else {
        typedef typename std::conditional<std::is_same<TS, __half>::value, __half2, __nv_bfloat162>::type Pair;
        const uint2 u = *reinterpret_cast<const uint2*>(sp);
        const Pair h0 = *reinterpret_cast<const Pair*>(&u.x);
        const Pair h1 = *reinterpret_cast<const Pair*>(&u.y);
        x[0] = __low2float(h0); x[1] = __high2float(h0);
        x[2] = __low2float(h1); x[3] = __high2float(h1);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < cols) x[j] = ld(sp + j);
    }
    __nv_bfloat16* dp = dst + r * ld_dst + c;
#pragma unroll
    for (int pl = 0; pl < PLANES; ++pl) {
      __nv_bfloat162 a = __floats2bfloat162_rn(x[0], x[1]);
      __nv_bfloat162 b = __floats2bfloat162_rn(x[2], x[3]);
      uint2 w;
      w.x = *reinterpret_cast<uint32_t*>(&a);
      w.y = *reinterpret_cast<uint32_t*>(&b);
      *reinterpret_cast<uint2*>(dp + pl * plane_stride) = w;
      x[0] -= __low2float(a); x[1] -= __high2float(a);
      x[2] -= __low2float(b); x[3] -= __high2float(b);
    }
  }
}

template <int PLANES, typename TS>
__global__ void split_planes_kernel(const SplitJob job0, const SplitJob job1) {
  split_planes<PLANES, TS>(job0, job1);
}
// In the place of fp16 planes, if one of `n` words asks for it; words[n] says so to the product.
__global__ void split_uneven_kernel(const SplitJob job0, const SplitJob job1, int* words, int n) {
  int w = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) w |= words[i];
  w = __syncthreads_or(w);
  if (blockIdx.x + blockIdx.y + threadIdx.x == 0) words[n] = w;
  if (w) split_planes<3, float>(job0, job1);
}

// ---- two fp16 planes per fp32 operand ---------------------------------------------------------
// x 2^s = p0 + p1, p0 and p1 the fp16 roundings of x 2^s and of what is left: 22 .. 23 bits of x where
// three bf16 planes keep 24, for three products instead of six and two thirds of the operand bytes.
// s makes the largest value of a row of A (a column of B) 2^14 .. 2^15, so that values down to 2^-17 of
// it keep all their bits and smaller ones an absolute error of 2^-40 of it; the epilogue takes the
// powers out again.  Such smaller values are one in 20000 of a normal distribution and do not show; but where
// a few values tower above all others of their row, and meet weights that are small or zero, they are the result.
// So the splits count them: with more than one in 32 of a row's or column's values other than zero, the
// operands are split into three bf16 planes after all and multiplied six times (decided on the device; where they
// are not, the look costs 4 us: a launch, and a word that the product waits for).  What is left: in up to one value of
// 32, an error of 2^-40 of the row's or column's largest value.
constexpr int F16_THREADS = 512, F16_ROW_QUADS = 8 * 32;  // quads of a row that a warp holds in registers

__device__ __forceinline__ int f16_shift(float most) {  // non-finite rows are non-finite either way
  if (!(most > 0.f) || isinf(most)) return 0;
  int e;
  frexpf(most, &e);  // most = f 2^e, 0.5 <= f < 1
  return max(-126, min(126, 15 - e));
}
__device__ __forceinline__ float abs_max4(float m, const float4& v) {
  return fmaxf(fmaxf(fmaxf(m, fabsf(v.x)), fmaxf(fabsf(v.y), fabsf(v.z))), fabsf(v.w));
}
__device__ __forceinline__ float4 load_quad(const float* row, int c, int cols, int vec_ok) {
  if (vec_ok && c + 3 < cols) return *reinterpret_cast<const float4*>(row + c);
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c < cols) v.x = row[c];
  if (c + 1 < cols) v.y = row[c + 1];
  if (c + 2 < cols) v.z = row[c + 2];
  if (c + 3 < cols) v.w = row[c + 3];
  return v;
}
// Returns how many of the values, in either half, are below 0.25 once scaled, zeros among them.
__device__ __forceinline__ __half2 store_f16_quad(__half* dst, long long plane_stride, const float4& v, float4 scale) {
  const float x[4] = {v.x * scale.x, v.y * scale.y, v.z * scale.z, v.w * scale.w};
  const __half2 a = __floats2half2_rn(x[0], x[1]), b = __floats2half2_rn(x[2], x[3]);
  const __half2 c = __floats2half2_rn(x[0] - __low2float(a), x[1] - __high2float(a));
  const __half2 d = __floats2half2_rn(x[2] - __low2float(b), x[3] - __high2float(b));
  *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  *reinterpret_cast<uint2*>(dst + plane_stride) =
      make_uint2(*reinterpret_cast<const uint32_t*>(&c), *reinterpret_cast<const uint32_t*>(&d));
  const __half2 few = __float2half2_rn(0.25f);
  return __hadd2(__hlt2(__habs2(a), few), __hlt2(__habs2(b), few));
}
// Adds to `score`, which is above zero for a row if more than one in 32 of its values other than zero, scaled
// by f, lose bits.
__device__ __forceinline__ void count_small(float x, float f, int& score) {
  const float v = fabsf(x) * f;
  score += v > 0.f ? (v < 0.25f ? 31 : -1) : 0;
}
__device__ __forceinline__ void count_small4(const float4& x, const float4& f, int (&score)[4]) {
  count_small(x.x, f.x, score[0]); count_small(x.y, f.y, score[1]);
  count_small(x.z, f.z, score[2]); count_small(x.w, f.w, score[3]);
}
// A warp takes 8 / QL rows at a time, of which it holds QL quads per lane; longer rows are read twice.  Returns whether
// a row has too many small values.
template <int QL>
__device__ __forceinline__ bool split_f16_rows(const SplitJob& a, int* __restrict__ a_exp) {
  bool uneven = false;
  constexpr int RW = 8 / QL;
  const int lane = threadIdx.x & 31, quads = (int)(a.ld_dst / 4), step = gridDim.x * (F16_THREADS / 32) * RW;
  for (int r0 = (blockIdx.x * (F16_THREADS / 32) + (threadIdx.x >> 5)) * RW; r0 < a.rows; r0 += step) {
    float4 v[RW][QL];
    float most[RW];
#pragma unroll
    for (int k = 0; k < RW; ++k) {
      const float* src = static_cast<const float*>(a.src) + (r0 + k) * a.ld_src;
      most[k] = 0.f;
#pragma unroll
      for (int i = 0; i < QL; ++i)
        v[k][i] = load_quad(src, (lane + 32 * i) * 4, r0 + k < a.rows ? a.cols : 0, a.vec_ok);
    }
#pragma unroll
    for (int k = 0; k < RW; ++k) {
#pragma unroll
      for (int i = 0; i < QL; ++i) most[k] = abs_max4(most[k], v[k][i]);
      if (QL == 8) {
        const float* src = static_cast<const float*>(a.src) + r0 * a.ld_src;
        for (int q = F16_ROW_QUADS + lane; q < quads; q += 32) most[k] = abs_max4(most[k], load_quad(src, q * 4, a.cols, a.vec_ok));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) most[k] = fmaxf(most[k], __shfl_xor_sync(0xffffffffu, most[k], o));
    }
#pragma unroll
    for (int k = 0; k < RW; ++k) {
      if (r0 + k >= a.rows) break;
      __half* dst = reinterpret_cast<__half*>(a.dst) + (r0 + k) * a.ld_dst;
      const int s = f16_shift(most[k]);
      const float f = exp2_int(s);
      const float4 scale = make_float4(f, f, f, f);
      if (lane == 0) a_exp[r0 + k] = -s;
      int score[4] = {0, 0, 0, 0};
      __half2 small = __float2half2_rn(0.f);
#pragma unroll
      for (int i = 0; i < QL; ++i)
        if (lane + 32 * i < quads)
          small = __hadd2(small, store_f16_quad(dst + (lane + 32 * i) * 4, a.plane_stride, v[k][i], scale));
      const bool held = QL < 8 || quads <= F16_ROW_QUADS;
      if (!held) {
        const float* src = static_cast<const float*>(a.src) + r0 * a.ld_src;
        for (int q = F16_ROW_QUADS + lane; q < quads; q += 32) {
          const float4 x = load_quad(src, q * 4, a.cols, a.vec_ok);
          store_f16_quad(dst + q * 4, a.plane_stride, x, scale);
          count_small4(x, scale, score);
        }
      }
      // (counted to the end only where zeros may be among the small ones)
      const int most_small = __reduce_add_sync(0xffffffffu, (int)(__low2float(small) + __high2float(small)));
      if (!held || 32 * most_small > a.cols - most_small) {
#pragma unroll
        for (int i = 0; i < QL; ++i) count_small4(v[k][i], scale, score);
        uneven |= __reduce_add_sync(0xffffffffu, score[0] + score[1] + score[2] + score[3]) > 0;
      }
    }
  }
  return uneven;
}
// blockIdx.y = 0: `a`, scaled by row, a warp per row or few; 1: `b`, scaled by column, 32 columns per block (its
// second reading comes from L2).  Bound by HBM: 256000 x 1024 takes one reading and one writing.  uneven: a word per
// block, whether its values ask for the bf16 planes.
__global__ void __launch_bounds__(F16_THREADS) split_f16_kernel(const SplitJob a, int* __restrict__ a_exp, const SplitJob b,
                                                                signed char* __restrict__ b_exp, int* __restrict__ uneven) {
  bool bad = false;
  if (blockIdx.y == 0) {
    const int quads = (int)(a.ld_dst / 4);
    if (quads <= 32) bad = split_f16_rows<1>(a, a_exp);
    else if (quads <= 64) bad = split_f16_rows<2>(a, a_exp);
    else if (quads <= 128) bad = split_f16_rows<4>(a, a_exp);
    else bad = split_f16_rows<8>(a, a_exp);
  } else {
    __shared__ float4 part[F16_THREADS];
    __shared__ int scores[32];
    const int q = threadIdx.x & 7, ry = threadIdx.x >> 3;
    constexpr int RY = F16_THREADS / 8;
    for (int c0 = blockIdx.x * 32; c0 < (int)b.ld_dst; c0 += gridDim.x * 32) {
      const int c = c0 + q * 4;
      const float* src = static_cast<const float*>(b.src);
      float4 most = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int r = ry; r < b.rows; r += RY) {
        const float4 v = load_quad(src + r * b.ld_src, c, b.cols, b.vec_ok);
        most = make_float4(fmaxf(most.x, fabsf(v.x)), fmaxf(most.y, fabsf(v.y)), fmaxf(most.z, fabsf(v.z)),
                           fmaxf(most.w, fabsf(v.w)));
      }
      __syncthreads();  // the columns before have been read
      part[threadIdx.x] = most;
      if (threadIdx.x < 32) scores[threadIdx.x] = 0;
      __syncthreads();
      for (int h = RY / 2; h > 0; h >>= 1) {
        if (ry < h) {
          const float4 o = part[threadIdx.x + h * 8];
          float4& m = part[threadIdx.x];
          m = make_float4(fmaxf(m.x, o.x), fmaxf(m.y, o.y), fmaxf(m.z, o.z), fmaxf(m.w, o.w));
        }
        __syncthreads();
      }
      most = part[q];
      const int4 s = make_int4(f16_shift(most.x), f16_shift(most.y), f16_shift(most.z), f16_shift(most.w));
      const float4 scale = make_float4(exp2_int(s.x), exp2_int(s.y), exp2_int(s.z), exp2_int(s.w));
      int score[4] = {0, 0, 0, 0};
      if (c < (int)b.ld_dst) {
        if (ry == 0) *reinterpret_cast<char4*>(b_exp + c) = make_char4(-s.x, -s.y, -s.z, -s.w);
#pragma unroll 4
        for (int r = ry; r < b.rows; r += RY) {
          const float4 x = load_quad(src + r * b.ld_src, c, b.cols, b.vec_ok);
          store_f16_quad(reinterpret_cast<__half*>(b.dst) + r * b.ld_dst + c, b.plane_stride, x, scale);
          count_small4(x, scale, score);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // over the warp's rows, then the block's
        score[i] += __shfl_xor_sync(0xffffffffu, score[i], 8);
        score[i] += __shfl_xor_sync(0xffffffffu, score[i], 16);
        if ((threadIdx.x & 31) < 8) atomicAdd(&scores[q * 4 + i], score[i]);
      }
      __syncthreads();
      if (threadIdx.x < 32) bad |= scores[threadIdx.x] > 0;
    }
  }
  const int any = __syncthreads_or(bad);
  if (threadIdx.x == 0) uneven[blockIdx.y * gridDim.x + blockIdx.x] = any;
}

// `dtype` of the sources.  __half: its 11 significant bits split exactly into two planes.  bf16: one
// plane, a copy with rows that TMA can address.  jobs: one or two.
bool wide_rows(const SplitJob& job, int dtype) {
  return (job.ld_src & 3) == 0 && (reinterpret_cast<uintptr_t>(job.src) & (dtype == HASTE_B200_F32 ? 15 : 7)) == 0;
}
int launch_split(SplitJob* jobs, int n, int dtype, int planes, cudaStream_t stream) {
  long long most = 0;
  for (int i = 0; i < n; ++i) {
    jobs[i].vec_ok = wide_rows(jobs[i], dtype);
    most = std::max(most, (long long)jobs[i].rows * (jobs[i].ld_dst / 4));
  }
  const dim3 grid(min(ceil_div(most, 256), 8 * sm_count()), n);
  const SplitJob a = jobs[0], b = jobs[n - 1];
  if (dtype == HASTE_B200_BF16) split_planes_kernel<1, __nv_bfloat16><<<grid, 256, 0, stream>>>(a, b);
  else if (dtype == HASTE_B200_F16 && planes == 3) split_planes_kernel<3, __half><<<grid, 256, 0, stream>>>(a, b);
  else if (dtype == HASTE_B200_F16) split_planes_kernel<2, __half><<<grid, 256, 0, stream>>>(a, b);
  else if (planes == 3) split_planes_kernel<3, float><<<grid, 256, 0, stream>>>(a, b);
  else split_planes_kernel<2, float><<<grid, 256, 0, stream>>>(a, b);
  HB_LAUNCH_OK();
  count_launch(1);
  return HASTE_B200_OK;
}

// Leaves in *uneven whether the planes are bf16 after all.  `words`: 8 per SM and one.
int launch_split_f16(SplitJob* jobs, int* a_exp, signed char* b_exp, int* words, const int** uneven, cudaStream_t stream) {
  for (int i = 0; i < 2; ++i) jobs[i].vec_ok = wide_rows(jobs[i], HASTE_B200_F32);
  const int per_warp = (int)(8 / max(1LL, min(8LL, (jobs[0].ld_dst + 127) / 128)));  // about what split_f16_rows takes
  const int blocks = max(ceil_div(jobs[0].rows, F16_THREADS / 32 * per_warp), ceil_div(jobs[1].cols, 32));
  const dim3 grid(min(blocks, 4 * sm_count()), 2);
  split_f16_kernel<<<grid, F16_THREADS, 0, stream>>>(jobs[0], a_exp, jobs[1], b_exp, words);
  HB_LAUNCH_OK();
  split_uneven_kernel<<<dim3(sm_count(), 2), 512, 0, stream>>>(jobs[0], jobs[1], words, 2 * grid.x);
  HB_LAUNCH_OK();
  count_launch(2);
  *uneven = words + 2 * grid.x;
  return HASTE_B200_OK;
}

// Adds up the partial tiles of a K split ([splits][M][ld], ld a multiple of 32) into C: four columns
// per thread, eight threads per 32-column chunk.  Vec: C's rows take 16-byte (8-byte) stores.
template <typename TC, bool Vec>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* __restrict__ part, int splits,
                                                            long long split_stride, int M, int N, int ld_part,
                                                            TC* __restrict__ c, long long ldc, int accumulate) {
  const unsigned quads = ld_part / 4, total = (unsigned)M * quads;
  for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) {
    const unsigned m = i / quads, n = (i - m * quads) * 4;
    if ((int)n >= N) continue;
    const float4* src = reinterpret_cast<const float4*>(part + (long long)m * ld_part + n);
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int k = 0; k < splits; ++k) {
      const float4 f = src[k * (split_stride / 4)];
      s.x += f.x; s.y += f.y; s.z += f.z; s.w += f.w;
    }
    float v[4] = {s.x, s.y, s.z, s.w};
    TC* dst = c + (long long)m * ldc + n;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (accumulate && (Vec || (int)n + e < N)) v[e] += ld(dst + e);
    if constexpr (Vec) {
      TC out[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) st(out + e, v[e]);
      typedef typename std::conditional<sizeof(TC) == 4, uint4, uint2>::type Word;
      Word w;
      memcpy(&w, out, sizeof(w));
      *reinterpret_cast<Word*>(dst) = w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if ((int)n + e < N) st(dst + e, v[e]);
    }
  }
}
template <typename TC>
void launch_reduce(const float* part, int splits, int M, int N, int ld_part, void* c, long long ldc, int accumulate,
                   int most, cudaStream_t stream) {
  const long long stride = (long long)M * ld_part;
  const int blocks = min(ceil_div(stride / 4, 256), most);
  const bool vec = N % 4 == 0 && ldc % 4 == 0 && reinterpret_cast<uintptr_t>(c) % (4 * sizeof(TC)) == 0;
  if (vec)
    splitk_reduce_kernel<TC, true><<<blocks, 256, 0, stream>>>(part, splits, stride, M, N, ld_part, (TC*)c, ldc, accumulate);
  else
    splitk_reduce_kernel<TC, false><<<blocks, 256, 0, stream>>>(part, splits, stride, M, N, ld_part, (TC*)c, ldc, accumulate);
}

// ----------------------------------------------------------------------------
// Host side
// ----------------------------------------------------------------------------
struct Operand {
  bool mn_major;          // contiguous along M (A) or N (B)
  long long ld;           // elements between consecutive outer indices
  long long plane_stride; // elements between planes
  const void* base;
};

// The opt-in to more than 48 KB of dynamic shared memory is a per-device (per-context)
// function attribute: one flag per device ordinal, so that a process driving several GPUs
// opts in on each of them.
constexpr int kMaxDevices = 64;
std::atomic<bool> g_attr_set[kMaxDevices];
std::atomic<int> g_max_pairs[kMaxDevices];  // 0: not asked yet, -1: no clusters, else the count

template <int NPROD>
constexpr int single_smem() { return Cfg<NPROD>::SMEM + 4 * EPI_TILE; }
template <int NPROD>
constexpr int pair_smem() { return Cfg<NPROD>::SMEM + PAIR_EPI_WARPS * EPI_TILE; }
static_assert(pair_smem<1>() <= 232448 && pair_smem<3>() <= 232448 && pair_smem<6>() <= 232448, "shared memory per CTA");

int set_kernel_attributes() {
  int dev = 0;
  HB_CUDA_OK(cudaGetDevice(&dev));
  if (dev >= 0 && dev < kMaxDevices && g_attr_set[dev].load(std::memory_order_acquire))
    return HASTE_B200_OK;
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  HB_CUDA_OK(cudaFuncSetAttribute(gemm_tcgen05_kernel<1>, attr, single_smem<1>()));
  HB_CUDA_OK(cudaFuncSetAttribute(gemm_tcgen05_kernel<3>, attr, single_smem<3>()));
  HB_CUDA_OK(cudaFuncSetAttribute(gemm_tcgen05_kernel<6>, attr, single_smem<6>()));
  HB_CUDA_OK(cudaFuncSetAttribute(gemm_tcgen05_pair_kernel<1>, attr, pair_smem<1>()));
  HB_CUDA_OK(cudaFuncSetAttribute(gemm_tcgen05_pair_kernel<3>, attr, pair_smem<3>()));
  HB_CUDA_OK(cudaFuncSetAttribute(gemm_tcgen05_pair_kernel<6>, attr, pair_smem<6>()));
  HB_CUDA_OK(cudaFuncSetAttribute(gemm_tcgen05_f16_kernel, attr, max(single_smem<3>(), single_smem<6>())));
  HB_CUDA_OK(cudaFuncSetAttribute(gemm_tcgen05_pair_f16_kernel, attr, max(pair_smem<3>(), pair_smem<6>())));
  if (dev >= 0 && dev < kMaxDevices) g_attr_set[dev].store(true, std::memory_order_release);
  return HASTE_B200_OK;
}

// How many clusters of two CTAs of the pair kernel the device holds at once (its persistent
// grid); 0 when cluster launch is not available.
int max_pairs() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  int n = g_max_pairs[dev].load(std::memory_order_acquire);
  if (n == 0) {
    n = -1;
    if (set_kernel_attributes() == HASTE_B200_OK) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(2 * sm_count());
      cfg.blockDim = dim3(PAIR_THREADS);
      cfg.dynamicSmemBytes = pair_smem<6>();
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, gemm_tcgen05_pair_kernel<6>, &cfg) ==
              cudaSuccess && clusters > 0)
        n = min(clusters, sm_count() / 2);
      cudaGetLastError();
    }
    g_max_pairs[dev].store(n, std::memory_order_release);
  }
  return n > 0 ? n : 0;
}

}  // namespace

// fp32 [rows, cols] (leading dimension ld_src) -> two bf16 planes of leading dimension ld_dst,
// plane_stride elements apart: the form GemmDesc::a_pl / b_pl takes, for an operand that
// several contractions read.
int gemm_split_planes(const float* src, long long ld_src, int rows, int cols,
                      __nv_bfloat16* dst, long long ld_dst, long long plane_stride,
                      cudaStream_t stream) {
  SplitJob job{src, ld_src, rows, cols, dst, ld_dst, plane_stride};
  return launch_split(&job, 1, HASTE_B200_F32, 2, stream);
}

namespace {
// Why this file's kernels do not take a contraction; null if they do.
const char* refusal(const GemmDesc& g) {
  if (!encode_fn()) return "cuTensorMapEncodeTiled not available";
  if (g.K <= 0) return "K == 0";
  // Small problems are launch-bound either way; keep them on the generic kernel.
  if ((long long)g.M * g.N * g.K < (1LL << 21) || g.M < 8 || g.N < 32)
    return "problem too small for the tensor-core path";
  if (g.dtype != HASTE_B200_BF16 && g.M < 32 && gemm_path() == HASTE_B200_GEMM_AUTO) return "few rows: fp32 sums";  // gemm.cu
  if ((g.a_cs != 1 && g.a_rs != 1) || (g.b_rs != 1 && g.b_cs != 1)) return "operand has no unit stride";
  return nullptr;
}
// fp32-accurate products go through two fp16 planes where half the products save more than the rows' and
// columns' scales and the look at their values cost (us with the splits, a LayerNorm and the scan over the result,
// six bf16 products / these: 256000 x 1024 x 1024 5527 / 4448, 16384 x 1024 x 1024 381 / 334, 65536 x 512 x 256
// 365 / 330, 16384 x 512 x 1024 298 / 278, 8000 x 1024 x 1024 193 / 179; M x K x N.  Below 8 G multiply-adds, or 256 of
// K, nothing is left).
bool f16_planes(const GemmDesc& g) {
  return g.precise && g.dtype == HASTE_B200_F32 && g.dtype_c == HASTE_B200_F32 && !g.accumulate && g.a_cs == 1 &&
         g.b_cs == 1 && g.b_rs != 1 && g.K >= 256 && (double)g.M * g.N * g.K >= 8e9;
}
}  // namespace

bool gemm_reads_planes(const GemmDesc& g) { return gemm_path() != HASTE_B200_GEMM_SIMT && !refusal(g); }

int gemm_sm100(const GemmDesc& g, cudaStream_t stream) {
  auto unsupported = [](const char* why) {
    set_last_error("gemm_sm100: %s", why);
    return HASTE_B200_ERR_UNSUPPORTED;
  };
  if (g.M <= 0 || g.N <= 0) return HASTE_B200_OK;
  if (const char* why = refusal(g)) return unsupported(why);
  // __half storage takes the split path too: a half splits exactly into two bf16 planes
  const bool half_src = g.dtype == HASTE_B200_F16;
  const bool f32 = g.dtype == HASTE_B200_F32 || half_src;
  const bool a_k = g.a_cs == 1, b_k = g.b_rs == 1;

  const int M = g.M, N = g.N, K = g.K;
  const bool f16 = f16_planes(g);
  Operand A, B;
  A.mn_major = !a_k;
  B.mn_major = !b_k;
  // extents in (outer rows, inner contiguous) form
  const long long a_rows = a_k ? M : K, a_cols = a_k ? K : M;
  const long long b_rows = b_k ? N : K, b_cols = b_k ? K : N;
  const long long a_ld_src = a_k ? g.a_rs : g.a_cs;
  const long long b_ld_src = b_k ? g.b_cs : g.b_rs;

  // scratch: planes for fp32 operands, partial tiles for split-K
  const int sms = sm_count();
  // CTA pairs on 256 x 256 tiles where the output is wide enough to fill them and the work is
  // worth the cluster launch and the coarser waves: 4 .. 7 us below 16 G multiply-adds, where only a
  // long K lets the pair's better rate make up for it (us, pair / single: fp32 2000 x 512 x 512 31 / 17,
  // 20000 x 512 x 512 66 / 58, 6400 x 512 x 2048 66 / 70, 30000 x 1024 x 1024 206 / 222; bf16 29 / 25 for the
  // second, 22 / 27 for the third).
  const double macs = (double)M * N * K;
  const bool large = macs >= 16e9 || (macs >= 4e9 && K >= 1024);
  const int pairs = (gemm_path() == HASTE_B200_GEMM_TCGEN05_SINGLE || M < 192 || N < 192 || !large)
                        ? 0 : max_pairs();
  const bool pair = pairs > 0;
  const int units = pair ? pairs : sms;
  const int tiles_m = ceil_div(M, pair ? PBM : BM), tiles_n = ceil_div(N, pair ? PBN : BN);
  const int kb_total = ceil_div(K, BK);
  int splits = 1;
  // (With K of 8192 and more also where a second or third wave would be nearly empty: 2048 x 3072 is 96 tiles
  // for 74 pairs; us at K = 64000 one split / three 734 / 601, 2000 x 2600, K = 20000 260 / 222.)
  if (kb_total >= 8 && tiles_m * tiles_n < (kb_total >= 128 ? 4 : 1) * units) {
    // Split K so that the work items fill whole waves of the persistent grid: pick the split
    // count with the smallest estimated time = (waves / splits) x K blocks x time per K block
    // + the traffic of the partial tiles (written once, read once by the reduction).
    const int tiles = tiles_m * tiles_n;
    const int max_splits = min(kb_total / 4, 64);
    const double products = g.dtype == HASTE_B200_BF16 ? 1.0 : (g.precise && !f16 ? 6.0 : 3.0);
    // us per K block and work unit (measured: the single-CTA kernel is bound by its operand
    // loads, the pair kernel by the tensor pipe)
    const double t_kb = pair ? 0.27 * products : (products == 1.0 ? 0.27 : 0.17 * products);
    const double t_part = 2.0 * (double)M * N * 4.0 / 6.0e6;          // us per split (HBM)
    double best = 1e30;
    for (int sp = 1; sp <= max_splits; ++sp) {
      const int per = ceil_div(kb_total, sp);
      const int real = ceil_div(kb_total, per);
      if (real != sp) continue;  // the same blocks per split as a smaller count: skip
      const double t = (double)ceil_div(tiles * sp, units) * per * t_kb + (sp > 1 ? sp * t_part : 0.0);
      if (t < best) { best = t; splits = sp; }
    }
  }
  int kb_per_split = ceil_div(kb_total, splits);
  splits = ceil_div(kb_total, kb_per_split);

  auto planes_usable = [&](const void* p, long long ld) {
    return f32 && !g.precise && p && (ld % 8) == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
  };
  const bool a_pre = planes_usable(g.a_pl, g.a_pl_ld) && (g.a_pl_stride % 8) == 0;
  const bool b_pre = planes_usable(g.b_pl, g.b_pl_ld) && (g.b_pl_stride % 8) == 0;
  // An operand goes through scratch if it has to be split or if TMA cannot address its rows
  // (bf16 with a row or a start that is no multiple of 16 bytes: the copy costs two passes over the
  // operand, the CUDA-core kernel that would take it as it is twenty times the contraction).
  const bool a_copy = f32 ? !a_pre : (a_ld_src % 8) != 0 || ((uintptr_t)g.a & 15) != 0;
  const bool b_copy = f32 ? !b_pre : (b_ld_src % 8) != 0 || ((uintptr_t)g.b & 15) != 0;
  const long long a_ld = a_pre ? g.a_pl_ld : (a_copy ? ((a_cols + 7) & ~7LL) : a_ld_src);
  const long long b_ld = b_pre ? g.b_pl_ld : (b_copy ? ((b_cols + 7) & ~7LL) : b_ld_src);
  const int planes = f32 ? (g.precise && !f16 ? 3 : 2) : 1, room = f16 ? 3 : planes;
  const size_t a_plane = a_copy ? Arena::pad((size_t)a_rows * a_ld * 2) : 0;
  const size_t b_plane = b_copy ? Arena::pad((size_t)b_rows * b_ld * 2) : 0;
  const int part_ld = (N + 31) & ~31;
  const bool via_partial = splits > 1;
  const size_t part_bytes = via_partial ? Arena::pad((size_t)splits * M * part_ld * 4) : 0;
  const size_t a_exps = f16 ? Arena::pad((size_t)M * 4) : 0, b_exps = f16 ? Arena::pad((size_t)tiles_n * PBN) : 0;
  const size_t words = f16 ? Arena::pad((size_t)(8 * sms + 1) * 4) : 0;
  const size_t bytes = room * (a_plane + b_plane) + part_bytes + a_exps + b_exps + words + 1024;
  Arena ws;
  HB_TRY(make_arena(&ws, stream, bytes, /*slot=*/1));
  int* err = device_error_word();
  if (!err) return unsupported("error word allocation failed");
  A.base = a_pre ? g.a_pl : g.a;
  A.plane_stride = a_pre ? g.a_pl_stride : 0;
  B.base = b_pre ? g.b_pl : g.b;
  B.plane_stride = b_pre ? g.b_pl_stride : 0;
  SplitJob jobs[2];
  int n_jobs = 0;
  auto through_scratch = [&](const void* src, long long ld_src, long long rows, long long cols, size_t plane,
                             long long ld, Operand* o) {
    __nv_bfloat16* to = ws.take<__nv_bfloat16>(room * plane / 2);
    jobs[n_jobs++] = SplitJob{src, ld_src, (int)rows, (int)cols, to, ld, (long long)(plane / 2)};
    o->base = to;
    o->plane_stride = plane / 2;
    return to != nullptr;
  };
  if (a_copy && !through_scratch(g.a, a_ld_src, a_rows, a_cols, a_plane, a_ld, &A)) return unsupported("scratch arena");
  if (b_copy && !through_scratch(g.b, b_ld_src, b_rows, b_cols, b_plane, b_ld, &B)) return unsupported("scratch arena");
  int* a_exp = nullptr;
  signed char* b_exp = nullptr;
  const int* uneven = nullptr;
  if (f16) {
    a_exp = ws.take<int>(a_exps / 4);
    b_exp = ws.take<signed char>(b_exps);
    int* w = ws.take<int>(words / 4);
    if (!a_exp || !b_exp || !w) return unsupported("scratch arena");
    HB_TRY(launch_split_f16(jobs, a_exp, b_exp, w, &uneven, stream));
  } else if (n_jobs) {
    HB_TRY(launch_split(jobs, n_jobs, g.dtype, planes, stream));
  }
  A.ld = a_ld;
  B.ld = b_ld;
  float* partial = nullptr;
  if (via_partial) {
    partial = ws.take<float>(part_bytes / 4);
    if (!partial) return unsupported("scratch arena");
  }

  Params p;
  p.M = M; p.N = N; p.K = K;
  p.a_mn_major = A.mn_major; p.b_mn_major = B.mn_major;
  p.tiles_m = tiles_m; p.tiles_n = tiles_n; p.splits = splits;
  p.kb_per_split = kb_per_split; p.kb_total = kb_total;
  p.c_is_bf16 = g.dtype_c == HASTE_B200_BF16 ? 1 : (g.dtype_c == HASTE_B200_F16 ? 2 : 0);
  p.accumulate = g.accumulate;
  p.c = g.c; p.ldc = g.ldc;
  p.wide = (g.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(g.c) & (4 * dtype_size(g.dtype_c) - 1)) == 0;
  p.a_exp = a_exp; p.b_exp = b_exp;
  p.uneven = uneven;
  p.partial = partial;
  p.partial_ld = part_ld;
  p.err = err;

  HB_TRY(set_kernel_attributes());
  // K-major: inner = K, box 64 (k) x 128 rows.  MN-major: inner = M/N, box 64 x 64 (k).
  CUtensorMap m_a, m_b, bf_a, bf_b;
  auto maps = [&](CUtensorMap* a, CUtensorMap* b, int n) {
    return make_map(a, A.base, a_cols, a_rows, A.ld, A.plane_stride, n, 64, A.mn_major ? 64 : BM) &&
           make_map(b, B.base, b_cols, b_rows, B.ld, B.plane_stride, n, 64, B.mn_major ? 64 : BN);
  };
  if (!maps(&m_a, &m_b, planes) || (f16 && !maps(&bf_a, &bf_b, 3)))
    return unsupported("tensor map encoding rejected the operand");
  if (pair) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * min(pairs, tiles_m * tiles_n * splits));
    cfg.blockDim = dim3(PAIR_THREADS);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (f16) {
      cfg.dynamicSmemBytes = max(pair_smem<3>(), pair_smem<6>());
      HB_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_tcgen05_pair_f16_kernel, m_a, m_b, bf_a, bf_b, p));
    } else if (planes == 3) {
      cfg.dynamicSmemBytes = pair_smem<6>();
      HB_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_tcgen05_pair_kernel<6>, m_a, m_b, p));
    } else if (planes == 2) {
      cfg.dynamicSmemBytes = pair_smem<3>();
      HB_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_tcgen05_pair_kernel<3>, m_a, m_b, p));
    } else {
      cfg.dynamicSmemBytes = pair_smem<1>();
      HB_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_tcgen05_pair_kernel<1>, m_a, m_b, p));
    }
  } else {
    const int grid = min(sms, tiles_m * tiles_n * splits);
    if (f16)
      gemm_tcgen05_f16_kernel<<<grid, THREADS, max(single_smem<3>(), single_smem<6>()), stream>>>(m_a, m_b, bf_a, bf_b, p);
    else if (planes == 3)
      gemm_tcgen05_kernel<6><<<grid, THREADS, single_smem<6>(), stream>>>(m_a, m_b, p);
    else if (planes == 2)
      gemm_tcgen05_kernel<3><<<grid, THREADS, single_smem<3>(), stream>>>(m_a, m_b, p);
    else
      gemm_tcgen05_kernel<1><<<grid, THREADS, single_smem<1>(), stream>>>(m_a, m_b, p);
  }
  HB_LAUNCH_OK();
  count_launch(1);
  if (via_partial) {
    auto reduce = g.dtype_c == HASTE_B200_BF16  ? launch_reduce<__nv_bfloat16>
                  : g.dtype_c == HASTE_B200_F16 ? launch_reduce<__half>
                                                : launch_reduce<float>;
    reduce(partial, splits, M, N, part_ld, g.c, g.ldc, g.accumulate, 16 * sms, stream);
    HB_LAUNCH_OK();
    count_launch(1);
  }
  return HASTE_B200_OK;
}

}  // namespace hb
