// LayerNormLSTM / LayerNormGRU recurrences over the whole grid, sm_100a: the sizes that do not fit the
// clusters of rec_ln_cluster.cuh - up to 512 units (bf16 storage: 1024), or many batch rows.
//
// A LayerNorm step is a chain of three hand-offs (GRU: two): the row statistics of h.R, of the cell
// state, and the new state - backward: partial dh, and two pairs of row sums.  Through L2 each of them
// takes 0.7 us from store to load and 1.2 .. 1.4 with what makes and takes it, however little is in it.
// The layout is therefore that of rec_grid_kernels.cuh - grid = (slices of 16 hidden units) x (row
// groups), the batch in chains of eight rows, product warps that hold R and finishing warps in two
// groups of four that take the chains in turn.  A group's chains are a stage apart - chain 0 A B C,
// chain 1 C' A B - so that the hand-offs of one are under way while another computes.  A bidirectional
// level runs as two such grids of half the GPU.
//   LayerNormLSTM fp32, 64 rows, H = 512, us per step forward / backward: 7.4 / 10.7 with 16 rows per CTA as
// one piece; here 6.5 / 6.9 with two chains per CTA, and 9.5 / 10.6 for both directions of a level side by
// side with four (one chain: 5.4 / 5.7).  What bounds it then is the finishing warps' own time, about
// 1200 instructions per warp, chain and step at the latency of dependent ones.
//
// The statistics of a CTA's 64 columns meet in its shared memory first (a barrier of the group's four
// warps); one 64-byte line per row chain and CTA then travels: 8 rows x (mean, M2) or (sum, sum).
//
// Arithmetic, fp32 storage: the operands of the step product are two fp16 planes each, h 2^14 and R
// scaled by a power of two per tile (values reach 2^15 at most), all four products.  That is 22 .. 23
// bits per operand, where the exchanged words carry 23; three bf16 planes took six products.  (With the
// gate functions of rec_ln_common.cuh outputs and gradients are as far from fp64 as before or nearer.)
// A chain with a state of 2 or more (an initial state may be) is multiplied in passes (product_by_size).
// Backward, the rows of d(h.R) are scaled by a bound on their largest value that falls out of the statistics'
// meeting.  bf16 storage: one bf16 plane.
#pragma once

#include "rec_grid_launch.cuh"
#include "rec_ln_cluster.cuh"

namespace hb {
namespace rec {

struct LnGridFwd : LnFwdParams {
  int CTAS, CH, K16, ring, throttle, wide;
};
struct LnGridBwd : LnBwdParams {
  int CTAS, CH, K16, wide;
  int pairs;       // the saved statistics start on whole pairs
  float* db_part;  // [2 x row groups][4][H]
};

// R on chip: N fragments of 16 gate columns x 16 units per tile.  Up to four of them stay in registers (one
// plane); the second plane and fragments beyond the fourth (bf16 storage, beyond 512 units) lie in shared
// memory.  P: registers per thread of the product warps; the finishing warps get the rest of 256.  (With all
// of R in registers they had 80, and spilled: LayerNormLSTM fp32, 64 rows, H = 512, two directions at a
// time, us per step forward / backward 11.3 / 13.1 -> 10.6 / 10.5.)  Backward beyond 512 units every warp keeps the 128 of
// the launch: with 104 the finishing warps bounded the step (us for a backward call of 60 steps with 104 / 128, LayerNormGRU
// bf16 H = 1024: 8 rows 785 / 721, 128 rows 2213 / 1770; H = 1001 128 rows 2504 / 2079; LayerNormLSTM H = 1024 128 rows
// 2896 / 2275).
template <int N>
struct LgRegs {
  static constexpr int KEEP = N < 4 ? N : 4, P = N <= 2 ? 112 : (N == 3 ? 120 : (N == 4 ? 136 : 152)), F = 256 - P;
};
template <int N>
__device__ __forceinline__ void reg_product() {
  if constexpr (LgRegs<N>::P > 128) reg_inc<LgRegs<N>::P>();
  else reg_dec<LgRegs<N>::P>();
}
template <int N>
__device__ __forceinline__ void reg_finish() {
  if constexpr (LgRegs<N>::F > 128) reg_inc<LgRegs<N>::F>();
  else reg_dec<LgRegs<N>::F>();
}
constexpr int LG_FWD_STASH = 6, LG_BWD_STASH = 19;  // floats per thread and chain

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }  // -126 .. 127
// The s for which most * 2^s is in [2^14, 2^15), as far as 2^s and 2^-s are floats.
__device__ __forceinline__ int f16_shift_of(float most) {
  return max(-126, min(126, 141 - (int)((__float_as_uint(most) >> 23) & 0xff)));
}
// (an infinity is one in either plane; the values beside it keep their scale)
__device__ __forceinline__ float finite_max(float m, float x) {
  x = fabsf(x);
  return x <= 3.402823466e38f ? fmaxf(m, x) : m;
}
// Two values -> the same pair in two fp16 planes.
__device__ __forceinline__ void f16_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const __half2 l = __floats2half2_rn(a - __low2float(h), b - __high2float(h));
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// A fragments of NS k-steps (x: row half 0 / 1, four consecutive k each): the first plane's first KEEP in
// registers, its others, or the second plane, in shared memory (512 bytes apart).  Returns the factor that
// takes their scale out of the product again.
template <int SPLIT, int NS, int KEEP>
__device__ __forceinline__ float scaled_fragments(float (&x)[NS][2][4], uint32_t (&hi)[KEEP][4], uint4* rest) {
  if constexpr (SPLIT == 1) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      uint32_t v[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) v[a] = pack_bf16(x[s][a & 1][(a >> 1) * 2], x[s][a & 1][(a >> 1) * 2 + 1]);
      if (s < KEEP) {
#pragma unroll
        for (int a = 0; a < 4; ++a) hi[s % KEEP][a] = v[a];
      } else {
        rest[(s - KEEP) * 32] = make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
    return 1.f;
  } else {
    static_assert(NS == KEEP, "both planes do not fit beyond 512 units");
    float most = 0.f;
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
      for (int i = 0; i < 8; ++i) most = finite_max(most, x[s][i >> 2][i & 3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
    const int sh = f16_shift_of(most);
    const float f = pow2(sh);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      uint32_t l[4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
        f16_pair(x[s][a & 1][(a >> 1) * 2] * f, x[s][a & 1][(a >> 1) * 2 + 1] * f, hi[s][a], l[a]);
      rest[s * 32] = make_uint4(l[0], l[1], l[2], l[3]);
    }
    return pow2(-sh);
  }
}
// The product of a chain with a state of 2 or more (x: this lane's values of row lane >> 2, in shared memory,
// because the registers are full).  An element is scaled by its own row and size, so that it keeps its 22 bits
// whatever lies beside it: a first pass takes what is smaller than 2, as the usual product does and with the same
// result, each further one what is within 2^-16 of the largest value that is left of a row.  Infinities and NaN
// go with the first pass.
template <int KSW, int NMT, int KEEP>
__device__ __forceinline__ void product_by_size(float4* x, const uint32_t (&wf)[NMT][KEEP][4], const uint4* rest,
                                                const float (&wscale)[NMT], float (&acc)[NMT][4]) {
  const int q = threadIdx.x & 3;
  const uint32_t at = smem_u32(x);
  bool some = false;
#pragma unroll
  for (int s = 0; s < KSW; ++s) some |= x[s * 32].x != 0.f || x[s * 32].y != 0.f || x[s * 32].z != 0.f || x[s * 32].w != 0.f;
  if (!__any_sync(0xffffffffu, some)) return;  // (the usual initial state)
  float least = 0.f, limit = 2.f;  // of what this pass takes
  int sh = 14;
  auto takes = [&](float v) {
    v = fabsf(v);
    return (v >= least && v < limit) || !(v <= 3.402823466e38f);
  };
#pragma unroll 1
  for (int pass = 0; pass < 32; ++pass) {  // (a float's 277 powers of two are 18 passes)
    const float f = pow2(sh);
    auto planes = [&](int s, uint32_t (&hi)[2], uint32_t (&lo)[2]) {
      float4 v;  // (volatile: made anew for each tile)
      asm volatile("ld.volatile.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                   : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at + s * 512) : "memory");
      f16_pair(takes(v.x) ? v.x * f : 0.f, takes(v.y) ? v.y * f : 0.f, hi[0], lo[0]);
      f16_pair(takes(v.z) ? v.z * f : 0.f, takes(v.w) ? v.w * f : 0.f, hi[1], lo[1]);
    };
    const float back = pow2(-sh);
    const float u0 = __shfl_sync(0xffffffffu, back, 8 * q), u1 = __shfl_sync(0xffffffffu, back, 8 * q + 4);
#pragma unroll
    for (int mt = 0; mt < NMT; ++mt) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};  // in the order of the usual product
#pragma unroll
      for (int s = 0; s < KSW; ++s) {
        uint32_t bh[2], bl[2];
        planes(s, bh, bl);
        const uint4 a = rest[(mt * KSW + s) * 32];
        mma_f16(d, wf[mt][s % KEEP], bl[0], bl[1]);
        mma_f16(d, a, bl[0], bl[1]);
        mma_f16(d, a, bh[0], bh[1]);
      }
#pragma unroll
      for (int s = 0; s < KSW; ++s) {
        uint32_t bh[2], bl[2];
        planes(s, bh, bl);
        mma_f16(d, wf[mt][s % KEEP], bh[0], bh[1]);
      }
      const float f0 = wscale[mt] * u0, f1 = wscale[mt] * u1;
      acc[mt][0] += d[0] * f0; acc[mt][1] += d[1] * f1;
      acc[mt][2] += d[2] * f0; acc[mt][3] += d[3] * f1;
    }
    float most = 0.f;  // of what is left
#pragma unroll
    for (int s = 0; s < KSW; ++s) {
      float4 v = x[s * 32];
      v.x = takes(v.x) ? 0.f : v.x; v.y = takes(v.y) ? 0.f : v.y;
      v.z = takes(v.z) ? 0.f : v.z; v.w = takes(v.w) ? 0.f : v.w;
      x[s * 32] = v;
      most = fmaxf(most, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
    if (!__any_sync(0xffffffffu, most > 0.f)) return;
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 1));
    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 2));
    sh = f16_shift_of(most);
    least = most * (1.0f / 65536.0f);
    limit = __uint_as_float(0x7f800000u);
  }
}
// How many fragments of a tile lie in shared memory.
template <int SPLIT, int NS>
constexpr int frag_rest() { return SPLIT == 2 ? NS : NS - LgRegs<NS>::KEEP; }

// Whether a phase has ended, without waiting.
__device__ __forceinline__ bool mb_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Barrier of a group's four warps; true if any of them has given up.
__device__ __forceinline__ bool group_barrier_or(int grp, bool flag) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, %2, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)flag), "r"(1 + grp)
      : "memory");
  return r != 0;
}

// ---- inputs and outputs of a finishing warp, in pieces of one quad of one row (rec_chain.cuh), NB blocks
// of four arrays per slot
constexpr int LN_PIECE = 16;
template <typename T, int NB>
struct LnIo {
  static constexpr int BLOCK = 32 * LN_PIECE, SLOT = NB * BLOCK;
  static constexpr int WARP = IO_RING * SLOT + BLOCK;  // + a block for the outputs
};
// 16-bit rows that start anywhere: up to three aligned words hold the piece, and the fourth word of its place says
// how many values lie before it.  Results leave in words too, as far as they go (LnOutput).  LayerNormGRU, 64 rows,
// 333 units, us per step forward / backward: loaded by value into registers and stored by value 5.2 / 6.5, loaded in
// words 5.1 / 6.0, both in words 4.0 / 4.6; 336 units 3.6 / 3.6.
template <typename T>
__device__ __forceinline__ void fetch_piece(uint32_t dst, const void* src, bool wide, int units) {
  if (wide) {
    cp_async_piece<4 * (int)sizeof(T)>(dst, src);
  } else if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < units)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * e), "l"(static_cast<const T*>(src) + e)
                     : "memory");
  } else {
    const uint32_t before = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src)) & 2u;
    const int bytes = (int)before + 2 * units;
#pragma unroll
    for (int e = 0; e < 3; ++e)
      if (4 * e < bytes)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * e),
                     "l"(static_cast<const char*>(src) - before + 4 * e), "r"(min(4, bytes - 4 * e))
                     : "memory");
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(dst + 12), "r"(before >> 1) : "memory");
  }
}
// Fetches the steps of chains grp, grp + 2, ... of every time step, IO_RING - 1 ahead.
template <typename T, int NB, bool BWD>
struct LnInputs {
  using Io = LnIo<T, NB>;
  const char* src[NB];   // this lane's piece at time 0 of chain row 0; null: none
  const char* pair;      // this lane's pair of values of a row (statistics), in its piece of the last block
  uint32_t step[NB];     // bytes per (time, row)
  uint32_t ring;
  int t, ch, slot_in, slot_out, units, pairs;

  __device__ __forceinline__ void init(uint8_t* buf, int lane, int T_, int grp, int units_) {
    ring = smem_u32(buf) + lane * LN_PIECE;
    t = BWD ? T_ - 1 : 0;
    ch = grp;
    slot_in = slot_out = 0;
    units = units_;
#pragma unroll
    for (int b = 0; b < NB; ++b) { src[b] = nullptr; step[b] = 0; }
    pair = nullptr;
    pairs = 1;
  }
  // array `base` (first element of the quad in row 0) with rows of `width` values, `first` rows on
  __device__ __forceinline__ void array(int b, const void* base, int u0, int width, int first, int lane) {
    step[b] = (uint32_t)width * sizeof(T);
    src[b] = (base && units > 0)
                 ? reinterpret_cast<const char*>(static_cast<const T*>(base) + u0) + (size_t)(first + (lane & 7)) * step[b]
                 : nullptr;
  }
  __device__ __forceinline__ void fetch(int T_, int N, bool wide, int lane, int tile0, int ch_n, int grp) {
    if (BWD ? t >= 0 : t < T_) {
      const int n0 = (tile0 + ch) * 8;
      const uint32_t row = (uint32_t)(t * N + n0), dst = ring + slot_in * Io::SLOT;
      if (n0 + (lane & 7) < N) {
#pragma unroll
        for (int b = 0; b < NB; ++b)
          if (src[b]) fetch_piece<T>(dst + b * Io::BLOCK, src[b] + (unsigned long long)row * step[b], wide, units);
        if (BWD && pair) {
          const char* from = pair + (unsigned long long)row * (2 * sizeof(T));
          const uint32_t to = dst + (NB - 1) * Io::BLOCK;
          if (pairs) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(from), "n"(2 * (int)sizeof(T)) : "memory");
          } else {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              if constexpr (sizeof(T) == 4)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + 4 * e), "l"(from + 4 * e) : "memory");
              else
                asm volatile("st.shared.u16 [%0], %1;" ::"r"(to + 2 * e), "h"(reinterpret_cast<const unsigned short*>(from)[e])
                             : "memory");
            }
          }
        }
      }
      if ((ch += 2) >= ch_n) {
        ch = grp;
        t += BWD ? -1 : 1;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++slot_in == IO_RING) slot_in = 0;
  }
  // The oldest step's slot; once this warp has read it, a fetch follows.
  __device__ __forceinline__ const uint8_t* wait(const uint8_t* buf) {
    asm volatile("cp.async.wait_group %0;" ::"n"(IO_RING - 2) : "memory");
    __syncwarp();
    const uint8_t* s = buf + slot_out * Io::SLOT;
    if (++slot_out == IO_RING) slot_out = 0;
    return s;
  }
};
template <typename T>
__device__ __forceinline__ float piece_value(const uint8_t* slot, int b, int a, int row, int ul, bool wide) {
  const uint8_t* at = slot + (b * 32 + a * 8 + row) * LN_PIECE;
  if constexpr (sizeof(T) == 2)
    if (!wide) ul += *reinterpret_cast<const int*>(at + 12);
  return ld(reinterpret_cast<const T*>(at) + ul);
}
// Results of a finishing warp, up to four arrays with rows of `width` values: a lane stores the piece of array
// lane >> 3 and row lane & 7.
template <typename T>
struct LnOutput {
  char* base;     // this lane's piece in row 0, null: none
  uint32_t step;  // bytes per row
  __device__ __forceinline__ void init(void* array, long long first, int u0, int width, int units, int lane) {
    step = (uint32_t)width * sizeof(T);
    base = (array && units > 0)
               ? reinterpret_cast<char*>(static_cast<T*>(array) + u0) + (size_t)(first + (lane & 7)) * step
               : nullptr;
  }
  template <int NA>
  __device__ __forceinline__ void put(uint8_t* out, const float (&v)[NA], uint32_t row0, int rows, int units, bool wide,
                                      int lane, int row, int ul) const {
    __syncwarp();  // the pieces before have been read
#pragma unroll
    for (int a = 0; a < NA; ++a) st(reinterpret_cast<T*>(out + (a * 8 + row) * 4 * (int)sizeof(T)) + ul, v[a]);
    __syncwarp();
    if ((lane >> 3) < NA && (lane & 7) < rows && base) {
      T* d = reinterpret_cast<T*>(base + (unsigned long long)row0 * step);
      const uint8_t* src = out + lane * 4 * (int)sizeof(T);
      if (wide) {
        copy_piece<T>(d, src);
      } else if (sizeof(T) == 2 && units == 4) {
        const uint16_t* v = reinterpret_cast<const uint16_t*>(src);
        uint16_t* to = reinterpret_cast<uint16_t*>(d);
        const uint32_t w0 = *reinterpret_cast<const uint32_t*>(v), w1 = *reinterpret_cast<const uint32_t*>(v + 2);
        if (reinterpret_cast<uintptr_t>(d) & 2u) {
          to[0] = v[0];
          *reinterpret_cast<uint32_t*>(to + 1) = __byte_perm(w0, w1, 0x5432);
          to[3] = v[3];
        } else {
          *reinterpret_cast<uint32_t*>(to) = w0;
          *reinterpret_cast<uint32_t*>(to + 2) = w1;
        }
      } else {
        for (int e = 0; e < units; ++e) d[e] = reinterpret_cast<const T*>(src)[e];
      }
    }
  }
};

// ---- statistics -----------------------------------------------------------------------------
// Words of a pair per row and CTA: [stat][parity][row tile][source CTA][8 rows][2 words] - lines that one CTA
// writes: with the words of several CTAs in a sector a step took half as long again.  Warp
// `quad` of a group takes the row pair 2 quad, 2 quad + 1 from all sources, a source (nHS > 32: two) per
// lane; the results meet in shared memory.  (Rows beyond the batch travel too.)  The loads are issued one
// stage ahead of their use: a look at L2 takes 800 cycles.  (Every warp on its own for all eight rows took
// four times the loads and twice the instructions.)
__device__ __forceinline__ size_t stat_at(int stat, int par, int tiles, int tile, int nHS) {
  return (size_t)((stat * 2 + par) * tiles + tile) * nHS * 16;
}
template <int NS>
struct StatWords {
  uint4 y[NS];
  const uint32_t* src;
  __device__ __forceinline__ void load(int nHS, int lane, uint32_t tag) {
#pragma unroll
    for (int k = 0; k < NS; ++k) y[k] = ld_relaxed_u32x4_if(lane + 32 * k < nHS, src + k * 512, tag);
  }
  // Until they are all there.
  __device__ __forceinline__ bool wait(int nHS, int lane, uint32_t tag, const Sync& sync, volatile int* s_abort, int code) {
    long long t0 = 0;
    unsigned int spins = 0;
    for (;;) {
      uint32_t bad = 0;
#pragma unroll
      for (int k = 0; k < NS; ++k) bad |= stale4(y[k], tag);
      if (__all_sync(0xffffffffu, (bad & 1u) == 0)) return true;
      if (__any_sync(0xffffffffu, !may_spin(spins, t0, sync, s_abort, code))) return false;
      load(nHS, lane, tag);
    }
  }
  // (first row's pair, second row's); a bare tag is zero
  __device__ __forceinline__ float4 value(int k) const {
    return make_float4(fword_value(y[k].x), fword_value(y[k].y), fword_value(y[k].z), fword_value(y[k].w));
  }
};
// A lane holds a value for either row of the pair; sums over the warp: the first row's in lanes 0 .. 15, the
// second's in the others.
__device__ __forceinline__ float pair_sum(float first, float second, int lane) {
  const bool own = lane >= 16;
  float s = (own ? second : first) + __shfl_xor_sync(0xffffffffu, own ? first : second, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// ---------------------------------------------------------------------------------------
template <int G, int KSW, int SPLIT, typename T>
__global__ void __launch_bounds__(GL_THREADS, 1) lg_fwd_kernel(const __grid_constant__ LnGridFwd p) {
  constexpr int NS = KSW <= 4 ? 1 : 2;  // sources of a lane in the exchange of statistics
  constexpr int NMT = 4, PART = GL_WARPS * NMT * 32, GT = 128;  // GT: threads of a finishing group
  using Io = LnIo<T, 2>;
  extern __shared__ __align__(16) uint8_t smem[];
  float4* part = reinterpret_cast<float4*>(smem);                              // [ring][warp][NMT][lane]
  uint4* planes = reinterpret_cast<uint4*>(part + p.ring * PART);              // [warp][NMT][what is not in registers][lane]
  float* stash = reinterpret_cast<float*>(planes + PART * frag_rest<SPLIT, KSW>());  // [CH][LG_FWD_STASH][GT]
  float* consts = stash + p.CH * LG_FWD_STASH * GT;                            // [3 G + 2][quad][unit]
  float2* meet = reinterpret_cast<float2*>(consts + (3 * G + 2) * 16);         // [2 groups][2][quad][8]
  float2* found = meet + 2 * 2 * NMT * 8;                                      // [2 groups][2][8] mean, 1/sigma
  uint64_t* barp = reinterpret_cast<uint64_t*>(found + 2 * 2 * 8);             // full[ring], empty[ring]
  const uint32_t pbar = smem_u32(barp), obar = pbar + 16 * p.ring;             // and, per chain: h has left
  uint8_t* io_base = reinterpret_cast<uint8_t*>(barp + 2 * p.ring + ((p.CH + 1) & ~1));
  __shared__ int s_abort_;
  volatile int* s_abort = &s_abort_;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, q = lane & 3;
  const int nHS = p.CTAS, hs = blockIdx.x % nHS, rg = blockIdx.x / nHS;
  const int H = p.H, N = p.N, u0 = hs * 16, tile0 = rg * p.CH, tiles = (N + 7) >> 3;
  const int ch_n = min(p.CH, tiles - tile0);
  if (tid == 0) {
    *s_abort = 0;
    for (int i = 0; i < p.ring; ++i) {
      mb_init(pbar + 8 * i, GL_WARPS);
      mb_init(pbar + 8 * (p.ring + i), NMT);
    }
    for (int i = 0; i < p.CH; ++i) mb_init(obar + 8 * i, NMT);
  }
  for (int i = tid; i < (3 * G + 2) * 16; i += GL_THREADS) {
    const int a = i / 16, unit = u0 + (i & 15);
    const void* src = a < G ? p.b : a < 2 * G ? (G == 3 ? p.b2 : nullptr) : a < 3 * G ? p.gamma_Rh
                                                                     : a == 3 * G ? p.gamma_h : p.beta_h;
    const int g = a < 3 * G ? a % G : 0;
    consts[i] = (src && unit < H) ? ld(static_cast<const T*>(src) + g * H + unit) : 0.f;
  }
  for (int i = tid; i < GL_WARPS * Io::WARP / 16; i += GL_THREADS)
    reinterpret_cast<uint4*>(io_base)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const int ring = min(p.ring, ch_n);  // a slot per chain, where they fit
  int slot = 0;
  uint32_t phase = 0;
  auto next_slot = [&]() {
    if (++slot == ring) { slot = 0; phase ^= 1u; }
  };
  constexpr uint32_t TAGBIT = SPLIT == 2 ? 1u : 0x40000000u;

  if (w < GL_WARPS) {
    // ------------------------------------------------------------------ product warps (as gl_fwd_kernel)
    reg_product<KSW>();
    constexpr int KEEP = LgRegs<KSW>::KEEP, REST = frag_rest<SPLIT, KSW>();
    uint32_t wf[NMT][KEEP][4];
    uint4* rest = planes + w * NMT * REST * 32 + lane;  // this lane's fragments that lie in shared memory
    float wscale[NMT];
#pragma unroll
    for (int mt = 0; mt < NMT; ++mt) {
      float x[KSW][2][4];
      const int unit = u0 + 4 * mt + (gq >> 1), ga = gq & 1;
#pragma unroll
      for (int s = 0; s < KSW; ++s) {
        const int k = ((w * KSW + s) * 4 + q) * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool ok = unit < H && k + i < H;
          const T* r = static_cast<const T*>(p.R) + (long long)(k + i) * G * H + unit;
          x[s][0][i] = ok ? ld(r + (long long)ga * H) : 0.f;
          x[s][1][i] = (ok && ga + 2 < G) ? ld(r + (long long)(ga + 2) * H) : 0.f;
        }
      }
      wscale[mt] = scaled_fragments<SPLIT, KSW, KEEP>(x, wf[mt], rest + mt * REST * 32);
    }
    const int kq = w * KSW * 4 + q;
    const uint32_t* src0 = p.xbuf + ((size_t)tile0 * p.K16 + w * KSW) * 128 + q * 32 + gq * 4;
    const uint32_t xtile = (uint32_t)p.K16 * 128, xpar = (uint32_t)tiles * xtile;
    const int nrow = N - tile0 * 8 - gq;
    auto fetch = [&](uint32_t par, uint32_t wt, int ch, uint4 (&y)[KSW], int s0, int s1) {
      const uint32_t* src = src0 + par * xpar + (uint32_t)ch * xtile;
      const bool rok = ch * 8 < nrow;
#pragma unroll
      for (int s = 0; s < KSW; ++s)
        if (s >= s0 && s < s1)
          y[s] = ld_relaxed_u32x4_if(rok && kq + s * 4 < nHS * NMT, src + s * 128, wt);
    };
    const bool throttle = p.throttle || w * KSW * 4 >= nHS * NMT;
    bool alive = true;
    uint4 y[KSW];
    auto tag_of = [](int t) {
      const uint32_t rt = (((uint32_t)t >> 1) & 1u) ^ 1u;
      return SPLIT == 2 ? rt : rt << 30;
    };
    fetch(0, tag_of(0), 0, y, 0, KSW);
    // Product warps that poll all the time fill the way to L2 for the statistics and for the words themselves.  So
    // after a first look they wait until this CTA's own h of the chain has left; the others' leaves at about
    // that time.  bf16 storage, whose next look falls behind the whole product, does not even take that first look before
    // (us per step, polling / this: LayerNormGRU bf16 8 rows H = 512 4.2 / 3.7, 32 rows H = 1024 7.1 / 5.8, 128 rows 18.2 /
    // 16.1; LayerNormLSTM fp32 64 rows H = 512 7.7 / 7.1; LayerNormGRU fp32 128 rows 8.0 / 7.9, without the first look 8.8).
    constexpr bool kAskAhead = SPLIT == 2;
    bool asked = true;
    for (int t = 0; t < p.T && alive; ++t) {
      const uint32_t wt = tag_of(t);
      for (int ch = 0; ch < ch_n; ++ch) {
        if (!asked) {
          if (!mb_wait_warp(obar + 8 * ch, (t - 1) & 1, p.sync, s_abort, 74)) { alive = false; break; }
          fetch(t & 1, wt, ch, y, 0, KSW);
        }
        long long t0 = 0;
        unsigned int spins = 0;
        uint32_t bad;
        for (;;) {
          bad = 0;
#pragma unroll
          for (int s = 0; s < KSW; ++s) bad |= stale4(y[s], wt);
          if (__all_sync(0xffffffffu, (bad & TAGBIT) == 0)) break;
          if (kAskAhead && spins == 0 && t > 0 && !mb_wait_warp(obar + 8 * ch, (t - 1) & 1, p.sync, s_abort, 74)) {
            alive = false;
            break;
          }
          if (__any_sync(0xffffffffu, !may_spin(spins, t0, p.sync, s_abort, 63))) { alive = false; break; }
          fetch(t & 1, wt, ch, y, 0, KSW);
        }
        if (!alive) break;
        // the next chain's words are on their way while this one's are multiplied (beyond the last step: words
        // that nobody waits for)
        const int ch2 = ch + 1 < ch_n ? ch + 1 : 0, t2 = ch + 1 < ch_n ? t : t + 1;
        auto fetch_next = [&]() {
          asked = kAskAhead || t2 == 0 || __all_sync(0xffffffffu, mb_test(obar + 8 * ch2, (t2 - 1) & 1));
          if (asked) fetch(t2 & 1, tag_of(t2), ch2, y, 0, KSW);
        };
        float acc[NMT][4];
#pragma unroll
        for (int mt = 0; mt < NMT; ++mt) acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.f;
        constexpr float kUsual = 1.0f / 16384.0f;  // takes the usual scale of h out again
        // (the tag lies in bit 0, so bit 30 of `bad` says that some state is 2 or more)
        const bool apart = SPLIT == 2 && __any_sync(0xffffffffu, (bad & 0x40000000u) != 0 || t == 0);
        if (__builtin_expect(apart, 0)) {
          if constexpr (SPLIT == 2) {
            // (the place of this warp's results: free as below)
            if (throttle &&
                !mb_wait_warp(pbar + 8 * (p.ring + slot), phase ^ 1u, p.sync, s_abort, 64)) { alive = false; break; }
            static_assert(KSW <= NMT, "a lane's values take the place of its results");
            float4* x = part + slot * PART + w * NMT * 32 + lane;
#pragma unroll
            for (int s = 0; s < KSW; ++s)
              x[s * 32] = make_float4(fword_value(y[s].x), fword_value(y[s].y), fword_value(y[s].z), fword_value(y[s].w));
            // The first step multiplies the initial state as the caller has it: its words, which say that the
            // others are there too, lack the last bit.
            if (t == 0 && ch * 8 < nrow) {
              const T* h0 = static_cast<const T*>(p.h) + (long long)((tile0 + ch) * 8 + gq) * H;
#pragma unroll
              for (int i = 0; i < KSW * 4; ++i) {
                const int k = (kq + (i >> 2) * 4) * 4 + (i & 3);
                if (k < H) reinterpret_cast<float*>(x + (i >> 2) * 32)[i & 3] = ld(h0 + k);
              }
            }
            product_by_size<KSW, NMT, KEEP>(x, wf, rest, wscale, acc);
            fetch_next();
          }
        } else if constexpr (SPLIT == 2) {
          constexpr float f = 1.0f / kUsual;
          uint32_t bh[KSW][2], bl[KSW][2];
#pragma unroll
          for (int s = 0; s < KSW; ++s) {
            f16_pair(fword_value(y[s].x) * f, fword_value(y[s].y) * f, bh[s][0], bl[s][0]);
            f16_pair(fword_value(y[s].z) * f, fword_value(y[s].w) * f, bh[s][1], bl[s][1]);
          }
          // the small products first
#pragma unroll
          for (int s = 0; s < KSW; ++s) {
#pragma unroll
            for (int mt = 0; mt < NMT; ++mt) mma_f16(acc[mt], wf[mt][s % KEEP], bl[s][0], bl[s][1]);
#pragma unroll
            for (int mt = 0; mt < NMT; ++mt) {
              const uint4 a = rest[(mt * REST + s) * 32];
              mma_f16(acc[mt], a, bl[s][0], bl[s][1]);
              mma_f16(acc[mt], a, bh[s][0], bh[s][1]);
            }
          }
          fetch_next();
#pragma unroll
          for (int s = 0; s < KSW; ++s)
#pragma unroll
            for (int mt = 0; mt < NMT; ++mt) mma_f16(acc[mt], wf[mt][s % KEEP], bh[s][0], bh[s][1]);
#pragma unroll
          for (int mt = 0; mt < NMT; ++mt)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[mt][i] *= wscale[mt] * kUsual;
        } else {
#pragma unroll
          for (int s = 0; s < KSW; ++s) {
            const uint32_t b0 = __byte_perm(y[s].x, y[s].y, 0x5410), b1 = __byte_perm(y[s].z, y[s].w, 0x5410);
#pragma unroll
            for (int mt = 0; mt < NMT; ++mt) {
              if (s < KEEP) {
                mma_bf16(acc[mt], wf[mt][s % KEEP], b0, b1);
              } else {
                const uint4 a = rest[(mt * REST + s - KEEP) * 32];
                const uint32_t af[4] = {a.x, a.y, a.z, a.w};
                mma_bf16(acc[mt], af, b0, b1);
              }
            }
          }
          fetch_next();
        }
        // (a slot per chain needs no look at `empty`: h of the next step took the statistics of this one,
        // which left after the group's barrier, and the partials are read before it)
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
    // ------------------------------------------------------------------ finishing warps: quad f & 3 of the
    // chains grp, grp + 2, ...; lane = (unit ul, row)
    reg_finish<KSW>();
    const int f = w - GL_WARPS, grp = f >> 2, quad = f & 3, gt = quad * 32 + lane;
    const int ul = lane >> 3, row = 2 * q + (gq & 1);
    const bool odd = gq & 1;
    const int uq = u0 + 4 * quad, unit = uq + ul, units = max(0, min(4, H - uq));
    const bool uok = unit < H;
    const long long NH = (long long)N * H;
    T *hb = static_cast<T*>(p.h), *cb = static_cast<T*>(p.c);
    const float* cst = consts + quad * 4 + ul;  // this unit's constants, 16 apart
    const size_t xtile = (size_t)p.K16 * 128;
    const int Q = hs * NMT + quad;
    uint32_t* xdst = p.xbuf + (size_t)(Q >> 2) * 128 + (Q & 3) * 32 + row * 4 + ul;
    const bool full = units == 4, cta_full = H - u0 >= 16;  // no ragged edge here
    const float cnt_last = (float)(H - (nHS - 1) * 16), rec_H = 1.0f / (float)H;
    float count[NS];  // units of this lane's sources
#pragma unroll
    for (int k = 0; k < NS; ++k) count[k] = lane + 32 * k < nHS - 1 ? 16.f : (lane + 32 * k == nHS - 1 ? cnt_last : 0.f);
    for (int ch = grp; ch < ch_n; ch += 2) {
      const int n = (tile0 + ch) * 8 + row;
      const bool ok = n < N && uok;
      float* sh = stash + (size_t)ch * LG_FWD_STASH * GT + gt;
      const float h0 = ok ? ld(hb + (long long)n * H + unit) : 0.f;
      if (n < N) gl_publish(xdst + (size_t)(tile0 + ch) * xtile, hword_encode<SPLIT>(h0, 1u));
      sh[0] = h0;
      sh[GT] = (G == 4 && ok) ? ld(cb + (long long)n * H + unit) : 0.f;
    }
    uint8_t* io = io_base + f * Io::WARP;
    uint8_t* out = io + IO_RING * Io::SLOT;
    LnInputs<T, 2, false> inputs;
    LnOutput<T> o_rh, o_v, o_state;  // h.R; gates; h, c, LN(c)
    inputs.init(io, lane, p.T, grp, units);
    {
      const int a = lane >> 3;
      inputs.array(0, a < G ? static_cast<const T*>(p.Wx) + (long long)a * H : nullptr, uq, G * H, 0, lane);
      inputs.array(1, (a == 0 && p.has_zoneout && p.training) ? p.mask : nullptr, uq, H, 0, lane);
      o_rh.init(static_cast<T*>(p.act_Rh) + (long long)a * H, 0, uq, G * H, a < G ? units : 0, lane);
      o_v.init(p.training && p.v ? static_cast<T*>(p.v) + (long long)a * H : nullptr, 0, uq, 4 * H, units, lane);
      o_state.init(a == 0 ? p.h : (G == 4 ? (a == 1 ? p.c : a == 2 ? p.act_c_norm : nullptr) : nullptr), a < 2 ? N : 0, uq, H,
                   units, lane);
    }
    if (grp < ch_n) {
#pragma unroll
      for (int i = 0; i < IO_RING - 1; ++i) inputs.fetch(p.T, N, p.wide, lane, tile0, ch_n, grp);
    }
    bool alive = true, stop = false;
    int turn = 0, fturn = 0;
    // A row's (mean, M2) over this CTA's columns (NV values per unit), on its way.  One group barrier.
    auto publish = [&](int stat, int t, int ch, const auto& v, uint32_t tag) {
      constexpr int NV = sizeof(v) / sizeof(float);
      float m = 0.f, d = 0.f;
      if (full) {
#pragma unroll
        for (int g = 0; g < NV; ++g) m += v[g];
        m *= 1.0f / NV;
#pragma unroll
        for (int g = 0; g < NV; ++g) d += (v[g] - m) * (v[g] - m);
        // equal parts: the mean is halfway, and half the squared distance times a part's count is added
        float mo = __shfl_xor_sync(0xffffffffu, m, 8), dd = __shfl_xor_sync(0xffffffffu, d, 8);
        d += dd + (mo - m) * (mo - m) * (0.5f * NV);
        m = 0.5f * (m + mo);
        mo = __shfl_xor_sync(0xffffffffu, m, 16);
        dd = __shfl_xor_sync(0xffffffffu, d, 16);
        d += dd + (mo - m) * (mo - m) * (1.0f * NV);
        m = 0.5f * (m + mo);
      } else {
        for (int g = 0; g < NV; ++g) m += v[g];
        m = uok ? m : 0.f;
        m += __shfl_xor_sync(0xffffffffu, m, 8);
        m += __shfl_xor_sync(0xffffffffu, m, 16);
        m = units > 0 ? m / (float)(units * NV) : 0.f;
        for (int g = 0; g < NV; ++g) d += (v[g] - m) * (v[g] - m);
        d = uok ? d : 0.f;
        d += __shfl_xor_sync(0xffffffffu, d, 8);
        d += __shfl_xor_sync(0xffffffffu, d, 16);
      }
      float2* at = meet + (grp * 2 + turn) * NMT * 8;
      turn ^= 1;
      if (ul == 0) at[quad * 8 + row] = make_float2(m, d);
      stop = group_barrier_or(grp, !alive);
      if (stop || quad != ((ch >> 1) & 3)) return;
      float2 y[NMT];
#pragma unroll
      for (int k = 0; k < NMT; ++k) y[k] = at[k * 8 + (lane & 7)];
      float mc = 0.f, m2 = 0.f;
      if (cta_full) {
        const float a = 0.5f * (y[0].x + y[1].x), b = 0.5f * (y[2].x + y[3].x);
        const float da = y[1].x - y[0].x, db = y[3].x - y[2].x;
        mc = 0.5f * (a + b);
        m2 = ((y[0].y + y[1].y) + (y[2].y + y[3].y)) + (da * da + db * db) * (2.0f * NV) + (b - a) * (b - a) * (4.0f * NV);
      } else {
#pragma unroll
        for (int k = 0; k < NMT; ++k) mc += (float)max(0, min(4, H - u0 - 4 * k)) * y[k].x;
        mc /= (float)(H - u0);
#pragma unroll
        for (int k = 0; k < NMT; ++k)
          m2 += y[k].y + (float)max(0, min(4, H - u0 - 4 * k)) * (float)NV * (y[k].x - mc) * (y[k].x - mc);
      }
      if (lane < 8)
        publish_u32x2(p.sbuf + stat_at(stat, t & 1, tiles, tile0 + ch, nHS) + hs * 16 + lane * 2,
                      fword_encode(mc, tag), fword_encode(m2, tag));
    };
    StatWords<NS> sw;
    auto look = [&](int stat, int t, int ch, uint32_t tag) {
      sw.src = p.sbuf + stat_at(stat, t & 1, tiles, tile0 + ch, nHS) + lane * 16 + quad * 4;
      sw.load(nHS, lane, tag);
    };
    // One group barrier.
    auto collect = [&](int nv, uint32_t tag, float& mean, float& inv, int code) {
      if (!sw.wait(nHS, lane, tag, p.sync, s_abort, code)) alive = false;
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int k = 0; k < NS; ++k) {
        s0 += count[k] * sw.value(k).x;
        s1 += count[k] * sw.value(k).z;
      }
      const float m = pair_sum(s0, s1, lane) * rec_H, mo = __shfl_xor_sync(0xffffffffu, m, 16);
      const float m0 = lane >= 16 ? mo : m, m1 = lane >= 16 ? m : mo;
      s0 = s1 = 0.f;
#pragma unroll
      for (int k = 0; k < NS; ++k) {
        const float c = count[k] * (float)nv;
        const float4 v = sw.value(k);
        s0 += v.y + c * (v.x - m0) * (v.x - m0);
        s1 += v.w + c * (v.z - m1) * (v.z - m1);
      }
      const float r = rsqrtf(pair_sum(s0, s1, lane) * rec_H * (1.0f / (float)nv) + kLnEps);
      float2* at = found + (grp * 2 + fturn) * 8;
      fturn ^= 1;
      if ((lane & 15) == 0) at[quad * 2 + (lane >> 4)] = make_float2(m, r);
      stop = group_barrier_or(grp, !alive);
      const float2 v = at[row];
      mean = v.x;
      inv = v.y;
    };
    // The stages of a group's chains, each chain after the first one stage (at most the last) behind the one
    // before: chain 0 A B C, chain 1 C' A B, ... - see the head of this file.
    constexpr int S = G == 4 ? 3 : 2;
    const int nc = (ch_n - grp + 1) / 2;
    auto stat_tag = [](int t) { return (((uint32_t)t >> 1) & 1u) ^ 1u; };
    bool looked = false;
    // the statistics of the stage after (k, i), if it waits for any
    auto look_ahead = [&](int k, int i) {
      if (++i == nc) { i = 0; ++k; }
      const int s = k - min(i, S - 1), t = s / S, stage = s - t * S;
      looked = s >= 0 && s < S * p.T && stage > 0;
      if (looked) look(stage - 1, t, grp + 2 * i, stat_tag(t));
    };
    for (int k = 0; k < S * p.T + min(nc, S) - 1 && !stop; ++k)
      for (int i = 0; i < nc && !stop; ++i) {
        const int s = k - min(i, S - 1), t = s / S, stage = s - t * S;
        if (s < 0 || s >= S * p.T) continue;
        const int ch = grp + 2 * i, tile = tile0 + ch, n0 = tile * 8;
        const uint32_t rt = stat_tag(t), e = (uint32_t)(t * N + n0);
        float* sh = stash + (size_t)ch * LG_FWD_STASH * GT + gt;
        if (stage > 0 && !looked) look(stage - 1, t, ch, rt);
        if (stage == 0) {
          // ---- stage A: h.R, its statistics
          const int n = t * ch_n + ch, sl = ring == ch_n ? ch : n % ring;
          if (!mb_wait_warp(pbar + 8 * sl, (ring == ch_n ? t : n / ring) & 1, p.sync, s_abort, 65)) alive = false;
          const float4* pr = part + sl * PART + quad * 32 + lane;
          float4 v[GL_WARPS];
#pragma unroll
          for (int w8 = 0; w8 < GL_WARPS; ++w8) v[w8] = pr[w8 * NMT * 32];
          float d[4], rh4[4], rh[G];
          d[0] = ((v[0].x + v[1].x) + (v[2].x + v[3].x)) + ((v[4].x + v[5].x) + (v[6].x + v[7].x));
          d[1] = ((v[0].y + v[1].y) + (v[2].y + v[3].y)) + ((v[4].y + v[5].y) + (v[6].y + v[7].y));
          d[2] = ((v[0].z + v[1].z) + (v[2].z + v[3].z)) + ((v[4].z + v[5].z) + (v[6].z + v[7].z));
          d[3] = ((v[0].w + v[1].w) + (v[2].w + v[3].w)) + ((v[4].w + v[5].w) + (v[6].w + v[7].w));
          swap_gates(d, odd, rh4);
#pragma unroll
          for (int g = 0; g < G; ++g) rh[g] = rh4[g];
          publish(0, t, ch, rh, rt);
          if (stop) break;
          look_ahead(k, i);
          // ---- off the chain
          if (lane == 0) mb_arrive(pbar + 8 * (p.ring + sl));
#pragma unroll
          for (int g = 0; g < G; ++g) sh[(2 + g) * GT] = rh[g];
          o_rh.template put<G>(out, rh, e, N - n0, units, p.wide, lane, row, ul);
        } else if (S == 3 && stage == 1) {
          // ---- stage B (LSTM): gates and the new cell state, its statistics
          const uint8_t* in = inputs.wait(io);
          float pre[4], v[4];
#pragma unroll
          for (int g = 0; g < 4; ++g) pre[g] = piece_value<T>(in, 0, g, row, ul, p.wide) + cst[g % G * 16];
          const float m = piece_value<T>(in, 1, 0, row, ul, p.wide);
          float mean1, inv1;
          collect(G, rt, mean1, inv1, 72);
          if (stop) break;
#pragma unroll
          for (int g = 0; g < 4; ++g)
            pre[g] = (sh[(2 + g) * GT] - mean1) * inv1 * cst[(2 * G + g % G) * 16] + pre[g];
          v[0] = ln_sigmoid<SPLIT>(pre[0]); v[1] = ln_tanh<SPLIT>(pre[1]);
          v[2] = ln_sigmoid<SPLIT>(pre[2]); v[3] = ln_sigmoid<SPLIT>(pre[3]);
          float c_new[1] = {v[2] * sh[GT] + v[0] * v[1]};
          publish(1, t, ch, c_new, rt);
          if (stop) break;
          look_ahead(k, i);
          // ---- off the chain
          sh[GT] = c_new[0];
          sh[2 * GT] = v[3];
          sh[3 * GT] = m;
          inputs.fetch(p.T, N, p.wide, lane, tile0, ch_n, grp);
          if (p.training) o_v.template put<4>(out, v, e, N - n0, units, p.wide, lane, row, ul);
          if (hs == 0 && quad == 0 && ul == 0 && n0 + row < N) {
            T* cc = static_cast<T*>(p.cache_Rh) + ((size_t)e + row) * 2;
            st(cc, mean1);
            st(cc + 1, inv1);
          }
        } else {
          // ---- last stage: the new state
          float wv[3] = {0.f, 0.f, 0.f}, m = 0.f;
          if constexpr (G == 4) {
            m = sh[3 * GT];
          } else {
            const uint8_t* in = inputs.wait(io);
#pragma unroll
            for (int g = 0; g < 3; ++g) wv[g] = piece_value<T>(in, 0, g, row, ul, p.wide) + cst[g * 16];
            m = piece_value<T>(in, 1, 0, row, ul, p.wide);
          }
          float mean, inv;
          collect(G == 4 ? 1 : G, rt, mean, inv, 73);
          if (stop) break;
          const float hp = sh[0];
          float h_new, c_norm = 0.f, v[4] = {0.f, 0.f, 0.f, 0.f};
          if constexpr (G == 4) {
            c_norm = (sh[GT] - mean) * inv * cst[3 * G * 16] + cst[(3 * G + 1) * 16];
            h_new = sh[2 * GT] * ln_tanh<SPLIT>(c_norm);
          } else {
            float rn[3];
#pragma unroll
            for (int g = 0; g < 3; ++g)
              rn[g] = (sh[(2 + g) * GT] - mean) * inv * cst[(2 * G + g) * 16] + cst[(G + g) * 16];
            v[0] = ln_sigmoid<SPLIT>(wv[0] + rn[0]);
            v[1] = ln_sigmoid<SPLIT>(wv[1] + rn[1]);
            v[3] = rn[2];
            v[2] = ln_tanh<SPLIT>(wv[2] + v[1] * v[3]);
            h_new = v[0] * hp + (1.0f - v[0]) * v[2];
          }
          if (p.has_zoneout)
            h_new = p.training ? zoneout<true>(h_new, hp, p.zoneout_prob, m) : zoneout<false>(h_new, hp, p.zoneout_prob, m);
          h_new = uok ? round_to_storage<T>(h_new) : 0.f;
          if (t + 1 < p.T && n0 + row < N)
            gl_publish(xdst + ((size_t)((t + 1) & 1) * tiles + tile) * xtile, hword_encode<SPLIT>(h_new, stat_tag(t + 1)));
          __syncwarp();
          if (lane == 0) mb_arrive(obar + 8 * ch);
          look_ahead(k, i);
          // ---- off the chain
          sh[0] = h_new;
          if constexpr (G == 4) {
            const float o[3] = {h_new, sh[GT], c_norm};
            o_state.template put<3>(out, o, e, N - n0, units, p.wide, lane, row, ul);
          } else {
            inputs.fetch(p.T, N, p.wide, lane, tile0, ch_n, grp);
            const float o[1] = {h_new};
            o_state.template put<1>(out, o, e, N - n0, units, p.wide, lane, row, ul);
            if (p.training) o_v.template put<4>(out, v, e, N - n0, units, p.wide, lane, row, ul);
          }
          if (hs == 0 && quad == 0 && ul == 0 && n0 + row < N) {
            T* cc = static_cast<T*>(G == 4 ? p.cache_c : p.cache_Rh) + ((size_t)e + row) * 2;
            st(cc, mean);
            st(cc + 1, inv);
          }
        }
      }
  }
}

// ---------------------------------------------------------------------------------------
// Exchange words: [2][row tiles][destination CTA][source CTA][4 quads][32], as gl_bwd_kernel.
template <int G, int TPW, int SPLIT, typename T>
__global__ void __launch_bounds__(GL_THREADS, 1) lg_bwd_kernel(const __grid_constant__ LnGridBwd p) {
  constexpr int NMT = 4, KSB = G, GT = 128;  // k-step kk: the sixteen units' gate kk
  constexpr int NS = TPW <= 4 ? 1 : 2;
  using Io = LnIo<T, 4>;
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t* gsm = smem;                                                    // [ring][KSB][512]
  uint4* planes = reinterpret_cast<uint4*>(gsm + GL_GRING * KSB * 512);   // [warp][what is not in registers][lane]
  float* rowf = reinterpret_cast<float*>(planes + GL_WARPS * frag_rest<SPLIT, TPW>() * KSB * 32);  // [ring][8], takes the rows' scale out
  float* consts = rowf + GL_GRING * 8;                                    // [G + 1][16]
  float4* meet = reinterpret_cast<float4*>(consts + (G + 1) * 16);        // [2 groups][2][quad][8]
  float2* found = reinterpret_cast<float2*>(meet + 2 * 2 * NMT * 8);      // [2 groups][2][8] row sums
  float* stash = reinterpret_cast<float*>(found + 2 * 2 * 8);             // [CH][LG_BWD_STASH][GT]
  uint64_t* barp = reinterpret_cast<uint64_t*>(stash + p.CH * LG_BWD_STASH * GT);  // full[ring], empty[ring]
  const uint32_t gbar = smem_u32(barp);
  uint8_t* io_base = reinterpret_cast<uint8_t*>(barp + 2 * GL_GRING);
  __shared__ int s_abort_;
  volatile int* s_abort = &s_abort_;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, q = lane & 3;
  const int nHS = p.CTAS, hs = blockIdx.x % nHS, rg = blockIdx.x / nHS;
  const int H = p.H, N = p.N, u0 = hs * 16, tile0 = rg * p.CH, tiles = (N + 7) >> 3;
  const int ch_n = min(p.CH, tiles - tile0);
  if (tid == 0) {
    *s_abort = 0;
    for (int i = 0; i < GL_GRING; ++i) {
      mb_init(gbar + 8 * i, NMT);
      mb_init(gbar + 8 * (GL_GRING + i), GL_WARPS);
    }
  }
  for (int i = tid; i < (G + 1) * 16; i += GL_THREADS) {
    const int g = i / 16, unit = u0 + (i & 15);
    const void* src = g < G ? p.gamma_Rh : p.gamma_h;
    consts[i] = (src && unit < H) ? ld(static_cast<const T*>(src) + (g < G ? g : 0) * H + unit) : 0.f;
  }
  for (int i = tid; i < GL_GRING * KSB * 512 / 16; i += GL_THREADS)
    reinterpret_cast<uint4*>(gsm)[i] = make_uint4(0u, 0u, 0u, 0u);
  for (int i = tid; i < GL_WARPS * Io::WARP / 16; i += GL_THREADS)
    reinterpret_cast<uint4*>(io_base)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const size_t line = (size_t)NMT * 32;
  RingPos<GL_GRING> gp;

  if (w < GL_WARPS) {
    // ------------------------------------------------------------------ product warps (as gl_bwd_kernel)
    if (TPW <= 4) reg_product<TPW>();
    const int rot = hs % p.K16;
    constexpr int KEEP = LgRegs<TPW>::KEEP, REST = frag_rest<SPLIT, TPW>();  // tiles
    uint32_t wf[KEEP][KSB][4];
    uint4* rest = planes + w * REST * KSB * 32 + lane;
    float wscale[TPW];
    uint32_t doff[TPW];
#pragma unroll
    for (int i = 0; i < TPW; ++i) {
      const int Lt = w + GL_WARPS * i;
      const bool live = Lt < p.K16;
      const int tile = Lt + rot < p.K16 ? Lt + rot : Lt + rot - p.K16;
      const int Q = tile * 4 + (gq >> 1), d = Q / NMT, qw = Q - d * NMT;
      doff[i] = live && d < nHS ? (uint32_t)(((d * nHS + hs) * NMT + qw) * 32 + ((gq & 1) * 4 + q) * 4) : ~0u;
      float x[KSB][2][4];
#pragma unroll
      for (int kk = 0; kk < KSB; ++kk) {
        const int j = Q * 4 + (gq & 1), k = u0 + 4 * q;
        const T* R = static_cast<const T*>(p.R);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const bool ok = live && j + 2 * hf < H && k + e < H;
            const long long col = (long long)kk * H + k + e;
            x[kk][hf][e] = ok ? ld(p.r_transposed ? R + col * H + j + 2 * hf : R + (long long)(j + 2 * hf) * G * H + col) : 0.f;
          }
      }
      if (SPLIT == 2 || i < KEEP) {
        wscale[i] = scaled_fragments<SPLIT, KSB, KSB>(x, wf[i % KEEP], rest + i * KSB * 32);
      } else {
        uint32_t f[KSB][4];
        wscale[i] = scaled_fragments<SPLIT, KSB, KSB>(x, f, nullptr);
#pragma unroll
        for (int kk = 0; kk < KSB; ++kk) rest[((i - KEEP) * KSB + kk) * 32] = make_uint4(f[kk][0], f[kk][1], f[kk][2], f[kk][3]);
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
        const float2 rf = SPLIT == 2 ? *reinterpret_cast<const float2*>(rowf + gp.slot * 8 + 2 * q) : make_float2(1.f, 1.f);
        __syncwarp();
        if (lane == 0) mb_arrive(gbar + 8 * (GL_GRING + gp.slot));  // the operand is in registers
        uint32_t* dst = p.exch + ((size_t)(ti & 1) * tiles + tile) * nHS * nHS * line;
        const bool send = tile * 8 + 2 * q < N;
#pragma unroll
        for (int i0 = 0; i0 < TPW; i0 += 4) {
          float acc[4][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
          if constexpr (SPLIT == 2) {
#pragma unroll
            for (int kk = 0; kk < KSB; ++kk) {
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (i0 + i < TPW) mma_f16(acc[i], wf[(i0 + i) % KEEP][kk], y[kk].z, y[kk].w);
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (i0 + i < TPW) {
                  const uint4 a = rest[((i0 + i) % TPW * KSB + kk) * 32];
                  mma_f16(acc[i], a, y[kk].z, y[kk].w);
                  mma_f16(acc[i], a, y[kk].x, y[kk].y);
                }
            }
#pragma unroll
            for (int kk = 0; kk < KSB; ++kk)
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (i0 + i < TPW) mma_f16(acc[i], wf[(i0 + i) % KEEP][kk], y[kk].x, y[kk].y);
          } else {
#pragma unroll
            for (int kk = 0; kk < KSB; ++kk)
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (i0 + i < TPW) {
                  if (i0 + i < KEEP) {
                    mma_bf16(acc[i], wf[(i0 + i) % KEEP][kk], y[kk].x, y[kk].y);
                  } else {
                    const uint4 a = rest[((i0 + i - KEEP) * KSB + kk) * 32];
                    const uint32_t af[4] = {a.x, a.y, a.z, a.w};
                    mma_bf16(acc[i], af, y[kk].x, y[kk].y);
                  }
                }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (i0 + i < TPW && send && doff[(i0 + i) % TPW] != ~0u) {
              float v[4] = {acc[i][0], acc[i][1], acc[i][2], acc[i][3]};
              if (SPLIT == 2) {
                const float f = wscale[(i0 + i) % TPW];
                v[0] = v[0] * f * rf.x; v[1] = v[1] * f * rf.y; v[2] = v[2] * f * rf.x; v[3] = v[3] * f * rf.y;
              }
              gl_publish4(dst + doff[(i0 + i) % TPW], fword_encode(v[0], tag), fword_encode(v[1], tag),
                          fword_encode(v[2], tag), fword_encode(v[3], tag));
            }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ finishing warps: quad f & 3 of the
    // chains grp, grp + 2, ...; lanes as in the cluster kernels
    if (TPW <= 4) reg_finish<TPW>();
    const int f = w - GL_WARPS, grp = f >> 2, quad = f & 3, gt = quad * 32 + lane;
    const int sub = lane >> 3, c8 = lane & 7;
    const int row = 2 * (c8 & 3) + (sub & 1), ul = (c8 >> 2) + 2 * (sub >> 1);
    const int uq = u0 + 4 * quad, unit = uq + ul, units = max(0, min(4, H - uq));
    const bool uok = unit < H, second = (c8 & 4) != 0;
    const long long NH = (long long)N * H;
    const float* cst = consts + quad * 4 + ul;
    const float inv_H = 1.0f / (float)H, inv_GH = 1.0f / (float)(G * H);
    const int NPS = (nHS + 3) / 4, j0 = sub * NPS, nj = max(0, min(NPS, nHS - j0));  // sources of a lane's gather
    for (int ch = grp; ch < ch_n; ch += 2) {
      const int n = (tile0 + ch) * 8 + row;
      const bool ok = n < N && uok;
      const long long o = (long long)n * H + unit;
      float* sh = stash + (size_t)ch * LG_BWD_STASH * GT + gt;
      sh[0] = ok ? p.dh_carry[o] : 0.f;
      sh[GT] = (G == 4 && ok) ? p.dc_carry[o] : 0.f;
      sh[2 * GT] = (G == 4 && ok) ? ld(static_cast<const T*>(p.c) + (long long)p.T * NH + o) : 0.f;
    }
    // (bias gradients in two levels, sixteen steps at a time: one long sum loses a tenth more)
    float acc_b[4] = {0.f, 0.f, 0.f, 0.f}, sum_b[4] = {0.f, 0.f, 0.f, 0.f}, acc_g1[G], acc_gh = 0.f, acc_bh = 0.f;
#pragma unroll
    for (int g = 0; g < G; ++g) acc_g1[g] = 0.f;
    bool alive = true, stop = false;
    int turn = 0, fturn = 0;
    const uint32_t* gsrc0 = p.exch + ((size_t)hs * nHS + j0) * line + quad * 32 + c8 * 4;
    const size_t tile_words = (size_t)nHS * nHS * line;
    auto gather = [&](int ch, int s, float& dh_c) {  // as gl_bwd_kernel
      uint4 y[8];
      const uint32_t want = (((uint32_t)s >> 1) & 1u) ^ 1u;
      const bool need = (tile0 + ch) * 8 + 2 * (c8 & 3) < N;
      float s4[4] = {0.f, 0.f, 0.f, 0.f};
      for (int b = 0; b < NPS && alive; b += 8) {
        const uint32_t* src = gsrc0 + ((size_t)(s & 1) * tiles + tile0 + ch) * tile_words + (size_t)b * line;
        long long t0 = 0;
        unsigned int spins = 0;
        for (;;) {
          uint32_t bad = 0;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            y[k] = ld_relaxed_u32x4_if(need && b + k < nj, src + (size_t)k * line, want);
#pragma unroll
          for (int k = 0; k < 8; ++k) bad |= stale4(y[k], want);
          if (__all_sync(0xffffffffu, (bad & 1u) == 0)) break;
          if (__any_sync(0xffffffffu, !may_spin(spins, t0, p.sync, s_abort, 66))) { alive = false; break; }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          s4[0] += fword_value(y[k].x); s4[1] += fword_value(y[k].y);
          s4[2] += fword_value(y[k].z); s4[3] += fword_value(y[k].w);
        }
      }
      dh_c += gather_reduce(s4, sub);
    };
    // Sums of a row's pair (x, y) over this CTA, on their way; with them the row's largest a and b, which
    // stay here.  One group barrier.
    auto publish = [&](int stat, int ti, int ch, float x, float y, float& a, float& b, uint32_t tag) {
      x += __shfl_xor_sync(0xffffffffu, x, 4);
      y += __shfl_xor_sync(0xffffffffu, y, 4);
      x += __shfl_xor_sync(0xffffffffu, x, 16);
      y += __shfl_xor_sync(0xffffffffu, y, 16);
      if (stat == 0 && SPLIT == 2) {
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 4));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, 4));
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 16));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, 16));
      }
      float4* at = meet + (grp * 2 + turn) * NMT * 8;
      turn ^= 1;
      if (ul == 0) at[quad * 8 + row] = make_float4(x, y, a, b);
      stop = group_barrier_or(grp, !alive);
      if (stop) return;
      if (stat == 0 && SPLIT == 2) {
#pragma unroll
        for (int k = 0; k < NMT; ++k) {
          const float4 v = at[k * 8 + row];
          a = fmaxf(a, v.z);
          b = fmaxf(b, v.w);
        }
      }
      if (quad == ((ch >> 1) & 3) && lane < 8) {
        float sx = 0.f, sy = 0.f;
#pragma unroll
        for (int k = 0; k < NMT; ++k) {
          const float4 v = at[k * 8 + lane];
          sx += v.x;
          sy += v.y;
        }
        publish_u32x2(p.sbuf + stat_at(stat, ti & 1, tiles, tile0 + ch, nHS) + hs * 16 + lane * 2,
                      fword_encode(sx, tag), fword_encode(sy, tag));
      }
    };
    StatWords<NS> sw;
    auto look = [&](int stat, int ti, int ch, uint32_t tag) {
      sw.src = p.sbuf + stat_at(stat, ti & 1, tiles, tile0 + ch, nHS) + lane * 16 + quad * 4;
      sw.load(nHS, lane, tag);
    };
    auto collect = [&](uint32_t tag, float& x, float& y, int code) {
      if (!sw.wait(nHS, lane, tag, p.sync, s_abort, code)) alive = false;
      float4 s = sw.value(0);
#pragma unroll
      for (int k = 1; k < NS; ++k) {
        const float4 v = sw.value(k);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
      const float2 v = make_float2(pair_sum(s.x, s.z, lane), pair_sum(s.y, s.w, lane));
      float2* at = found + (grp * 2 + fturn) * 8;
      fturn ^= 1;
      if ((lane & 15) == 0) at[quad * 2 + (lane >> 4)] = v;
      stop = group_barrier_or(grp, !alive);
      x = at[row].x;
      y = at[row].y;
    };
    // blocks: gates; h.R; dh_new, mask, c or h before, dc_new; LN(c), statistics of h.R, of c
    uint8_t* io = io_base + f * Io::WARP;
    uint8_t* out = io + IO_RING * Io::SLOT;
    LnInputs<T, 4, true> inputs;
    LnOutput<T> o_rh, o_v, o_q;  // d(h.R); LSTM gate gradients / GRU dp; GRU dq
    inputs.init(io, lane, p.T, grp, units);
    {
      const int a = lane >> 3;
      o_rh.init(static_cast<T*>(p.act_Rh) + (long long)a * H, 0, uq, G * H, a < G ? units : 0, lane);
      o_v.init(static_cast<T*>(G == 4 ? p.v : p.dp) + (long long)a * H, 0, uq, G * H, a < G ? units : 0, lane);
      o_q.init(G == 4 ? nullptr : static_cast<T*>(p.dq) + (long long)a * H, 0, uq, G * H, a < G ? units : 0, lane);
      inputs.array(0, static_cast<const T*>(p.v) + (long long)a * H, uq, 4 * H, 0, lane);
      inputs.array(1, a < G ? static_cast<const T*>(p.act_Rh) + (long long)a * H : nullptr, uq, G * H, 0, lane);
      inputs.array(2, a == 0 ? p.dh_new : a == 1 ? (p.has_zoneout ? p.mask : nullptr) : a == 2 ? (G == 4 ? p.c : p.h) : p.dc_new,
                   uq, H, (a == 0 || a == 3) ? N : 0, lane);
      inputs.array(3, (G == 4 && a == 0) ? p.act_c_norm : nullptr, uq, H, 0, lane);
      const void* pairs = a == 1 ? p.cache_Rh : (a == 2 && G == 4) ? p.cache_c : nullptr;
      if (pairs) inputs.pair = static_cast<const char*>(pairs) + (lane & 7) * 2 * sizeof(T);
      inputs.pairs = p.pairs;
    }
    if (grp < ch_n) {
#pragma unroll
      for (int i = 0; i < IO_RING - 1; ++i) inputs.fetch(p.T, N, p.wide, lane, tile0, ch_n, grp);
    }
    // stash: 0 dh, 1 dc, 2 c carried; 3.. gate gradients (LSTM before stage B: gates i, g, f and d_o);
    // 7.. h.R - mean; 11 its 1/sigma; 12 dc arriving, 13 c before, 14 c - mean, 15 its 1/sigma,
    // 16 gamma_h d(LN c); 17, 18 bounds of gamma d(gates) and of h.R - mean
    float* const sh0 = stash + gt;
    constexpr int S = G == 4 ? 3 : 2;  // stages, in the order of lg_fwd_kernel
    const int nc = (ch_n - grp + 1) / 2;
    auto stat_tag = [](int ti) { return (((uint32_t)ti >> 1) & 1u) ^ 1u; };
    bool looked = false;
    auto look_ahead = [&](int k, int i) {
      if (++i == nc) { i = 0; ++k; }
      const int s = k - min(i, S - 1), ti = s / S, stage = s - ti * S;
      looked = s >= 0 && s < S * p.T && stage > 0;
      if (looked) look(S - 1 - stage, ti, grp + 2 * i, stat_tag(ti));
    };
    for (int k = 0; k < S * p.T + min(nc, S) - 1 && !stop; ++k)
      for (int i = 0; i < nc && !stop; ++i) {
        const int s = k - min(i, S - 1), ti = s / S, stage = s - ti * S;
        if (s < 0 || s >= S * p.T) continue;
        const int ch = grp + 2 * i, n0 = (tile0 + ch) * 8, t = p.T - 1 - ti;
        const uint32_t tag = stat_tag(ti), e = (uint32_t)(t * N + n0);
        const bool ok = n0 + row < N && uok;
        float* sh = sh0 + (size_t)ch * LG_BWD_STASH * GT;
        if (stage > 0 && !looked) look(S - 1 - stage, ti, ch, tag);
        if (stage == 0 && i == 0 && (ti & 15) == 15) {
#pragma unroll
          for (int g = 0; g < 4; ++g) { sum_b[g] += acc_b[g]; acc_b[g] = 0.f; }
        }
        auto norm_sums = [&](const float (&dg)[G], const float (&cx)[G], float inv1) {
          float s1 = 0.f, s2 = 0.f, a = 0.f, b = 0.f;
#pragma unroll
          for (int g = 0; g < G; ++g) {
            const float db = cst[g * 16] * dg[g];
            if (ok) {
              s1 += cx[g] * db;
              s2 += db;
              a = fmaxf(a, fabsf(db));
              b = fmaxf(b, fabsf(cx[g]));
              acc_g1[g] += cx[g] * inv1 * dg[g];
            }
          }
          publish(0, ti, ch, s1, s2, a, b, tag);
          sh[17 * GT] = a;
          sh[18 * GT] = b;
        };
        if (stage == 0) {
          // ---- stage A
          const uint8_t* in = inputs.wait(io);
          const float mean1 = piece_value<T>(in, 3, 1, row, 0, p.wide), inv1 = piece_value<T>(in, 3, 1, row, 1, p.wide);
          const float mean3 = piece_value<T>(in, 3, 2, row, 0, p.wide), inv3 = piece_value<T>(in, 3, 2, row, 1, p.wide);
          float gv[4], cx[G];
#pragma unroll
          for (int g = 0; g < 4; ++g) gv[g] = piece_value<T>(in, 0, g, row, ul, p.wide);
#pragma unroll
          for (int g = 0; g < G; ++g) {
            cx[g] = piece_value<T>(in, 1, g, row, ul, p.wide) - mean1;
            sh[(7 + g) * GT] = cx[g];
          }
          sh[11 * GT] = inv1;
          const float dhn = piece_value<T>(in, 2, 0, row, ul, p.wide), m = piece_value<T>(in, 2, 1, row, ul, p.wide);
          const float prev = piece_value<T>(in, 2, 2, row, ul, p.wide), dcn = piece_value<T>(in, 2, 3, row, ul, p.wide);
          const float cn = piece_value<T>(in, 3, 0, row, ul, p.wide);
          float dh_c = sh[0];
          if (ti > 0) gather(ch, ti - 1, dh_c);
          float dh_total = dhn + dh_c, keep = 0.f;
          if (p.has_zoneout) {
            keep = (1.0f - m) * dh_total;
            dh_total = m * dh_total;
          }
          if constexpr (G == 4) {
            const float cx3 = ok ? sh[2 * GT] - mean3 : 0.f;
            const float c_tanh = ln_tanh<SPLIT>(cn);
            const float d_norm = ok ? d_tanh(c_tanh) * (gv[3] * dh_total) : 0.f;
            const float db3 = cst[G * 16] * d_norm;
            if (ok) {
              acc_gh += cx3 * inv3 * d_norm;
              acc_bh += d_norm;
            }
            float a = 0.f, b = 0.f;
            publish(1, ti, ch, ok ? cx3 * db3 : 0.f, ok ? db3 : 0.f, a, b, tag);
            if (stop) break;
            look_ahead(k, i);
            sh[0] = ok ? keep : 0.f;
            sh[3 * GT] = gv[0]; sh[4 * GT] = gv[1]; sh[5 * GT] = gv[2];
            sh[6 * GT] = d_sigmoid(gv[3]) * (c_tanh * dh_total);
            sh[12 * GT] = p.dc_new ? dcn : 0.f;
            sh[13 * GT] = prev;
            sh[14 * GT] = cx3; sh[15 * GT] = inv3; sh[16 * GT] = db3;
          } else {
            const float z = gv[0], r = gv[1], gg = gv[2], qg = gv[3];
            const float dp_g = ok ? d_tanh(gg) * ((1.0f - z) * dh_total) : 0.f;
            float dg[G];
            dg[0] = ok ? d_sigmoid(z) * ((prev - gg) * dh_total) : 0.f;
            dg[1] = ok ? d_sigmoid(r) * (dp_g * qg) : 0.f;
            dg[2] = ok ? dp_g * r : 0.f;
            norm_sums(dg, cx, inv1);
            if (stop) break;
            look_ahead(k, i);
            sh[0] = ok ? keep + z * dh_total : 0.f;
#pragma unroll
            for (int g = 0; g < G; ++g) sh[(3 + g) * GT] = dg[g];
            const float op[3] = {dg[0], dg[1], dp_g}, oq[3] = {dg[0], dg[1], dg[2]};
            o_v.template put<3>(out, op, e, N - n0, units, p.wide, lane, row, ul);
            o_q.template put<3>(out, oq, e, N - n0, units, p.wide, lane, row, ul);
            acc_b[0] += dg[0]; acc_b[1] += dg[1]; acc_b[2] += dp_g; acc_b[3] += dg[2];
          }
          inputs.fetch(p.T, N, p.wide, lane, tile0, ch_n, grp);
        } else if (S == 3 && stage == 1) {
          // ---- stage B (LSTM): the cell state's LayerNorm, the gate gradients
          float S1, S2;
          collect(tag, S1, S2, 70);
          if (stop) break;
          const float r = sh[15 * GT];
          const float dsigma = -0.5f * S1 * r * r * r, dmu = -S2 * r;
          const float dcl = 2.0f * sh[14 * GT] * dsigma * inv_H + r * sh[16 * GT] + dmu * inv_H;
          const float ig = sh[3 * GT], gg = sh[4 * GT], fg = sh[5 * GT], cprev = sh[13 * GT];
          const float dc_total = ok ? sh[12 * GT] + sh[GT] + dcl : 0.f;
          float dg[G], cx[G];
          dg[0] = ok ? d_sigmoid(ig) * (gg * dc_total) : 0.f;
          dg[1] = ok ? d_tanh(gg) * (ig * dc_total) : 0.f;
          dg[2] = ok ? d_sigmoid(fg) * (cprev * dc_total) : 0.f;
          dg[G - 1] = ok ? sh[6 * GT] : 0.f;
#pragma unroll
          for (int g = 0; g < G; ++g) cx[g] = sh[(7 + g) * GT];
          norm_sums(dg, cx, sh[11 * GT]);
          if (stop) break;
          look_ahead(k, i);
          sh[GT] = ok ? fg * dc_total : 0.f;
          sh[2 * GT] = cprev;
#pragma unroll
          for (int g = 0; g < G; ++g) {
            sh[(3 + g) * GT] = dg[g];
            acc_b[g] += dg[g];
          }
          o_v.template put<G>(out, dg, e, N - n0, units, p.wide, lane, row, ul);
        } else {
          // ---- stage C: d(h.R), the operand of the product
          float S1, S2;
          collect(tag, S1, S2, 71);
          if (stop) break;
          const float r = sh[11 * GT];
          const float dsigma = -0.5f * S1 * r * r * r, dmu = -S2 * r;
          float x[G];
#pragma unroll
          for (int g = 0; g < G; ++g)
            x[g] = ok ? 2.0f * sh[(7 + g) * GT] * dsigma * inv_GH + r * (cst[g * 16] * sh[(3 + g) * GT]) + dmu * inv_GH : 0.f;
          const int n = ti * ch_n + ch, sl = n & (GL_GRING - 1);
          static_assert((GL_GRING & (GL_GRING - 1)) == 0, "ring position");
          if (!mb_wait_warp(gbar + 8 * (GL_GRING + sl), ((n / GL_GRING) & 1) ^ 1, p.sync, s_abort, 67)) alive = false;
          uint8_t* gb = gsm + sl * KSB * 512;
          float scale = 1.f;
          if (SPLIT == 2) {
            const float bound = 2.0f * sh[18 * GT] * fabsf(dsigma) * inv_GH + r * sh[17 * GT] + fabsf(dmu) * inv_GH;
            const int sc = f16_shift_of(bound);
            scale = pow2(sc);
            if (quad == 0 && ul == 0) rowf[sl * 8 + row] = pow2(-sc);
          }
#pragma unroll
          for (int g = 0; g < G; ++g) {
            uint32_t own;
            if (SPLIT == 2) {
              const float v = x[g] * scale;
              const __half hi = __float2half_rn(v);
              const __half2 both = __halves2half2(hi, __float2half_rn(v - __half2float(hi)));
              own = *reinterpret_cast<const uint32_t*>(&both);
            } else {
              own = pack_bf16(x[g], 0.f);
            }
            const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 4);
            *reinterpret_cast<uint32_t*>(gb + g * 512 + quad_piece(quad, row) + (second ? 8 : 0) + (sub >> 1) * 4) =
                second ? __byte_perm(other, own, 0x7632) : __byte_perm(own, other, 0x5410);
          }
          __syncwarp();
          if (lane == 0) mb_arrive(gbar + 8 * sl);
          look_ahead(k, i);
          o_rh.template put<G>(out, x, e, N - n0, units, p.wide, lane, row, ul);
        }
      }
    // ---- what is left of dh: the recurrent part of step 0, then the carries go out
    for (int ch = grp; ch < ch_n && alive && !stop; ch += 2) {
      const int n = (tile0 + ch) * 8 + row;
      float* sh = sh0 + (size_t)ch * LG_BWD_STASH * GT;
      float dh_c = sh[0];
      gather(ch, p.T - 1, dh_c);
      if (alive && n < N && uok) {
        p.dh_carry[(long long)n * H + unit] = dh_c;
        if (G == 4) p.dc_carry[(long long)n * H + unit] = sh[GT];
      }
    }
    // ---- parameter gradients of this group's chains: over the eight rows
    auto rows = [&](float v) {
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      return v + __shfl_xor_sync(0xffffffffu, v, 8);
    };
    const bool first = row == 0 && uok;
    const size_t pr = (size_t)rg * 2 + grp;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float s = rows(sum_b[g] + acc_b[g]);
      if (first) p.db_part[(pr * 4 + g) * H + unit] = s;
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float s = rows(acc_g1[g]);
      if (first) p.dgRh_part[(pr * G + g) * H + unit] = s;
    }
    if (G == 4) {
      const float s = rows(acc_gh), b = rows(acc_bh);
      if (first) {
        p.dgh_part[pr * H + unit] = s;
        p.dbh_part[pr * H + unit] = b;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// Host side (the tiling is chosen in recurrent_host.cu).
template <int G, int KSW, int SPLIT, typename T>
int lg_fwd_go(LnGridFwd& p, int nRG, cudaStream_t s) {
  static std::atomic<int> set[kChainMaxDevices];
  const size_t slot = (size_t)GL_WARPS * 4 * 512 + 16;
  const size_t rest = (size_t)GL_WARPS * 4 * frag_rest<SPLIT, KSW>() * 512 + (size_t)p.CH * LG_FWD_STASH * 512 +
                      (3 * G + 2) * 64 + 2 * 2 * (4 + 1) * 8 * 8 + (size_t)((p.CH + 1) & ~1) * 8 + (size_t)GL_WARPS * LnIo<T, 2>::WARP;
  p.ring = min(p.CH, (int)(((size_t)kGlMaxSmem - rest) / slot));
  p.throttle = p.ring < p.CH;  // (a group's four warps have read their partials before its statistics leave)
  return gl_launch(lg_fwd_kernel<G, KSW, SPLIT, T>, p, p.CTAS * nRG, p.ring * slot + rest, set, s);
}
template <int G, int SPLIT, typename T>
int run_ln_grid_fwd(const LnFwdParams& q, const LnGridGeometry& g, int wide, cudaStream_t s) {
  LnGridFwd p;
  static_cast<LnFwdParams&>(p) = q;
  p.CTAS = p.K16 = g.nHS;
  p.CH = g.CH;
  p.wide = wide;
  const int ksw = ceil_div(p.K16, GL_WARPS);
  if (ksw <= 2) return lg_fwd_go<G, 2, SPLIT, T>(p, g.nRG, s);
  if (ksw <= 3) return lg_fwd_go<G, 3, SPLIT, T>(p, g.nRG, s);
  if (ksw <= 4) return lg_fwd_go<G, 4, SPLIT, T>(p, g.nRG, s);
  if constexpr (SPLIT == 1) return lg_fwd_go<G, 8, SPLIT, T>(p, g.nRG, s);
  return HASTE_B200_ERR_UNSUPPORTED;
}

template <int G, int TPW, int SPLIT, typename T>
int lg_bwd_go(LnGridBwd& p, int nRG, cudaStream_t s) {
  static std::atomic<int> set[kChainMaxDevices];
  const size_t smem = (size_t)GL_GRING * (G * 512 + 32) + (size_t)GL_WARPS * frag_rest<SPLIT, TPW>() * G * 512 +
                      (G + 1) * 64 + 2 * 2 * 4 * 8 * 16 + 2 * 2 * 8 * 8 + (size_t)p.CH * LG_BWD_STASH * 512 +
                      2 * GL_GRING * 8 + (size_t)GL_WARPS * LnIo<T, 4>::WARP;
  return gl_launch(lg_bwd_kernel<G, TPW, SPLIT, T>, p, p.CTAS * nRG, smem, set, s);
}
template <int G, int SPLIT, typename T>
int run_ln_grid_bwd(const LnBwdParams& q, float* db_part, const LnGridGeometry& g, int wide, cudaStream_t s) {
  LnGridBwd p;
  static_cast<LnBwdParams&>(p) = q;
  p.CTAS = p.K16 = g.nHS;
  p.CH = g.CH;
  p.wide = wide;
  p.pairs = ((reinterpret_cast<uintptr_t>(q.cache_Rh) | reinterpret_cast<uintptr_t>(q.cache_c)) & (2 * sizeof(T) - 1)) == 0;
  p.db_part = db_part;
  const int tpw = ceil_div(p.K16, GL_WARPS);
  if (tpw <= 2) return lg_bwd_go<G, 2, SPLIT, T>(p, g.nRG, s);
  if (tpw <= 3) return lg_bwd_go<G, 3, SPLIT, T>(p, g.nRG, s);
  if (tpw <= 4) return lg_bwd_go<G, 4, SPLIT, T>(p, g.nRG, s);
  if constexpr (SPLIT == 1) return lg_bwd_go<G, 8, SPLIT, T>(p, g.nRG, s);
  return HASTE_B200_ERR_UNSUPPORTED;
}

}  // namespace rec
}  // namespace hb
