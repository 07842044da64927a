// Shared parts of the persistent recurrences, sm_100a: tagged exchange words, polling loads, mma.sync
// wrappers, gate functions, the abort protocol and the cooperative launch.
//
// One launch covers all T steps of a layer pass; R stays on chip for the whole pass and nothing is
// launched per time step, where the reference issues a cuBLAS call and a pointwise kernel per step
// (lib/lstm_forward_gpu.cu.cc:210-310, lib/lstm_backward_gpu.cu.cc:246-316,
//  lib/gru_forward_gpu.cu.cc:214-308, lib/gru_backward_gpu.cu.cc:252-320).
//
// fp32 storage: operands are split into bf16 (hi, lo) pairs and three products
// (hi.hi, hi.lo, lo.hi) are accumulated in fp32, which keeps the step product within
// ~1e-5 of fp32 arithmetic.  bf16 storage: one product.
//
// Step-to-step data flow carries its own readiness: everything a CTA hands to another
// CTA is written as 32-bit words that hold the value and a tag that alternates every time
// a buffer is reused.  h_t (forward) travels as a bf16 (hi, lo) pair with the tag in bit 14 of the
// lo half, always zero for a genuine lo, whose magnitude is below 2^-8 of the value; partial dh
// (backward) travels as fp32 with the tag in the lowest mantissa bit.  A consumer simply re-reads
// a word until the tag is the one it expects.  There is no counter, no fence and no grid-wide
// barrier on the critical path, and 32-bit stores cannot tear.
//
// Every wait is bounded: when the limit runs out the warp raises the CTA's and the
// grid's abort flags and the process error word; all CTAs leave their loops and the host
// reports HASTE_B200_ERR_TIMEOUT.
#pragma once

#include "cells.cuh"

namespace hb {
namespace rec {

constexpr int U = 16;          // hidden units per CTA
constexpr int WARPS = 8;
constexpr int THREADS = WARPS * 32;
constexpr long long SPIN_LIMIT_CYCLES = 4000000000LL;

struct Sync {
  int* abort_flag;  // device-global
  int* err;         // process error word (pinned host memory)
};

// ---------------------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo_elem, float hi_elem) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo_elem, hi_elem);  // .x = lower address
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void split_bf16(float x, float& hi, float& lo) {
  hi = __bfloat162float(__float2bfloat16_rn(x));
  lo = x - hi;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  const uint32_t f[4] = {a.x, a.y, a.z, a.w};
  mma_bf16(d, f, b0, b1);
}
// Polling loads: relaxed, gpu scope, so that every poll is served by L2.
__device__ __forceinline__ uint4 ld_relaxed_u32x4(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

// The same under a condition, without a branch; else four times `other`.
__device__ __forceinline__ uint4 ld_relaxed_u32x4_if(bool ok, const uint32_t* p, uint32_t other) {
  uint4 v = make_uint4(other, other, other, other);
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %5, 0;\n\t"
      "@p ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
      : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
      : "l"(p), "r"((uint32_t)ok)
      : "memory");
  return v;
}

__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Publishing stores of the exchange: `volatile` with a memory clobber, so that the compiler
// issues them exactly where they are written - ahead of the bulky activation stores of the same
// stage, never behind them.  .cg: the word goes to L2, where the consumers poll.
__device__ __forceinline__ void publish_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.global.cg.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void publish_u32x2(uint32_t* p, uint32_t a, uint32_t b) {
  asm volatile("st.global.cg.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}

// Exchange word: bits 0-15 hi (bf16), bits 16-31 lo (bf16) with bit 30 replaced by `tag`.
__device__ __forceinline__ uint32_t xword_encode(float x, uint32_t tag) {
  float hi, lo;
  split_bf16(x, hi, lo);
  if (!(fabsf(lo) < 1.0f)) lo = 0.0f;  // NaN/Inf/huge values travel in hi alone
  return (pack_bf16(hi, lo) & 0xBFFFFFFFu) | (tag << 30);
}
__device__ __forceinline__ float xword_value(uint32_t w) {
  return __uint_as_float(w << 16) + __uint_as_float(w & 0xBFFF0000u);
}

// Tagged fp32 word: the value with its lowest mantissa bit replaced by the tag (22 explicit
// mantissa bits survive).  One logic instruction to encode or decode; used wherever the
// consumer wants the number itself rather than ready-made bf16 planes.
__device__ __forceinline__ uint32_t fword_encode(float x, uint32_t tag) {
  return (__float_as_uint(x) & ~1u) | tag;
}
__device__ __forceinline__ float fword_value(uint32_t w) { return __uint_as_float(w & ~1u); }

// Fast gate functions (ex2.approx based): error ~1e-6 absolute, far inside the parity bar.
__device__ __forceinline__ float sigmoid_fast(float x) {
  return __fdividef(1.0f, 1.0f + __expf(-x));
}
__device__ __forceinline__ float tanh_fast(float x) {
  // 1 - 2/(1+e^{2x}); clamp keeps e^{2x} finite
  const float e = __expf(2.0f * fminf(fmaxf(x, -15.0f), 15.0f));
  return 1.0f - __fdividef(2.0f, 1.0f + e);
}

// Marks the grid as failed; the first reporter also leaves four words of detail.
__device__ __forceinline__ void raise_abort(const Sync& s, int* s_abort, int code, int d0 = 0,
                                            int d1 = 0, int d2 = 0, int d3 = 0) {
  *reinterpret_cast<volatile int*>(s_abort) = 1;
  if (atomicExch(s.abort_flag, 1) == 0) {
    volatile int* e = reinterpret_cast<volatile int*>(s.err);
    e[1] = d0; e[2] = d1; e[3] = d2; e[4] = d3;
    __threadfence_system();
    e[0] = code;
  }
  __threadfence_system();
}

// Whether a recurrence with `half` chains per CTA within an SM budget of up to half of the GPU, two directions
// side by side, is ahead of the whole GPU with `whole` chains for one direction after the other.  Side by side one
// direction's hand-offs are under way while the other computes, until the chains are enough to fill that time
// by themselves.  Both directions of 100 steps, us in turn / side by side, forward and backward:
//   LSTM fp32 H = 1024    16 rows, 2 chains for 2  519 / 461, 1394 / 1136    64 rows, 8 for 4  1483 / 1549, 2897 / 2935
//        H = 640          32 rows, 4 for 2  635 / 680, 1205 / 1197            48 rows, 6 for 2  652 / 976, 1339 / 1616
//   GRU fp32 H = 1024     32 rows, 4 for 2  802 / 775, 1641 / 1378            64 rows, 8 for 4  1524 / 1484, 2186 / 2449
//        H = 640          48 rows, 6 for 2  622 / 867, 1196 / 1618            96 rows, 12 for 4 1186 / 1689, 2021 / 3022
//   LayerNormLSTM fp32 H = 512  64 rows, 4 for 2  1346 / 1117, 2032 / 1866    128 rows, 8 for 4  2032 / 2014, 3141 / 3403
//        H = 400          80 rows, 5 for 2  1310 / 1366, 1985 / 2250          96 rows, 6 for 3  1661 / 1473, 2461 / 2448
//   LayerNormGRU bf16 H = 768   24 rows, 3 for 1  870 / 752, 1272 / 1354      48 rows, 6 for 2  1084 / 1218, 1474 / 1958
inline bool budget_pays(bool bwd, int budget, int half, int whole) {
  if (2 * budget > sm_count()) return true;  // a budget for another reason than a second direction
  return bwd ? half <= 2 * whole && half <= 6 : half <= 2 * whole || half <= 3;
}

}  // namespace rec
}  // namespace hb
