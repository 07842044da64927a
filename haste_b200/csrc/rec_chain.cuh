// Shared parts of the chain recurrences (rec_cluster_kernels.cuh, rec_grid_kernels.cuh): kernel
// parameters, the cell's arithmetic, tagged words, bounded waits and the input / output warps.
//
// A "chain" is eight batch rows: the N dimension of mma.m16n8k16, whose A operand is the
// recurrent matrix in registers.  A gate-stage warp owns a quad of hidden units for the eight rows
// of a chain, one element per lane.  What it reads from the big tensors comes through a ring in
// shared memory that it fills itself with cp.async a few steps ahead - the four gates of a quad
// and eight rows are one 16-byte piece per lane - and its results leave the same way, as 16-byte
// stores.  (Element-wise loads and stores in this place cost a backward step at N=32, H=512 1100
// cycles of store issue and 2000 more until its loads were through, out of 5700.)
#pragma once

#include "recurrent_common.cuh"

namespace hb {
namespace rec {

struct ChainParams {
  int T, N, H;
  int CTAS;      // CTAs that share the hidden dimension of one row group
  int CH;        // chains per CTA
  int K16;       // 16-unit tiles of the hidden dimension, CTAS * units per CTA / 16 rounded up
  int ring;      // grid forward: partial tiles in flight
  int throttle;  // grid forward: a slot may come round before it is known to be free
  int training, has_zoneout, r_transposed;
  int zero_init; // backward: dh and dc start at zero instead of what they hold
  int wide;      // rows and pointers allow whole-quad accesses (H a multiple of 4)
  float zoneout_prob;
  const void *R, *b, *b2;
  const void* gin;    // forward: x.W [T,N,G*H]; backward: gate cache [T,N,4H]
  const void* mask;   // [T,N,H] or null
  void *h, *c;        // [T+1,N,H]; forward: slot 0 in, the rest out; backward: in
  void* gout;         // forward: gate cache out [T,N,4H] or null
  const void *dh_new, *dc_new;  // backward [T+1,N,H]; dc_new may be null
  void *dv;           // LSTM backward: gate gradients [T,N,4H] (may alias gin)
  void *dp, *dq;      // GRU backward [T,N,3H]
  __nv_bfloat16 *gpl, *gpl2;  // fp32 storage, optional: bf16 planes of dv / dp and dq
  long long gpl_stride;
  void *dh, *dc;      // backward [N,H] in/out
  float* db_part;     // backward [row groups][4H]
  uint32_t* xbuf;     // grid: exchange words, zeroed before launch
  Sync sync;          // cluster kernels use the error word only
};

// ---- gate functions: ex2.approx and rcp.approx (relative error about 2^-22 each)
__device__ __forceinline__ float ex2_(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float chain_sigmoid(float x) { return rcp_(1.0f + ex2_(-1.4426950408889634f * x)); }
__device__ __forceinline__ float chain_tanh(float x) {  // 1 - 2 / (1 + e^2x); e^2x may be inf
  return fmaf(-2.0f, rcp_(1.0f + ex2_(2.8853900817779268f * x)), 1.0f);
}

// The cell: pre-activations of the recurrent product rh and of the input wv, previous state.
template <int G>
__device__ __forceinline__ void cell_fwd(const float (&rh)[4], const float (&wv)[G], const float (&bias)[4],
                                         float hp, float cp, float (&gate)[4], float& h_new, float& c_new) {
  if (G == 4) {
    gate[0] = chain_sigmoid(wv[0] + bias[0] + rh[0]);
    gate[1] = chain_tanh(wv[1] + bias[1] + rh[1]);
    gate[2] = chain_sigmoid(wv[2] + bias[2] + rh[2]);
    gate[3] = chain_sigmoid(wv[G - 1] + bias[3] + rh[3]);
    c_new = gate[2] * cp + gate[0] * gate[1];
    h_new = gate[3] * chain_tanh(c_new);
  } else {  // bias: bx_z + br_z, bx_r + br_r, bx_g, br_g
    gate[0] = chain_sigmoid(wv[0] + bias[0] + rh[0]);
    gate[1] = chain_sigmoid(wv[1] + bias[1] + rh[1]);
    gate[3] = rh[2] + bias[3];
    gate[2] = chain_tanh(wv[2] + bias[2] + gate[1] * gate[3]);
    h_new = gate[0] * hp + (1.0f - gate[0]) * gate[2];
    c_new = 0.f;
  }
}

template <int G, typename T>
__device__ __forceinline__ void load_bias(const ChainParams& p, int unit, float (&bias)[4]) {
  const T *b = reinterpret_cast<const T*>(p.b), *b2 = reinterpret_cast<const T*>(p.b2);
  const int H = p.H;
  bias[0] = bias[1] = bias[2] = bias[3] = 0.f;
  if (unit >= H) return;
  if (G == 4) {
#pragma unroll
    for (int g = 0; g < 4; ++g) bias[g] = ld(b + g * H + unit);
  } else {
    bias[0] = ld(b + unit) + ld(b2 + unit);
    bias[1] = ld(b + H + unit) + ld(b2 + H + unit);
    bias[2] = ld(b + 2 * H + unit);
    bias[3] = ld(b2 + 2 * H + unit);
  }
}

// The cell's gradient: gate values gv, gradients of h and c -> gate gradients dg (LSTM d(i,g,f,o);
// GRU dp_z, dp_r, dp_g, dq_g), carried gradients.  TANH: `cnew` is already tanh(c).
template <int G, bool TANH = false>
__device__ __forceinline__ void cell_bwd(const float (&gv)[4], float prev /* c or h before */, float cnew,
                                         float dh_total, float dcv, bool zo, float m, float& dh_c,
                                         float& dc_c, float (&dg)[4]) {
  float keep = 0.f;
  if (zo) {
    keep = (1.0f - m) * dh_total;
    dh_total = m * dh_total;
  }
  if (G == 4) {
    const float c_tanh = TANH ? cnew : chain_tanh(cnew);
    const float dc_total = dcv + dc_c + d_tanh(c_tanh) * (gv[3] * dh_total);
    dg[0] = d_sigmoid(gv[0]) * (gv[1] * dc_total);
    dg[1] = d_tanh(gv[1]) * (gv[0] * dc_total);
    dg[2] = d_sigmoid(gv[2]) * (prev * dc_total);
    dg[3] = d_sigmoid(gv[3]) * (c_tanh * dh_total);
    dc_c = gv[2] * dc_total;
    dh_c = keep;
  } else {
    const float dp_g = d_tanh(gv[2]) * ((1.0f - gv[0]) * dh_total);
    dg[0] = d_sigmoid(gv[0]) * ((prev - gv[2]) * dh_total);
    dg[1] = d_sigmoid(gv[1]) * (dp_g * gv[3]);
    dg[2] = dp_g;
    dg[3] = dp_g * gv[1];
    dh_c = keep + gv[0] * dh_total;
  }
}

// ---- operand layout --------------------------------------------------------------------
// A k-step is 16 units = four quads; a lane's B fragment is the four words of one (row, quad).
// Byte offset of the 16-byte piece of `row` inside the 128-byte line of quad j (mod 4): rotated
// by 2j so that the eight lanes of a load phase - two rows, four quads - touch all banks once.
__device__ __forceinline__ uint32_t quad_piece(int j, int row) {
  return (uint32_t)(j * 128 + ((row + 2 * j) & 7) * 16);
}
// hi / lo B fragments of one k-step from the four tagged words of a lane
template <int SPLIT>
__device__ __forceinline__ void unpack_words(const uint4& x, uint32_t (&bh)[2], uint32_t (&bl)[2]) {
  bh[0] = __byte_perm(x.x, x.y, 0x5410);
  bh[1] = __byte_perm(x.z, x.w, 0x5410);
  if (SPLIT == 2) {
    bl[0] = __byte_perm(x.x, x.y, 0x7632) & 0xBFFFBFFFu;
    bl[1] = __byte_perm(x.z, x.w, 0x7632) & 0xBFFFBFFFu;
  }
}
// A fragment (hi plane, lo plane) of rows half 0 / 1, four consecutive k each
template <int SPLIT>
__device__ __forceinline__ void pack_weights(const float (&x)[2][4], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
#pragma unroll
  for (int a = 0; a < 4; ++a) {  // fragment register a: rows half a & 1, k half a >> 1
    const float v0 = x[a & 1][(a >> 1) * 2], v1 = x[a & 1][(a >> 1) * 2 + 1];
    if (SPLIT == 2) {
      float h0, l0, h1, l1;
      split_bf16(v0, h0, l0);
      split_bf16(v1, h1, l1);
      hi[a] = pack_bf16(h0, h1);
      lo[a] = pack_bf16(l0, l1);
    } else {
      hi[a] = pack_bf16(v0, v1);
    }
  }
}
// Forward weights: gate columns of `unit` (lane's row pair: gates ga, ga + 2), k .. k+3
template <int G, int SPLIT, typename T>
__device__ __forceinline__ void fwd_weights(const ChainParams& p, int unit, int ga, int k, bool live,
                                            uint32_t (&hi)[4], uint32_t (&lo)[4]) {
  const T* R = reinterpret_cast<const T*>(p.R);
  const int H = p.H;
  float x[2][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool ok = live && unit < H && k + i < H;
    const T* r = R + (long long)(k + i) * G * H + unit;
    x[0][i] = ok ? ld(r + (long long)ga * H) : 0.f;
    x[1][i] = (ok && ga + 2 < G) ? ld(r + (long long)(ga + 2) * H) : 0.f;
  }
  pack_weights<SPLIT>(x, hi, lo);
}
// Backward weights: output units j, j + 2; gate columns (gate, k .. k+3)
template <int G, int SPLIT, typename T>
__device__ __forceinline__ void bwd_weights(const ChainParams& p, int j, int gate, int k, bool live,
                                            uint32_t (&hi)[4], uint32_t (&lo)[4]) {
  const T* R = reinterpret_cast<const T*>(p.R);
  const int H = p.H;
  float x[2][4];
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const bool ok = live && gate < G && j + 2 * hf < H && k + e < H;
      const long long col = (long long)gate * H + k + e;
      x[hf][e] = ok ? ld(p.r_transposed ? R + col * H + j + 2 * hf : R + (long long)(j + 2 * hf) * G * H + col) : 0.f;
    }
  }
  pack_weights<SPLIT>(x, hi, lo);
}
// Even gq holds gates 0 and 2 of rows 2q, 2q+1, its odd partner gates 1 and 3: swap, so that each
// lane has the four gates of one row.
__device__ __forceinline__ void swap_gates(const float (&d)[4], bool odd, float (&rh)[4]) {
  const float r0 = __shfl_xor_sync(0xffffffffu, odd ? d[0] : d[1], 4);
  const float r1 = __shfl_xor_sync(0xffffffffu, odd ? d[2] : d[3], 4);
  rh[0] = odd ? r0 : d[0];
  rh[1] = odd ? d[1] : r0;
  rh[2] = odd ? r1 : d[2];
  rh[3] = odd ? d[3] : r1;
}
// Gate gradients of one (unit, row) -> B operand line of (gate, quad).  Lanes c8 and c8 ^ 4 hold a
// pair of units: the even one writes the pair's hi halves, the odd one the lo halves.
template <int G, int NQ>
__device__ __forceinline__ void store_gate_operand(uint8_t* gb, const float (&dg)[4], int quad, int row,
                                                   int sub, bool second) {
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float hi, lo;
    split_bf16(dg[(G == 3 && g == 2) ? 3 : g], hi, lo);
    const uint32_t own = pack_bf16(hi, lo);
    const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 4);
    const int lq = g * NQ + quad;
    *reinterpret_cast<uint32_t*>(gb + (lq >> 2) * 512 + quad_piece(lq & 3, row) + (second ? 8 : 0) + (sub >> 1) * 4) =
        second ? __byte_perm(other, own, 0x7632) : __byte_perm(own, other, 0x5410);
  }
}
// Sums over the four lane groups of a gather (sub = lane / 8); a lane keeps word `sub`.
__device__ __forceinline__ float gather_reduce(const float (&s4)[4], int sub) {
  const float a0 = __shfl_xor_sync(0xffffffffu, (sub & 2) ? s4[0] : s4[2], 16);
  const float a1 = __shfl_xor_sync(0xffffffffu, (sub & 2) ? s4[1] : s4[3], 16);
  const float b0 = ((sub & 2) ? s4[2] : s4[0]) + a0, b1 = ((sub & 2) ? s4[3] : s4[1]) + a1;
  const float e = __shfl_xor_sync(0xffffffffu, (sub & 1) ? b0 : b1, 8);
  return ((sub & 1) ? b1 : b0) + e;
}
__device__ __forceinline__ uint32_t stale4(const uint4& v, uint32_t want) {
  return (v.x ^ want) | (v.y ^ want) | (v.z ^ want) | (v.w ^ want);
}

// ---- bounded waits ----------------------------------------------------------------------
__device__ __forceinline__ void mb_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mb_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mb_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// While a wait may go on: false once this CTA or the grid has given up, or this wait's limit ran
// out.  (The cluster kernels have no flag of the grid: a CTA that stops publishing lets its peers
// run into their own limits.)  `t0` is set at the first look at the clock.
__device__ __forceinline__ bool may_spin(unsigned int& spins, long long& t0, const Sync& s, volatile int* s_abort,
                                         int code) {
  if ((++spins & 63u) != 0) return true;
  if (*s_abort != 0 || (s.abort_flag && *reinterpret_cast<volatile int*>(s.abort_flag) != 0)) {
    *s_abort = 1;
    return false;
  }
  const long long now = clock64();
  if (spins == 64u) t0 = now;
  if (now - t0 <= SPIN_LIMIT_CYCLES) return true;
  *s_abort = 1;
  if (!s.abort_flag || atomicExch(s.abort_flag, 1) == 0) {
    volatile int* e = reinterpret_cast<volatile int*>(s.err);
    e[1] = blockIdx.x;
    e[2] = threadIdx.x;
    __threadfence_system();
    e[0] = code;
  }
  __threadfence_system();
  return false;
}
__device__ __forceinline__ bool mb_wait(uint32_t bar, uint32_t parity, const Sync& s, volatile int* s_abort, int code) {
  if (mb_try(bar, parity)) return true;
  long long t0 = 0;
  unsigned int spins = 0;
  while (!mb_try(bar, parity))
    if (!may_spin(spins, t0, s, s_abort, code)) return false;
  return true;
}
// The whole warp waits and agrees on the outcome.
__device__ __forceinline__ bool mb_wait_warp(uint32_t bar, uint32_t parity, const Sync& s, volatile int* s_abort,
                                             int code) {
  return __all_sync(0xffffffffu, mb_wait(bar, parity, s, s_abort, code));
}

// Position in a ring: slot and the parity of its current phase.
template <int R>
struct RingPos {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void next() {
    if (++slot == R) {
      slot = 0;
      phase ^= 1u;
    }
  }
};

// ---- inputs and outputs of a gate-stage warp -------------------------------------------------
// Per warp in shared memory: IO_RING slots of two blocks of 32 pieces (a piece: one quad of one
// row, 16 or 8 bytes) - block 0 the gate values, piece = gate * 8 + row; block 1 single values,
// piece = array * 8 + row - and one such slot for the outputs.
constexpr int IO_RING = 4;
template <typename T>
struct IoBytes {
  static constexpr int PIECE = 4 * (int)sizeof(T), SLOT = 64 * PIECE, WARP = (IO_RING + 1) * SLOT;
};

template <int B>
__device__ __forceinline__ void cp_async_piece(uint32_t dst, const void* src) {
  if (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

// Inputs, in the order of the steps this warp takes (chain c0, c0 + cs, ... of each time step;
// time runs down when BWD).  NG gate arrays in rows of S values; singles: forward {mask}, backward
// {dh_new, c or h, mask, dc_new}.
template <typename T, int NG, bool BWD>
struct WarpInputs {
  const char *gsrc, *ssrc;  // this lane's piece of block 0 / 1 at time 0 of chain row 0, null: none
  uint32_t gstep, sstep;    // bytes per (time, row)
  uint32_t ring;
  int t, ch;                // next step to fetch
  int slot_in, slot_out;

  __device__ __forceinline__ void init(const ChainParams& p, uint8_t* buf, int lane, int u0, int S, int c0) {
    ring = smem_u32(buf) + lane * IoBytes<T>::PIECE;
    slot_in = slot_out = 0;
    t = BWD ? p.T - 1 : 0;
    ch = c0;
    const int a = lane >> 3, r = lane & 7;
    gstep = (uint32_t)S * sizeof(T);
    sstep = (uint32_t)p.H * sizeof(T);
    gsrc = ssrc = nullptr;
    if (u0 >= p.H || !p.wide) return;
    if (a < NG)
      gsrc = reinterpret_cast<const char*>(reinterpret_cast<const T*>(p.gin) + a * p.H + u0) + (size_t)r * gstep;
    const void* single = nullptr;
    if (!BWD) single = (a == 0 && p.has_zoneout && p.training) ? p.mask : nullptr;
    else if (a == 0) single = p.dh_new;
    else if (a == 1) single = NG == 4 && p.c ? p.c : p.h;
    else if (a == 2) single = p.has_zoneout ? p.mask : nullptr;
    else single = p.dc_new;
    if (single)
      ssrc = reinterpret_cast<const char*>(reinterpret_cast<const T*>(single) + u0) +
             (size_t)(r + ((BWD && (a == 0 || a == 3)) ? p.N : 0)) * sstep;
  }
  __device__ __forceinline__ void fetch(const ChainParams& p, int lane, int tile0, int ch_n, int c0, int cs) {
    if (p.wide && (BWD ? t >= 0 : t < p.T)) {
      const int n0 = (tile0 + ch) * 8;
      const uint32_t row = (uint32_t)(t * p.N + n0), dst = ring + slot_in * IoBytes<T>::SLOT;
      if (n0 + (lane & 7) < p.N) {
        if (gsrc) cp_async_piece<IoBytes<T>::PIECE>(dst, gsrc + (unsigned long long)row * gstep);
        if (ssrc) cp_async_piece<IoBytes<T>::PIECE>(dst + IoBytes<T>::SLOT / 2, ssrc + (unsigned long long)row * sstep);
      }
      if ((ch += cs) >= ch_n) {
        ch = c0;
        t += BWD ? -1 : 1;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++slot_in == IO_RING) slot_in = 0;
  }
  // The oldest step's slot (this warp's lanes may read it), and the fetch of the step IO_RING - 1
  // further on.
  __device__ __forceinline__ const uint8_t* take(const ChainParams& p, const uint8_t* buf, int lane, int tile0,
                                                 int ch_n, int c0, int cs) {
    asm volatile("cp.async.wait_group %0;" ::"n"(IO_RING - 2) : "memory");
    __syncwarp();  // every lane's pieces are there, and every lane has read the slot before
    const uint8_t* s = buf + slot_out * IoBytes<T>::SLOT;
    if (++slot_out == IO_RING) slot_out = 0;
    fetch(p, lane, tile0, ch_n, c0, cs);
    return s;
  }
};

// Value a of block b at (row, ul) of a slot.
template <typename T>
__device__ __forceinline__ float slot_value(const uint8_t* slot, int b, int a, int row, int ul) {
  return ld(reinterpret_cast<const T*>(slot + b * (IoBytes<T>::SLOT / 2) + (a * 8 + row) * IoBytes<T>::PIECE) + ul);
}
template <typename T>
__device__ __forceinline__ void slot_store(uint8_t* slot, int b, int a, int row, int ul, float v) {
  st(reinterpret_cast<T*>(slot + b * (IoBytes<T>::SLOT / 2) + (a * 8 + row) * IoBytes<T>::PIECE) + ul, v);
}
template <typename T>
__device__ __forceinline__ void copy_piece(T* dst, const uint8_t* src) {
  if (sizeof(T) == 4) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
  else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(src);
}

// Inputs of one forward step for the lane's (row n, unit).
template <typename T, int G>
__device__ __forceinline__ void fwd_inputs(const ChainParams& p, const uint8_t* slot, int t, int n, int unit, int row,
                                           int ul, float (&wv)[G], float& m) {
  const bool zt = p.has_zoneout && p.training;
  if (p.wide) {
#pragma unroll
    for (int g = 0; g < G; ++g) wv[g] = slot_value<T>(slot, 0, g, row, ul);
    if (zt) m = slot_value<T>(slot, 1, 0, row, ul);
  } else if (n < p.N && unit < p.H) {
    const long long e = (long long)t * p.N + n;
    const T* x = reinterpret_cast<const T*>(p.gin) + e * G * p.H + unit;
#pragma unroll
    for (int g = 0; g < G; ++g) wv[g] = ld(x + (long long)g * p.H);
    if (zt) m = ld(reinterpret_cast<const T*>(p.mask) + e * p.H + unit);
    if (t + 1 < p.T) {
#pragma unroll
      for (int g = 0; g < G; ++g) prefetch_l2(x + ((long long)p.N * G + g) * p.H);
      if (zt) prefetch_l2(reinterpret_cast<const T*>(p.mask) + (e + p.N) * p.H + unit);
    }
  } else {
#pragma unroll
    for (int g = 0; g < G; ++g) wv[g] = 0.f;
  }
}

// Results of one forward step: h, c (LSTM), the gate cache.
template <typename T, int G>
__device__ __forceinline__ void fwd_outputs(const ChainParams& p, uint8_t* slot, int lane, int t, int n0, int u0,
                                            int row, int ul, float h, float c, const float (&gate)[4]) {
  const bool cache = p.training && p.gout;
  const int H = p.H;
  T *hb = reinterpret_cast<T*>(p.h), *cb = reinterpret_cast<T*>(p.c), *vb = reinterpret_cast<T*>(p.gout);
  if (p.wide) {
    __syncwarp();  // the last step's pieces have been read
    slot_store<T>(slot, 1, 0, row, ul, h);
    if (G == 4) slot_store<T>(slot, 1, 1, row, ul, c);
    if (cache) {
#pragma unroll
      for (int g = 0; g < 4; ++g) slot_store<T>(slot, 0, g, row, ul, gate[g]);
    }
    __syncwarp();
    const int a = lane >> 3, n = n0 + (lane & 7);
    if (n < p.N && u0 < H) {
      const long long e = (long long)t * p.N + n;
      const uint8_t* src = slot + lane * IoBytes<T>::PIECE;
      if (cache) copy_piece<T>(vb + (e * 4 + a) * H + u0, src);
      if (a < (G == 4 ? 2 : 1)) copy_piece<T>((a == 0 ? hb : cb) + (e + p.N) * H + u0, src + IoBytes<T>::SLOT / 2);
    }
  } else if (n0 + row < p.N && u0 + ul < H) {
    const long long e = (long long)t * p.N + n0 + row;
    st(hb + (e + p.N) * H + u0 + ul, h);
    if (G == 4) st(cb + (e + p.N) * H + u0 + ul, c);
    if (cache) {
#pragma unroll
      for (int g = 0; g < 4; ++g) st(vb + (e * 4 + g) * H + u0 + ul, gate[g]);
    }
  }
}

// Inputs of one backward step.  prev: c (LSTM) or h (GRU) before the step.
template <typename T, int G>
__device__ __forceinline__ void bwd_inputs(const ChainParams& p, const uint8_t* slot, int t, int n, int unit, int row,
                                           int ul, float (&gv)[4], float& dhv, float& prev, float& m, float& dcv) {
  m = 1.f;
  dcv = 0.f;
  if (p.wide) {
#pragma unroll
    for (int g = 0; g < 4; ++g) gv[g] = slot_value<T>(slot, 0, g, row, ul);
    dhv = slot_value<T>(slot, 1, 0, row, ul);
    prev = slot_value<T>(slot, 1, 1, row, ul);
    if (p.has_zoneout) m = slot_value<T>(slot, 1, 2, row, ul);
    if (G == 4 && p.dc_new) dcv = slot_value<T>(slot, 1, 3, row, ul);
  } else if (n < p.N && unit < p.H) {
    const long long e = (long long)t * p.N + n, o = e * p.H + unit, NH = (long long)p.N * p.H;
    const T* v = reinterpret_cast<const T*>(p.gin) + e * 4 * p.H + unit;
    const T *dhn = reinterpret_cast<const T*>(p.dh_new) + o, *dcn = reinterpret_cast<const T*>(p.dc_new) + o;
    const T *pv = reinterpret_cast<const T*>(G == 4 ? p.c : p.h) + o, *mk = reinterpret_cast<const T*>(p.mask) + o;
#pragma unroll
    for (int g = 0; g < 4; ++g) gv[g] = ld(v + (long long)g * p.H);
    dhv = ld(dhn + NH);
    prev = ld(pv);
    if (p.has_zoneout) m = ld(mk);
    if (G == 4 && p.dc_new) dcv = ld(dcn + NH);
    if (t > 0) {
#pragma unroll
      for (int g = 0; g < 4; ++g) prefetch_l2(v - 4 * NH + (long long)g * p.H);
      prefetch_l2(dhn);
      prefetch_l2(pv - NH);
      if (p.has_zoneout) prefetch_l2(mk - NH);
      if (G == 4 && p.dc_new) prefetch_l2(dcn);
    }
  } else {
    gv[0] = gv[1] = gv[2] = gv[3] = dhv = prev = 0.f;
  }
}

// Results of one backward step: the gate gradients and, for fp32 storage, their bf16 planes.
template <typename T, int G>
__device__ __forceinline__ void bwd_outputs(const ChainParams& p, uint8_t* slot, int lane, int t, int n0, int u0,
                                            int row, int ul, const float (&dg)[4]) {
  const int H = p.H;
  T *dv = reinterpret_cast<T*>(p.dv), *dp = reinterpret_cast<T*>(p.dp), *dq = reinterpret_cast<T*>(p.dq);
  if (p.wide) {
    __syncwarp();  // the last step's pieces have been read
#pragma unroll
    for (int g = 0; g < 4; ++g) slot_store<T>(slot, 0, g, row, ul, dg[g]);
    __syncwarp();
    const int a = lane >> 3, n = n0 + (lane & 7);
    if (n < p.N && u0 < H) {
      const long long e = (long long)t * p.N + n;
      const uint8_t* src = slot + lane * IoBytes<T>::PIECE;
      // LSTM: gate a of dv.  GRU: dp holds values 0, 1, 2 and dq values 0, 1, 3.
      const long long o1 = (G == 4 ? e * 4 + a : e * 3 + a) * H + u0, o2 = (e * 3 + (a == 3 ? 2 : a)) * H + u0;
      if (G == 4) copy_piece<T>(dv + o1, src);
      if (G == 3 && a < 3) copy_piece<T>(dp + o1, src);
      if (G == 3 && a != 2) copy_piece<T>(dq + o2, src);
      if (sizeof(T) == 4 && p.gpl) {
        const float4 f = *reinterpret_cast<const float4*>(src);
        float h0, h1, h2, h3, l0, l1, l2, l3;
        split_bf16(f.x, h0, l0); split_bf16(f.y, h1, l1); split_bf16(f.z, h2, l2); split_bf16(f.w, h3, l3);
        const uint2 hi = make_uint2(pack_bf16(h0, h1), pack_bf16(h2, h3));
        const uint2 lo = make_uint2(pack_bf16(l0, l1), pack_bf16(l2, l3));
        if (G == 4 || a < 3) {
          *reinterpret_cast<uint2*>(p.gpl + o1) = hi;
          *reinterpret_cast<uint2*>(p.gpl + p.gpl_stride + o1) = lo;
        }
        if (G == 3 && a != 2) {
          *reinterpret_cast<uint2*>(p.gpl2 + o2) = hi;
          *reinterpret_cast<uint2*>(p.gpl2 + p.gpl_stride + o2) = lo;
        }
      }
    }
  } else if (n0 + row < p.N && u0 + ul < H) {
    const long long e = (long long)t * p.N + n0 + row;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const long long o1 = (G == 4 ? e * 4 + a : e * 3 + a) * H + u0 + ul, o2 = (e * 3 + (a == 3 ? 2 : a)) * H + u0 + ul;
      float hi, lo;
      split_bf16(dg[a], hi, lo);
      if (G == 4) st(dv + o1, dg[a]);
      if (G == 3 && a < 3) st(dp + o1, dg[a]);
      if (G == 3 && a != 2) st(dq + o2, dg[a]);
      if (sizeof(T) == 4 && p.gpl) {
        if (G == 4 || a < 3) {
          p.gpl[o1] = __float2bfloat16_rn(hi);
          p.gpl[p.gpl_stride + o1] = __float2bfloat16_rn(lo);
        }
        if (G == 3 && a != 2) {
          p.gpl2[o2] = __float2bfloat16_rn(hi);
          p.gpl2[p.gpl_stride + o2] = __float2bfloat16_rn(lo);
        }
      }
    }
  }
}

}  // namespace rec
}  // namespace hb
