#include "util.cuh"

#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <utility>
#include <vector>

namespace hb {

// ---------------------------------------------------------------------------
// Error text (thread-local) and launch counter.
// ---------------------------------------------------------------------------
static thread_local char g_err[512] = "";

void set_last_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}
const char* last_error() { return g_err; }

static std::atomic<long long> g_launches{0};
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launch_count() { return g_launches.load(std::memory_order_relaxed); }

int sm_count() {
  static std::atomic<int> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return 148;
  }
  if (dev >= 0 && dev < 64) {
    const int c = cached[dev].load(std::memory_order_relaxed);
    if (c > 0) return c;
  }
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    n = 148;
  }
  if (dev >= 0 && dev < 64) cached[dev].store(n, std::memory_order_relaxed);
  return n;
}

// ---------------------------------------------------------------------------
// Error word shared with the kernels.
// ---------------------------------------------------------------------------
namespace {
std::once_flag g_errw_once;
int* g_errw = nullptr;
}  // namespace

int* device_error_word() {
  std::call_once(g_errw_once, [] {
    void* p = nullptr;
    if (cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
      g_errw = static_cast<int*>(p);
      *g_errw = 0;
    } else {
      cudaGetLastError();
    }
  });
  return g_errw;  // unified addressing: the host pointer is valid on every device
}

int take_error_word(int* detail) {
  if (!g_errw) return 0;
  volatile int* w = g_errw;
  const int v = *w;
  if (v) {
    if (detail)
      for (int i = 0; i < 4; ++i) detail[i] = w[1 + i];
    *w = 0;
  }
  return v;
}

// ---------------------------------------------------------------------------
// Per-phase timing.
// ---------------------------------------------------------------------------
namespace {
struct ProfRec { int phase; cudaEvent_t a, b; bool closed; };
std::mutex g_prof_mu;
std::vector<ProfRec> g_prof;
std::atomic<bool> g_prof_on{false};
}  // namespace

void profile_enable(bool on) { g_prof_on.store(on); }
bool profile_enabled() { return g_prof_on.load(std::memory_order_relaxed); }

void profile_mark(int phase, bool begin, cudaStream_t s) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  if (begin) {
    ProfRec r{phase, nullptr, nullptr, false};
    cudaEventCreate(&r.a);
    cudaEventCreate(&r.b);
    cudaEventRecord(r.a, s);
    g_prof.push_back(r);
  } else {
    for (auto it = g_prof.rbegin(); it != g_prof.rend(); ++it)
      if (it->phase == phase && !it->closed) {
        cudaEventRecord(it->b, s);
        it->closed = true;
        break;
      }
  }
}

void profile_read(float* ms, int n) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  for (int i = 0; i < n; ++i) ms[i] = 0.f;
  for (auto& r : g_prof) {
    if (r.closed) {
      cudaEventSynchronize(r.b);
      float t = 0.f;
      if (cudaEventElapsedTime(&t, r.a, r.b) == cudaSuccess && r.phase < n) ms[r.phase] += t;
    }
    cudaEventDestroy(r.a);
    cudaEventDestroy(r.b);
  }
  g_prof.clear();
}

// ---------------------------------------------------------------------------
// Scratch pool.
// ---------------------------------------------------------------------------
namespace {
struct Block { void* p = nullptr; size_t n = 0; };
std::mutex g_ws_mu;
// (device, stream, slot, and for the handle that names another stream in every thread the thread)
std::map<std::tuple<int, cudaStream_t, int, const void*>, Block> g_ws;
thread_local char t_self;
}  // namespace

void* workspace(cudaStream_t stream, size_t bytes, int slot) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    set_last_error("cudaGetDevice failed");
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(g_ws_mu);
  const void* thread = stream == cudaStreamPerThread ? &t_self : nullptr;
  Block& b = g_ws[std::make_tuple(dev, stream, slot, thread)];
  if (b.n >= bytes && b.p) return b.p;
  if (b.p) {
    // Work already queued on this stream may still read the old block.
    cudaStreamSynchronize(stream);
    cudaFree(b.p);
    b.p = nullptr;
    b.n = 0;
  }
  size_t want = bytes + bytes / 4 + (1 << 20);
  cudaError_t e = cudaMalloc(&b.p, want);
  if (e != cudaSuccess) {
    want = bytes;
    e = cudaMalloc(&b.p, want);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    b.p = nullptr;
    set_last_error("scratch allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
    return nullptr;
  }
  b.n = want;
  return b.p;
}

int make_arena(Arena* a, cudaStream_t stream, size_t bytes, int slot) {
  a->base = static_cast<char*>(workspace(stream, bytes, slot));
  a->cap = bytes;
  a->off = 0;
  return a->base ? HASTE_B200_OK : HASTE_B200_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// Column sums.
// ---------------------------------------------------------------------------
namespace {

constexpr int CS_THREADS = 128;  // threads per block, four columns each
constexpr int CS_ROWS = 8;       // rows whose loads are in flight together
constexpr int CS_CHUNKS = 128;   // row chunks (partials per column)

inline int cs_chunks(int rows) {
  const int c = ceil_div(rows, CS_ROWS);
  return c < CS_CHUNKS ? (c > 0 ? c : 1) : CS_CHUNKS;
}

// A stream over the matrix, bound by HBM: 8- or 16-byte loads where rows and start allow them
// (Vec), CS_ROWS of them ahead.  One column per thread and four rows ahead read a [64000 x 3072]
// bf16 matrix at 2.1 TB/s.  The order of every sum is fixed by rows and width.
template <typename T, bool Vec>
__global__ void __launch_bounds__(CS_THREADS) colsum_stage1(const T* __restrict__ in, long long lda, int rows,
                                                            int width, int chunks, float* __restrict__ part) {
  const int j = (blockIdx.x * CS_THREADS + threadIdx.x) * 4;
  if (j >= width) return;
  const int c = blockIdx.y;
  const int per = (rows + chunks - 1) / chunks;
  const int r0 = c * per, r1 = min(rows, r0 + per);
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  for (int r = r0; r < r1; r += CS_ROWS) {
    float x[CS_ROWS][4];
#pragma unroll
    for (int k = 0; k < CS_ROWS; ++k) {
      const T* q = in + (long long)(r + k) * lda + j;
      const bool ok = r + k < r1;
      if constexpr (Vec) {
        typedef typename std::conditional<sizeof(T) == 4, uint4, uint2>::type Word;
        Word w{};
        if (ok) w = *reinterpret_cast<const Word*>(q);
        const T* e = reinterpret_cast<const T*>(&w);
#pragma unroll
        for (int i = 0; i < 4; ++i) x[k][i] = ld(e + i);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[k][i] = ok && j + i < width ? ld(q + i) : 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float a = 0.f;
#pragma unroll
      for (int k = 0; k < CS_ROWS; ++k) a += x[k][i];
      s[i] += a;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (j + i < width) part[(long long)c * width + j + i] = s[i];
}

// 32 columns x 8 groups of chunks.  The first w2 columns go to out2 as well.
template <typename T>
__global__ void __launch_bounds__(256) colsum_stage2(const float* __restrict__ part, int width, int chunks,
                                                     T* __restrict__ out, T* __restrict__ out2, int w2,
                                                     int accumulate) {
  __shared__ float sums[8][32];
  const int col = threadIdx.x & 31, grp = threadIdx.x >> 5, j = blockIdx.x * 32 + col;
  float s = 0.f;
  if (j < width)
    for (int c = grp; c < chunks; c += 8) s += part[(long long)c * width + j];
  sums[grp][col] = s;
  __syncthreads();
  if (grp != 0 || j >= width) return;
#pragma unroll
  for (int k = 1; k < 8; ++k) s += sums[k][col];
  if (j < w2) st(out2 + j, accumulate ? s + ld(out2 + j) : s);
  st(out + j, accumulate ? s + ld(out + j) : s);
}

template <typename T>
__global__ void bias_grad_kernel(int gates, const float* __restrict__ part, int rows, int H,
                                 T* __restrict__ db, T* __restrict__ db2, int accumulate) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= 4 * H) return;
  float s = 0.f;
  for (int r = 0; r < rows; ++r) s += part[(long long)r * 4 * H + j];
  if (gates == 4 || j < 3 * H) st(db + j, accumulate ? ld(db + j) + s : s);
  if (gates == 3 && (j < 2 * H || j >= 3 * H)) {
    T* d = db2 + (j < 2 * H ? j : j - H);
    st(d, accumulate ? ld(d) + s : s);
  }
}

template <typename T>
__global__ void to_float_kernel(const T* __restrict__ src, float* __restrict__ dst, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = ld(src + i);
}
template <typename T>
__global__ void from_float_kernel(const float* __restrict__ src, T* __restrict__ dst, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) st(dst + i, src[i]);
}

template <typename T>
__global__ void add_float_into_kernel(const float* __restrict__ src, T* __restrict__ dst, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) st(dst + i, ld(dst + i) + src[i]);
}

}  // namespace

int add_float_into(int dtype, const float* src, void* dst, size_t n, cudaStream_t stream) {
  if (n == 0) return HASTE_B200_OK;
  const int blocks = ceil_div((long long)n, 256);
  if (dtype == HASTE_B200_F32)
    add_float_into_kernel<float><<<blocks, 256, 0, stream>>>(src, (float*)dst, n);
  else if (dtype == HASTE_B200_F16)
    add_float_into_kernel<__half><<<blocks, 256, 0, stream>>>(src, (__half*)dst, n);
  else
    add_float_into_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(src, (__nv_bfloat16*)dst, n);
  HB_LAUNCH_OK();
  count_launch(1);
  return HASTE_B200_OK;
}

size_t colsum_scratch_floats(int rows, int width) { return (size_t)cs_chunks(rows) * width; }

namespace {
template <typename T>
void colsum_first(const void* in, long long lda, int rows, int width, int chunks, float* part, cudaStream_t stream) {
  const dim3 grid(ceil_div(width, 4 * CS_THREADS), chunks);
  const bool vec = width % 4 == 0 && lda % 4 == 0 && reinterpret_cast<uintptr_t>(in) % (4 * sizeof(T)) == 0;
  if (vec) colsum_stage1<T, true><<<grid, CS_THREADS, 0, stream>>>((const T*)in, lda, rows, width, chunks, part);
  else colsum_stage1<T, false><<<grid, CS_THREADS, 0, stream>>>((const T*)in, lda, rows, width, chunks, part);
}
}  // namespace

int colsum(int in_dtype, const void* in, long long ld_, int rows, int width, int out_dtype,
           void* out, int accumulate, float* scratch, cudaStream_t stream, void* out2, int w2) {
  if (width <= 0) return HASTE_B200_OK;
  const int chunks = cs_chunks(rows), blocks = ceil_div(width, 32);
  if (in_dtype == HASTE_B200_F32) colsum_first<float>(in, ld_, rows, width, chunks, scratch, stream);
  else if (in_dtype == HASTE_B200_F16) colsum_first<__half>(in, ld_, rows, width, chunks, scratch, stream);
  else colsum_first<__nv_bfloat16>(in, ld_, rows, width, chunks, scratch, stream);
  HB_LAUNCH_OK();
  if (out_dtype == HASTE_B200_F32)
    colsum_stage2<float><<<blocks, 256, 0, stream>>>(scratch, width, chunks, (float*)out, (float*)out2, w2,
                                                     accumulate);
  else if (out_dtype == HASTE_B200_F16)
    colsum_stage2<__half><<<blocks, 256, 0, stream>>>(scratch, width, chunks, (__half*)out, (__half*)out2, w2,
                                                      accumulate);
  else
    colsum_stage2<__nv_bfloat16><<<blocks, 256, 0, stream>>>(scratch, width, chunks, (__nv_bfloat16*)out,
                                                             (__nv_bfloat16*)out2, w2, accumulate);
  HB_LAUNCH_OK();
  count_launch(2);
  return HASTE_B200_OK;
}

int bias_grad_finish(int gates, const float* part, int rows, int H, int dtype, void* db, void* db2,
                     int accumulate, cudaStream_t stream) {
  const int blocks = ceil_div(4LL * H, 128);
  if (dtype == HASTE_B200_F32)
    bias_grad_kernel<float><<<blocks, 128, 0, stream>>>(gates, part, rows, H, (float*)db, (float*)db2, accumulate);
  else if (dtype == HASTE_B200_F16)
    bias_grad_kernel<__half><<<blocks, 128, 0, stream>>>(gates, part, rows, H, (__half*)db, (__half*)db2,
                                                        accumulate);
  else
    bias_grad_kernel<__nv_bfloat16><<<blocks, 128, 0, stream>>>(gates, part, rows, H,
                                                                (__nv_bfloat16*)db, (__nv_bfloat16*)db2, accumulate);
  HB_LAUNCH_OK();
  count_launch(1);
  return HASTE_B200_OK;
}

int to_float(int dtype, const void* src, float* dst, size_t n, cudaStream_t stream) {
  if (n == 0) return HASTE_B200_OK;
  const int blocks = ceil_div((long long)n, 256);
  if (dtype == HASTE_B200_F32)
    to_float_kernel<float><<<blocks, 256, 0, stream>>>((const float*)src, dst, n);
  else if (dtype == HASTE_B200_F16)
    to_float_kernel<__half><<<blocks, 256, 0, stream>>>((const __half*)src, dst, n);
  else
    to_float_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)src, dst, n);
  HB_LAUNCH_OK();
  count_launch(1);
  return HASTE_B200_OK;
}

int from_float(int dtype, const float* src, void* dst, size_t n, cudaStream_t stream) {
  if (n == 0) return HASTE_B200_OK;
  const int blocks = ceil_div((long long)n, 256);
  if (dtype == HASTE_B200_F32)
    from_float_kernel<float><<<blocks, 256, 0, stream>>>(src, (float*)dst, n);
  else if (dtype == HASTE_B200_F16)
    from_float_kernel<__half><<<blocks, 256, 0, stream>>>(src, (__half*)dst, n);
  else
    from_float_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(src, (__nv_bfloat16*)dst, n);
  HB_LAUNCH_OK();
  count_launch(1);
  return HASTE_B200_OK;
}

}  // namespace hb
