// haste_b200_native: the host path of the layers in rnn.py - output allocation, the library call and
// the autograd node - in one C++ call per layer call.
//
// A layer call on a small batch is bound by its host work: argument checks, a dozen tensor
// operations and the autograd glue cost 90 us per call in Python, ten times the kernels of a
// single time step.  Here a call without gradients allocates its outputs and launches; a call with
// gradients also records one autograd node whose backward pass allocates the gradients
// uninitialised (the library assigns them) and reads the incoming gradient where autograd left
// it: the node's outputs are the sequences h_1..h_T (c_1..c_T) themselves, kept behind a slot for
// the initial state, so no [T+1] gradient is assembled and no gradient of c is made up of zeros.
#include <torch/extension.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>

#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "haste_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
namespace py = pybind11;

enum Cell { LSTM, GRU, INDRNN, LN_LSTM, LN_GRU, LN_INDRNN };

bool has_c(int cell) { return cell == LSTM || cell == LN_LSTM; }

// The library functions, resolved once from the shared object that the ctypes binding has loaded
// (so that both use one copy of it and its settings).
#define HB_FUNCTIONS(X)                                                                              \
  X(last_error) X(exchange_sm_budget) X(exchange_assign_gradients) X(lstm_forward) X(lstm_backward)  \
  X(gru_forward) X(gru_backward) X(indrnn_forward) X(indrnn_backward) X(layer_norm_lstm_forward)     \
  X(layer_norm_lstm_backward) X(layer_norm_gru_forward) X(layer_norm_gru_backward)                   \
  X(layer_norm_indrnn_forward) X(layer_norm_indrnn_backward) X(lstm_forward_iterate)                 \
  X(gru_forward_iterate)
struct Library {
#define HB_FIELD(f) decltype(&haste_b200_##f) f = nullptr;
  HB_FUNCTIONS(HB_FIELD)
#undef HB_FIELD
} lib;
PyObject* haste_error = nullptr;  // _C.HasteError, kept for the life of the process

void load(const std::string& path, py::object error) {
  void* so = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!so) throw std::runtime_error(dlerror());
#define HB_RESOLVE(f)                                                                      \
  lib.f = reinterpret_cast<decltype(&haste_b200_##f)>(dlsym(so, "haste_b200_" #f));        \
  if (!lib.f) throw std::runtime_error("haste_b200_" #f " is missing from " + path);
  HB_FUNCTIONS(HB_RESOLVE)
#undef HB_RESOLVE
  haste_error = error.release().ptr();
}

struct LibraryError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
void ok(const char* name, int status) {
  if (status != HASTE_B200_OK)
    throw LibraryError("haste_b200_" + std::string(name) + " failed with status " + std::to_string(status) + ": " +
                       lib.last_error());
}
#define CALL(f, ...) ok(#f, lib.f(__VA_ARGS__))

void cuda_ok(cudaError_t e) { TORCH_CHECK(e == cudaSuccess, "haste_b200: ", cudaGetErrorString(e)); }

int dtype_of(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return HASTE_B200_F32;
    case at::kBFloat16: return HASTE_B200_BF16;
    case at::kHalf: return HASTE_B200_F16;  // GRU only; the other entry points reject it
    default: break;
  }
  throw py::type_error(std::string("haste_b200 supports float32, bfloat16 and (GRU only) float16 tensors, got ") +
                       c10::toString(t.scalar_type()));
}

// LayerNormLSTM keeps its saved activations in float32 also for bfloat16 layers (BF16_WIDE).
at::TensorOptions saved_options(const Tensor& x, int cell) {
  return cell == LN_LSTM && x.scalar_type() == at::kBFloat16 ? x.options().dtype(at::kFloat) : x.options();
}
int lib_dtype(const Tensor& x, int cell) {
  const int d = dtype_of(x);
  return cell == LN_LSTM && d == HASTE_B200_BF16 ? HASTE_B200_BF16_WIDE : d;
}

void* ptr(const Tensor& t) { return t.defined() && t.numel() ? t.data_ptr() : nullptr; }

// Settings of this thread's calls, put back as they were.
struct SmBudget {
  int sms, was;
  explicit SmBudget(int n) : sms(n), was(sms ? lib.exchange_sm_budget(sms) : 0) {}
  ~SmBudget() { if (sms) lib.exchange_sm_budget(was); }
};
struct AssignGradients {
  int was = lib.exchange_assign_gradients(1);
  ~AssignGradients() { lib.exchange_assign_gradients(was); }
};

void check(const Tensor& x, at::ArrayRef<Tensor> ts) {
  TORCH_CHECK(x.is_cuda(), "haste_b200: tensor must be a CUDA tensor");
  for (const Tensor& t : ts) {
    if (!t.defined() || !t.numel()) continue;
    TORCH_CHECK(t.is_cuda(), "haste_b200: tensor must be a CUDA tensor");
    TORCH_CHECK(t.is_contiguous(), "haste_b200: tensor must be contiguous");
    TORCH_CHECK(t.device() == x.device() && t.scalar_type() == x.scalar_type(),
                "haste_b200: all tensors must share one device and dtype");
  }
}

// (Numbers are put into messages with std::to_string: an ostream of this object may meet the locale
// of another copy of the C++ library.)
std::string shape_of(const Tensor& t) {
  std::string s = "[";
  for (int64_t n : t.sizes()) s += (s.size() > 1 ? "," : "") + std::to_string(n);
  return s + "]";
}

// The library takes pointers and sizes, so what the tensors hold has to be said here: x [T,N,C] with
// the layer's weights, and the mask where it is read.  (The states are checked where they are taken.)
void check_sizes(int cell, const Tensor& x, int64_t H, const std::vector<Tensor>& P, const Tensor* mask) {
  static const int kGates[] = {4, 3, 1, 4, 3, 1};
  const int64_t GH = kGates[cell] * H, C = x.size(2);
  auto wrong = [&](const Tensor& t, const char* name, const std::string& want) {
    TORCH_CHECK(false, "haste_b200: " + std::string(name) + " must be " + want + " for an input " + shape_of(x) +
                           " and " + std::to_string(H) + " units, got " + shape_of(t));
  };
  auto matrix = [&](const Tensor& t, const char* name, int64_t rows, int64_t cols) {
    if (t.dim() != 2 || t.size(0) != rows || t.size(1) != cols)
      wrong(t, name, "[" + std::to_string(rows) + "," + std::to_string(cols) + "]");
  };
  auto holds = [&](const Tensor& t, const char* name, int64_t n) {
    if (t.numel() != n) wrong(t, name, std::to_string(n) + " values");
  };
  matrix(P[0], "kernel", C, GH);
  if (GH != H) matrix(P[1], "recurrent kernel", H, GH);
  else holds(P[1], "recurrent scale", H);
  holds(P[2], "bias", GH);
  if (cell == GRU || cell == LN_GRU) holds(P[3], "recurrent bias", GH);
  if (cell == LN_LSTM) {
    holds(P[3], "gamma", 2 * GH);
    holds(P[4], "gamma_h", H);
    holds(P[5], "beta_h", H);
  }
  if (cell == LN_GRU) holds(P[4], "gamma", 2 * GH);
  if (cell == LN_INDRNN && P[3].numel() < H) wrong(P[3], "gamma", "[2,H]");  // only its first row is read
  if (mask && mask->defined() && mask->numel()) holds(*mask, "zoneout mask", x.size(0) * x.size(1) * H);
}

struct Dims { int T, N, C, H; };

// A sequence [T,N,H] with room for the state before it: slot 0 of the buffer, filled with `s0` or
// zeros.  The returned tensor starts at slot 1 and is no view of the buffer to autograd.
Tensor sequence(const Dims& d, const Tensor& like, const Tensor& s0, cudaStream_t stream) {
  const int64_t slot = (int64_t)d.N * d.H;
  Tensor buf = at::empty({d.T + 1, d.N, d.H}, like.options());
  const size_t bytes = slot * buf.element_size();
  if (s0.defined()) cuda_ok(cudaMemcpyAsync(buf.data_ptr(), s0.data_ptr(), bytes, cudaMemcpyDeviceToDevice, stream));
  else cuda_ok(cudaMemsetAsync(buf.data_ptr(), 0, bytes, stream));
  Tensor y = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(buf.storage()), buf.key_set(), buf.dtype());
  y.unsafeGetTensorImpl()->set_sizes_and_strides(c10::IntArrayRef{d.T, d.N, d.H}, c10::IntArrayRef{slot, d.H, 1}, slot);
  return y;
}
// Start of the buffer behind a tensor of sequence().
void* slot0(const Tensor& y) {
  return static_cast<char*>(y.data_ptr()) - y.size(1) * y.size(2) * y.element_size();
}
// The whole buffer [T+1,N,H] behind a tensor of sequence(), as the backward pass keeps it: slot 0 is
// part of what saved-tensor hooks (offloading, checkpointing) copy, and the version counter is that
// of `y`, so that a change of the output in place is noticed.
Tensor whole(const Tensor& y) {
  Tensor buf = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(y.storage()), y.key_set(), y.dtype());
  c10::TensorImpl* impl = buf.unsafeGetTensorImpl();
  impl->set_sizes_and_strides(c10::IntArrayRef{y.size(0) + 1, y.size(1), y.size(2)}, y.strides(), 0);
  impl->set_version_counter(y.unsafeGetTensorImpl()->version_counter());
  return buf;
}

struct Forward {
  Tensor y, c;
  std::vector<Tensor> saved;  // what only the backward pass needs
};

// params: LSTM {W,R,b}  GRU {W,R,bx,br}  IndRNN {W,u,b}  LayerNormLSTM {W,R,b,gamma,gamma_h,beta_h}
// LayerNormGRU {W,R,bx,br,gamma}  LayerNormIndRNN {W,u,b,gamma}
Forward run_forward(int cell, bool training, double zoneout, const Tensor& x, const Tensor& h0, const Tensor& c0,
                    const Tensor& mask, at::TensorList P) {
  const Dims d{(int)x.size(0), (int)x.size(1), (int)x.size(2),
               (int)(cell == INDRNN || cell == LN_INDRNN ? P[0].size(1) : P[1].size(0))};
  cudaStream_t st = c10::cuda::getCurrentCUDAStream().stream();
  void* s = (void*)st;
  const bool zo = zoneout != 0.0 && mask.defined() && mask.numel();
  const float zp = zo ? (float)zoneout : 0.0f;
  const void* mp = zo ? mask.data_ptr() : nullptr;
  const int dt = lib_dtype(x, cell), tr = training;
  const auto o = x.options(), so = saved_options(x, cell);
  Forward f;
  f.y = sequence(d, x, h0, st);
  void *h = slot0(f.y), *c = nullptr;
  if (has_c(cell)) {
    f.c = sequence(d, x, c0, st);
    c = slot0(f.c);
  }
  const int64_t T = d.T, N = d.N, H = d.H;
  switch (cell) {
    case LSTM: {
      Tensor v = at::empty({T, N, 4 * H}, o), tmp = at::empty({N, 4 * H}, o);
      CALL(lstm_forward, dt, tr, d.T, d.N, d.C, d.H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(x), h, c, ptr(v),
                                 ptr(tmp), zp, mp, s);
      f.saved = {v};
      break;
    }
    case GRU: {
      Tensor v = training ? at::empty({T, N, 4 * H}, o) : Tensor(), wx = at::empty({T, N, 3 * H}, o),
             tmp = at::empty({N, 3 * H}, o);
      CALL(gru_forward, dt, tr, d.T, d.N, d.C, d.H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(P[3]), ptr(x), h,
                                ptr(v), ptr(wx), ptr(tmp), zp, mp, s);
      f.saved = {v};
      break;
    }
    case INDRNN: {
      Tensor ws = at::empty({T, N, H}, o);
      CALL(indrnn_forward, dt, tr, d.T, d.N, d.C, d.H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(x), h, ptr(ws), zp,
                                   mp, s);
      break;
    }
    case LN_LSTM: {
      Tensor wx = at::empty({T, N, 4 * H}, so), wxn = at::empty({T, N, 4 * H}, so), k1 = at::empty({T, N, 2}, so),
             rh = at::empty({T, N, 4 * H}, so), k2 = at::empty({T, N, 2}, so), cn = at::empty({T, N, H}, so),
             k3 = at::empty({T, N, 2}, so), tmp = at::empty({N, 4 * H}, so);
      char* g = static_cast<char*>(P[3].data_ptr());
      CALL(layer_norm_lstm_forward, dt, tr, d.T, d.N, d.C, d.H, ptr(P[0]), ptr(P[1]), ptr(P[2]), g,
                                            g + 4 * H * P[3].element_size(), ptr(P[4]), ptr(P[5]), ptr(x), h, c, ptr(wx),
                                            ptr(wxn), ptr(k1), ptr(rh), ptr(k2), ptr(cn), ptr(k3), ptr(tmp), zp, mp, s);
      f.saved = {wx, wxn, k1, rh, k2, cn, k3};
      break;
    }
    case LN_GRU: {
      Tensor v = training ? at::empty({T, N, 4 * H}, o) : Tensor(), wx = at::empty({T, N, 3 * H}, o),
             wxn = at::empty({T, N, 3 * H}, o), k1 = at::empty({T, N, 2}, o), rh = at::empty({T, N, 3 * H}, o),
             tmp = at::empty({N, 3 * H}, o), k2 = at::empty({T, N, 2}, o);
      char* g = static_cast<char*>(P[4].data_ptr());
      CALL(layer_norm_gru_forward, dt, tr, d.T, d.N, d.C, d.H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(P[3]), g,
                                           g + 3 * H * P[4].element_size(), ptr(x), h, ptr(v), ptr(wx), ptr(k1),
                                           ptr(wxn), ptr(rh), ptr(k2), ptr(tmp), zp, mp, s);
      f.saved = {v, wx, k1, rh, k2};
      break;
    }
    default: {
      Tensor ws = at::empty({T, N, H}, o), wx = at::empty({T, N, H}, o), k1 = at::empty({T, N, 2}, o);
      CALL(layer_norm_indrnn_forward, dt, tr, d.T, d.N, d.C, d.H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(P[3]),
                                              ptr(x), h, ptr(ws), ptr(wx), ptr(k1), zp, mp, s);
      f.saved = {wx, k1};
    }
  }
  return f;
}

// Incoming gradient of a sequence as the library takes it: a pointer one slot before it (the library
// never reads that slot).  Undefined: `zero` makes it zeros, else null.
void* incoming(Tensor& g, const Tensor& hs, bool zero) {
  if (!g.defined()) {
    if (!zero) return nullptr;
    g = at::zeros({hs.size(0) - 1, hs.size(1), hs.size(2)}, hs.options());
  }
  g = g.contiguous();
  return slot0(g);
}

struct RnnNode : public torch::autograd::Function<RnnNode> {
  static variable_list forward(AutogradContext* ctx, int64_t cell, bool training, double zoneout, int64_t budget,
                               Tensor x, c10::optional<Tensor> h0, c10::optional<Tensor> c0,
                               c10::optional<Tensor> mask_, at::TensorList params) {
    const Tensor mask = mask_.value_or(Tensor());
    Forward f = run_forward((int)cell, training, zoneout, x, h0.value_or(Tensor()), c0.value_or(Tensor()), mask, params);
    variable_list save = {x, mask, whole(f.y)};
    if (f.c.defined()) save.push_back(whole(f.c));
    for (const Tensor& t : params) save.push_back(t);
    int64_t kept = 0;
    for (const Tensor& t : f.saved) {
      save.push_back(t);
      kept += t.defined() ? t.numel() : 0;
    }
    ctx->saved_data["kept"] = kept;
    ctx->save_for_backward(std::move(save));
    ctx->saved_data["cell"] = cell;
    ctx->saved_data["training"] = training;
    ctx->saved_data["budget"] = budget;
    ctx->saved_data["has_h0"] = h0.has_value();
    ctx->saved_data["has_c0"] = c0.has_value();
    ctx->saved_data["params"] = (int64_t)params.size();
    ctx->set_materialize_grads(false);
    variable_list out = {f.y};
    if (f.c.defined()) out.push_back(f.c);
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grad) {
    try {
      return gradients(ctx, grad);
    } catch (const LibraryError& e) {  // keeps its Python type on the way through the engine
      py::gil_scoped_acquire gil;
      PyErr_SetString(haste_error, e.what());
      python_error error;
      error.persist();
      throw error;
    }
  }

  static variable_list gradients(AutogradContext* ctx, variable_list& grad) {
    const int cell = (int)ctx->saved_data["cell"].toInt();
    static const char* names[] = {"LSTM", "GRU", "IndRNN", "LayerNormLSTM", "LayerNormGRU", "LayerNormIndRNN"};
    TORCH_CHECK(ctx->saved_data["training"].toBool(), names[cell], " backward can only be called in training mode");
    const SmBudget sm((int)ctx->saved_data["budget"].toInt());
    const size_t np = (size_t)ctx->saved_data["params"].toInt();
    variable_list sv = ctx->get_saved_variables();
    for (Tensor& t : sv)  // hooks may hand back tensors of their own
      if (t.defined()) t = t.contiguous();
    const Tensor x = sv[0], mask = sv[1], hs = sv[2];
    size_t i = 3;
    const Tensor cs = has_c(cell) ? sv[i++] : Tensor();
    const variable_list P(sv.begin() + i, sv.begin() + i + np);
    const variable_list S(sv.begin() + i + np, sv.end());
    const int T = (int)x.size(0), N = (int)x.size(1), C = (int)x.size(2), H = (int)hs.size(2);
    check(x, P);
    check(x, {mask, hs, cs});
    check_sizes(cell, x, H, P, &mask);
    const int64_t values = (int64_t)(T + 1) * N * H;
    bool same = hs.numel() == values && (!cs.defined() || cs.numel() == values);
    int64_t kept = 0;
    for (const Tensor& t : S) {
      kept += t.defined() ? t.numel() : 0;
      same &= !t.defined() || (t.device() == x.device() && t.dtype() == saved_options(x, cell).dtype());
    }
    TORCH_CHECK(same && kept == ctx->saved_data["kept"].toInt(), "haste_b200: a saved tensor has changed its kind");
    const c10::cuda::CUDAGuard guard(x.device());
    void* s = (void*)c10::cuda::getCurrentCUDAStream().stream();
    const auto o = x.options();
    const int dt = lib_dtype(x, cell);
    void* gh = incoming(grad[0], hs, true);
    void* gc = has_c(cell) ? incoming(grad[1], hs, false) : nullptr;
    const bool want_x = cell == LN_LSTM || cell == LN_GRU || ctx->needs_input_grad(0);
    Tensor dx = want_x ? at::empty(x.sizes(), o) : Tensor();
    Tensor dh = at::empty({N, H}, o), dc = has_c(cell) ? at::empty({N, H}, o) : Tensor();
    variable_list D;
    for (const Tensor& t : P) D.push_back(at::empty(t.sizes(), o));
    const AssignGradients assign;
    switch (cell) {
      case LSTM:
        CALL(lstm_backward, dt, 0, T, N, C, H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(x), ptr(hs), ptr(cs), gh,
                                    gc, ptr(dx), ptr(D[0]), ptr(D[1]), ptr(D[2]), ptr(dh), ptr(dc), ptr(S[0]), ptr(mask),
                                    s);
        break;
      case GRU: {
        Tensor dp = at::empty({T, N, 3 * H}, o), dq = at::empty({T, N, 3 * H}, o);
        CALL(gru_backward, dt, 0, T, N, C, H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(P[3]), ptr(x), ptr(hs),
                                   ptr(S[0]), gh, ptr(dx), ptr(D[0]), ptr(D[1]), ptr(D[2]), ptr(D[3]), ptr(dh), ptr(dp),
                                   ptr(dq), ptr(mask), s);
        break;
      }
      case INDRNN: {
        Tensor ws = at::empty({T, N, H}, o);
        CALL(indrnn_backward, dt, 0, T, N, C, H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(x), ptr(hs), gh, ptr(dx),
                                      ptr(D[0]), ptr(D[1]), ptr(D[2]), ptr(dh), ptr(ws), ptr(mask), s);
        break;
      }
      case LN_LSTM: {
        const size_t row = (size_t)4 * H * P[3].element_size();
        char *g = static_cast<char*>(P[3].data_ptr()), *dg = static_cast<char*>(D[3].data_ptr());
        CALL(layer_norm_lstm_backward, dt, 0, T, N, C, H, ptr(P[0]), ptr(P[1]), ptr(P[2]), g, g + row, ptr(P[4]),
                                               ptr(P[5]), ptr(x), ptr(hs), ptr(cs), gh, gc, ptr(dx), ptr(D[0]),
                                               ptr(D[1]), ptr(D[2]), dg, dg + row, ptr(D[4]), ptr(D[5]), ptr(dh), ptr(dc),
                                               ptr(S[0]), ptr(S[1]), ptr(S[2]), ptr(S[3]), ptr(S[4]), ptr(S[5]),
                                               ptr(S[6]), ptr(mask), s);
        break;
      }
      case LN_GRU: {
        Tensor dp = at::empty({T, N, 3 * H}, o), dq = at::empty({T, N, 3 * H}, o);
        const size_t row = (size_t)3 * H * P[4].element_size();
        char *g = static_cast<char*>(P[4].data_ptr()), *dg = static_cast<char*>(D[4].data_ptr());
        CALL(layer_norm_gru_backward, dt, 0, T, N, C, H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(P[3]), g, g + row,
                                              ptr(x), ptr(hs), ptr(S[0]), gh, ptr(dx), ptr(D[0]), ptr(D[1]), ptr(D[2]),
                                              ptr(D[3]), dg, dg + row, ptr(dh), ptr(dp), ptr(dq), ptr(S[1]), ptr(S[2]),
                                              ptr(S[3]), ptr(S[4]), ptr(mask), s);
        break;
      }
      default: {
        Tensor ws = at::empty({T, N, H}, o);
        // gamma is [2,H]; its second row takes no part and has a zero gradient
        cuda_ok(cudaMemsetAsync(D[3].data_ptr(), 0, D[3].numel() * D[3].element_size(), (cudaStream_t)s));
        CALL(layer_norm_indrnn_backward, dt, 0, T, N, C, H, ptr(P[0]), ptr(P[1]), ptr(P[2]), ptr(P[3]), ptr(x),
                                                 ptr(hs), gh, ptr(dx), ptr(D[0]), ptr(D[1]), ptr(D[2]), ptr(D[3]),
                                                 ptr(dh), ptr(ws), ptr(S[0]), ptr(S[1]), ptr(mask), s);
      }
    }
    variable_list out(4);  // cell, training, zoneout, budget
    out.push_back(dx);
    out.push_back(ctx->saved_data["has_h0"].toBool() ? dh : Tensor());
    out.push_back(ctx->saved_data["has_c0"].toBool() ? dc : Tensor());
    out.push_back(Tensor());  // mask
    out.insert(out.end(), D.begin(), D.end());
    return out;
  }
};

// One call of a layer with at least one row and one step: x [T,N,C] ([N,T,C] with batch_first),
// h0 / c0 [1,N,H] or None.  Returns (output, final h, final c or None) as BaseRNN.forward hands
// them out; `lengths` (a device tensor [N]) only without gradients.
std::tuple<Tensor, Tensor, c10::optional<Tensor>> forward(
    int cell, Tensor x, const c10::optional<Tensor>& h0_, const c10::optional<Tensor>& c0_,
    const c10::optional<Tensor>& lengths, std::vector<Tensor> params, const c10::optional<Tensor>& mask_, bool training,
    double zoneout, bool batch_first, bool state_sequence, int budget) {
  TORCH_CHECK(x.dim() == 3, "haste_b200: input must have three dimensions, got " + shape_of(x));
  if (batch_first) x = x.transpose(0, 1);
  x = x.contiguous();
  const int64_t T = x.size(0), N = x.size(1);
  const int64_t H = cell == INDRNN || cell == LN_INDRNN ? params[0].size(1) : params[1].size(0);
  auto state = [&](const c10::optional<Tensor>& t) {
    if (!t) return Tensor();
    TORCH_CHECK(t->dim() == 3 && t->size(0) == 1 && t->size(1) == N && t->size(2) == H, "haste_b200: state must be [1,N,H]");
    return t->requires_grad() ? t->select(0, 0).contiguous() : t->contiguous();  // [1,N,H] lies like [N,H]
  };
  Tensor h0 = state(h0_), c0 = state(c0_);
  Tensor mask = mask_ ? mask_->contiguous() : Tensor();
  bool graph = false;
  for (Tensor& p : params) p = p.contiguous();
  if (at::GradMode::is_enabled()) {
    graph = x.requires_grad() || (h0.defined() && h0.requires_grad()) || (c0.defined() && c0.requires_grad());
    for (const Tensor& p : params) graph |= p.requires_grad();
  }
  check(x, params);
  check(x, {h0, c0, mask});
  check_sizes(cell, x, H, params, training && zoneout != 0.0 ? &mask : nullptr);
  const c10::cuda::CUDAGuard guard(x.device());
  const SmBudget sm(budget);
  Tensor y, c;
  if (graph) {
    auto given = [](const Tensor& t) { return t.defined() ? c10::optional<Tensor>(t) : c10::nullopt; };
    const variable_list out = RnnNode::apply((int64_t)cell, training, zoneout, (int64_t)budget, x, given(h0), given(c0),
                                             given(mask), at::TensorList(params));
    y = out[0];
    if (out.size() > 1) c = out[1];
  } else if (T == 1 && !training && !lengths && (cell == LSTM || cell == GRU)) {
    // a single step: the state goes from buffer to buffer
    const int dt = dtype_of(x), n = (int)N, hh = (int)H, cc = (int)x.size(2), G = cell == LSTM ? 4 : 3;
    void* s = (void*)c10::cuda::getCurrentCUDAStream().stream();
    const bool zo = zoneout != 0.0 && mask.defined() && mask.numel();
    const float zp = zo ? (float)zoneout : 0.0f;
    const void* mp = zo ? mask.data_ptr() : nullptr;
    y = at::empty({1, N, H}, x.options());
    if (!h0.defined()) h0 = at::zeros({N, H}, x.options());
    if (cell == LSTM) {
      if (!c0.defined()) c0 = at::zeros({N, H}, x.options());
      c = at::empty({1, N, H}, x.options());
    }
    auto step = [&](void* t0, void* t1) {
      return cell == LSTM ? lib.lstm_forward_iterate(dt, 0, n, cc, hh, ptr(params[0]), ptr(params[1]), ptr(params[2]),
                                                     ptr(x), ptr(h0), ptr(c0), ptr(y), ptr(c), t0, t1, zp, mp, s)
                          : lib.gru_forward_iterate(dt, 0, n, cc, hh, ptr(params[0]), ptr(params[1]), ptr(params[2]),
                                                    ptr(params[3]), ptr(x), ptr(h0), ptr(y), nullptr, t0, t1, zp, mp, s);
    };
    // up to 64 rows the step is one kernel without scratch; what it does not take comes back at once
    int status = N > 64 ? HASTE_B200_ERR_INVALID : step(nullptr, nullptr);
    if (status == HASTE_B200_ERR_INVALID) {
      Tensor tmp = at::empty({2, N, G * H}, x.options());
      status = step(tmp.data_ptr(), static_cast<char*>(tmp.data_ptr()) + N * G * H * tmp.element_size());
    }
    ok(cell == LSTM ? "lstm_forward_iterate" : "gru_forward_iterate", status);
  } else {
    Forward f = run_forward(cell, training, zoneout, x, h0, c0, mask, params);
    y = f.y;
    c = f.c;
  }
  auto final_state = [&](const Tensor& seq) {
    if (state_sequence) return (batch_first ? seq.transpose(0, 1) : seq).unsqueeze(0);
    if (!lengths) return T == 1 && !graph ? seq : seq.narrow(0, T - 1, 1);
    // the state after lengths[n] steps: slot 0, the initial state, belongs to length 0
    const Tensor slots = seq.as_strided({T + 1, N, H}, {N * H, H, 1}, 0);
    return at::index(slots, {*lengths, at::arange(N, lengths->options().dtype(at::kLong))}).unsqueeze(0);
  };
  c10::optional<Tensor> cf;
  if (c.defined()) cf = final_state(c);
  return {batch_first ? y.transpose(0, 1) : y, final_state(y), cf};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const LibraryError& e) {
      PyErr_SetString(haste_error, e.what());
    }
  });
  m.def("load", &load);
  m.def("forward", &forward, py::call_guard<py::gil_scoped_release>());
}
