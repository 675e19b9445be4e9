// Host path of the Python modules in native code: the autograd nodes around the C ABI (include/spion_b200.h).
//
// A call through torch.autograd.Function costs 30 - 60 us of interpreter time in each direction, and an attention layer is six of
// them (projections, attention, output projection) plus casts, copies and reductions: 1.1 ms per forward + backward of a layer
// whose kernels take 50 us.  Here a layer is one node: projections, attention and output projection call the library
// back to back, in the layouts the next kernel reads, and the backward does the same.
//
// Only orchestration lives here; every kernel is behind the C ABI.
#include <torch/extension.h>
#include <ATen/SavedTensorHooks.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/Exceptions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <memory>
#include <mutex>
#include <vector>

#include "../../include/spion_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;
using c10::optional;

struct Failure : std::runtime_error { using std::runtime_error::runtime_error; };

void check(int rc, const char* what) {
  if (rc != 0) throw Failure(std::string(what) + " failed: " + spion_status_string(rc) + " (" + std::to_string(rc) + ")");
}

py::object& error_type() {
  static py::object* type = new py::object(py::module_::import("spion_b200._lib").attr("SpionError"));      // never destroyed
  return *type;
}
// A backward runs on a thread of the autograd engine, which turns C++ exceptions into RuntimeError: raise the library's own
// error there, as the forward does through the module's exception translator.
template <class F>
variable_list as_backward(F f) {
  try {
    return f();
  } catch (const Failure& e) {
    py::gil_scoped_acquire gil;
    PyErr_SetString(error_type().ptr(), e.what());
    python_error raised;
    raised.persist();
    throw raised;
  }
}

void* stream_of(const Tensor& t) { return (void*)c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
void* p(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
const float* pf(const Tensor& t) { return t.defined() ? (const float*)t.data_ptr() : nullptr; }

// The nodes below work on memory: they form no forward-mode tangents, and tracers, dispatch modes and transforms would not see what
// they do.  Calls under one of those take the way over torch operators and Python autograd functions, which they know.
bool plain(const Tensor& t) {
  static const c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::FuncTorchGradWrapper,
                                            c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::Functionalize, c10::DispatchKey::Negative,
                                            c10::DispatchKey::ZeroTensor});
  return !t.key_set().has_any(wrapped) && !t._fw_grad(0).defined();
}
bool plain(std::initializer_list<at::ArrayRef<Tensor>> lists) {
  if (torch::jit::tracer::isTracing() || c10::impl::TorchDispatchModeTLS::any_modes_set()) return false;
  for (const auto& ts : lists)
    for (const Tensor& t : ts)
      if (!plain(t)) return false;
  return true;
}

// ------------------------------------------------------------------------------------------------ token matrices
spion_tokens tok(const std::vector<Tensor>& ts, int cols) {
  spion_tokens t = {};
  t.count = (int)ts.size();
  for (int i = 0; i < t.count; ++i) t.ptr[i] = ts[i].data_ptr();
  t.cols = cols;
  t.is_bf16 = ts[0].scalar_type() == at::kBFloat16;
  return t;
}
spion_tokens tok_heads(const std::vector<Tensor>& ts, int H, int d, int L) {
  spion_tokens t = tok(ts, H * d);
  t.heads = H; t.head_dim = d; t.seq_len = L;
  return t;
}
bool aligned32(const Tensor& t) { return ((uintptr_t)t.data_ptr() & 31) == 0; }

struct Weights {                        // up to three stacked linear layers
  std::vector<Tensor> W, b;
  const float* copy = nullptr;          // instead of W: the stacked weights of `layers` equal layers
  int layers = 0, copy_in = 0, copy_out = 0;
  Weights() {}
  Weights(std::vector<Tensor> W_, std::vector<Tensor> b_) : W(std::move(W_)), b(std::move(b_)) {}
  Weights(const float* p, int n_layers, int64_t in_features, int64_t out_features)
      : copy(p), layers(n_layers), copy_in((int)in_features), copy_out((int)out_features) {}
  int n() const { return copy ? layers : (int)W.size(); }
  int in() const { return copy ? copy_in : (int)W[0].size(1); }
  int out() const { return copy ? copy_out : (int)(W[0].size(0) * W.size()); }
  const float* at(int i) const { return copy ? copy + (int64_t)i * (copy_out / layers) * copy_in : pf(W[i]); }
};

// What a mixed-precision backward reads in place of the input and the weights: as under the framework's own autocast, the caller may
// change both in between.  The forward's kernels write the copies on the way.
struct Kept {
  Tensor x, w;
  float* w_to = nullptr;                // where the weights go: w, or a part of a buffer that several layers share
  // x: the input (bf16 input is kept as it is); fp32 layers keep nothing
  Kept() {}
  Kept(bool need, bool fp32, const Tensor& X, const Weights& l, float* shared = nullptr) {
    if (!need || fp32) return;
    if (!shared) w = at::empty({l.out(), l.in()}, l.W[0].options());
    w_to = shared ? shared : (float*)w.data_ptr();
    if (X.scalar_type() == at::kFloat) x = at::empty(X.sizes(), X.options().dtype(at::kBFloat16));
  }
};
void linear_forward(const spion_tokens& X, const Weights& w, bool fp32, const spion_tokens& Y, void* gelu_out, int64_t T, void* st,
                    const Kept& kept = Kept()) {
  const float *W[3], *b[3];
  for (int i = 0; i < w.n(); ++i) { W[i] = pf(w.W[i]); b[i] = pf(w.b[i]); }
  check(spion_linear_forward_keep(&X, W, b, w.n(), fp32, &Y, gelu_out, p(kept.x), kept.w_to, T, w.in(), w.out(), st),
        "spion_linear_forward_keep");
}
// the projections of a layer with padded keys, and the penalties of its attention
void linear_forward_keypad(const spion_tokens& X, const Weights& w, bool fp32, const spion_tokens& Y, int64_t T, void* st, const Kept& kept,
                           const Tensor& mask, int B, int H, int L, const Tensor& pen) {
  const float *W[3], *b[3];
  for (int i = 0; i < w.n(); ++i) { W[i] = pf(w.W[i]); b[i] = pf(w.b[i]); }
  check(spion_linear_forward_keypad(&X, W, b, w.n(), fp32, &Y, p(kept.x), kept.w_to, T, w.in(), w.out(), pf(mask), B, H, L, (float*)p(pen), st),
        "spion_linear_forward_keypad");
}
void linear_backward_input(const spion_tokens& dY, const Weights& w, bool fp32, const void* gelu_in, const spion_tokens& dX, int64_t T, void* st) {
  const float* W[3];
  for (int i = 0; i < w.n(); ++i) W[i] = w.at(i);
  check(spion_linear_backward_input(&dY, W, w.n(), fp32, gelu_in, &dX, T, w.in(), w.out(), st), "spion_linear_backward_input");
}
// Weight and bias gradients of the stacked layers from dY (one [T, per] matrix per layer, or their head-split form) and X.
// fp32 tokens (or the copy kept of them): the library's kernel, views of one buffer.  bf16 tokens (a layer inside a mixed-precision
// encoder): the framework's bf16 products and the column-sum kernel, so that a training step repeats bit for bit what separate layers give.
void linear_backward_weight(const std::vector<Tensor>& dY, const spion_tokens& tY, const Tensor& X, const spion_tokens& tX, const Weights& w,
                            bool fp32, int64_t T, void* st, std::vector<Tensor>& dW, std::vector<Tensor>& db, bool copied = false) {
  const int64_t in = w.in(), out = w.out(), per = out / w.n();
  const auto opt = X.options().dtype(at::kFloat);
  if (tX.is_bf16 && !copied && tY.heads == 0 && tX.heads == 0) {
    Tensor x2 = X.view({T, in});
    const int n = w.n();
    Tensor prod = at::empty({out, in}, x2.options());        // the products side by side: one conversion for all of them, beside the sums
    std::vector<const void*> dys;
    for (int i = 0; i < n; ++i) {
      Tensor dy2 = dY[i].view({T, per}), part = prod.narrow(0, i * per, per);
      at::mm_out(part, dy2.t(), x2);
      dys.push_back(dy2.data_ptr());
    }
    Tensor g32, sums;
    const bool kernel = per == 64 || per == 128 || per == 256 || per == 512;
    if (kernel) {
      sums = at::empty({out}, opt);
      Tensor ws = at::empty({(int64_t)n * spion_layernorm_workspace_floats((int)per)}, opt);
      g32 = at::empty({out, in}, opt);
      check(spion_column_sums_convert(dys.data(), n, 1, (float*)sums.data_ptr(), (float*)ws.data_ptr(), T, (int)per, prod.data_ptr(),
                                      (float*)g32.data_ptr(), out * in, st), "spion_column_sums_convert");
    } else {
      g32 = prod.to(at::kFloat);
    }
    for (int i = 0; i < n; ++i) {
      dW.push_back(g32.narrow(0, i * per, per));
      db.push_back(kernel ? sums.narrow(0, i * per, per) : dY[i].view({T, per}).sum(0).to(at::kFloat));
    }
    return;
  }
  Tensor g = at::empty({out * in + out}, opt);
  Tensor ws = at::empty({(int64_t)spion_linear_workspace_floats(T, (int)in, (int)out, fp32)}, opt);
  float* gp = (float*)g.data_ptr();
  check(spion_linear_backward_weight(&tY, &tX, fp32, gp, gp + out * in, (float*)ws.data_ptr(), T, (int)in, (int)out, st),
        "spion_linear_backward_weight");
  for (int i = 0; i < w.n(); ++i) {
    dW.push_back(g.narrow(0, i * per * in, per * in).view({per, in}));
    db.push_back(g.narrow(0, out * in + i * per, per));
  }
}

bool weights_ok(const std::vector<Tensor>& W, const std::vector<Tensor>& b, const Tensor& like, bool fp32) {
  const int64_t in = W[0].size(1), out = W[0].size(0);
  for (size_t i = 0; i < W.size(); ++i) {
    if (W[i].scalar_type() != at::kFloat || !W[i].is_contiguous() || W[i].device() != like.device() || !aligned32(W[i])) return false;
    if (!b[i].defined() || b[i].scalar_type() != at::kFloat || !b[i].is_contiguous() || b[i].device() != like.device()) return false;
    if (W[i].size(0) != out || W[i].size(1) != in) return false;
  }
  return spion_linear_supported((int)in, (int)(out * W.size()), fp32) != 0;
}

// ------------------------------------------------------------------------------------------------ attention context
enum Mode { NATIVE = 0, DROPIN_SPARSE = 1, DROPIN_DENSE = 2 };

// What the Python modules keep per attention context: the C ABI's handle and the sizes it was created with.  The handle has a
// stream, a head layout and a mask of its own: `mutex` is held from setting them to the last launch that reads them, and never
// waited for by a thread that holds the interpreter's lock (the holder may need that one).
struct Context {
  int64_t handle = 0;
  int mode = NATIVE;
  int64_t B = 0, H = 0, L = 0, d = 0;
  int device = 0;
  bool bf16 = false, keypad = false, fused = false, recompute = false, return_probs = true, needs_scratch = false;
  bool rounded = false;                 // not recompute: rebuilt tiles too, but of the rounded probabilities
  bool owned = false;                   // destroys the handle
  int64_t nnz = 0;                      // selected elements per (b,h) matrix
  Tensor sum_mat, offsets, columns;     // element CSR of the drop-in layout
  Tensor mask;                          // native: the block mask [nb, nb] the handle is set to; generation counts the masks
  int64_t generation = 0;
  std::mutex mutex;
  spion_ctx* ctx() const { return reinterpret_cast<spion_ctx*>(handle); }
  at::ScalarType type() const { return bf16 ? at::kBFloat16 : at::kFloat; }
  void close() { if (owned && handle) { spion_destroy(ctx()); } handle = 0; }
  ~Context() { close(); }
};
using ContextPtr = std::shared_ptr<Context>;

std::string shape_str(const Tensor& t) {
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + ")";
}

// Names the contents of a mask tensor, so that the structure derived from it can be kept: storage, view of it and version.  The alias
// keeps the storage alive (its address cannot be handed to another mask) and shares the version counter.
struct MaskKey {
  Tensor alias;
  int64_t version = -1;
  bool matches(const Tensor& t) const {
    return alias.defined() && t.data_ptr() == alias.data_ptr() && (int64_t)t._version() == version && t.sizes() == alias.sizes() &&
           t.strides() == alias.strides() && t.scalar_type() == alias.scalar_type() && t.device() == alias.device();
  }
  void set(const Tensor& t) {
    alias = t.detach();
    version = (int64_t)t._version();
  }
};

// native contexts: a new block mask (uint8 [nb, nb] on the context's device, owned by the caller's module and never changed)
void set_pattern(const ContextPtr& c, const Tensor& mask, int64_t bs) {
  py::gil_scoped_release nogil;
  if (mask.numel() < (c->L / bs) * (c->L / bs))
    throw Failure("block mask has shape " + shape_str(mask) + ", this module needs " + std::to_string(c->L / bs) + " blocks per side");
  c10::cuda::CUDAGuard guard(c->device);
  std::lock_guard<std::mutex> hold(c->mutex);
  check(spion_set_stream(c->ctx(), (void*)c10::cuda::getCurrentCUDAStream(c->device).stream()), "spion_set_stream");
  c->mask = mask;
  ++c->generation;
  check(spion_set_pattern(c->ctx(), (const uint8_t*)mask.data_ptr()), "spion_set_pattern");
  c->nnz = (int64_t)spion_pattern_nnzb(c->ctx()) * bs * bs;
}

void check_operand(const Context& c, const Tensor& t, const char* name) {
  if (t.dim() != 4 || t.size(0) != c.B || t.size(1) != c.H || t.size(2) != c.L || t.size(3) != c.d)
    throw Failure(std::string(name) + " has shape " + shape_str(t) + ", this module was built for (" + std::to_string(c.B) + ", " +
                  std::to_string(c.H) + ", " + std::to_string(c.L) + ", " + std::to_string(c.d) +
                  ") (batch_size, num_head, max_seq_len, head_dim of its config)");
  if (!t.is_cuda() || t.device().index() != c.device)
    throw Failure(std::string(name) + " is on " + t.device().str() + ", the module's context is on cuda:" + std::to_string(c.device));
}

// key-padding mask [B, L] of 1 / 0 as floats.  The drop-in modules expand a mask of one sequence or of one key.
Tensor key_mask(const Context& c, const Tensor& mask, const Tensor& like) {
  auto fits = [&](int i, int64_t n) { return mask.size(i) == n || (c.mode != NATIVE && mask.size(i) == 1); };
  if (!mask.defined() || mask.dim() != 2 || !fits(0, c.B) || !fits(1, c.L))
    throw Failure("key-padding mask must have shape (" + std::to_string(c.B) + ", " + std::to_string(c.L) + ")");
  return mask.to(like.device(), at::kFloat).expand({c.B, c.L}).contiguous();
}
Tensor empty_penalty(const Context& c, const Tensor& like) { return at::empty({c.B, c.H, c.L}, like.options().dtype(at::kFloat)); }
// ... -> penalty per (b,h) matrix [BH, L]
Tensor penalty(const Context& c, const Tensor& mask, const Tensor& like, void* st) {
  Tensor m = key_mask(c, mask, like), pen = empty_penalty(c, like);
  check(spion_expand_keypad(pf(m), (int)c.B, (int)c.H, (int)c.L, (float*)pen.data_ptr(), st), "spion_expand_keypad");
  return pen;
}

// One forward call: operands in, results out (everything the backward needs).
struct Attn {
  Tensor q, k, v, pen, O, lse, P, stat; // stat: what the rounded P are rebuilt from
  int heads = 0;                        // 0: operands [B, H, L, d] contiguous; H: views of [B, L, H, d]
  // the mask the forward ran on (drop-in: as element CSR); the context may move on to another before the backward
  Tensor sum_mat, offsets, columns, mask;
  int64_t nnz = 0, generation = 0;
};

Tensor empty_operand(const Context& c, int heads, const Tensor& like) {
  const auto opt = like.options().dtype(c.type());
  if (heads) return at::empty({c.B, c.L, c.H, c.d}, opt).transpose(1, 2);
  return at::empty({c.B, c.H, c.L, c.d}, opt);
}
// 0: contiguous [B, H, L, d]; H: the head-split view of a contiguous [B, L, H, d] tensor; -1: neither
int operand_form(const Context& c, const Tensor& t) {
  if (t.is_contiguous()) return 0;
  if (t.stride(0) == c.L * c.H * c.d && t.stride(1) == c.d && t.stride(2) == c.H * c.d && t.stride(3) == 1) return (int)c.H;
  return -1;
}

// need: a backward may follow
void attn_forward(Context& c, Attn& a, bool need, void* st) {
  spion_ctx* x = c.ctx();
  const auto f32 = a.q.options().dtype(at::kFloat);
  std::lock_guard<std::mutex> hold(c.mutex);
  a.nnz = c.nnz;
  check(spion_set_stream(x, st), "spion_set_stream");
  if (c.mode == DROPIN_SPARSE) {
    a.sum_mat = c.sum_mat; a.offsets = c.offsets; a.columns = c.columns;
    a.O = empty_operand(c, 0, a.q);
    a.P = at::empty({c.B * c.H * a.nnz}, f32);
    check(spion_block_attn_forward_rm(x, pf(a.q), pf(a.k), pf(a.v), pf(a.pen), (float*)a.P.data_ptr(), (float*)a.O.data_ptr(),
                                      (const int*)a.offsets.data_ptr(), (const int*)a.columns.data_ptr(),
                                      (const int*)a.sum_mat.data_ptr(), (int)a.nnz), "spion_block_attn_forward_rm");
    return;
  }
  if (c.mode == DROPIN_DENSE) {
    a.O = empty_operand(c, 0, a.q);
    a.P = at::empty({c.B, c.H, c.L, c.L}, f32);
    check(spion_dense_attn_forward_rm(x, pf(a.q), pf(a.k), pf(a.v), pf(a.pen), (float*)a.P.data_ptr(), (float*)a.O.data_ptr()),
          "spion_dense_attn_forward_rm");
    return;
  }
  a.mask = c.mask; a.generation = c.generation;
  check(spion_set_head_layout(x, a.heads), "spion_set_head_layout");
  a.O = empty_operand(c, a.heads, a.q);
  if (c.fused) {
    a.lse = at::empty({c.B * c.H * c.L}, f32);
    // under hooks on saved tensors the backward reads the P that they hand back
    if (need && c.rounded && !c.recompute && !at::SavedTensorDefaultHooks::get_hooks()) {
      a.stat = at::empty({2 * c.B * c.H * c.L}, f32);
      if (c.return_probs) a.P = at::empty({c.B * c.H * a.nnz}, a.q.options());
      check(spion_attn_forward_probs(x, p(a.q), p(a.k), p(a.v), pf(a.pen), p(a.O), (float*)a.lse.data_ptr(), p(a.P), (float*)a.stat.data_ptr()),
            "spion_attn_forward_probs");
      return;
    }
    // the probabilities are stored only for callers that want them back and for a backward that reads them
    if (c.return_probs || (need && !c.recompute)) a.P = at::empty({c.B * c.H * a.nnz}, a.q.options());
    check(spion_attn_forward_fused(x, p(a.q), p(a.k), p(a.v), pf(a.pen), p(a.O), (float*)a.lse.data_ptr(), p(a.P)),
          "spion_attn_forward_fused");
  } else {
    a.P = at::empty({c.B * c.H * a.nnz}, a.q.options());
    Tensor scratch;
    if (c.needs_scratch) scratch = at::empty({c.B * c.H * a.nnz}, f32);
    check(spion_attn_forward_ex(x, p(a.q), p(a.k), p(a.v), pf(a.pen), p(a.P), p(a.O), (float*)p(scratch)), "spion_attn_forward_ex");
  }
}

// Runs f with the handle set to the forward's mask.  A module that has been given another mask since takes it back afterwards; both
// read the mask's size back, so such a backward cannot be captured.
template <class F>
void on_mask_of(const Context& c, const Attn& a, F f) {
  if (c.mode != NATIVE || a.generation == c.generation) return f();
  check(spion_set_pattern(c.ctx(), (const uint8_t*)a.mask.data_ptr()), "spion_set_pattern");
  try {
    f();
  } catch (...) {
    spion_set_pattern(c.ctx(), (const uint8_t*)c.mask.data_ptr());
    throw;
  }
  check(spion_set_pattern(c.ctx(), (const uint8_t*)c.mask.data_ptr()), "spion_set_pattern");
}

void attn_backward_on(const Context& c, const Attn& a, const Tensor& dO, Tensor& dq, Tensor& dk, Tensor& dv);
void attn_backward(Context& c, const Attn& a, const Tensor& dO, Tensor& dq, Tensor& dk, Tensor& dv, void* st) {
  std::lock_guard<std::mutex> hold(c.mutex);
  check(spion_set_stream(c.ctx(), st), "spion_set_stream");
  on_mask_of(c, a, [&] { attn_backward_on(c, a, dO, dq, dk, dv); });
}

void attn_backward_on(const Context& c, const Attn& a, const Tensor& dO, Tensor& dq, Tensor& dk, Tensor& dv) {
  spion_ctx* x = c.ctx();
  const auto f32 = a.q.options().dtype(at::kFloat);
  dq = empty_operand(c, a.heads, a.q); dk = empty_operand(c, a.heads, a.q); dv = empty_operand(c, a.heads, a.q);
  if (c.mode == DROPIN_SPARSE) {
    Tensor dS = at::empty({c.B * c.H * a.nnz}, f32);
    Tensor dP;
    if (spion_block_attn_needs_scratch(x)) dP = at::empty({c.B * c.H * a.nnz}, f32);
    check(spion_block_attn_backward_rm(x, pf(a.q), pf(a.k), pf(a.v), pf(a.P), pf(a.O), pf(dO), (float*)p(dP), (float*)dS.data_ptr(),
                                       (float*)dq.data_ptr(), (float*)dk.data_ptr(), (float*)dv.data_ptr(),
                                       (const int*)a.offsets.data_ptr(), (const int*)a.columns.data_ptr(),
                                       (const int*)a.sum_mat.data_ptr(), (int)a.nnz), "spion_block_attn_backward_rm");
    return;
  }
  if (c.mode == DROPIN_DENSE) {
    const long long n = spion_dense_attn_scratch_floats(x);
    Tensor s1, s3;
    if (n > 0) { s1 = at::empty({n}, f32); s3 = at::empty({n}, f32); }
    check(spion_dense_attn_backward_rm(x, pf(a.q), pf(a.k), pf(a.v), pf(a.P), pf(a.O), pf(dO), (float*)p(s1), (float*)p(s3),
                                       (float*)dq.data_ptr(), (float*)dk.data_ptr(), (float*)dv.data_ptr()),
          "spion_dense_attn_backward_rm");
    return;
  }
  check(spion_set_head_layout(x, a.heads), "spion_set_head_layout");
  if (a.stat.defined()) {
    check(spion_attn_backward_probs(x, p(a.q), p(a.k), p(a.v), p(a.O), p(dO), pf(a.stat), pf(a.pen), p(dq), p(dk), p(dv)),
          "spion_attn_backward_probs");
    return;
  }
  if (c.fused && !a.P.defined()) {
    check(spion_attn_backward_fused(x, p(a.q), p(a.k), p(a.v), p(a.O), p(dO), pf(a.lse), pf(a.pen), p(dq), p(dk), p(dv)),
          "spion_attn_backward_fused");
    return;
  }
  Tensor dS = at::empty({c.B * c.H * a.nnz}, a.q.options()), scratch;
  if (!c.fused && c.needs_scratch) scratch = at::empty({c.B * c.H * a.nnz}, f32);
  check(spion_attn_backward_ex(x, p(a.q), p(a.k), p(a.v), p(a.P), p(a.O), p(dO), p(dS), (float*)p(scratch), nullptr, p(dq), p(dk), p(dv)),
        "spion_attn_backward_ex");
}

// ------------------------------------------------------------------------------------------------ autograd nodes
SavedVariable save(const Tensor& t) { return SavedVariable(t, false); }

// What a backward reads of its forward, as saved variables: a tensor that a caller also holds (the output, the probabilities) is
// checked for changes since, and hooks on saved tensors see all of them.
struct SavedAttn {
  // P is saved beside stat as well: a change of what the caller holds is an error
  SavedVariable q, k, v, pen, O, lse, P, stat, sum_mat, offsets, columns;
  Attn rest;
  // q_in, k_in, v_in: the caller's tensors where the kernels read them in place, else what a holds
  void save_all(const Attn& a, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in) {
    q = save(q_in); k = save(k_in); v = save(v_in);
    pen = save(a.pen); O = save(a.O); lse = save(a.lse); P = save(a.P); stat = save(a.stat);
    sum_mat = save(a.sum_mat); offsets = save(a.offsets); columns = save(a.columns);
    rest.heads = a.heads; rest.mask = a.mask; rest.nnz = a.nnz; rest.generation = a.generation;
  }
  Attn unpack(const Context& c) const {
    Attn a = rest;
    // a hook may hand a tensor back in other strides
    auto operand = [&](const SavedVariable& s) {
      Tensor t = s.unpack();
      if (!a.heads) return t.contiguous();
      return operand_form(c, t) == a.heads ? t : t.transpose(1, 2).contiguous().transpose(1, 2);
    };
    auto values = [](const SavedVariable& s) { Tensor t = s.unpack(); return t.defined() ? t.contiguous() : t; };
    a.q = operand(q); a.k = operand(k); a.v = operand(v); a.O = operand(O);
    a.pen = values(pen); a.lse = values(lse); a.P = values(P); a.stat = values(stat);
    a.sum_mat = values(sum_mat); a.offsets = values(offsets); a.columns = values(columns);
    return a;
  }
  void reset() {
    for (SavedVariable* s : {&q, &k, &v, &pen, &O, &lse, &P, &stat, &sum_mat, &offsets, &columns}) s->reset_data();
    rest = Attn();
  }
};

// A backward that is itself recorded (create_graph) is formed by torch operators from tensors that are part of the graph, as far as
// the forward was: linear layers are differentiated again, the attention's gradients are constants, as they have always been.
bool recorded() { return at::GradMode::is_enabled(); }
struct OutsideAutocast { c10::impl::ExcludeDispatchKeyGuard guard{c10::autocast_dispatch_keyset}; };

struct AttnNode : public Node {
  ContextPtr c;
  SavedAttn saved;
  at::ScalarType tq, tk, tv;
  bool released = false;
  std::string name() const override { return "BlockSparseAttentionBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    saved.reset();
    released = true;
  }
  variable_list apply(variable_list&& grads) override {
    return as_backward([&] { return backward(grads); });
  }
  variable_list backward(const variable_list& grads) {
    std::lock_guard<std::mutex> lock(mutex_);
    TORCH_CHECK(!released, "Trying to backward through the graph a second time (the saved tensors have been freed)");
    variable_list out(3);
    if (!grads[0].defined()) return out;
    c10::cuda::CUDAGuard guard(c->device);
    const Attn s = saved.unpack(*c);
    Tensor go = grads[0].to(c->type());
    if (s.heads && operand_form(*c, go) != s.heads) go = go.transpose(1, 2).contiguous().transpose(1, 2);
    else if (!s.heads) go = go.contiguous();
    Tensor dq, dk, dv;
    attn_backward(*c, s, go, dq, dk, dv, stream_of(go));
    out[0] = dq.to(tq); out[1] = dk.to(tk); out[2] = dv.to(tv);
    return out;
  }
};

struct Result {
  Tensor out;
  Attn a;
};
// out, probs (None when none were stored), lse, pen, q used, k used, heads; f runs without the interpreter's lock
template <class F>
py::tuple as_tuple(F f) {
  Result r;
  {
    py::gil_scoped_release nogil;
    r = f();
  }
  auto or_none = [](const Tensor& t) -> py::object { return t.defined() ? py::cast(t) : py::none(); };
  return py::make_tuple(r.out, or_none(r.a.P), or_none(r.a.lse), or_none(r.a.pen), r.a.q, r.a.k, r.a.heads);
}

// attention(q, k, v)
Result attention(const ContextPtr& c, const Tensor& query, const Tensor& key, const Tensor& value, const optional<Tensor>& mask) {
  check_operand(*c, query, "query");
  check_operand(*c, key, "key");
  check_operand(*c, value, "value");
  c10::cuda::CUDAGuard guard(c->device);
  void* st = stream_of(query);
  const bool need = at::GradMode::is_enabled() && (query.requires_grad() || key.requires_grad() || value.requires_grad());
  Attn a;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (c->keypad) a.pen = penalty(*c, mask.has_value() ? *mask : Tensor(), query, st);
    a.q = query.detach().to(c->type()); a.k = key.detach().to(c->type()); a.v = value.detach().to(c->type());
    // head-split views of [B, L, H*d] projections are read where they lie; anything else is packed
    if (c->fused && operand_form(*c, a.q) == c->H && operand_form(*c, a.k) == c->H && operand_form(*c, a.v) == c->H) a.heads = (int)c->H;
    if (!a.heads) { a.q = a.q.contiguous(); a.k = a.k.contiguous(); a.v = a.v.contiguous(); }
    attn_forward(*c, a, need, st);
  }
  Tensor out = a.O;
  if (need) {
    auto node = std::shared_ptr<AttnNode>(new AttnNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(query, key, value));
    node->c = c;
    node->tq = query.scalar_type(); node->tk = key.scalar_type(); node->tv = value.scalar_type();
    Attn kept = a;
    if (c->fused && c->recompute) kept.P = Tensor();
    auto in_place = [](const Tensor& in, const Tensor& used) { return used.data_ptr() == in.data_ptr() ? in : used; };
    node->saved.save_all(kept, in_place(query, a.q), in_place(key, a.k), in_place(value, a.v));
    out = a.O.detach();                  // shares the version counter of what was saved
    torch::autograd::set_history(out, node);
  }
  return Result{out, a};
}

struct LinearNode : public Node {
  bool fp32 = false;
  SavedVariable x, w;
  at::ScalarType out_type, x_type;
  std::string name() const override { return "TokenLinearBackward"; }
  void release_variables() override { std::lock_guard<std::mutex> lock(mutex_); x.reset_data(); w.reset_data(); }
  variable_list apply(variable_list&& grads) override {
    return as_backward([&] { return backward(grads); });
  }
  variable_list backward(const variable_list& grads) {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(3);
    if (!grads[0].defined()) return out;
    Tensor X = x.unpack();
    Weights l; l.W.push_back(w.unpack());
    c10::cuda::CUDAGuard guard(X.device());
    if (recorded()) {
      OutsideAutocast outside;
      const Tensor go = grads[0].to(out_type).reshape({-1, l.out()}), x2 = X.to(out_type).reshape({-1, l.in()});
      if (task_should_compute_output(0)) out[0] = go.matmul(l.W[0].to(out_type)).reshape(X.sizes()).to(x_type);
      if (task_should_compute_output(1)) out[1] = go.t().matmul(x2).to(at::kFloat);
      if (task_should_compute_output(2)) out[2] = go.sum(0).to(at::kFloat);
      return out;
    }
    if (!X.is_contiguous() || !aligned32(X)) X = X.contiguous().clone();
    Tensor go = grads[0].to(out_type).contiguous();
    if (!aligned32(go)) go = go.clone();
    void* st = stream_of(X);
    const int64_t T = X.numel() / l.in();
    const spion_tokens tg = tok({go}, l.out());
    if (task_should_compute_output(1) || task_should_compute_output(2)) {
      std::vector<Tensor> dW, db;
      linear_backward_weight({go}, tg, X, tok({X}, l.in()), l, fp32, T, st, dW, db, X.scalar_type() != x_type);
      out[1] = dW[0]; out[2] = db[0];
    }
    if (task_should_compute_output(0)) {
      out[0] = at::empty(X.sizes(), X.options().dtype(x_type));
      linear_backward_input(tg, l, fp32, nullptr, tok({out[0]}, l.in()), T, st);
    }
    return out;
  }
};

// The attention call of a forward that has been made, as a node over other (equal) operands
Tensor as_node(const ContextPtr& c, const Attn& a, const Tensor& query, const Tensor& key, const Tensor& value) {
  auto node = std::shared_ptr<AttnNode>(new AttnNode(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(query, key, value));
  node->c = c;
  node->tq = query.scalar_type(); node->tk = key.scalar_type(); node->tv = value.scalar_type();
  node->saved.save_all(a, a.q, a.k, a.v);
  Tensor out = a.O.detach();
  torch::autograd::set_history(out, node);
  return out;
}
// The same for a linear layer; its inputs are given by their edges, its operands by what was saved of them.
Tensor as_linear_node(const Tensor& y, bool fp32, const Tensor& x, const Tensor& w, at::ScalarType x_type, torch::autograd::edge_list edges) {
  auto node = std::shared_ptr<LinearNode>(new LinearNode(), torch::autograd::deleteNode);
  node->set_next_edges(std::move(edges));
  node->fp32 = fp32; node->x = save(x); node->w = save(w); node->out_type = y.scalar_type(); node->x_type = x_type;
  Tensor out = y.detach();
  torch::autograd::set_history(out, node);
  return out;
}

// Column sums of dk [T, n]: the gradient of the key projection's bias in dense attention is zero, what comes out is the rounding of all that
// leads to it.  Summed as the stages sum it, so that a layer in one node and its stages give the same one.
Tensor key_bias_grad(const Context& c, const Tensor& dk, void* st) {
  const int64_t T = dk.size(0), n = dk.size(1);
  if (c.mode == DROPIN_DENSE || !(n == 64 || n == 128 || n == 256 || n == 512)) return dk.sum(0);
  Tensor sums = at::empty({n}, dk.options()), ws = at::empty({(int64_t)spion_layernorm_workspace_floats((int)n)}, dk.options());
  check(spion_column_sums(dk.data_ptr(), 0, (float*)sums.data_ptr(), (float*)ws.data_ptr(), T, (int)n, st), "spion_column_sums");
  return sums;
}

// A whole multi-head attention layer: x [B, L, dim] -> projections -> attention -> output projection [B, L, dim_out].
// noise: dense attention in fp32.  What the gradient of the key projection's bias consists of (above) stays as the stages form it: the
// projections to Q, K and V and the way from the output's gradient to dO are the framework's products, the rest is the library's: products of
// three bf16 parts where the framework has fp32 ones.  Error against 64 bits ÷ that of the framework's, twelve layers of 350 to 24000 tokens, of
// normal tokens and of positive ones: output 0.3 - 1.0, gradients of the tokens 0.7 - 1.0, of the weights 0.2 - 1.0, of the biases (fp32 sums in another
// order) 0.5 - 1.3.
struct LayerNode : public Node {
  ContextPtr c;
  bool fp32 = false, noise = false;
  SavedAttn saved;
  SavedVariable x, w[4];                 // Wq, Wk, Wv, Wf; mixed precision: w[0] is the copy of all four, one after another
  int64_t dim_out = 0;
  at::ScalarType out_type, x_type;
  bool released = false;
  std::string name() const override { return "SparseAttentionLayerBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    x.reset_data();
    for (auto& s : w) s.reset_data();
    saved.reset();
    released = true;
  }
  // stage by stage: the saved results of the stages become outputs of nodes of their own
  variable_list recorded_backward(const Tensor& grad, void* st) {
    OutsideAutocast outside;
    variable_list out(9);
    const auto type = fp32 ? at::kFloat : at::kBFloat16;
    const Attn a = saved.unpack(*c);
    const Tensor X = x.unpack(), x2 = X.to(type).reshape({c->B * c->L, X.size(2)});
    const int64_t HD = c->H * c->d, dim = X.size(2);
    Tensor W[4];
    for (int i = 0; i < 4; ++i) {
      if (fp32) W[i] = w[i].unpack();
      else W[i] = w[0].unpack().narrow(0, i * HD * dim, i < 3 ? HD * dim : dim_out * HD).view({i < 3 ? HD : dim_out, i < 3 ? dim : HD});
    }
    auto rows = [&](const Tensor& t) { return t.transpose(1, 2).reshape({c->B, c->L, c->H * c->d}); };
    auto operand = [&](const Tensor& t, int i) {
      const Tensor y = as_linear_node(rows(t), fp32, X, W[i], x_type, {next_edge(0), next_edge(1 + 2 * i), next_edge(2 + 2 * i)});
      return y.view({c->B, c->L, c->H, c->d}).transpose(1, 2);
    };
    const Tensor O = rows(as_node(c, a, operand(a.q, 0), operand(a.k, 1), operand(a.v, 2))).to(type);
    const Tensor go = grad.to(out_type).reshape({c->B * c->L, W[3].size(0)});
    if (task_should_compute_output(7)) out[7] = go.t().matmul(O.reshape({c->B * c->L, -1})).to(at::kFloat);
    if (task_should_compute_output(8)) out[8] = go.sum(0).to(at::kFloat);
    Tensor dO = go.matmul(W[3].to(type)).view({c->B, c->L, c->H, c->d}).transpose(1, 2), g[3];
    {
      at::NoGradGuard constant;
      dO = dO.to(c->type());
      if (!a.heads) dO = dO.contiguous();
      attn_backward(*c, a, dO, g[0], g[1], g[2], st);
    }
    for (int i = 0; i < 3; ++i) {
      const Tensor gi = rows(g[i]).reshape({c->B * c->L, c->H * c->d}).to(type);
      if (task_should_compute_output(1 + 2 * i)) out[1 + 2 * i] = gi.t().matmul(x2).to(at::kFloat);
      if (task_should_compute_output(2 + 2 * i)) out[2 + 2 * i] = gi.sum(0).to(at::kFloat);
      if (task_should_compute_output(0)) {
        const Tensor dx = gi.matmul(W[i].to(type));
        out[0] = out[0].defined() ? out[0] + dx : dx;
      }
    }
    if (out[0].defined()) out[0] = out[0].view(X.sizes()).to(x_type);
    return out;
  }
  // inputs: x, Wq, bq, Wk, bk, Wv, bv, Wf, bf
  variable_list apply(variable_list&& grads) override {
    return as_backward([&] { return backward(grads); });
  }
  variable_list backward(const variable_list& grads) {
    std::lock_guard<std::mutex> lock(mutex_);
    TORCH_CHECK(!released, "Trying to backward through the graph a second time (the saved tensors have been freed)");
    variable_list out(9);
    if (!grads[0].defined()) return out;
    c10::cuda::CUDAGuard guard(c->device);
    if (recorded()) return recorded_backward(grads[0], stream_of(grads[0]));
    const int H = (int)c->H, d = (int)c->d, L = (int)c->L;
    const int64_t T = c->B * c->L;
    const Attn a = saved.unpack(*c);
    Tensor X = x.unpack();
    if (!X.is_contiguous() || !aligned32(X)) X = X.contiguous().clone();
    const int dim = (int)X.size(2);
    Weights qkv, ff;
    const Tensor w0 = w[0].unpack();
    if (fp32) {
      qkv.W = {w0, w[1].unpack(), w[2].unpack()};
      ff.W = {w[3].unpack()};
    } else {
      const int64_t n = 3 * (int64_t)H * d * dim;
      qkv = Weights(pf(w0), 3, dim, 3 * H * d);
      ff = Weights(pf(w0) + n, 1, H * d, dim_out);
    }
    Tensor go = grads[0].to(out_type).contiguous();
    if (!aligned32(go)) go = go.clone();
    void* st = stream_of(go);
    auto form = [&](const std::vector<Tensor>& ts) { return a.heads ? tok(ts, H * d) : tok_heads(ts, H, d, L); };
    auto rows = [&](const Tensor& t) { return a.heads ? t.transpose(1, 2).view({T, H * d}) : t; };
    const spion_tokens tgo = tok({go}, (int)dim_out);
    const spion_tokens tO = form({a.O});
    std::vector<Tensor> dW, db;
    if (task_should_compute_output(7) || task_should_compute_output(8)) {
      linear_backward_weight({go}, tgo, rows(a.O), tO, ff, fp32, T, st, dW, db);
      out[7] = dW[0]; out[8] = db[0];
    }
    Tensor dO;
    if (noise) {
      OutsideAutocast outside;
      dO = at::mm(go.view({T, dim_out}), ff.W[0]).view({c->B, c->L, H, d}).transpose(1, 2).contiguous();
    } else {
      dO = empty_operand(*c, a.heads, a.q);
      linear_backward_input(tgo, ff, fp32, nullptr, form({dO}), T, st);
    }
    Tensor dq, dk, dv;
    attn_backward(*c, a, dO, dq, dk, dv, st);
    const spion_tokens tg = form({dq, dk, dv});
    bool any = false;
    for (int i = 1; i < 7; ++i) any = any || task_should_compute_output(i);
    if (any) {
      dW.clear(); db.clear();
      linear_backward_weight({rows(dq), rows(dk), rows(dv)}, tg, X, tok({X}, dim), qkv, fp32, T, st, dW, db, X.scalar_type() != x_type);
      for (int i = 0; i < 3; ++i) { out[1 + 2 * i] = dW[i]; out[2 + 2 * i] = db[i]; }
      if (noise && task_should_compute_output(4)) out[4] = key_bias_grad(*c, dk.transpose(1, 2).reshape({T, H * d}), st);
    }
    if (task_should_compute_output(0)) {
      Tensor dX = at::empty(X.sizes(), X.options().dtype(x_type));
      linear_backward_input(tg, qkv, fp32, nullptr, tok({dX}, dim), T, st);
      out[0] = dX;
    }
    return out;
  }
};

// Can the layer run as one node?  fp32: everything in fp32; else bf16 operands (mixed precision).
bool layer_supported(const ContextPtr& c, const Tensor& x, const std::vector<Tensor>& W, const std::vector<Tensor>& b, bool fp32) {
  if (c->bf16 == fp32 || !plain({x, W, b})) return false;
  if (!x.is_cuda() || x.device().index() != c->device || x.dim() != 3 || x.size(0) != c->B || x.size(1) != c->L) return false;
  if (x.scalar_type() != at::kFloat && (fp32 || x.scalar_type() != at::kBFloat16)) return false;
  if ((c->d & (c->d - 1)) || c->d < 32 || x.size(2) != W[0].size(1) || W[3].size(1) != c->H * c->d || W[0].size(0) != c->H * c->d) return false;
  if (x.scalar_type() == at::kBFloat16 && (W[0].size(0) % 64 || !c->fused)) return false;      // see spion_linear_backward_input
  return weights_ok({W[0], W[1], W[2]}, {b[0], b[1], b[2]}, x, fp32) && weights_ok({W[3]}, {b[3]}, x, fp32);
}

Result attention_layer(const ContextPtr& c, const Tensor& x, const optional<Tensor>& mask, const std::vector<Tensor>& W,
                          const std::vector<Tensor>& b, bool fp32, bool noise) {
  c10::cuda::CUDAGuard guard(c->device);
  void* st = stream_of(x);
  const int H = (int)c->H, d = (int)c->d, L = (int)c->L;
  const int64_t T = c->B * c->L;
  bool need = x.requires_grad();
  for (int i = 0; i < 4; ++i) need = need || W[i].requires_grad() || b[i].requires_grad();
  need = need && at::GradMode::is_enabled();
  Attn a;
  Tensor out;
  Kept kept_in, kept_out;
  Tensor kept_w;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    Tensor X = x.detach();
    if (!X.is_contiguous() || !aligned32(X)) X = X.contiguous().clone();
    const auto opt = X.options().dtype(c->type());
    Tensor keys;
    if (c->keypad && (noise || T * H > 0x7fffffffLL)) a.pen = penalty(*c, mask.has_value() ? *mask : Tensor(), X, st);
    else if (c->keypad) { keys = key_mask(*c, mask.has_value() ? *mask : Tensor(), X); a.pen = empty_penalty(*c, X); }
    // bf16 tokens: operands stay [B, L, H, d], whose rows the weight gradients' matrix products read
    a.heads = X.scalar_type() == at::kBFloat16 && c->fused ? H : 0;
    auto form = [&](const std::vector<Tensor>& ts) { return a.heads ? tok(ts, H * d) : tok_heads(ts, H, d, L); };
    Weights qkv{{W[0].detach(), W[1].detach(), W[2].detach()}, {b[0].detach(), b[1].detach(), b[2].detach()}};
    Weights ff{{W[3].detach()}, {b[3].detach()}};
    const int64_t n_in = (int64_t)qkv.out() * qkv.in();
    if (need && !fp32) kept_w = at::empty({n_in + (int64_t)ff.out() * ff.in()}, W[0].options());
    if (noise) {
      auto operand = [&](int i) { return at::linear(X, qkv.W[i], qkv.b[i]).view({c->B, c->L, H, d}).transpose(1, 2).contiguous(); };
      a.q = operand(0); a.k = operand(1); a.v = operand(2);
    } else {
      const Tensor like = at::empty({0}, opt);
      a.q = empty_operand(*c, a.heads, like); a.k = empty_operand(*c, a.heads, like); a.v = empty_operand(*c, a.heads, like);
      kept_in = Kept(need, fp32, X, qkv, (float*)p(kept_w));
      const spion_tokens in = tok({X}, (int)X.size(2)), operands = form({a.q, a.k, a.v});
      if (keys.defined()) linear_forward_keypad(in, qkv, fp32, operands, T, st, kept_in, keys, (int)c->B, H, L, a.pen);
      else linear_forward(in, qkv, fp32, operands, nullptr, T, st, kept_in);
    }
    attn_forward(*c, a, need, st);
    out = at::empty({c->B, c->L, ff.out()}, opt);
    kept_out = Kept(need, fp32, a.O, ff, kept_w.defined() ? (float*)p(kept_w) + n_in : nullptr);
    linear_forward(form({a.O}), ff, fp32, tok({out}, ff.out()), nullptr, T, st, kept_out);
  }
  if (need) {
    auto node = std::shared_ptr<LayerNode>(new LayerNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, W[0], b[0], W[1], b[1], W[2], b[2], W[3], b[3]));
    node->c = c; node->fp32 = fp32; node->noise = noise; node->out_type = out.scalar_type();
    Attn kept = a;
    if (c->mode == NATIVE && c->fused && c->recompute) kept.P = Tensor();
    node->saved.save_all(kept, a.q, a.k, a.v);
    node->x_type = x.scalar_type();
    node->x = save(kept_in.x.defined() ? kept_in.x : x);
    node->dim_out = W[3].size(0);
    if (kept_w.defined()) node->w[0] = save(kept_w);
    else for (int i = 0; i < 4; ++i) node->w[i] = save(W[i]);
    torch::autograd::set_history(out, node);
  }
  return Result{out, a};
}

// ------------------------------------------------------------------------------------------------ linear layers on their own
bool linear_supported(const Tensor& x, const Tensor& W, const Tensor& b, bool fp32) {
  if (!x.is_cuda() || !plain({x, W, b}) || x.numel() == 0 || x.dim() < 2 || x.size(-1) != W.size(1)) return false;
  if (x.scalar_type() != at::kFloat && (fp32 || x.scalar_type() != at::kBFloat16)) return false;
  return x.numel() / W.size(1) < 0x7fffff00LL && weights_ok({W}, {b}, x, fp32);
}

bool mlp_supported(const Tensor& x, const Tensor& W1, const Tensor& b1, const Tensor& W2, const Tensor& b2) {
  return linear_supported(x, W1, b1, false) && plain({W2, b2}) && W2.dim() == 2 && W2.size(1) == W1.size(0) && weights_ok({W2}, {b2}, x, false);
}

Tensor linear(const Tensor& x, const Tensor& W, const Tensor& b, bool fp32) {
  c10::cuda::CUDAGuard guard(x.device());
  const bool need = at::GradMode::is_enabled() && (x.requires_grad() || W.requires_grad() || b.requires_grad());
  Tensor out;
  Kept kept;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    Tensor X = x.detach();
    if (!X.is_contiguous() || !aligned32(X)) X = X.contiguous().clone();
    Weights l{{W.detach()}, {b.detach()}};
    kept = Kept(need, fp32, X, l);
    auto sizes = x.sizes().vec();
    sizes.back() = l.out();
    out = at::empty(sizes, X.options().dtype(fp32 ? at::kFloat : at::kBFloat16));
    linear_forward(tok({X}, l.in()), l, fp32, tok({out}, l.out()), nullptr, X.numel() / l.in(), stream_of(X), kept);
  }
  if (need) {
    auto node = std::shared_ptr<LinearNode>(new LinearNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, W, b));
    node->fp32 = fp32; node->out_type = out.scalar_type(); node->x_type = x.scalar_type();
    node->x = save(kept.x.defined() ? kept.x : x);
    node->w = save(kept.w.defined() ? kept.w : W);
    torch::autograd::set_history(out, node);
  }
  return out;
}

// Feed-forward block Linear -> GELU -> Linear under mixed precision, the activation inside the first product's kernel.
struct MlpNode : public Node {
  SavedVariable x, w1, w2, h_s, g_s;     // h_s, g_s: pre-activation and activation, bf16
  at::ScalarType x_type;
  bool released = false;
  std::string name() const override { return "FeedForwardBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&x, &w1, &w2, &h_s, &g_s}) s->reset_data();
    released = true;
  }
  // inputs: x, W1, b1, W2, b2
  variable_list apply(variable_list&& grads) override {
    return as_backward([&] { return backward(grads); });
  }
  variable_list backward(const variable_list& grads) {
    std::lock_guard<std::mutex> lock(mutex_);
    TORCH_CHECK(!released, "Trying to backward through the graph a second time (the saved tensors have been freed)");
    variable_list out(5);
    if (!grads[0].defined()) return out;
    Tensor X = x.unpack();
    c10::cuda::CUDAGuard guard(X.device());
    if (recorded()) {
      OutsideAutocast outside;
      auto half = [](const Tensor& t) { return t.to(at::kBFloat16); };
      const Tensor W1 = w1.unpack(), W2 = w2.unpack(), x2 = half(X).reshape({-1, W1.size(1)});
      auto sizes = X.sizes().vec();
      sizes.back() = W1.size(0);
      const Tensor pre = as_linear_node(h_s.unpack().reshape(sizes), false, X, W1, x_type, {next_edge(0), next_edge(1), next_edge(2)}).reshape({-1, W1.size(0)});
      const Tensor go = half(grads[0]).reshape({-1, W2.size(0)}), dh = at::gelu_backward(go.matmul(half(W2)), pre);
      if (task_should_compute_output(0)) out[0] = dh.matmul(half(W1)).reshape(X.sizes()).to(x_type);
      if (task_should_compute_output(1)) out[1] = dh.t().matmul(x2).to(at::kFloat);
      if (task_should_compute_output(2)) out[2] = dh.sum(0).to(at::kFloat);
      if (task_should_compute_output(3)) out[3] = go.t().matmul(at::gelu(pre)).to(at::kFloat);
      if (task_should_compute_output(4)) out[4] = go.sum(0).to(at::kFloat);
      return out;
    }
    if (!X.is_contiguous() || !aligned32(X)) X = X.contiguous().clone();
    const Tensor h = h_s.unpack().contiguous(), g = g_s.unpack().contiguous();
    Weights l1, l2;
    l1.W.push_back(w1.unpack()); l2.W.push_back(w2.unpack());
    Tensor go = grads[0].to(at::kBFloat16).contiguous();
    if (!aligned32(go)) go = go.clone();
    void* st = stream_of(X);
    const int64_t T = X.numel() / l1.in();
    std::vector<Tensor> dW, db;
    const spion_tokens tg = tok({go}, l2.out());
    linear_backward_weight({go}, tg, g, tok({g}, l2.in()), l2, false, T, st, dW, db);
    Tensor dh = at::empty(h.sizes(), h.options());
    linear_backward_input(tg, l2, false, p(h), tok({dh}, l2.in()), T, st);
    const spion_tokens th = tok({dh}, l1.out());
    linear_backward_weight({dh}, th, X, tok({X}, l1.in()), l1, false, T, st, dW, db, X.scalar_type() != x_type);
    if (task_should_compute_output(0)) {
      out[0] = at::empty(X.sizes(), X.options().dtype(x_type));
      linear_backward_input(th, l1, false, nullptr, tok({out[0]}, l1.in()), T, st);
    }
    out[1] = dW[1]; out[2] = db[1]; out[3] = dW[0]; out[4] = db[0];
    return out;
  }
};

Tensor mlp(const Tensor& x, const Tensor& W1, const Tensor& b1, const Tensor& W2, const Tensor& b2) {
  c10::cuda::CUDAGuard guard(x.device());
  const bool need = at::GradMode::is_enabled() &&
                    (x.requires_grad() || W1.requires_grad() || b1.requires_grad() || W2.requires_grad() || b2.requires_grad());
  Tensor out, h, g;
  Kept kept1, kept2;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    Tensor X = x.detach();
    if (!X.is_contiguous() || !aligned32(X)) X = X.contiguous().clone();
    Weights l1{{W1.detach()}, {b1.detach()}}, l2{{W2.detach()}, {b2.detach()}};
    const int64_t T = X.numel() / l1.in();
    const auto opt = X.options().dtype(at::kBFloat16);
    h = at::empty({T, l1.out()}, opt);
    g = at::empty({T, l1.out()}, opt);
    void* st = stream_of(X);
    kept1 = Kept(need, false, X, l1); kept2 = Kept(need, false, g, l2);
    linear_forward(tok({X}, l1.in()), l1, false, tok({h}, l1.out()), g.data_ptr(), T, st, kept1);
    auto sizes = x.sizes().vec();
    sizes.back() = l2.out();
    out = at::empty(sizes, opt);
    linear_forward(tok({g}, l2.in()), l2, false, tok({out}, l2.out()), nullptr, T, st, kept2);
  }
  if (need) {
    auto node = std::shared_ptr<MlpNode>(new MlpNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, W1, b1, W2, b2));
    node->x_type = x.scalar_type();
    node->x = save(kept1.x.defined() ? kept1.x : x); node->w1 = save(kept1.w); node->w2 = save(kept2.w);
    node->h_s = save(h); node->g_s = save(g);
    torch::autograd::set_history(out, node);
  }
  return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  error_type();
  py::register_local_exception_translator([](std::exception_ptr e) {
    try {
      if (e) std::rethrow_exception(e);
    } catch (const Failure& f) {
      PyErr_SetString(error_type().ptr(), f.what());
    }
  });
  py::class_<Context, ContextPtr>(m, "Context")
      .def(py::init<>())
      .def("close", &Context::close)
      .def("set_pattern", &set_pattern)
      .def_readwrite("handle", &Context::handle)
      .def_readwrite("mode", &Context::mode)
      .def_readwrite("B", &Context::B).def_readwrite("H", &Context::H).def_readwrite("L", &Context::L).def_readwrite("d", &Context::d)
      .def_readwrite("device", &Context::device)
      .def_readwrite("bf16", &Context::bf16).def_readwrite("keypad", &Context::keypad).def_readwrite("fused", &Context::fused)
      .def_readwrite("recompute", &Context::recompute).def_readwrite("rounded", &Context::rounded).def_readwrite("return_probs", &Context::return_probs)
      .def_readwrite("needs_scratch", &Context::needs_scratch).def_readwrite("owned", &Context::owned)
      .def_readwrite("nnz", &Context::nnz)
      .def_readwrite("sum_mat", &Context::sum_mat).def_readwrite("offsets", &Context::offsets).def_readwrite("columns", &Context::columns);
  py::class_<MaskKey>(m, "MaskKey").def(py::init<>()).def("matches", &MaskKey::matches).def("set", &MaskKey::set);
  // None, unless `inside` (an autograd function that stands for the call), where something wants to see the call (plain())
  m.def("attention", [](const ContextPtr& c, const Tensor& q, const Tensor& k, const Tensor& v, const optional<Tensor>& mask, bool inside) -> py::object {
    if (!inside && !plain({q, k, v})) return py::none();
    return as_tuple([&] { return attention(c, q, k, v, mask); });
  }, py::arg("context"), py::arg("query"), py::arg("key"), py::arg("value"), py::arg("mask"), py::arg("inside") = false);
  m.def("layer_supported", &layer_supported);
  m.def("attention_layer", [](const ContextPtr& c, const Tensor& x, const optional<Tensor>& mask, const std::vector<Tensor>& W,
                              const std::vector<Tensor>& b, bool fp32, bool noise) {
    return as_tuple([&] { return attention_layer(c, x, mask, W, b, fp32, noise); });
  });
  m.def("linear_supported", &linear_supported);
  m.def("linear", &linear);
  m.def("mlp_supported", &mlp_supported);
  m.def("mlp", &mlp);
}
