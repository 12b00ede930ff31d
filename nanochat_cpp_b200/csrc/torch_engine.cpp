// Native host path of the engine's public entry points: argument checks, buffers, launch order and the autograd nodes of
// the MX Linears, as a Python extension over libmxb200's C ABI. Mirrors the reference's C++ host code
// (src/nanochat/model/fp8/fp8.cpp:113-171, 240-338, 424-571; ops/softcap_ce.cpp:27-205; ops/residual_norm.cpp:33-96).
//
// Why native: every launch of a small Linear takes 3 to 15 us on the device, while a Python autograd function with a
// ctypes call and a handful of tensor objects per launch cost the host 30 to 50 us each, so every shape up to a few
// thousand tokens was bound by the host (fp8_matmul of 2048 x 768 -> 3072, forward and backward: 59 us of kernels in a
// 250 us pass). Here a call costs a few allocations from torch's caching allocator and the launches. Tensors that
// nobody outside sees (quantized operands) are one byte buffer per lifetime, data then scales. The launches run without the
// GIL: a full launch queue blocks its own thread only, and threads that drive several GPUs do not wait for one another.
#include <optional>
#include <stdexcept>
#include <utility>
#include <vector>

#include <ATen/FuncTorchTLS.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/util/SmallVector.h>
#include <torch/csrc/Exceptions.h>
#include <torch/extension.h>

#include "mxb200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr auto kE4M3 = at::kFloat8_e4m3fn;
constexpr auto kE8M0 = at::kFloat8_e8m0fnu;

// ---------------------------------------------------------------------------------------------------- plumbing

// The library's status as the Python error it is everywhere (capi.Mxb200Error), from an autograd worker's thread too.
[[noreturn]] void raise_status(int status, const char* what) {
  py::gil_scoped_acquire gil;
  const py::object type = py::module_::import("nanochat_cpp_b200.capi").attr("Mxb200Error");
  const py::object error = type(status, what);
  PyErr_SetObject(type.ptr(), error.ptr());
  python_error e;
  e.persist();
  throw e;
}

inline void check(int status, const char* what) {
  if (status != MXB200_OK)
    raise_status(status, what);
}

[[noreturn]] void fail(const char* message) {
  throw std::runtime_error(message);
}

inline void require(bool ok, const char* message) {
  if (!ok)
    fail(message);
}

inline void require_cuda(const Tensor& t, const char* what) {
  if (!t.is_cuda())
    throw std::runtime_error(std::string(what) + ": expected a CUDA tensor; this engine has no CPU path");
}

inline void* stream() {
  return c10::cuda::getCurrentCUDAStream().stream();
}

inline Tensor empty(at::IntArrayRef size, at::ScalarType dtype, at::Device device) {
  return at::detail::empty_cuda(size, dtype, device, std::nullopt);
}

inline bool fits(int64_t rows, int64_t cols) {
  return rows % 128 == 0 && cols % 128 == 0;
}

// One layout of a quantized (R, C) tensor by address: data row-major, then its scales.
struct Layout {
  void* data = nullptr;
  void* scale = nullptr;
};

constexpr int64_t mx_bytes(int64_t R, int64_t C) {
  return R * C + R * C / 32;
}

// An (R, C) layout in one byte buffer; R * C is a multiple of 16384, so the scales start aligned.
inline Tensor layout_buffer(int64_t R, int64_t C, at::Device device) {
  return empty({mx_bytes(R, C)}, at::kByte, device);
}

inline Layout layout_of(const Tensor& buffer, int64_t R, int64_t C) {
  auto* p = static_cast<unsigned char*>(buffer.data_ptr());
  return {p, p + R * C};
}

inline Layout layout_of(const Tensor& data, const Tensor& scale) {
  return {data.data_ptr(), scale.data_ptr()};
}

// The kernels' view of a layout whose rows have `ld` values, from (row, col) on; both multiples of 128.
inline mxb200_mx_out view(const Layout& l, int64_t ld, int64_t row = 0, int64_t col = 0) {
  const int64_t tiles = ld / 128;
  return {static_cast<unsigned char*>(l.data) + row * ld + col, ld,
          static_cast<unsigned char*>(l.scale) + (row / 128 * tiles + col / 128) * 512, tiles};
}

constexpr mxb200_mx_out kNoLayout{nullptr, 0, nullptr, 0};

// The four tensors of a quantized matrix as Python sees them.
struct Mx {
  Tensor data, data_t, scale, scale_t;
  Layout rows() const { return layout_of(data, scale); }
  Layout cols() const { return layout_of(data_t, scale_t); }
};

Mx empty_mx(int64_t R, int64_t C, at::Device device, bool rows = true, bool cols = true) {
  Mx q;
  if (rows)
    q.data = empty({R, C}, kE4M3, device), q.scale = empty({R * C / 32}, kE8M0, device);
  if (cols)
    q.data_t = empty({C, R}, kE4M3, device), q.scale_t = empty({R * C / 32}, kE8M0, device);
  return q;
}

void check_quantizable(const Tensor& x) {
  require_cuda(x, "quantize_mx");
  require(x.dim() == 2 && x.is_contiguous() && fits(x.size(0), x.size(1)) &&
                (x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kFloat),
          "MX: expected an aligned, contiguous 2D tensor with dims % 128");
}

void quantize(const Tensor& x, const mxb200_mx_out& out, const mxb200_mx_out& out_t) {
  check_quantizable(x);
  check(mxb200_quantize_mx(x.data_ptr(), x.scalar_type() == at::kBFloat16, x.size(0), x.size(1), out, out_t,
                           MXB200_PROLOGUE_NONE, MXB200_SCALE_REFERENCE, stream()),
        "quantize_mx");
}

// d (M, N) = a (M, K) . b (N, K)^T, bf16 or fp32 (alpha, +=).
mxb200_gemm_desc gemm_desc(void* d, at::ScalarType dtype, const Layout& a, const Layout& b, int64_t M, int64_t N, int64_t K,
                           const float* alpha = nullptr, bool accumulate = false) {
  return {a.data, a.scale, b.data, b.scale, d, nullptr, alpha, M, N, K,
          dtype == at::kFloat ? MXB200_OUT_F32 : MXB200_OUT_BF16, accumulate};
}

// GEMMs in one launch where the library can, split along K where it says so.
void run_gemms(const mxb200_gemm_desc* g, int n, at::Device device) {
  const size_t bytes = mxb200_gemm_group_workspace_bytes(g, n);
  Tensor ws;  // K slices: the caching allocator hands it on along this stream only, behind the launches that use it
  if (bytes > 0)
    ws = empty({static_cast<int64_t>(bytes)}, at::kByte, device);
  check(mxb200_gemm_group(g, n, bytes > 0 ? ws.data_ptr() : nullptr, bytes, stream()), "mx_gemm");
}

void gemm(void* d, at::ScalarType dtype, const Layout& a, const Layout& b, int64_t M, int64_t N, int64_t K, at::Device device) {
  const mxb200_gemm_desc g = gemm_desc(d, dtype, a, b, M, N, K);
  run_gemms(&g, 1, device);
}

Tensor gemm_bf16(const Layout& a, const Layout& b, int64_t M, int64_t N, int64_t K, at::Device device) {
  Tensor d = empty({M, N}, at::kBFloat16, device);
  gemm(d.data_ptr(), at::kBFloat16, a, b, M, N, K, device);
  return d;
}

// fp8.h:114-116. The Linears ask in forward: a weight frozen there gets no gradient from that pass, whatever it is in backward.
bool grad_direct(const Tensor& w) {
  return w.is_leaf() && w.requires_grad() && w.scalar_type() == at::kFloat && w.is_contiguous();
}

// A weight gradient dW = alpha * go_t (n, K) . in_t (C, K)^T of weights whose rows concatenate to n, as the GEMM that makes
// it and what follows. Direct (fp32 leaves): into their .grad, allocated (=) when undefined, else accumulated (+=); several
// whose gradients share one buffer take one += (fp8.cpp:470-514). Else: returned to autograd in the weights' type.
class WeightGrad {
 public:
  WeightGrad(const Layout& go_t, const Layout& in_t, int64_t n, int64_t C, int64_t K, std::vector<Tensor> weights,
             bool direct, const float* alpha, at::Device device)
      : ws_(std::move(weights)), direct_(direct) {
    int64_t total = 0;
    bool shapes = true, all = direct, bf16 = !direct && alpha == nullptr;
    for (const Tensor& w : ws_) {
      total += w.size(0), shapes &= w.size(1) == C;
      all = all && w.grad().defined();
      bf16 &= w.scalar_type() == at::kBFloat16;
    }
    require(shapes && total == n, "mx_grad_weights: weight rows must concatenate to the gradient's");
    if (all) {
      const Tensor& g0 = ws_[0].grad();
      const char* base = static_cast<const char*>(g0.data_ptr());
      bool contiguous = true;
      int64_t row = 0;
      for (const Tensor& w : ws_) {
        const Tensor& g = w.grad();
        contiguous &= g.is_contiguous() && g.scalar_type() == at::kFloat && g.data_ptr() == base + row * C * 4;
        row += w.size(0);
      }
      if (contiguous && (ws_.size() == 1 || (g0.is_view() && g0._base().numel() == n * C))) {
        done_ = true;
        desc_ = gemm_desc(const_cast<char*>(base), at::kFloat, go_t, in_t, n, C, K, alpha, true);
        return;
      }
    }
    // bf16 weights: rounded once in the epilogue, as the cast of an fp32 result would round it
    const auto dtype = bf16 ? at::kBFloat16 : at::kFloat;
    buf_ = empty({n, C}, dtype, device);
    desc_ = gemm_desc(buf_.data_ptr(), dtype, go_t, in_t, n, C, K, alpha, false);
  }

  const mxb200_gemm_desc& desc() const { return desc_; }

  // After the GEMM has been launched: the gradients autograd gets, undefined where .grad already has them.
  variable_list finish() {
    variable_list out(ws_.size());
    int64_t row = 0;
    for (size_t i = 0; i < ws_.size() && !done_; ++i) {
      const Tensor& w = ws_[i];
      // row blocks of one buffer, as the reference's merged q/k/v
      Tensor part = ws_.size() == 1 ? buf_ : buf_.narrow(0, row, w.size(0));
      row += w.size(0);
      if (!direct_)
        out[i] = part.scalar_type() == w.scalar_type() ? part : part.to(w.scalar_type());
      else if (w.grad().defined())
        w.mutable_grad().add_(part);
      else
        w.mutable_grad() = part;
    }
    return out;
  }

 private:
  std::vector<Tensor> ws_;
  bool direct_, done_ = false;
  Tensor buf_;
  mxb200_gemm_desc desc_{};
};

// ---------------------------------------------------------------------------------------------------- weight cache

// FP8 copies of weights, remade only when a weight changes: in-place updates bump the tensor's version (fp8.h:18-38,
// fp8.cpp:516-536). Used with the GIL held only.
class WeightCache {
 public:
  explicit WeightCache(bool on) : enabled(on) {}
  bool enabled;

  py::object get(int kind, const std::vector<Tensor>& weights, const py::object& make) {
    if (!enabled)
      return make();
    if (!hit(kind, weights)) {
      py::object made = make();
      store(kind, weights, made);
    }
    return value_;
  }

  bool hit(int kind, const std::vector<Tensor>& weights) const {
    if (kind != kind_ || weights.size() != keys_.size())
      return false;
    for (size_t i = 0; i < weights.size(); ++i)
      if (!keys_[i].is(weights[i]))
        return false;
    return true;
  }

  void store(int kind, const std::vector<Tensor>& weights, py::object value) {
    value_ = std::move(value);
    kind_ = kind;
    keys_.clear();
    for (const Tensor& w : weights)
      keys_.emplace_back(w);
  }

  Mx mx() const {
    const auto t = value_.cast<std::vector<Tensor>>();
    return {t.at(0), t.at(1), t.at(2), t.at(3)};
  }

 private:
  // The weak reference keeps a dead weight's address from being another tensor's while the key stands.
  struct Key {
    c10::weak_intrusive_ptr<c10::TensorImpl, c10::UndefinedTensorImpl> impl;
    const void* data;
    int64_t version;
    explicit Key(const Tensor& w)
        : impl(w.getIntrusivePtr()), data(w.data_ptr()), version(static_cast<int64_t>(w._version())) {}
    bool is(const Tensor& w) const {
      return impl._unsafe_get_target() == w.unsafeGetTensorImpl() && data == w.data_ptr() &&
             version == static_cast<int64_t>(w._version());
    }
  };
  int kind_ = -1;
  std::vector<Key> keys_;
  py::object value_;
};

// An (R, C) tensor quantized by the caller. The transposed layout is read by the backward only. The scales' type is the
// caller's: any of one byte.
Mx given_mx(const std::vector<Tensor>& t, int64_t R, int64_t C, at::Device device, bool grad, const char* what) {
  const Mx q{t.at(0), t.at(1), t.at(2), t.at(3)};
  const auto layout = [&](const Tensor& data, const Tensor& scale, int64_t rows, int64_t cols) {
    for (const Tensor* p : {&data, &scale}) {
      require_cuda(*p, what);
      if (p->device() != device || !p->is_contiguous())
        throw std::runtime_error(std::string(what) + ": expected contiguous operands on the input's device");
    }
    if (data.sizes() != at::IntArrayRef{rows, cols} || data.scalar_type() != kE4M3)
      throw std::runtime_error(std::string(what) + ": shape mismatch");
    if (scale.numel() != rows * cols / 32 || scale.element_size() != 1)
      throw std::runtime_error(std::string(what) + ": expected e4m3 operands with their MX scales");
  };
  layout(q.data, q.scale, R, C);
  if (grad)
    layout(q.data_t, q.scale_t, C, R);
  return q;
}

// The quantized copy of a (merged) weight: from the cache when it holds it, else to be quantized by the caller, into
// `keep` when a cache wants it afterwards and into unnamed buffers otherwise.
struct WeightUse {
  WeightCache* cache = nullptr;  // null: no caching
  std::vector<Tensor> weights;
  Mx mx;        // cached or given, or freshly made for the cache
  bool ready = false;
  Tensor rows_buffer, cols_buffer;  // without a cache

  // `from`: a cache or a list of the four tensors that a cache of another class gave (with the GIL held), or None or null.
  WeightUse(const py::object* from, std::vector<Tensor> ws, bool grad) : weights(std::move(ws)) {
    if (from == nullptr || from->is_none())
      return;
    if (!py::isinstance<WeightCache>(*from)) {
      mx = given_mx(from->cast<std::vector<Tensor>>(), out_features(), in_features(), weights[0].device(), grad, "mx_gemm");
      ready = true;
    } else if (auto* c = from->cast<WeightCache*>(); c->enabled) {
      cache = c;
      if (c->hit(1, weights))
        mx = c->mx(), ready = true;
    }
  }

  int64_t out_features() const {
    int64_t n = 0;
    for (const Tensor& w : weights)
      n += w.size(0);
    return n;
  }
  int64_t in_features() const { return weights[0].size(1); }

  void allocate(at::Device device, bool need_cols) {
    const int64_t n = out_features(), C = in_features();
    if (cache != nullptr) {
      mx = empty_mx(n, C, device);
    } else {
      rows_buffer = layout_buffer(n, C, device);
      if (need_cols)
        cols_buffer = layout_buffer(C, n, device);
    }
  }
  Layout rows() const {
    return rows_buffer.defined() ? layout_of(rows_buffer, out_features(), in_features()) : mx.rows();
  }
  Layout cols() const {
    return cols_buffer.defined() ? layout_of(cols_buffer, in_features(), out_features())
                                 : (mx.data_t.defined() ? mx.cols() : Layout{});
  }
  // what backward reads: {buffer} or {data_t, scale_t}
  void save(variable_list& to) const {
    if (cols_buffer.defined()) {
      to.push_back(cols_buffer);
      to.emplace_back();
    } else {
      to.push_back(mx.data_t);
      to.push_back(mx.scale_t);
    }
  }
  void publish() {
    if (cache != nullptr && !ready) {
      py::gil_scoped_acquire gil;
      py::list l;
      for (const Tensor& t : {mx.data, mx.data_t, mx.scale, mx.scale_t})
        l.append(py::cast(t));
      cache->store(1, weights, l);
    }
  }
};

// A saved layout: one buffer holding data then scales, or a data tensor and a scale tensor.
inline Layout saved_layout(const Tensor& a, const Tensor& b, int64_t R, int64_t C) {
  return b.defined() ? layout_of(a, b) : layout_of(a, R, C);
}

// ---------------------------------------------------------------------------------------------------- quantizer jobs

// Quantizations that do not depend on one another, issued together.
class QuantizeJobs {
 public:
  void add(const Tensor& x, const mxb200_mx_out& out, const mxb200_mx_out& out_t) {
    check_quantizable(x);
    items_.push_back({{x.data_ptr(), x.size(0), x.size(1), out, out_t}, x.scalar_type() == at::kBFloat16});
    hold_.push_back(x);
  }
  void add(const Tensor& x, const Layout& rows, const Layout& cols, bool need_cols = true) {
    add(x, view(rows, x.size(1)), need_cols ? view(cols, x.size(0)) : kNoLayout);
  }
  // a weight's parts into their row ranges of one buffer (fp8.cpp:155-171)
  void add(WeightUse& w, at::Device device, bool need_cols) {
    if (w.ready)
      return;
    w.allocate(device, need_cols);
    const Layout rows = w.rows(), cols = w.cols();
    const int64_t n = w.out_features(), C = w.in_features();
    int64_t row = 0;
    for (const Tensor& part : w.weights) {
      const Tensor p = part.detach().contiguous();
      add(p, view(rows, C, row, 0), cols.data != nullptr ? view(cols, n, 0, row) : kNoLayout);
      row += part.size(0);
    }
  }
  void run() {
    if (!items_.empty())
      check(mxb200_quantize_mx_items(items_.data(), static_cast<int>(items_.size()), MXB200_SCALE_REFERENCE, stream()),
            "quantize_mx");
  }

 private:
  c10::SmallVector<mxb200_quantize_item, 8> items_;
  c10::SmallVector<Tensor, 8> hold_;
};

// ---------------------------------------------------------------------------------------------------- Linear

// Whether a call of these inputs gets an autograd node. What a node refuses, forward-mode tangents and function transforms
// (vmap, jvp), is refused without one too: the outputs would come back as constants.
inline bool grad_mode(std::initializer_list<const Tensor*> inputs) {
  for (const Tensor* t : inputs)
    TORCH_CHECK_NOT_IMPLEMENTED(!t->_fw_grad(0).defined(), "MX: forward-mode differentiation is not implemented");
  if (const auto& transforms = at::functorch::functorchTLSAccessor())
    transforms->checkSupportsCppAutogradFunction();
  if (!at::GradMode::is_enabled())
    return false;
  for (const Tensor* t : inputs)
    if (t->requires_grad())
      return true;
  return false;
}

// One Linear under MX: y = x . w^T, dX = dY . w, dW = dY^T . x, every operand E4M3 with per-32 scales along the
// contraction (fp8.cpp:240-260).
Tensor linear_forward(const Tensor& x, WeightUse& w, bool grad, Tensor* x_cols) {
  const auto device = x.device();
  const int64_t N = x.size(0), C = x.size(1), O = w.out_features();
  const Tensor x_rows = layout_buffer(N, C, device);
  if (grad)
    *x_cols = layout_buffer(C, N, device);
  QuantizeJobs jobs;
  jobs.add(x, layout_of(x_rows, N, C), grad ? layout_of(*x_cols, C, N) : Layout{}, grad);
  jobs.add(w, device, grad);
  jobs.run();
  w.publish();
  return gemm_bf16(layout_of(x_rows, N, C), w.rows(), N, O, C, device);
}

struct Float8Matmul : torch::autograd::Function<Float8Matmul> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, WeightUse* use) {
    Tensor x_cols;
    Tensor y = linear_forward(x, *use, true, &x_cols);
    variable_list saved{x_cols};
    use->save(saved);
    ctx->save_for_backward(std::move(saved));
    ctx->saved_data["w"] = w;
    ctx->saved_data["direct"] = grad_direct(w);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor w = ctx->saved_data["w"].toTensor();
    const Tensor go = grads[0].contiguous();
    const auto device = go.device();
    const int64_t N = go.size(0), O = w.size(0), C = w.size(1);
    const Tensor g_rows = layout_buffer(N, O, device), g_cols = layout_buffer(O, N, device);
    QuantizeJobs jobs;
    jobs.add(go, layout_of(g_rows, N, O), layout_of(g_cols, O, N));
    jobs.run();
    // the weight gradient first: with K = tokens its tiles are the longer ones of the launch
    mxb200_gemm_desc gemms[2];
    int n = 0;
    const bool direct = ctx->saved_data["direct"].toBool();
    std::optional<WeightGrad> wgrad;
    if (direct || ctx->needs_input_grad(1)) {
      wgrad.emplace(layout_of(g_cols, O, N), layout_of(saved[0], C, N), O, C, N, std::vector<Tensor>{w}, direct, nullptr, device);
      gemms[n++] = wgrad->desc();
    }
    Tensor dx, dw;
    if (ctx->needs_input_grad(0)) {
      dx = empty({N, C}, at::kBFloat16, device);
      gemms[n++] = gemm_desc(dx.data_ptr(), at::kBFloat16, layout_of(g_rows, N, O), saved_layout(saved[1], saved[2], C, O), N, C, O);
    }
    run_gemms(gemms, n, device);
    if (wgrad.has_value())
      dw = wgrad->finish()[0];
    return {dx, dw, Tensor()};
  }
};

Tensor fp8_matmul(const Tensor& input, const Tensor& w, const py::object& cache) {
  require(input.dim() == 2 && w.dim() == 2 && fits(input.size(0), input.size(1)) && fits(w.size(0), w.size(1)),
          "fp8_matmul: MX needs N, in, out % 128");
  require(input.size(1) == w.size(1), "mx_gemm: shape mismatch");
  require_cuda(input, "quantize_mx");
  const Tensor x = input.contiguous();
  const bool grad = grad_mode({&x, &w});
  WeightUse use(&cache, {w}, grad);
  const py::gil_scoped_release nogil;
  if (!grad)
    return linear_forward(x, use, false, nullptr);
  return Float8Matmul::apply(x, w, &use);
}

// ---------------------------------------------------------------------------------------------------- q, k, v

// Attention's three projections of one input, merged: MX scales run along K, so the weights concatenate along their
// rows and the output gradients along their columns (fp8.cpp:424-462).
variable_list qkv_forward(const Tensor& x, WeightUse& w, int64_t gate_cols, const Mx* x_mx, bool grad, variable_list* saved) {
  const auto device = x.device();
  const int64_t N = x.size(0), C = x.size(1), n = w.out_features();
  Tensor x_rows, x_cols;
  QuantizeJobs jobs;
  if (x_mx == nullptr) {
    x_rows = layout_buffer(N, C, device);
    if (grad)
      x_cols = layout_buffer(C, N, device);
    jobs.add(x, layout_of(x_rows, N, C), grad ? layout_of(x_cols, C, N) : Layout{}, grad);
  }
  jobs.add(w, device, grad);
  jobs.run();
  w.publish();
  const Tensor qkv = gemm_bf16(x_mx != nullptr ? x_mx->rows() : layout_of(x_rows, N, C), w.rows(), N, n, C, device);
  variable_list out;
  int64_t row = 0;
  for (const Tensor& part : w.weights) {
    out.push_back(qkv.narrow(1, row, part.size(0)));
    row += part.size(0);
  }
  if (gate_cols > 0) {
    if (x.scalar_type() == at::kBFloat16) {
      out.push_back(empty({N, gate_cols}, at::kBFloat16, device));
      check(mxb200_copy_columns(out.back().data_ptr(), gate_cols, x.data_ptr(), C, N, gate_cols, stream()), "fp8_qkv");
    } else {
      out.push_back(x.narrow(1, 0, gate_cols).contiguous());
    }
  }
  if (saved != nullptr) {
    if (x_mx != nullptr)
      *saved = {x_mx->data_t, x_mx->scale_t};
    else
      *saved = {x_cols, Tensor()};
    w.save(*saved);
  }
  return out;
}

struct MxQkv : torch::autograd::Function<MxQkv> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& wq, const Tensor& wk, const Tensor& wv,
                               int64_t gate_cols, WeightUse* use, const Mx* x_mx) {
    variable_list saved;
    variable_list out = qkv_forward(x, *use, gate_cols, x_mx, true, &saved);
    ctx->save_for_backward(std::move(saved));
    ctx->saved_data["w"] = std::vector<Tensor>{wq, wk, wv};
    ctx->saved_data["gate_cols"] = gate_cols;
    ctx->saved_data["tokens"] = x.size(0);
    ctx->saved_data["direct"] = grad_direct(wq) && grad_direct(wk) && grad_direct(wv);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const std::vector<Tensor> ws = ctx->saved_data["w"].toTensorVector();
    const int64_t gate_cols = ctx->saved_data["gate_cols"].toInt(), N = ctx->saved_data["tokens"].toInt();
    const auto device = ws[0].device();
    const int64_t C = ws[0].size(1);
    const bool direct = ctx->saved_data["direct"].toBool();
    int64_t n = 0;
    for (const Tensor& w : ws)
      n += w.size(0);
    const Tensor g_rows = layout_buffer(N, n, device), g_cols = layout_buffer(n, N, device);
    const Layout g = layout_of(g_rows, N, n), g_t = layout_of(g_cols, n, N);
    QuantizeJobs jobs;
    int64_t row = 0;
    for (size_t i = 0; i < 3; ++i) {
      const Tensor gi = grads[i].defined() ? grads[i].contiguous()
                                           : at::zeros({N, ws[i].size(0)}, ws[i].options().dtype(at::kBFloat16));
      jobs.add(gi, view(g, n, 0, row), view(g_t, N, row, 0));
      row += ws[i].size(0);
    }
    jobs.run();
    mxb200_gemm_desc gemms[2];
    int count = 0;
    WeightGrad wgrad(g_t, saved_layout(saved[0], saved[1], C, N), n, C, N, ws, direct, nullptr, device);
    gemms[count++] = wgrad.desc();
    Tensor dx;
    if (ctx->needs_input_grad(0)) {
      dx = empty({N, C}, at::kBFloat16, device);
      gemms[count++] = gemm_desc(dx.data_ptr(), at::kBFloat16, g, saved_layout(saved[2], saved[3], C, n), N, C, n);
    }
    run_gemms(gemms, count, device);
    if (dx.defined() && gate_cols > 0 && grads[3].defined()) {
      const Tensor gate = grads[3].contiguous();
      if (gate.scalar_type() == at::kBFloat16)
        check(mxb200_add_columns(dx.data_ptr(), C, gate.data_ptr(), gate_cols, N, gate_cols, stream()), "fp8_qkv");
      else  // of an fp32 input: added in fp32, rounded once
        dx.narrow(1, 0, gate_cols).add_(gate);
    }
    variable_list out{dx};
    for (Tensor& dw : wgrad.finish())
      out.push_back(std::move(dw));
    out.resize(7);
    return out;
  }
};

variable_list fp8_qkv(const Tensor& x_2d, const Tensor& wq, const Tensor& wk, const Tensor& wv, int64_t gate_cols,
                      const py::object& cache, const std::optional<std::vector<Tensor>>& x_mx) {
  bool ok = x_2d.dim() == 2 && fits(x_2d.size(0), x_2d.size(1)) && gate_cols >= 0 && gate_cols <= x_2d.size(1);
  for (const Tensor* w : {&wq, &wk, &wv})
    ok &= w->dim() == 2 && w->size(0) % 128 == 0;
  require(ok, "fp8_qkv: MX needs N, in and every weight's rows % 128");
  require(wk.size(1) == wq.size(1) && wv.size(1) == wq.size(1), "q/k/v weights must share the input dim");
  require(wq.size(1) == x_2d.size(1), "mx_gemm: shape mismatch");
  require_cuda(x_2d, "quantize_mx");
  const Tensor x = x_2d.contiguous();
  const bool grad = grad_mode({&x, &wq, &wk, &wv});
  const Mx given = x_mx.has_value() ? given_mx(*x_mx, x.size(0), x.size(1), x.device(), grad, "mx_gemm") : Mx{};
  WeightUse use(&cache, {wq, wk, wv}, grad);
  const Mx* mx = x_mx.has_value() ? &given : nullptr;
  const py::gil_scoped_release nogil;
  if (!grad)
    return qkv_forward(x, use, gate_cols, mx, false, nullptr);
  return MxQkv::apply(x, wq, wk, wv, gate_cols, &use, mx);
}

// ---------------------------------------------------------------------------------------------------- relu^2 MLP

// c_proj(relu(c_fc(x))^2): the forward quantizes relu(h)^2 in c_fc's epilogue, the backward quantizes
// dh = (go . w_proj) * 2h in the dgrad GEMM's epilogue without writing it; h is what is saved (fp8.cpp:262-338).
Tensor mlp_forward(const Tensor& x, WeightUse& fc, WeightUse& proj, const Mx* x_mx, bool grad, variable_list* saved) {
  const auto device = x.device();
  const int64_t N = x.size(0), C = x.size(1), H = fc.out_features(), O = proj.out_features();
  Tensor x_rows, x_cols;
  QuantizeJobs jobs;
  if (x_mx == nullptr) {
    x_rows = layout_buffer(N, C, device);
    if (grad)
      x_cols = layout_buffer(C, N, device);
    jobs.add(x, layout_of(x_rows, N, C), grad ? layout_of(x_cols, C, N) : Layout{}, grad);
  }
  jobs.add(fc, device, grad);
  jobs.add(proj, device, grad);
  jobs.run();
  fc.publish();
  proj.publish();
  const Tensor h = empty({N, H}, at::kBFloat16, device);
  const Tensor a_rows = layout_buffer(N, H, device), a_cols = layout_buffer(H, N, device);
  const Layout xq = x_mx != nullptr ? x_mx->rows() : layout_of(x_rows, N, C), w = fc.rows();
  const Layout a = layout_of(a_rows, N, H), a_t = layout_of(a_cols, H, N);
  check(mxb200_gemm_relu_square(xq.data, xq.scale, w.data, w.scale, h.data_ptr(), a.data, a.scale, a_t.data, a_t.scale, N,
                                H, C, stream()),
        "mx_gemm_relu_square");
  if (saved != nullptr) {
    if (x_mx != nullptr)
      *saved = {x_mx->data_t, x_mx->scale_t};
    else
      *saved = {x_cols, Tensor()};
    fc.save(*saved);
    proj.save(*saved);
    saved->push_back(h);
    saved->push_back(a_cols);
  }
  return gemm_bf16(a, proj.rows(), N, O, H, device);
}

struct Fp8ReluSquareMlp : torch::autograd::Function<Fp8ReluSquareMlp> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w_fc, const Tensor& w_proj, WeightUse* fc,
                        WeightUse* proj, const Mx* x_mx) {
    variable_list saved;
    Tensor y = mlp_forward(x, *fc, *proj, x_mx, true, &saved);
    ctx->save_for_backward(std::move(saved));
    ctx->saved_data["w_fc"] = w_fc;
    ctx->saved_data["w_proj"] = w_proj;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor w_fc = ctx->saved_data["w_fc"].toTensor(), w_proj = ctx->saved_data["w_proj"].toTensor();
    const Tensor grad = grads[0].contiguous();
    const auto device = grad.device();
    const Tensor& h = saved[6];
    const int64_t N = h.size(0), H = h.size(1), C = w_fc.size(1), O = w_proj.size(0);
    const Tensor go_rows = layout_buffer(N, O, device), go_cols = layout_buffer(O, N, device);
    const Layout go = layout_of(go_rows, N, O), go_t = layout_of(go_cols, O, N);
    QuantizeJobs jobs;
    jobs.add(grad, go, go_t);
    jobs.run();
    const Tensor dh_rows = layout_buffer(N, H, device), dh_cols = layout_buffer(H, N, device);
    const Layout dh = layout_of(dh_rows, N, H), dh_t = layout_of(dh_cols, H, N);
    const Layout proj_t = saved_layout(saved[4], saved[5], H, O);
    check(mxb200_gemm_relu_square_bwd(go.data, go.scale, proj_t.data, proj_t.scale, h.data_ptr(), dh.data, dh.scale,
                                      dh_t.data, dh_t.scale, N, H, O, stream()),
          "mx_gemm_relu_square_bwd");
    // the three remaining GEMMs share a launch; fc's weight gradient and the input gradient read dh while it is in L2
    mxb200_gemm_desc gemms[3];
    int n = 0;
    std::optional<WeightGrad> fc, proj;
    const bool fc_direct = grad_direct(w_fc), proj_direct = grad_direct(w_proj);
    const auto fc_grad = [&] {
      if (fc_direct || ctx->needs_input_grad(1)) {
        fc.emplace(dh_t, saved_layout(saved[0], saved[1], C, N), H, C, N, std::vector<Tensor>{w_fc}, fc_direct, nullptr, device);
        gemms[n++] = fc->desc();
      }
    };
    const bool tied = w_fc.is_same(w_proj);  // both into one .grad, in the order of the Linears' backwards
    if (!tied)
      fc_grad();
    if (proj_direct || ctx->needs_input_grad(2)) {
      proj.emplace(go_t, layout_of(saved[7], H, N), O, H, N, std::vector<Tensor>{w_proj}, proj_direct, nullptr, device);
      gemms[n++] = proj->desc();
    }
    if (tied)
      fc_grad();
    Tensor dx;
    if (ctx->needs_input_grad(0)) {
      dx = empty({N, C}, at::kBFloat16, device);
      gemms[n++] = gemm_desc(dx.data_ptr(), at::kBFloat16, dh, saved_layout(saved[2], saved[3], C, H), N, C, H);
    }
    run_gemms(gemms, n, device);
    return {dx, fc.has_value() ? fc->finish()[0] : Tensor(), proj.has_value() ? proj->finish()[0] : Tensor(), Tensor(),
            Tensor(), Tensor()};
  }
};

Tensor fp8_relu_square_mlp(const Tensor& x_2d, const Tensor& w_fc, const Tensor& w_proj, const py::object& fc_cache,
                           const py::object& proj_cache, const std::optional<std::vector<Tensor>>& x_mx) {
  require(x_2d.dim() == 2 && w_fc.dim() == 2 && w_proj.dim() == 2 && fits(x_2d.size(0), x_2d.size(1)) &&
                fits(w_fc.size(0), w_fc.size(1)) && fits(w_proj.size(0), w_proj.size(1)) &&
                w_fc.size(1) == x_2d.size(1) && w_proj.size(1) == w_fc.size(0),
          "fp8_relu_square_mlp: MX needs N, in, hidden, out % 128");
  require_cuda(x_2d, "quantize_mx");
  const Tensor x = x_2d.contiguous();
  const bool grad = grad_mode({&x, &w_fc, &w_proj});
  const Mx given = x_mx.has_value() ? given_mx(*x_mx, x.size(0), x.size(1), x.device(), grad, "mx_gemm_relu_square") : Mx{};
  WeightUse fc(&fc_cache, {w_fc}, grad), proj(&proj_cache, {w_proj}, grad);
  const Mx* mx = x_mx.has_value() ? &given : nullptr;
  const py::gil_scoped_release nogil;
  if (!grad)
    return mlp_forward(x, fc, proj, mx, false, nullptr);
  return Fp8ReluSquareMlp::apply(x, w_fc, w_proj, &fc, &proj, mx);
}

// ---------------------------------------------------------------------------------------------------- chunked lm_head

struct LossArgs {
  int64_t vocab, chunk_rows;
  double softcap;
};

struct ChunkOutputs {
  float* losses = nullptr;             // (N), or null
  void* grad_x = nullptr;              // (N, C) bf16, or null: loss only
  const float* grad_scale = nullptr;   // upstream gradient of the losses, one value or one per row
  int64_t grad_scale_stride = 0;
  const int64_t* num_valid = nullptr;  // divides the scale
};

// Per chunk of rows: logits = xq[chunk] . wq^T, the loss pass, the gradient quantized straight from the logits (row-wise
// into a chunk buffer, transposed into one (padded, N) buffer), grad_x[chunk] = gq . wq_t^T (softcap_ce.cpp:27-110). With
// grad_x, x_cols and g_cols receive the transposes: the operands of the single weight-gradient GEMM.
void run_chunks(const Tensor& x, WeightUse& w, const Tensor& targets, const LossArgs& args, const ChunkOutputs& out,
                Tensor* x_cols, Tensor* g_cols) {
  const auto device = x.device();
  const int64_t N = x.size(0), C = x.size(1), V = w.out_features();
  const bool grad = out.grad_x != nullptr;
  const Tensor x_rows = layout_buffer(N, C, device);
  if (grad)
    *x_cols = layout_buffer(C, N, device);
  QuantizeJobs jobs;
  jobs.add(x, layout_of(x_rows, N, C), grad ? layout_of(*x_cols, C, N) : Layout{}, grad);
  jobs.add(w, device, grad);
  jobs.run();
  w.publish();
  const int64_t rows_max = std::min(N, args.chunk_rows);
  const Tensor logits = empty({rows_max, V}, at::kBFloat16, device);
  const Tensor row_floats = empty({2, rows_max}, at::kFloat, device);  // lse, and the losses nobody asked for
  auto* lse = static_cast<float*>(row_floats.data_ptr());
  Tensor g_rows;
  Layout g_t;
  if (grad) {
    g_rows = layout_buffer(rows_max, V, device);
    *g_cols = layout_buffer(V, N, device);
    g_t = layout_of(*g_cols, V, N);
  }
  const Layout xq = layout_of(x_rows, N, C), wq = w.rows();
  const auto* t = static_cast<const int64_t*>(targets.data_ptr());
  void* s = stream();
  const auto logits_gemm = [&](int64_t begin) {
    const mxb200_mx_out x_chunk = view(xq, C, begin);
    return gemm_desc(logits.data_ptr(), at::kBFloat16, {x_chunk.data, x_chunk.scale}, wq, std::min(N - begin, args.chunk_rows),
                     V, C);
  };
  for (int64_t begin = 0; begin < N; begin += args.chunk_rows) {
    const int64_t rows = std::min(N - begin, args.chunk_rows);
    if (!grad || begin == 0) {
      const mxb200_gemm_desc g = logits_gemm(begin);
      run_gemms(&g, 1, device);
    }
    check(mxb200_softcap_ce_loss(logits.data_ptr(), rows, V, t + begin, static_cast<int>(args.vocab), static_cast<int>(V),
                                 static_cast<float>(args.softcap), out.losses != nullptr ? out.losses + begin : lse + rows_max,
                                 lse, s),
          "softcap_ce_loss");
    if (!grad)
      continue;
    const Layout g = layout_of(g_rows, rows, V);
    const float* scale = out.grad_scale != nullptr ? out.grad_scale + begin * out.grad_scale_stride : nullptr;
    check(mxb200_softcap_ce_grad_mx(logits.data_ptr(), rows, V, t + begin, lse, static_cast<int>(args.vocab),
                                    static_cast<int>(V), static_cast<float>(args.softcap), scale, out.grad_scale_stride,
                                    out.num_valid, view(g, V), view(g_t, N, 0, begin), MXB200_SCALE_REFERENCE, s),
          "softcap_ce_grad_mx");
    // The input gradient has few long tiles (rows x C, K = V): the next chunk's logits, whose buffer has been read, share its
    // launch and fill the rest of the machine. 16384 x 1536 in chunks of 2048 over 32768 columns, where the gradient alone has
    // 64 tiles for 74 CTA pairs: 3454 -> 3367 us forward + backward on one GPU.
    mxb200_gemm_desc gemms[2] = {
          gemm_desc(static_cast<char*>(out.grad_x) + begin * C * 2, at::kBFloat16, g, w.cols(), rows, C, V)};
    int n = 1;
    if (begin + args.chunk_rows < N)
      gemms[n++] = logits_gemm(begin + args.chunk_rows);
    run_gemms(gemms, n, device);
  }
}

// For mean and sum the incoming gradient is a scalar, so the forward computes grad_x and the weight gradient's operands
// at once and the backward only scales: one GEMM with alpha = that gradient, straight into .grad when the weight is an
// fp32 leaf (softcap_ce.cpp:118-205).
Tensor reduced_loss(const Tensor& losses, const Tensor& num_valid, bool mean) {
  Tensor loss = empty({}, at::kFloat, losses.device());
  check(mxb200_reduce_losses(static_cast<const float*>(losses.data_ptr()), losses.numel(),
                             mean ? static_cast<const int64_t*>(num_valid.data_ptr()) : nullptr,
                             static_cast<float*>(loss.data_ptr()), stream()),
        "softcap_cross_entropy");
  return loss;
}

Tensor count_valid(const Tensor& targets) {
  Tensor n = empty({}, at::kLong, targets.device());
  check(mxb200_count_valid(static_cast<const int64_t*>(targets.data_ptr()), targets.numel(),
                           static_cast<int64_t*>(n.data_ptr()), stream()),
        "softcap_cross_entropy");
  return n;
}

struct SoftcapReduced : torch::autograd::Function<SoftcapReduced> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& targets,
                        const LossArgs* args, bool mean, WeightUse* use) {
    const Tensor num_valid = mean ? count_valid(targets) : Tensor();
    const Tensor losses = empty({x.size(0)}, at::kFloat, x.device());
    const Tensor grad_x = empty(x.sizes(), at::kBFloat16, x.device());
    ChunkOutputs out;
    out.losses = static_cast<float*>(losses.data_ptr());
    out.grad_x = grad_x.data_ptr();
    out.num_valid = mean ? static_cast<const int64_t*>(num_valid.data_ptr()) : nullptr;
    Tensor x_cols, g_cols;
    run_chunks(x, *use, targets, *args, out, &x_cols, &g_cols);
    ctx->save_for_backward({grad_x, g_cols, x_cols});
    ctx->saved_data["w"] = weight;
    return reduced_loss(losses, num_valid, mean);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor weight = ctx->saved_data["w"].toTensor();
    const Tensor& grad_x = saved[0];
    const auto device = grad_x.device();
    const int64_t N = grad_x.size(0), C = grad_x.size(1), V = weight.size(0);
    const Tensor g = grads[0].to(at::kFloat).contiguous();
    const auto* alpha = static_cast<const float*>(g.data_ptr());
    const Layout g_t = layout_of(saved[1], V, N), x_t = layout_of(saved[2], C, N);
    Tensor dw;
    const bool direct = grad_direct(weight);
    if (direct || ctx->needs_input_grad(1)) {
      WeightGrad wgrad(g_t, x_t, V, C, N, {weight}, direct, alpha, device);
      run_gemms(&wgrad.desc(), 1, device);
      dw = wgrad.finish()[0];
    }
    Tensor dx;
    if (ctx->needs_input_grad(0)) {
      dx = empty({N, C}, at::kBFloat16, device);
      check(mxb200_scale_bf16(grad_x.data_ptr(), alpha, dx.data_ptr(), N * C, stream()), "softcap_cross_entropy");
    }
    return {dx, dw, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// A cache kept alive by a graph node, which may be destroyed without the GIL.
struct CacheHolder : torch::CustomClassHolder {
  PyObject* object;
  explicit CacheHolder(py::object o) : object(o.release().ptr()) {}
  ~CacheHolder() override {
    py::gil_scoped_acquire gil;
    Py_XDECREF(object);
  }
};

// Reduction none: the backward re-runs the chunks with the per-row gradient.
struct SoftcapPerToken : torch::autograd::Function<SoftcapPerToken> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const Tensor& targets,
                        const LossArgs* args, WeightUse* use, const py::object* cache) {
    const Tensor losses = empty({x.size(0)}, at::kFloat, x.device());
    ChunkOutputs out;
    out.losses = static_cast<float*>(losses.data_ptr());
    run_chunks(x, *use, targets, *args, out, nullptr, nullptr);
    ctx->save_for_backward({x, weight, targets});
    ctx->saved_data["vocab"] = args->vocab;
    ctx->saved_data["chunk_rows"] = args->chunk_rows;
    ctx->saved_data["softcap"] = args->softcap;
    if (!cache->is_none()) {
      py::gil_scoped_acquire gil;
      ctx->saved_data["cache"] = c10::IValue::make_capsule(c10::make_intrusive<CacheHolder>(*cache));
    }
    return losses;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &weight = saved[1], &targets = saved[2];
    const auto device = x.device();
    const int64_t N = x.size(0), C = x.size(1), V = weight.size(0);
    const LossArgs args{ctx->saved_data["vocab"].toInt(), ctx->saved_data["chunk_rows"].toInt(),
                        ctx->saved_data["softcap"].toDouble()};
    const Tensor g = grads[0].to(at::kFloat).contiguous();
    const Tensor grad_x = empty({N, C}, at::kBFloat16, device);
    ChunkOutputs out;
    out.grad_x = grad_x.data_ptr();
    out.grad_scale = static_cast<const float*>(g.data_ptr());
    out.grad_scale_stride = 1;
    Tensor x_cols, g_cols;
    std::optional<WeightUse> use;
    if (const auto cache = ctx->saved_data.find("cache"); cache != ctx->saved_data.end()) {
      py::gil_scoped_acquire gil;
      const auto object = py::reinterpret_borrow<py::object>(static_cast<CacheHolder*>(cache->second.toCapsule().get())->object);
      use.emplace(&object, std::vector<Tensor>{weight}, true);
    } else {
      use.emplace(nullptr, std::vector<Tensor>{weight}, true);
    }
    run_chunks(x, *use, targets, args, out, &x_cols, &g_cols);
    WeightGrad wgrad(layout_of(g_cols, V, N), layout_of(x_cols, C, N), V, C, N, {weight}, false, nullptr, device);
    run_gemms(&wgrad.desc(), 1, device);
    return {grad_x, wgrad.finish()[0], Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor softcap_cross_entropy(const Tensor& x_in, const Tensor& weight, const Tensor& targets_in, int64_t vocab,
                             double softcap, int64_t chunk_rows, int reduction, const py::object& cache_object) {
  const Tensor x = x_in.contiguous(), targets = targets_in.to(at::kLong).contiguous();
  require_cuda(targets, "softcap_cross_entropy");
  const LossArgs args{vocab, chunk_rows, softcap};
  const bool mean = reduction == 0, none = reduction == 2, grad = grad_mode({&x, &weight});
  WeightUse use(&cache_object, {weight}, grad);
  const py::gil_scoped_release nogil;
  if (grad)
    return none ? SoftcapPerToken::apply(x, weight, targets, &args, &use, &cache_object)
                : SoftcapReduced::apply(x, weight, targets, &args, mean, &use);
  const Tensor losses = empty({x.size(0)}, at::kFloat, x.device());
  ChunkOutputs out;
  out.losses = static_cast<float*>(losses.data_ptr());
  run_chunks(x, use, targets, args, out, nullptr, nullptr);
  return none ? losses : reduced_loss(losses, mean ? count_valid(targets) : Tensor(), mean);
}

// ---------------------------------------------------------------------------------------------------- other entry points

// Forward of the fused residual step with MX output (residual_norm.cpp:36-96). Returns (res, n, n_mx..., rstd, s).
std::vector<std::optional<Tensor>> residual_norm_mx(const Tensor& x, const std::optional<Tensor>& r,
                                                    const std::optional<Tensor>& x0, const std::optional<Tensor>& lr,
                                                    const std::optional<Tensor>& l0, int64_t layer, int64_t gate_cols,
                                                    double eps) {
  const auto device = x.device();
  const int64_t cols = x.size(-1), rows = x.numel() / cols;
  const Tensor res = empty(x.sizes(), at::kBFloat16, device), n = empty(x.sizes(), at::kBFloat16, device);
  const Tensor rstd = empty({rows}, at::kFloat, device);
  std::optional<Tensor> s;
  if (r.has_value() && x0.has_value())
    s = empty(x.sizes(), at::kBFloat16, device);
  const Mx q = empty_mx(rows, cols, device);
  mxb200_residual_norm_mx a{};
  a.x = x.data_ptr();
  a.r = r.has_value() ? r->data_ptr() : nullptr;
  if (x0.has_value()) {
    a.x0 = x0->data_ptr();
    a.lr = static_cast<const float*>(lr->data_ptr()) + layer;
    a.l0 = static_cast<const float*>(l0->data_ptr()) + layer;
  }
  a.s = s.has_value() ? s->data_ptr() : nullptr;
  a.res = res.data_ptr();
  a.n = n.data_ptr();
  a.rstd = static_cast<float*>(rstd.data_ptr());
  a.rows = rows, a.cols = static_cast<int32_t>(cols), a.eps = static_cast<float>(eps);
  a.out = view(q.rows(), cols), a.out_t = view(q.cols(), rows);
  a.n_cols = static_cast<int32_t>(gate_cols);
  check(mxb200_residual_norm_mx_fwd(&a, stream()), "residual_norm_mx");
  return {res, n, q.data, q.data_t, q.scale, q.scale_t, rstd, s};
}

// (x, out, out_t) jobs; out and out_t are ctypes structures laid out as mxb200_mx_out.
mxb200_mx_out mx_out_of(PyObject* o) {
  Py_buffer b;
  if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0)
    throw py::error_already_set();
  const bool ok = b.len == static_cast<Py_ssize_t>(sizeof(mxb200_mx_out));
  mxb200_mx_out out = kNoLayout;
  if (ok)
    std::memcpy(&out, b.buf, sizeof(out));
  PyBuffer_Release(&b);
  require(ok, "MX: expected an MxOut");
  return out;
}

void quantize_mx_batch_into(const py::sequence& jobs, int scale_rule) {
  const size_t count = jobs.size();
  if (count == 0)
    return;
  std::vector<mxb200_quantize_job> list;
  list.reserve(count);
  std::optional<at::ScalarType> dtype;
  std::optional<at::Device> device;
  for (size_t i = 0; i < count; ++i) {
    const py::object item = jobs[i];
    const auto job = py::reinterpret_borrow<py::sequence>(item);
    require(job.size() == 3, "MX: a job is (x, out, out_t)");
    const py::object px = job[0], po = job[1], pt = job[2];
    const Tensor x = px.cast<Tensor>();
    if (i == 0)
      require_cuda(x, "quantize_mx_batch"), dtype = x.scalar_type(), device = x.device();
    require(x.is_cuda() && x.dim() == 2 && x.is_contiguous() && fits(x.size(0), x.size(1)) && x.scalar_type() == *dtype &&
                  (*dtype == at::kBFloat16 || *dtype == at::kFloat) && x.device() == *device,
            "MX: expected aligned, contiguous 2D tensors of one dtype with dims % 128");
    list.push_back({x.data_ptr(), x.size(0), x.size(1), mx_out_of(po.ptr()), mx_out_of(pt.ptr())});
  }
  const py::gil_scoped_release nogil;
  check(mxb200_quantize_mx_batch(list.data(), static_cast<int>(count), *dtype == at::kBFloat16, scale_rule, stream()),
        "quantize_mx_batch");
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.doc() = "Native host path of nanochat_cpp_b200.engine.";
  m.attr("built_for") = MXB200_BUILT_FOR;  // build.py looks for it in the file
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p)
        std::rethrow_exception(p);
    } catch (python_error& e) {
      e.restore();
    }
  });
  py::class_<WeightCache>(m, "WeightCache")
        .def(py::init<bool>(), py::arg("enabled") = false)
        .def_readwrite("enabled", &WeightCache::enabled)
        .def("get", &WeightCache::get, py::arg("kind"), py::arg("weights"), py::arg("make"));
  m.def("fp8_matmul", &fp8_matmul);
  m.def("fp8_qkv", &fp8_qkv);
  m.def("fp8_relu_square_mlp", &fp8_relu_square_mlp);
  m.def("softcap_cross_entropy", &softcap_cross_entropy);
  m.def("residual_norm_mx", &residual_norm_mx, py::call_guard<py::gil_scoped_release>());
  m.def("quantize_mx_batch_into", &quantize_mx_batch_into);
}
