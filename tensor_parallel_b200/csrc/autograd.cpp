// Autograd nodes of the layers whose training calls are bound by the host at ordinary sizes: linear and norms.
//
// A small call (100 tokens through a 768 x 3072 projection with bias, forward and backward) keeps the GPU busy for 37 us.  As Python
// autograd functions over ctypes it took 176 us: each of its launches cost 10 to 20 us of interpreter work, and the backward nodes
// ran under the interpreter lock on the autograd thread.  The same nodes in C++ enqueue the same kernels, with the same shapes,
// copies and saved tensors, without entering the interpreter.
//
// The module has no link to the kernel library: `bind` receives the entry points of the library that ops/native.py loaded
// (a variant with index checks, for instance), and the two callbacks that need Python objects.
#include <torch/extension.h>

#include <c10/cuda/CUDAStream.h>

#include <atomic>
#include <stdexcept>
#include <string>

#include "tpb_api.h"

namespace py = pybind11;
using at::Tensor;

namespace {

struct Library {
  decltype(&tpb_gemm_plan_ex) plan = nullptr;
  decltype(&tpb_gemm_bf16_ex) gemm = nullptr;
  decltype(&tpb_norm_fwd) norm_fwd = nullptr;
  decltype(&tpb_norm_bwd) norm_bwd = nullptr;
  decltype(&tpb_norm_bwd_parts) norm_bwd_parts = nullptr;
  decltype(&tpb_col_sum_parts) col_sum_parts = nullptr;
  decltype(&tpb_col_sum) col_sum = nullptr;
};
Library lib;
PyObject* error_text = nullptr;     // (code, what) -> message
PyObject* reserve_slots = nullptr;  // (device index, fp32 elements) -> address of the device's reduction context
constexpr int MAX_DEVICES = 64;
std::atomic<tpb_reduce_ctx_t*> contexts[MAX_DEVICES];
std::atomic<long long> launched{0};

void check(int code, const char* what) {
  if (code == TPB_OK) return;
  std::string text = std::string(what) + " failed: " + std::to_string(code);
  {
    py::gil_scoped_acquire gil;
    try {
      text = py::reinterpret_borrow<py::function>(error_text)(code, what).cast<std::string>();
    } catch (py::error_already_set& e) {
      e.discard_as_unraisable("error text of a native kernel");
    }
  }
  throw std::runtime_error(text);
}

// The reduction context of a device, with at least `elems` fp32 elements per slot.  It lives as long as the process.
tpb_reduce_ctx_t* context(const Tensor& t, size_t elems) {
  const int device = t.is_cuda() ? t.get_device() : 0;
  TORCH_CHECK(device >= 0 && device < MAX_DEVICES, "device index out of range");
  tpb_reduce_ctx_t* c = contexts[device].load(std::memory_order_acquire);
  if (c && elems <= c->slot_stride) return c;
  std::string problem;
  {
    py::gil_scoped_acquire gil;
    try {
      const auto address = py::reinterpret_borrow<py::function>(reserve_slots)(device, elems).cast<uintptr_t>();
      c = reinterpret_cast<tpb_reduce_ctx_t*>(address);
    } catch (py::error_already_set& e) {
      problem = e.what();
    }
  }
  if (!problem.empty()) throw std::runtime_error(problem);
  contexts[device].store(c, std::memory_order_release);
  return c;
}

void* stream_of(const Tensor& t) {
  return t.is_cuda() ? static_cast<void*>(c10::cuda::getCurrentCUDAStream().stream()) : nullptr;
}

Tensor or_undefined(const std::optional<Tensor>& t) { return t.has_value() ? *t : Tensor(); }
const void* data(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }

// TMA needs a unit inner stride, a 16-byte aligned base and a row pitch that is a multiple of 16 bytes; other operands are copied.
Tensor tma_ready(const Tensor& t) {
  if (t.stride(1) == 1 && t.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0) return t;
  const int64_t rows = t.size(0), cols = t.size(1);
  Tensor view = at::empty({rows, (cols + 7) / 8 * 8}, t.options()).slice(1, 0, cols);
  view.copy_(t);
  return view;
}

// out[tokens, features] = x w^T + bias; x_t / w_t: that operand lies transposed in memory ([k, tokens] / [k, features]).  `sum`, if defined, is
// what the product is added to, and what is returned.
Tensor gemm(const Tensor& x_in, const Tensor& w_in, const Tensor& bias, bool x_t, bool w_t, const Tensor& sum = Tensor()) {
  if (x_in.scalar_type() != at::kBFloat16 || w_in.scalar_type() != at::kBFloat16)  // (the kernel takes its operands' element size for granted)
    throw py::type_error("native GEMMs take bf16 operands, got " + std::string(at::toString(x_in.scalar_type())) + " and " + at::toString(w_in.scalar_type()));
  const int64_t tokens = x_in.size(x_t ? 1 : 0), k = x_in.size(x_t ? 0 : 1), features = w_in.size(w_t ? 1 : 0);
  TORCH_CHECK(x_in.dim() == 2 && w_in.dim() == 2 && w_in.size(w_t ? 0 : 1) == k, "operands of a native GEMM of ", x_in.sizes(), " and ", w_in.sizes(),
              " do not contract");
  const Tensor x = tma_ready(x_in), w = tma_ready(w_in);
  Tensor out = sum.defined() ? sum : at::empty({tokens, features}, x.options());
  tpb_gemm_plan_t plan;
  check(lib.plan(int(tokens), int(features), int(k), 1, 0, 0, int(x_t || w_t), &plan), "gemm_plan");
  tpb_reduce_ctx_t* rc = context(x, plan.reduce && !plan.stream ? size_t(tokens) * size_t(out.stride(0)) : 0);
  tpb_gemm_opts_t opts = {};
  opts.x_mn = x_t;
  opts.w_mn = w_t;
  check(lib.gemm(x.const_data_ptr(), w.const_data_ptr(), out.mutable_data_ptr(), data(bias), data(sum), int(tokens), int(features), int(k), int(x.stride(0)),
                 int(w.stride(0)), int(out.stride(0)), 0, 1.f, &plan, rc, x_t || w_t ? &opts : nullptr, stream_of(x)),
        "tpb_gemm_bf16");
  launched.fetch_add(1, std::memory_order_relaxed);
  return out;
}

// What a call costs beside its launches is tensor operations that change nothing, 0.5 to 1 us each: a view or a conversion is taken only where
// shape or type ask for it.
Tensor rows_of(const Tensor& x) { return x.dim() == 2 ? x : x.reshape({-1, x.size(-1)}); }
Tensor as_type(const Tensor& t, at::ScalarType dtype) { return t.scalar_type() == dtype ? t : t.to(dtype); }

// Rows as the leading dimensions of x have it.
Tensor shaped_as(const Tensor& rows, const Tensor& x) {
  if (x.dim() == 2) return rows;
  std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = rows.size(1);
  return rows.view(shape);
}
// The shape of an input, kept for its gradient where that is not its rows' (empty otherwise).
std::vector<int64_t> shape_of(const Tensor& x) { return x.dim() == 2 ? std::vector<int64_t>() : x.sizes().vec(); }
Tensor in_shape(const Tensor& rows, const c10::IValue& shape) {
  const auto sizes = shape.toIntVector();
  return sizes.empty() ? rows : rows.view(sizes);
}

// Whether something goes on around a gradient that a kernel would drop out of: a graph of its own (create_graph), a batch of gradients
// (is_grads_batched) or another transform, a tensor subclass.
bool more_than_numbers(const Tensor& g) {
  return (at::GradMode::is_enabled() && g.requires_grad()) || !g.has_storage() || g.unsafeGetTensorImpl()->is_python_dispatch();
}

// The gradient of a bias: column sums of g in fp32, as `dtype`.
Tensor column_sums(const Tensor& g, at::ScalarType dtype) {
  if (!lib.col_sum || more_than_numbers(g) || g.size(0) == 0 || g.size(1) % 8 || (dtype != at::kBFloat16 && dtype != at::kFloat) ||
      reinterpret_cast<uintptr_t>(g.const_data_ptr()) % 16)
    return g.sum(at::IntArrayRef{0}, false, at::kFloat).to(dtype);  // (summed in fp32 without an fp32 copy of the gradient)
  const int rows = int(g.size(0)), cols = int(g.size(1)), parts = lib.col_sum_parts(rows, cols);
  Tensor out = at::empty({cols}, g.options().dtype(dtype)), partials = parts > 1 ? at::empty({parts, cols}, g.options().dtype(at::kFloat)) : Tensor();
  check(lib.col_sum(g.const_data_ptr(), out.mutable_data_ptr(), parts > 1 ? partials.data_ptr<float>() : nullptr, rows, cols, dtype == at::kFloat, stream_of(g)),
        "tpb_col_sum");  // (not among the launches: those of a linear layer are its GEMMs)
  return out;
}

struct LinearFn : torch::autograd::Function<LinearFn> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& weight, const std::optional<Tensor>& bias_) {
    const Tensor bias = or_undefined(bias_);
    const Tensor x2d = rows_of(x);
    const Tensor out = gemm(x2d, weight, bias, false, false);
    ctx->save_for_backward({x2d, weight});
    ctx->saved_data["shape"] = shape_of(x);
    ctx->saved_data["bias"] = bias.defined();
    return shaped_as(out, x);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2d = saved[0], &weight = saved[1], &grad = grads[0];
    const Tensor g = as_type(rows_of(grad), at::kBFloat16).contiguous();
    Tensor gx, gw, gb;
    if (ctx->needs_input_grad(0)) gx = in_shape(gemm(g, weight, Tensor(), false, true), ctx->saved_data["shape"]);
    if (ctx->needs_input_grad(1)) gw = gemm(g, x2d, Tensor(), true, true);
    if (ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(2))
      gb = column_sums(g, grad.scalar_type());
    return {gx, gw, gb};
  }
};

// Several projections of one input, without biases.  As nodes of their own they leave the sum of their gradients of the input to the engine, which
// reads and writes each of them once more (three of 8192 x 4096: 59 us); here the second and third GEMM add to what the one before stored.
struct LinearsFn : torch::autograd::Function<LinearsFn> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& x, at::TensorList weights) {
    const Tensor x2d = rows_of(x);
    torch::autograd::variable_list outs, saved{x2d};
    for (const Tensor& w : weights) {
      outs.push_back(shaped_as(gemm(x2d, w, Tensor(), false, false), x));
      saved.push_back(w);
    }
    ctx->save_for_backward(saved);
    ctx->saved_data["shape"] = shape_of(x);
    ctx->set_materialize_grads(false);
    return outs;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    torch::autograd::variable_list out(1 + grads.size());
    Tensor gx;
    for (size_t i = grads.size(); i-- > 0;) {  // (the engine's order, so that there are only roundings fewer; q, the largest where k and v have fewer heads, last)
      if (!grads[i].defined()) continue;       // (nobody used that projection)
      const Tensor g = as_type(rows_of(grads[i]), at::kBFloat16).contiguous();
      if (ctx->needs_input_grad(0)) gx = gemm(g, saved[1 + i], Tensor(), false, true, gx);
      if (ctx->needs_input_grad(1 + i)) out[1 + i] = gemm(g, saved[0], Tensor(), true, true);
    }
    if (gx.defined()) out[0] = in_shape(gx, ctx->saved_data["shape"]);
    return out;
  }
};

std::vector<Tensor> linears(const Tensor& x, const std::vector<Tensor>& weights) { return LinearsFn::apply(x, at::TensorList(weights)); }

Tensor linear(const Tensor& x, const Tensor& weight, const std::optional<Tensor>& bias_) {
  const Tensor bias = or_undefined(bias_);
  if (at::GradMode::is_enabled() && (x.requires_grad() || weight.requires_grad() || (bias.defined() && bias.requires_grad())))
    return LinearFn::apply(x, weight, bias_);
  return shaped_as(gemm(rows_of(x), weight, bias, false, false), x);
}

int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16) return 0;
  if (t.scalar_type() == at::kFloat) return 1;
  throw py::type_error("native kernels take bf16 or fp32 tensors, got " + std::string(at::toString(t.scalar_type())));
}

// mode 0: RMSNorm, 1: LayerNorm, of bf16 or fp32 rows.
struct NormFn : torch::autograd::Function<NormFn> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const std::optional<Tensor>& weight_, const std::optional<Tensor>& bias_,
                        double eps, int64_t mode) {
    const Tensor weight = or_undefined(weight_), bias = or_undefined(bias_);
    const int dtype = dtype_code(x);
    const Tensor x2d = rows_of(x).contiguous();
    const Tensor w = weight.defined() ? as_type(weight, x.scalar_type()).contiguous() : Tensor();
    const Tensor b = bias.defined() ? as_type(bias, x.scalar_type()).contiguous() : Tensor();
    const int64_t rows = x2d.size(0), cols = x2d.size(1);
    Tensor out = at::empty_like(x2d);
    Tensor stats = at::empty({mode == 1 ? 2 : 1, rows}, x2d.options().dtype(at::kFloat));  // 1 / deviation, and for LayerNorm the mean, of every row
    float* rstd = stats.data_ptr<float>();
    check(lib.norm_fwd(x2d.const_data_ptr(), nullptr, data(w), data(b), out.mutable_data_ptr(), nullptr, rstd, mode == 1 ? rstd + rows : nullptr, int(rows),
                       int(cols), float(eps), int(mode), dtype, stream_of(x2d)),
          "tpb_norm_fwd");
    launched.fetch_add(1, std::memory_order_relaxed);
    ctx->save_for_backward({x2d, w, stats});
    ctx->saved_data["shape"] = shape_of(x);
    ctx->saved_data["meta"] = std::vector<int64_t>{mode, weight.defined() ? int64_t(weight.scalar_type()) : int64_t(-1),
                                                   bias.defined() ? int64_t(bias.scalar_type()) : int64_t(-1)};
    return shaped_as(out, x);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x2d = saved[0], &w = saved[1], &stats = saved[2];
    const auto meta = ctx->saved_data["meta"].toIntVector();
    const int64_t mode = meta[0], wdtype = meta[1], bdtype = meta[2];
    const Tensor g = as_type(rows_of(grads[0]), x2d.scalar_type()).contiguous();
    const int64_t rows = x2d.size(0), cols = x2d.size(1);
    Tensor dx = at::empty_like(x2d);
    // column sums: one fp32 partial row per CTA, added up by a second kernel that writes the gradients in their own dtype
    const bool has_w = wdtype >= 0, has_b = bdtype >= 0;
    const bool narrow = has_w && (!has_b || bdtype == wdtype) && wdtype == int64_t(at::kBFloat16);
    const int parts = lib.norm_bwd_parts(int(rows), int(cols));
    const auto fp32 = x2d.options().dtype(at::kFloat);
    const auto as_grad = narrow ? x2d.options().dtype(at::kBFloat16) : fp32;
    Tensor partials = has_w || has_b ? at::empty({int(has_w) + int(has_b), parts, cols}, fp32) : Tensor();
    float* part_w = has_w ? partials.data_ptr<float>() : nullptr;
    float* part_b = has_b ? partials.data_ptr<float>() + (has_w ? int64_t(parts) * cols : 0) : nullptr;
    const float* rstd = stats.const_data_ptr<float>();
    Tensor dw = has_w ? at::empty({cols}, as_grad) : Tensor(), db = has_b ? at::empty({cols}, as_grad) : Tensor();
    auto out = [](Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; };
    check(lib.norm_bwd(g.const_data_ptr(), x2d.const_data_ptr(), data(w), rstd, mode == 1 ? rstd + rows : nullptr, dx.mutable_data_ptr(), part_w, part_b, out(dw),
                       out(db), int(rows), int(cols), int(mode), dtype_code(x2d), narrow ? 0 : 1, stream_of(x2d)),
          "tpb_norm_bwd");
    launched.fetch_add(has_w || has_b ? 2 : 1, std::memory_order_relaxed);
    if (has_w) dw = as_type(dw, at::ScalarType(wdtype));
    if (has_b) db = as_type(db, at::ScalarType(bdtype));
    return {in_shape(dx, ctx->saved_data["shape"]), dw, db, Tensor(), Tensor()};
  }
};

Tensor norm(const Tensor& x, const std::optional<Tensor>& weight, const std::optional<Tensor>& bias, double eps, int64_t mode) {
  return NormFn::apply(x, weight, bias, eps, mode);
}

template <typename F>
void entry(F& f, const py::dict& addresses, const char* name) {
  f = reinterpret_cast<F>(addresses[name].cast<uintptr_t>());
}

void bind(const py::dict& addresses, py::function text, py::function reserve) {
  entry(lib.plan, addresses, "tpb_gemm_plan_ex");
  entry(lib.gemm, addresses, "tpb_gemm_bf16_ex");
  entry(lib.norm_fwd, addresses, "tpb_norm_fwd");
  entry(lib.norm_bwd, addresses, "tpb_norm_bwd");
  entry(lib.norm_bwd_parts, addresses, "tpb_norm_bwd_parts");
  if (addresses.contains("tpb_col_sum")) {
    entry(lib.col_sum_parts, addresses, "tpb_col_sum_parts");
    entry(lib.col_sum, addresses, "tpb_col_sum");
  } else {
    lib.col_sum = nullptr;
  }
  Py_XDECREF(error_text);
  Py_XDECREF(reserve_slots);
  error_text = text.release().ptr();  // (kept for the life of the process, beyond the interpreter's teardown of module globals)
  reserve_slots = reserve.release().ptr();
  for (auto& c : contexts) c.store(nullptr, std::memory_order_release);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("bind", &bind);
  m.def("layout", [] { return TPB_API_LAYOUT; });  // of the structures that it hands to the library it is bound to
  m.def("launches", [] { return launched.load(std::memory_order_relaxed); });
  const auto unlocked = py::call_guard<py::gil_scoped_release>();
  m.def("linear", &linear, unlocked);
  m.def("linears", &linears, unlocked);
  m.def("norm", &norm, unlocked);
}
