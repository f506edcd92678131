// Native autograd nodes for the calls a training program makes most: linear, RMSNorm (with and without residual),
// SwiGLU, cross entropy and attention.
//
// Same kernels, outputs and gradients as the Python nodes of ops/functional.py and ops/attention.py, without their
// interpreter time: small layers are bound by it (linear forward + backward of 512 x 256 -> 512: 24 us of kernels, 146 us a
// pass through the Python node and 65 through this one).  Every entry takes the plain case only -- dense bf16 CUDA tensors of the
// exact tensor type, aligned, no tracing, no function transform, no dispatch mode, no forward-mode gradient, no engine
// attributes on the weight -- and returns None for anything else; the caller then runs the Python node, which handles or
// refuses it as it always did.
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <atomic>
#include <cstdint>
#include <string>

namespace py = pybind11;
using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

namespace {

// ------------------------------------------------------------------ the kernel library's entry points
using P = const void*;
struct Kernels {
  int (*gemm)(P, P, P, int, int, int, int, int, int, int, int, int, int, P, P, P);
  int (*gemm_workspace)(int, int, int);
  int (*rmsnorm_parts)(int);
  int (*rmsnorm_fwd)(P, P, P, P, P, P, int, int, float, P);
  int (*rmsnorm_bwd)(P, P, P, P, P, P, P, P, int, int, int, P);
  int (*swiglu_fwd)(P, P, int64_t, int, P);
  int (*swiglu_bwd)(P, P, P, int64_t, int, P);
  int (*xent)(P, P, P, int, int, int, float, int64_t, P);
  int (*attn_fwd)(P, P, P, P, P, int, int, int, int, int, int, int, int, float, P, P);
  int (*attn_bwd)(P, P, P, P, P, P, P, P, P, P, int, int, int, int, int, int, int, int, int, int, int, float, P, P, int);
};
Kernels kernels;
PyObject* kernel_error = nullptr;     // KernelError
PyObject* status_of = nullptr;        // device index -> address of its status word, which lives as long as the process
PyObject* linear_wgrad = nullptr;     // (weight, dy, x) -> gradient or None: the Python node's weight gradient
PyObject* norm_wgrad_target = nullptr;  // weight -> (buffer or None, accumulate)
std::atomic<int64_t> launched{0};

constexpr int kMaxDevices = 64;
std::atomic<const void*> status_words[kMaxDevices];

const void* status_word(const Tensor& t) {
  const int dev = t.get_device();
  const void* p = status_words[dev].load(std::memory_order_acquire);
  if (p == nullptr) {
    py::gil_scoped_acquire gil;
    p = reinterpret_cast<const void*>(py::cast<uintptr_t>(py::handle(status_of)(dev)));
    status_words[dev].store(p, std::memory_order_release);
  }
  return p;
}

const void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

void check(int code, const char* what) {
  if (code == 0) return;
  py::gil_scoped_acquire gil;
  PyErr_SetString(kernel_error, (std::string(what) + " failed with CUDA error code " + std::to_string(code)).c_str());
  throw py::error_already_set();
}

// ------------------------------------------------------------------ the plain case
bool plain_context() {
  // the front mode is included while any function transform (grad, vmap, jvp, ...) runs
  return !c10::impl::dispatch_mode_enabled() &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
         !torch::jit::tracer::isTracing();
}
bool plain(const py::handle& h, at::ScalarType type = at::kBFloat16) {
  if (!THPVariable_CheckExact(h.ptr())) return false;
  const Tensor& t = THPVariable_Unpack(h.ptr());
  return t.is_cuda() && t.scalar_type() == type && t.has_storage() && t.layout() == at::kStrided && !t.is_neg() && !t.is_conj() &&
         t.get_device() < kMaxDevices && t.numel() > 0 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && !t._fw_grad(0).defined();
}
// A weight that carries `main_grad` at the forward pass belongs to the Python nodes.  The buffer may also be given to it
// between the passes, and the weight's own attributes decide: what a saved-tensor hook (offloading, activation
// checkpointing) unpacks is another tensor without them.  So the weight itself travels beside the saved tensors.
bool has_main_grad(py::handle weight) { return PyObject_HasAttrString(weight.ptr(), "main_grad") != 0; }
void keep_weight(AutogradContext* ctx, const Tensor& w) { ctx->saved_data["weight"] = w; }
Tensor kept_weight(AutogradContext* ctx) { return ctx->saved_data["weight"].toTensor(); }
bool has_main_grad(const Tensor& weight) {
  py::gil_scoped_acquire gil;
  return has_main_grad(py::reinterpret_steal<py::object>(THPVariable_Wrap(weight)));
}
// Runs a node's forward pass as torch runs its own operators and ctypes its calls: without the interpreter lock.  An allocation
// or a launch may block behind a collective that hangs, and the Python thread that aborts it has to run.
template <typename Apply>
auto unlocked(Apply apply) {
  py::gil_scoped_release no_gil;
  return apply();
}
bool fits_int(int64_t v) { return v >= 0 && v <= INT32_MAX; }

// The kernels read dense rows in vectors of 16 bytes.
bool aligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
Tensor dense(const Tensor& t) {
  if (!t.is_contiguous()) return t.contiguous();
  return aligned(t) ? t : t.clone();
}

// A saved tensor in the backward pass.  A hook may have unpacked another one than the forward pass looked at: of any strides
// and at any address, which a copy mends, or of another kind, which is refused.
bool is_operand(const Tensor& t, at::IntArrayRef sizes, const Tensor& grad, at::ScalarType type) {
  return t.defined() && t.is_cuda() && t.device() == grad.device() && t.layout() == at::kStrided && t.scalar_type() == type &&
         t.sizes() == sizes;
}
Tensor operand(const Tensor& t, at::IntArrayRef sizes, const Tensor& grad, at::ScalarType type = at::kBFloat16) {
  TORCH_CHECK(is_operand(t, sizes, grad, type), "a saved tensor is another in the backward pass (replaced, or unpacked by a saved-tensor hook) than the forward pass saved");
  return dense(t);
}

// ------------------------------------------------------------------ linear
// out [M, N] = op(a) op(b): a is [M, K], or [K, M] with a_mn; b is [N, K], or [K, N] with b_mn.  All dense.
void gemm(const Tensor& a, const Tensor& b, const Tensor& out, int64_t M, int64_t N, int64_t K, bool a_mn, bool b_mn) {
  const int floats = kernels.gemm_workspace(M, N, K);
  const Tensor workspace = floats ? at::empty({floats}, a.options().dtype(at::kFloat)) : Tensor();
  check(kernels.gemm(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a_mn ? M : K, b_mn ? N : K, N, a_mn, b_mn, 0, 0,
                     status_word(a), floats ? workspace.data_ptr() : nullptr, stream()),
        "tft_gemm_bf16");
  launched += floats ? 2 : 1;
}

struct Linear : public Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w) {
    const int64_t N = w.size(0), K = w.size(1), M = x.numel() / K;
    auto sizes = x.sizes().vec();
    sizes.back() = N;
    Tensor y = at::empty(sizes, x.options());
    gemm(x, w, y, M, N, K, false, false);
    ctx->save_for_backward({x, w});
    keep_weight(ctx, w);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor dy = dense(grads[0]), weight = kept_weight(ctx);
    // the gradient's shape is the output's; a weight whose data was replaced since is refused with the saved one
    const int64_t N = dy.size(-1), K = weight.size(-1), M = dy.numel() / N;
    auto sizes = dy.sizes().vec();
    sizes.back() = K;
    const Tensor x = operand(saved[0], sizes, dy), w = operand(saved[1], {N, K}, dy);
    Tensor dx, dw;
    if (ctx->needs_input_grad(0)) {
      dx = at::empty_like(x);
      gemm(dy, w, dx, M, K, N, false, true);
    }
    if (ctx->needs_input_grad(1)) {
      if (has_main_grad(weight)) {  // given to it since the forward pass
        py::gil_scoped_acquire gil;
        const py::object g = py::handle(linear_wgrad)(weight, dy.view({M, N}), x.view({M, K}));
        if (!g.is_none()) dw = g.cast<Tensor>();
      } else {
        dw = at::empty({N, K}, w.options());
        gemm(dy, x, dw, N, K, M, true, true);
      }
    }
    return {dx, dw};
  }
};

py::object linear(py::handle hx, py::handle hw) {
  if (!plain(hx) || !plain(hw) || !plain_context()) return py::none();
  const Tensor &x = THPVariable_Unpack(hx.ptr()), &w = THPVariable_Unpack(hw.ptr());
  if (w.dim() != 2 || x.dim() < 1 || x.size(-1) != w.size(1) || !x.is_contiguous() || !w.is_contiguous() || w.size(0) % 8 ||
      w.size(1) % 8 || !fits_int(x.numel() / w.size(1)) || !fits_int(w.size(0)) || !fits_int(w.size(1)) ||
      x.get_device() != w.get_device())
    return py::none();
  if (has_main_grad(hw) || PyObject_HasAttrString(hw.ptr(), "gather_comm")) return py::none();
  return py::cast(unlocked([&] { return Linear::apply(x, w); }));
}

// ------------------------------------------------------------------ RMSNorm
// The kernel's split of a row over threads: dim = threads * 8 * v with 32 | threads <= 512 and v <= 4.
bool norm_dim(int64_t dim) {
  for (int v = 1; v <= 4; ++v)
    if (dim % (8 * v) == 0 && dim / (8 * v) % 32 == 0 && dim / (8 * v) <= 512) return true;
  return false;
}

// (dx, dw) of y = rmsnorm(h) * w; dres is added to dx.
std::pair<Tensor, Tensor> norm_backward(const Tensor& weight, const Tensor& grad_y, const variable_list& saved, const Tensor& grad_h) {
  const Tensor dy = dense(grad_y), dres = grad_h.defined() ? dense(grad_h) : grad_h;
  const int64_t dim = dy.size(-1), rows = dy.numel() / dim;
  const Tensor h = operand(saved[0], dy.sizes(), dy), w = operand(saved[1], {dim}, dy), rstd = operand(saved[2], {rows}, dy, at::kFloat);
  Tensor dx = at::empty_like(h), dw, out;
  bool accumulate = false;
  if (has_main_grad(weight)) {  // given to it since the forward pass
    py::gil_scoped_acquire gil;
    const py::tuple target = py::handle(norm_wgrad_target)(weight);
    if (!target[0].is_none()) out = target[0].cast<Tensor>();
    accumulate = target[1].cast<bool>();
  }
  if (!out.defined()) out = dw = at::empty_like(w);
  const Tensor partial = at::empty({kernels.rmsnorm_parts(static_cast<int>(rows)) * dim}, h.options().dtype(at::kFloat));
  check(kernels.rmsnorm_bwd(dy.data_ptr(), h.data_ptr(), w.data_ptr(), rstd.data_ptr(), dres.defined() ? dres.data_ptr() : nullptr,
                            dx.data_ptr(), out.data_ptr(), partial.data_ptr(), rows, dim, accumulate, stream()),
        "tft_rmsnorm_bwd");
  launched += 2;
  return {dx, dw};
}

struct RMSNorm : public Function<RMSNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps) {
    const int64_t dim = x.size(-1), rows = x.numel() / dim;
    Tensor y = at::empty_like(x), rstd = at::empty({rows}, x.options().dtype(at::kFloat));
    check(kernels.rmsnorm_fwd(x.data_ptr(), nullptr, w.data_ptr(), y.data_ptr(), nullptr, rstd.data_ptr(), rows, dim, eps, stream()),
          "tft_rmsnorm_fwd");
    ++launched;
    ctx->save_for_backward({x, w, rstd});
    keep_weight(ctx, w);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto [dx, dw] = norm_backward(kept_weight(ctx), grads[0], ctx->get_saved_variables(), Tensor());
    return {dx, dw, Tensor()};
  }
};

struct AddRMSNorm : public Function<AddRMSNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& res, const Tensor& w, double eps) {
    const int64_t dim = x.size(-1), rows = x.numel() / dim;
    Tensor y = at::empty_like(x), h = at::empty_like(x), rstd = at::empty({rows}, x.options().dtype(at::kFloat));
    check(kernels.rmsnorm_fwd(x.data_ptr(), res.data_ptr(), w.data_ptr(), y.data_ptr(), h.data_ptr(), rstd.data_ptr(), rows, dim, eps,
                              stream()),
          "tft_rmsnorm_fwd");
    ++launched;
    ctx->save_for_backward({h, w, rstd});
    keep_weight(ctx, w);
    return {y, h};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    // an output that took no part in the loss arrives as zeros, as in the Python node
    auto [dx, dw] = norm_backward(kept_weight(ctx), grads[0], ctx->get_saved_variables(), grads[1]);
    return {dx, dx, dw, Tensor()};
  }
};

bool plain_norm(py::handle hx, py::handle hw) {
  if (!plain(hx) || !plain(hw) || !plain_context()) return false;
  const Tensor &x = THPVariable_Unpack(hx.ptr()), &w = THPVariable_Unpack(hw.ptr());
  return x.dim() >= 1 && w.dim() == 1 && x.size(-1) == w.size(0) && x.is_contiguous() && w.is_contiguous() && norm_dim(w.size(0)) &&
         fits_int(x.numel() / w.size(0)) && x.get_device() == w.get_device() && !has_main_grad(hw);
}
py::object rmsnorm(py::handle hx, py::handle hw, double eps) {
  if (!plain_norm(hx, hw)) return py::none();
  const Tensor &x = THPVariable_Unpack(hx.ptr()), &w = THPVariable_Unpack(hw.ptr());
  return py::cast(unlocked([&] { return RMSNorm::apply(x, w, eps); }));
}
py::object add_rmsnorm(py::handle hx, py::handle hr, py::handle hw, double eps) {
  if (!plain_norm(hx, hw) || !plain(hr)) return py::none();
  const Tensor &x = THPVariable_Unpack(hx.ptr()), &res = THPVariable_Unpack(hr.ptr()), &w = THPVariable_Unpack(hw.ptr());
  if (!res.is_contiguous() || res.sizes() != x.sizes() || res.get_device() != x.get_device()) return py::none();
  const variable_list out = unlocked([&] { return AddRMSNorm::apply(x, res, w, eps); });
  return py::make_tuple(out[0], out[1]);
}

// ------------------------------------------------------------------ SwiGLU
struct SwiGLU : public Function<SwiGLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gu) {
    const int64_t F = gu.size(-1) / 2, rows = gu.numel() / (2 * F);
    auto sizes = gu.sizes().vec();
    sizes.back() = F;
    Tensor out = at::empty(sizes, gu.options());
    check(kernels.swiglu_fwd(gu.data_ptr(), out.data_ptr(), rows, F, stream()), "tft_swiglu_fwd");
    ++launched;
    ctx->save_for_backward({gu});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor dout = dense(grads[0]);
    const int64_t F = dout.size(-1), rows = dout.numel() / F;
    auto sizes = dout.sizes().vec();
    sizes.back() = 2 * F;
    const Tensor gu = operand(ctx->get_saved_variables()[0], sizes, dout);
    Tensor dgu = at::empty_like(gu);
    check(kernels.swiglu_bwd(gu.data_ptr(), dout.data_ptr(), dgu.data_ptr(), rows, F, stream()), "tft_swiglu_bwd");
    ++launched;
    return {dgu};
  }
};
py::object swiglu(py::handle h) {
  if (!plain(h) || !plain_context()) return py::none();
  const Tensor& gu = THPVariable_Unpack(h.ptr());
  if (gu.dim() < 1 || !gu.is_contiguous() || gu.size(-1) % 16 || !fits_int(gu.size(-1))) return py::none();
  return py::cast(unlocked([&] { return SwiGLU::apply(gu); }));
}

// ------------------------------------------------------------------ attention
int64_t token_stride(const Tensor& t) { return t.stride(1); }
bool plain_heads(const Tensor& t) {  // [B, S, H, D], heads packed inside a token row, sequences one after another
  return t.dim() == 4 && t.stride(3) == 1 && t.stride(2) == t.size(3) && t.stride(0) == t.stride(1) * t.size(1) &&
         t.stride(1) % 8 == 0 && fits_int(t.stride(1)) && t.stride(1) > 0;
}
Tensor heads_operand(const Tensor& t, at::IntArrayRef sizes, const Tensor& grad) {  // strided as it is where the kernel can
  return is_operand(t, sizes, grad, at::kBFloat16) && plain_heads(t) && aligned(t) ? t : operand(t, sizes, grad);
}
struct Attention : public Function<Attention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, double scale) {
    const int64_t B = q.size(0), S = q.size(1), Hq = q.size(2), D = q.size(3), Hkv = k.size(2);
    Tensor o = at::empty({B, S, Hq, D}, q.options()), lse = at::empty({B, Hq, S}, q.options().dtype(at::kFloat));
    check(kernels.attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), B, S, Hq, Hkv, D, token_stride(q),
                           token_stride(k), token_stride(v), scale, status_word(q), stream()),
          "tft_attn_fwd");
    ++launched;
    ctx->save_for_backward({q, k, v, o, lse});
    ctx->saved_data["scale"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor d_o = dense(grads[0]);
    const int64_t B = d_o.size(0), S = d_o.size(1), Hq = d_o.size(2), D = d_o.size(3), Hkv = s[1].size(2);
    const Tensor q = heads_operand(s[0], {B, S, Hq, D}, d_o), k = heads_operand(s[1], {B, S, Hkv, D}, d_o);
    const Tensor v = heads_operand(s[2], {B, S, Hkv, D}, d_o), o = operand(s[3], d_o.sizes(), d_o);
    const Tensor lse = operand(s[4], {B, Hq, S}, d_o, at::kFloat);
    Tensor dq = at::empty({B, S, Hq, D}, q.options()), dk = at::empty({B, S, Hkv, D}, q.options());
    Tensor dv = at::empty({B, S, Hkv, D}, q.options()), delta = at::empty({B, Hq, S}, lse.options());
    check(kernels.attn_bwd(d_o.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), delta.data_ptr(),
                           dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), B, S, Hq, Hkv, D, token_stride(q), token_stride(k),
                           token_stride(v), Hq * D, Hkv * D, Hkv * D, ctx->saved_data["scale"].toDouble(), status_word(q), stream(), 7),
          "tft_attn_bwd_tmem");
    launched += 3;
    return {dq, dk, dv, Tensor()};
  }
};
py::object attention(py::handle hq, py::handle hk, py::handle hv, double scale) {
  if (!plain(hq) || !plain(hk) || !plain(hv) || !plain_context()) return py::none();
  const Tensor &q = THPVariable_Unpack(hq.ptr()), &k = THPVariable_Unpack(hk.ptr()), &v = THPVariable_Unpack(hv.ptr());
  if (!plain_heads(q) || !plain_heads(k) || !plain_heads(v) || k.sizes() != v.sizes() || q.size(0) != k.size(0) ||
      q.size(1) != k.size(1) || q.size(3) != k.size(3) || (q.size(3) != 64 && q.size(3) != 128) || q.size(2) % k.size(2) || !(scale > 0) ||
      !fits_int(q.size(1)) || !fits_int(q.size(0)) || q.get_device() != k.get_device() || q.get_device() != v.get_device())
    return py::none();
  return py::cast(unlocked([&] { return Attention::apply(q, k, v, scale); }));
}

// ------------------------------------------------------------------ cross entropy (mean over all rows)
struct CrossEntropy : public Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& targets) {
    const int64_t V = logits.size(-1), rows = logits.numel() / V;
    const double scale = 1.0 / rows;
    Tensor loss_rows = at::empty({rows}, logits.options().dtype(at::kFloat));
    check(kernels.xent(logits.data_ptr(), targets.data_ptr(), loss_rows.data_ptr(), rows, V, V, scale, -100, stream()), "tft_xent");
    ++launched;
    ctx->save_for_backward({logits});  // now holds d loss / d logits
    return loss_rows.sum() * scale;
  }
  static variable_list backward(AutogradContext* ctx, variable_list) { return {ctx->get_saved_variables()[0], Tensor()}; }
};
py::object cross_entropy(py::handle hl, py::handle ht) {
  if (!plain(hl) || !plain(ht, at::kLong) || !plain_context()) return py::none();
  const Tensor &logits = THPVariable_Unpack(hl.ptr()), &targets = THPVariable_Unpack(ht.ptr());
  if (logits.dim() < 1 || !logits.is_contiguous() || !targets.is_contiguous() || logits.size(-1) % 8 || !fits_int(logits.size(-1)) ||
      !fits_int(logits.numel() / logits.size(-1)) || targets.numel() != logits.numel() / logits.size(-1) ||
      logits.get_device() != targets.get_device())
    return py::none();
  return py::cast(unlocked([&] { return CrossEntropy::apply(logits, targets); }));
}

template <typename F>
void take(const py::dict& entries, const char* name, F& fn) {
  fn = reinterpret_cast<F>(py::cast<uintptr_t>(entries[name]));
}

void setup(const py::dict& entries, py::object error, py::object status, py::object wgrad, py::object norm_target) {
  take(entries, "tft_gemm2_bf16", kernels.gemm);
  take(entries, "tft_gemm2_workspace", kernels.gemm_workspace);
  take(entries, "tft_rmsnorm_bwd_parts", kernels.rmsnorm_parts);
  take(entries, "tft_rmsnorm_fwd", kernels.rmsnorm_fwd);
  take(entries, "tft_rmsnorm_bwd", kernels.rmsnorm_bwd);
  take(entries, "tft_swiglu_fwd", kernels.swiglu_fwd);
  take(entries, "tft_swiglu_bwd", kernels.swiglu_bwd);
  take(entries, "tft_xent", kernels.xent);
  take(entries, "tft_attn_fwd_pair", kernels.attn_fwd);
  take(entries, "tft_attn_bwd_tmem", kernels.attn_bwd);
  kernel_error = error.release().ptr();
  status_of = status.release().ptr();
  linear_wgrad = wgrad.release().ptr();
  norm_wgrad_target = norm_target.release().ptr();
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.doc() = "Autograd nodes of the plain cases; every function returns None for a call that the Python node has to take.";
  m.attr("torch_mark") = TFT_TORCH_MARK;  // which torch this was built against (utils/build.py)
  m.def("setup", &setup);
  m.def("launches", [] { return launched.load(); });
  m.def("linear", &linear);
  m.def("rmsnorm", &rmsnorm);
  m.def("add_rmsnorm", &add_rmsnorm);
  m.def("swiglu", &swiglu);
  m.def("attention", &attention);
  m.def("cross_entropy", &cross_entropy);
}
