// Autograd nodes of the training path without Python in them: token table, norms, SwiGLU, rotation of a fused projection, attention, vocabulary
// loss and the linear layer of one rank.  Each does what the torch.autograd.Function of the same name in ops/ or parallel_layers/layers.py does
// (the same kernels on the same tensors, the same tensors saved); those stay for CPU tensors, tensor subclasses, recording, tracing,
// functorch and forward-mode AD, which the callers ask about (ops/_ext.py native()).  A node in Python costs about 20 us forward and 40 us
// backward (its context, the interpreter's lock in the engine's thread, a dozen calls), a small training step had 23 of them: 2750 us a step
// with them, 1900 with the first of these.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <atomic>

#include "bindings.h"
#include "kernels.h"

namespace py = pybind11;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

namespace {

std::atomic<int64_t> g_launches{0};                        // kernels of this package that were launched from here
void count(int64_t n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }

Tensor rows(const Tensor& t) { return t.reshape({-1, t.size(-1)}); }
bool aligned(const Tensor& t) { return (uintptr_t)t.data_ptr() % 16 == 0; }

// ---------------------------------------------------------------------------------------------------------------- norms
struct RmsNorm : Function<RmsNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps) {
    const Tensor x2 = rows(x);
    count();
    auto o = rmsnorm_fwd(x2.contiguous(), w.contiguous(), eps);
    ctx->save_for_backward({x2, w, o[1]});
    return o[0].view(x.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    count(2);
    auto o = rmsnorm_bwd(rows(g[0]).contiguous(), s[0].contiguous(), s[1].contiguous(), s[2]);
    return {o[0].view(g[0].sizes()), o[1], Tensor()};
  }
};

struct AddRmsNorm : Function<AddRmsNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& r, const Tensor& w, double eps) {
    count();
    auto o = add_rmsnorm_fwd(rows(x).contiguous(), rows(r).contiguous(), w.contiguous(), eps);
    ctx->save_for_backward({o[1], w, o[2]});
    return {o[0].view(x.sizes()), o[1].view(x.sizes())};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    count(2);
    auto o = add_rmsnorm_bwd(rows(g[0]).contiguous(), rows(g[1]).contiguous(), s[0], s[1].contiguous(), s[2]);
    const Tensor dh = o[0].view(g[0].sizes());
    return {dh, dh, o[1], Tensor()};
  }
};

// --------------------------------------------------------------------------------------------------------------- SwiGLU
struct SwiGLU : Function<SwiGLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gate_up) {
    ctx->save_for_backward({gate_up});
    count();
    auto shape = gate_up.sizes().vec();
    shape.back() /= 2;
    return swiglu_fwd(rows(gate_up).contiguous()).view(shape);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const Tensor gate_up = ctx->get_saved_variables()[0];
    count();
    return {swiglu_bwd(rows(g[0]).contiguous(), rows(gate_up).contiguous()).view(gate_up.sizes())};
  }
};

// -------------------------------------------------------------------------------------- rotation of a fused projection
Tensor packets(const Tensor& t) {
  const int64_t per = 16 / t.element_size();
  bool ok = t.stride(3) == 1 && aligned(t);
  for (int d = 0; d < 3; ++d) ok = ok && (t.size(d) == 1 || t.stride(d) % per == 0);
  return ok ? t : t.contiguous();
}

struct RopeQKV : Function<RopeQKV> {
  static variable_list forward(AutogradContext* ctx, const Tensor& qkv, const Tensor& cos_, const Tensor& sin_, int64_t heads, int64_t kv_heads) {
    const Tensor c = cos_.contiguous().to(at::kFloat), s = sin_.contiguous().to(at::kFloat);
    ctx->save_for_backward({c, s});
    count();
    auto o = rope_qkv_fwd(qkv, c, s, heads, kv_heads);
    const int64_t D = o[0].size(-1);
    const Tensor v = qkv.slice(-1, (heads + kv_heads) * D).unflatten(-1, {kv_heads, D}).transpose(0, 1);
    return {o[0], o[1], v};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    count();
    return {rope_qkv_bwd(packets(g[0]), packets(g[1]), packets(g[2]), s[0], s[1]), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------------------ attention
// What the kernels' maps take as it is: head_dim contiguous, sequences and heads whole rows apart or beside one another within a row; anything
// else is copied once (ops/attention.py _tma_view).
Tensor map_view(const Tensor& t) {
  if (t.stride(3) != 1 || !aligned(t)) return t.contiguous();
  const int64_t ss = t.stride(1);
  if (ss % 8) return t.contiguous();
  int64_t cols = 128;
  for (int d : {0, 2}) {
    const int64_t n = t.size(d), st = t.stride(d);
    if (n > 1 && !(st >= ss && st % std::max<int64_t>(ss, 1) == 0)) {
      if (st % 8) return t.contiguous();
      cols += (n - 1) * st;
    }
  }
  return cols > ss && t.size(1) > 1 ? t.contiguous() : t;
}

struct FlashAttention : Function<FlashAttention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_, bool causal, double scale) {
    const Tensor q = map_view(q_), k = map_view(k_), v = map_view(v_);
    count();
    auto o = flash_attn_fwd(q, k, v, causal, scale, true);
    ctx->save_for_backward({q, k, v, o[0], o[1]});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["scale"] = scale;
    return o[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    const bool causal = ctx->saved_data["causal"].toBool();
    const int H = (int)s[0].size(2), Hkv = (int)s[1].size(2);
    const int parts = H == Hkv ? 1 : nxd::flash_attn_bwd_parts((int)s[0].size(0), (int)s[0].size(1), (int)s[1].size(1), H, Hkv, causal);
    count(parts > 1 ? 4 : 3);
    auto o = flash_attn_bwd(map_view(g[0]), s[0], s[1], s[2], s[3], s[4], causal, ctx->saved_data["scale"].toDouble(), true, c10::nullopt, 0);
    return {o[0], o[1], o[2], Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------- vocabulary loss of one whole shard
struct CrossEntropy : Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& target) {
    const Tensor logits2 = rows(logits), tgt = target.reshape({-1});
    count();
    auto o = ce_loss(logits2.contiguous(), tgt.contiguous().to(at::kLong));
    ctx->save_for_backward({logits2, tgt, o[1]});
    ctx->saved_data["shape"] = logits.sizes();
    return o[0].view(target.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    count();
    const Tensor d = ce_backward(s[0].contiguous(), s[1].contiguous().to(at::kLong), s[2], g[0].reshape({-1}).to(at::kFloat).contiguous(), 0, 0.0,
                                 s[0].size(1));
    return {d.view(ctx->saved_data["shape"].toIntVector()), Tensor()};
  }
};

// Rows of a token table; the gradient (csrc/embedding_grad.cu) goes through autograd like the lookup's own, and only the ids are kept.
struct TableLookup : Function<TableLookup> {
  static Tensor forward(AutogradContext* ctx, const Tensor& ids, const Tensor& weight) {
    ctx->save_for_backward({ids});
    ctx->saved_data["rows"] = weight.size(0);
    return at::embedding(weight, ids);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const Tensor ids = ctx->get_saved_variables()[0];
    const int64_t n = ctx->saved_data["rows"].toInt();
    if (at::GradMode::is_enabled() || g[0].scalar_type() != at::kBFloat16)      // create_graph: the gradient is differentiated again
      return {Tensor(), at::embedding_dense_backward(g[0], ids, n, -1, false)};
    Tensor gy = rows(g[0]).contiguous();
    if (!aligned(gy)) gy = gy.clone();
    count(3);
    const Tensor out = at::empty({n, gy.size(1)}, gy.options());
    embedding_grad(ids.reshape({-1}).contiguous(), gy, out, true);
    return {Tensor(), out};
  }
};

// Mean of the losses of a causal language model's positions whose label is not -100: logits [S, B, V] of a whole vocabulary, labels [B, S].
// The labels are read in forward alone, so that their buffer may take the next batch at once.
struct CausalLoss : Function<CausalLoss> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& labels, bool shift) {
    const Tensor logits2 = rows(logits).contiguous();
    c10::cuda::CUDAGuard guard(logits.device());
    const auto st = c10::cuda::getCurrentCUDAStream().stream();
    const int64_t S = labels.size(1), B = labels.size(0), T = S * B;
    const Tensor target = at::empty({T}, labels.options()), mask = at::empty({T}, logits.options().dtype(at::kFloat));
    const Tensor mean = at::empty({}, mask.options()), divisor = at::empty({}, mask.options());
    nxd::lm_targets(labels.data_ptr<int64_t>(), labels.stride(0), labels.stride(1), target.data_ptr<int64_t>(), mask.data_ptr<float>(), (int)S, (int)B,
                    shift, st);
    auto o = ce_loss(logits2, target);
    nxd::lm_mean(o[0].data_ptr<float>(), mask.data_ptr<float>(), mean.data_ptr<float>(), divisor.data_ptr<float>(), (int)T, st);
    count(3);
    ctx->save_for_backward({logits2, target, o[1], mask, divisor});
    ctx->saved_data["shape"] = logits.sizes();
    return mean;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    c10::cuda::CUDAGuard guard(s[0].device());
    const Tensor gout = g[0].to(at::kFloat).contiguous(), grads = at::empty_like(s[3]);
    nxd::lm_row_grads(gout.data_ptr<float>(), s[4].data_ptr<float>(), s[3].data_ptr<float>(), grads.data_ptr<float>(), (int)grads.numel(),
                      c10::cuda::getCurrentCUDAStream().stream());
    count(2);
    const Tensor d = ce_backward(s[0], s[1], s[2], grads, 0, 0.0, s[0].size(1));
    return {d.view(ctx->saved_data["shape"].toIntVector()), Tensor(), Tensor()};
  }
};

// --------------------------------------------------------------------------------------------------------------- linear
// y = x Wᵀ of one rank.  The weight's gradient goes into its fp32 buffer where the optimizer gave it one (wgrad in
// parallel_layers/layers.py, which is called for whatever the kernels do not take as it is).
PyObject* g_wgrad = nullptr;                               // layers.wgrad
PyObject* g_fused_wgrad_enabled = nullptr;                 // ops.gemm.fused_wgrad_enabled

bool pairs(int64_t M, int64_t N) { return M > 128 || N <= 16384; }      // ops/gemm.py _pairs

void product(const Tensor& a, const Tensor& b, const Tensor& out, bool ta, bool tb, bool acc) {
  count();
  if (pairs(out.size(0), out.size(1))) gemm_bf16_2cta(a, b, out, ta, tb, acc);
  else gemm_bf16(a, b, out, ta, tb, acc);
}

// an attribute, or null where there is none
py::object attribute(PyObject* o, const char* name) {
  PyObject* v = PyObject_GetAttrString(o, name);
  if (!v) {
    if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw py::error_already_set();
    PyErr_Clear();
  }
  return py::reinterpret_steal<py::object>(v);
}

Tensor weight_gradient(const Tensor& go, const Tensor& x, const Tensor& weight) {
  py::gil_scoped_acquire gil;
  const py::object w = py::reinterpret_steal<py::object>(THPVariable_Wrap(weight));
  const py::object buf = attribute(w.ptr(), "main_grad");
  if (buf && THPVariable_Check(buf.ptr())) {
    const Tensor mg = THPVariable_Unpack(buf.ptr());
    if (mg.scalar_type() == at::kFloat && mg.is_contiguous() && mg.sizes() == weight.sizes() && mg.device() == go.device() && aligned(mg) &&
        go.size(0) % 8 == 0 && py::reinterpret_borrow<py::object>(g_fused_wgrad_enabled)().cast<bool>()) {
      const py::object fresh = attribute(w.ptr(), "main_grad_fresh");
      const int is_fresh = fresh ? PyObject_IsTrue(fresh.ptr()) : 0;
      if (is_fresh < 0) throw py::error_already_set();
      product(go, x, mg, true, false, !is_fresh);
      if (PyObject_SetAttrString(w.ptr(), "main_grad_fresh", Py_False)) throw py::error_already_set();
      const py::object ready = attribute(w.ptr(), "_nxd_grad_ready");      // ZeRO-1 overlapped reduce-scatter: this gradient is final
      if (ready && !ready.is_none()) ready(w);
      return Tensor();
    }
  }
  const py::object r = py::reinterpret_borrow<py::object>(g_wgrad)(go, x, w);
  return r.is_none() ? Tensor() : r.cast<Tensor>();
}

struct Linear : Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, bool few) {
    ctx->save_for_backward({x, weight});
    ctx->saved_data["x"] = x.requires_grad();
    const Tensor x2 = rows(x);
    auto shape = x.sizes().vec();
    shape.back() = weight.size(0);
    if (x2.size(0) <= 8) { count(); return gemv(x2, weight, c10::nullopt).view(shape); }
    if (few) { count(); return gemm_few_rows(x2, weight, 0).view(shape); }
    const Tensor y = at::empty({x2.size(0), weight.size(0)}, x.options());
    product(x2, weight, y, false, true, false);
    return y.view(shape);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    auto o = gradients(rows(g[0].contiguous()), s[0], s[1], ctx->saved_data["x"].toBool());
    return {o.first, o.second, Tensor()};
  }
  static std::pair<Tensor, Tensor> gradients(Tensor go, const Tensor& x, const Tensor& weight, bool of_x) {
    Tensor x2 = rows(x).contiguous();
    if (!aligned(go)) go = go.clone();
    if (!aligned(x2)) x2 = x2.clone();
    Tensor gx, gw;
    if (of_x) {
      gx = at::empty({go.size(0), weight.size(1)}, go.options());
      product(go, weight, gx, false, false, false);
      gx = gx.view(x.sizes());
    }
    if (weight.requires_grad()) gw = weight_gradient(go, x2, weight);
    return {gx, gw};
  }
};

// The nodes of a product and of SwiGLU for results that a kernel has left already (`products`, `y`).  Two of them, so that the products and the
// incoming gradient are given back before the gradients of the input and the weights need memory: in one node they were not, 51 MB at
// the peak of a step of 4096 tokens through 4096 x 11008, 540 at 8192 tokens in a micro-batch of a whole 7B model.
struct ProductsOf : Function<ProductsOf> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, Tensor* products) {
    ctx->save_for_backward({x, weight});
    ctx->saved_data["x"] = x.requires_grad();
    return *products;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto s = ctx->get_saved_variables();
    auto o = Linear::gradients(rows(g[0].contiguous()), s[0], s[1], ctx->saved_data["x"].toBool());
    return {o.first, o.second, Tensor()};
  }
};
struct SwiGLUOf : Function<SwiGLUOf> {
  static Tensor forward(AutogradContext* ctx, const Tensor& products, Tensor* y) {
    ctx->save_for_backward({products});
    return *y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    return {SwiGLU::backward(ctx, std::move(g))[0], Tensor()};
  }
};

// SwiGLU of x · [gate; up]ᵀ in one kernel: the products are kept for the backward pass as they leave the tensor cores, and not read again for it
Tensor linear_swiglu_node(const Tensor& x, const Tensor& weight) {
  Tensor products;
  auto y = linear_swiglu(x, weight, false, &products);
  TORCH_CHECK(y.has_value(), "linear_swiglu: no kernel for these operands");
  count();
  return SwiGLUOf::apply(ProductsOf::apply(x, weight, &products), &*y);
}

c10::optional<Tensor> linear(const Tensor& x, const Tensor& weight, bool few) {
  if (!x.is_cuda() || x.device() != weight.device() || x.scalar_type() != at::kBFloat16 || weight.scalar_type() != at::kBFloat16 || x.dim() < 2 ||
      weight.dim() != 2 || !x.is_contiguous() || !weight.is_contiguous() || x.size(-1) != weight.size(1) || !aligned(x) || !aligned(weight))
    return c10::nullopt;
  const int64_t K = weight.size(1), N = weight.size(0), M = K ? x.numel() / K : 0;
  const bool grads = at::GradMode::is_enabled() && (x.requires_grad() || weight.requires_grad());
  const bool rows = M % 8 == 0 || (!grads && (M <= 8 || (few && M <= 64)));      // others as ops/gemm.py matmul takes them
  if (M < 1 || N % 8 || K % 8 || N < 8 || !rows) return c10::nullopt;
  return Linear::apply(x, weight, few);
}

}  // namespace

void bind_native_autograd(py::module_& m) {
  auto n = m.def_submodule("native", "autograd nodes without Python in them");
  n.def("rms_norm", [](const Tensor& x, const Tensor& w, double eps) { return RmsNorm::apply(x, w, eps); });
  n.def("add_rms_norm", [](const Tensor& x, const Tensor& r, const Tensor& w, double eps) {
    auto o = AddRmsNorm::apply(x, r, w, eps);
    return py::make_tuple(o[0], o[1]);
  });
  n.def("swiglu", [](const Tensor& gu) { return SwiGLU::apply(gu); });
  n.def("rope_qkv", [](const Tensor& qkv, const Tensor& c, const Tensor& s, int64_t heads, int64_t kv_heads) {
    auto o = RopeQKV::apply(qkv, c, s, heads, kv_heads);
    return py::make_tuple(o[0], o[1], o[2]);
  });
  n.def("flash_attention", [](const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale) {
    return FlashAttention::apply(q, k, v, causal, scale);
  });
  n.def("cross_entropy", [](const Tensor& logits, const Tensor& target) { return CrossEntropy::apply(logits, target); });
  n.def("causal_loss", [](const Tensor& logits, const Tensor& labels, bool shift) { return CausalLoss::apply(logits, labels, shift); });
  n.def("table_lookup", [](const Tensor& ids, const Tensor& weight) { return TableLookup::apply(ids, weight); });
  n.def("linear", &linear);
  n.def("linear_swiglu", &linear_swiglu_node);
  n.def("swiglu_of", [](const Tensor& products, Tensor y) { return SwiGLUOf::apply(products, &y); });
  n.def("pairs", &pairs);
  n.def("launches", [] { return g_launches.load(); });
  n.def("set_weight_gradient", [](py::object wgrad, py::object enabled) {      // kept for the life of the process
    g_wgrad = wgrad.release().ptr();
    g_fused_wgrad_enabled = enabled.release().ptr();
  });
}
