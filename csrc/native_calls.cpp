// Host paths in native code: autograd nodes of the single operators that programs call by themselves, and the whole
// forward pass of a dense model where no gradient is recorded. The kernels are those of the Python operators, in the same
// order; with small tensors the Python between them takes longer than they do. Measured, us, through Python / here:
// forward of 4 layers of width 576 on 33 tokens 749 / 289 (190 of kernels); forward and backward of attention, 256 tokens
// x 9 heads, 105 / 88; of a linear of 1999 x 960 x 2560, 96 / 74.
#include <ATen/core/grad_mode.h>
#include <torch/csrc/autograd/custom_function.h>

#include <atomic>
#include <cmath>

#include "torch_ops.h"

namespace pico_torch {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// kernels launched by the calls of this file, in forward passes and in the backward passes of their nodes
static std::atomic<int64_t> g_launches{0};

// The Python form of the weight gradient: it accumulates into main_grad, runs hooks or postpones, and returns None, or
// gives the gradient. Needed where the parameter or the caller asks for any of that.
static bool python_wgrad(const at::Tensor& w, const at::Tensor& dy2, const at::Tensor& x2, at::Tensor& dw) {
  pybind11::gil_scoped_acquire gil;
  pybind11::object ops = pybind11::module_::import("picotron_b200.ops.gemm");
  pybind11::object weight = pybind11::cast(w);
  const bool plain = ops.attr("_DEFER_QUEUE").is_none() &&
                     (!pybind11::hasattr(weight, "main_grad") || weight.attr("main_grad").is_none());
  if (plain) return false;
  pybind11::object got = ops.attr("wgrad_into")(weight, pybind11::cast(dy2), pybind11::cast(x2));
  if (!got.is_none()) dw = got.cast<at::Tensor>();
  return true;
}

// y = x w^T
struct LinearNode : torch::autograd::Function<LinearNode> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& x, const at::Tensor& w) {
    auto [y, x2, launches] = linear_fwd(x, w);
    g_launches += launches;
    ctx->save_for_backward({x2, w});
    ctx->saved_data["shape"] = x.sizes().vec();
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &x2 = saved[0], &w = saved[1];
    const at::Tensor dy2 = rows_of(grads[0]);
    at::Tensor dx, dw;
    if (ctx->needs_input_grad(0)) {
      auto [d, launches] = gemm_new(dy2, w, true);
      g_launches += launches;
      dx = d.view(ctx->saved_data["shape"].toIntVector());
    }
    if (ctx->needs_input_grad(1) && !python_wgrad(w, dy2, x2, dw)) {
      const int64_t K = dy2.size(0), M = dy2.size(1), N = x2.size(1);
      dw = at::empty({M, N}, dy2.options());
      g_launches += gemm(dy2, x2, dw, M, N, K, dy2.stride(0), x2.stride(0), N, true, true, 0, 0);
    }
    return {dx, dw};
  }
};

// whole-sequence attention on [b, s, heads, d]
struct AttentionNode : torch::autograd::Function<AttentionNode> {
  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                            bool causal, double sm_scale) {
    auto [out, lse] = attention_fwd_new(q, k, v, sm_scale, causal, 0, 0);
    ++g_launches;
    ctx->save_for_backward({q, k, v, out, lse});
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["sm_scale"] = sm_scale;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    auto [dq, dk, dv] = attention_bwd_new(grads[0], saved[0], saved[1], saved[2], saved[3], saved[4],
                                          ctx->saved_data["sm_scale"].toDouble(), ctx->saved_data["causal"].toBool(),
                                          0, 0, c10::nullopt, c10::nullopt, 0);
    g_launches += 3;
    return {dq, dk, dv, at::Tensor(), at::Tensor()};
  }
};

// Logits [b, s, V] of a dense decoder without gradients; a layer is (norm, q | k | v, output projection, norm, gate | up,
// down projection, the two norms' eps). Each residual add rides in the norm that follows it (the sum is
// rounded to bf16 there as a separate add would round it).
static at::Tensor dense_forward(const at::Tensor& ids, const at::Tensor& embedding,
                                const std::vector<std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor,
                                                             at::Tensor, double, double>>& layers,
                                const at::Tensor& final_norm, double final_eps, const at::Tensor& head, int64_t heads,
                                int64_t kv_heads, int64_t head_dim, const at::Tensor& cos, const at::Tensor& sin,
                                int64_t pos0) {
  at::NoGradGuard no_grad;
  TORCH_CHECK(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.dim() == 2 && embedding.is_cuda() &&
                  embedding.is_contiguous() && embedding.scalar_type() == at::kBFloat16,
              "dense_forward: int64 ids [b, s] and a bf16 embedding on the GPU");
  const int64_t b = ids.size(0), s = ids.size(1), T = b * s, hidden = embedding.size(1);
  const double scale = 1.0 / std::sqrt((double)head_dim);
  int64_t launches = 1;
  auto product = [&](const at::Tensor& x, const at::Tensor& w) {
    auto [y, n] = gemm_new(x, w, false);
    launches += n;
    return y;
  };
  at::Tensor x = at::empty({T, hidden}, embedding.options());       // the residual stream
  const at::Tensor flat = ids.reshape({-1}).contiguous();
  embedding_fwd(embedding, flat, x, T, hidden, embedding.size(0), 0);
  c10::optional<at::Tensor> branch;                                  // what is to be added to it
  auto norm = [&](const at::Tensor& w, double eps) {
    auto [y, h, rstd] = branch.has_value() ? rmsnorm_new(*branch, x, w, eps) : rmsnorm_new(x, c10::nullopt, w, eps);
    ++launches;
    x = h;
    return y;
  };
  for (const auto& [norm1, qkv, out, norm2, gate_up, down, eps1, eps2] : layers) {
    at::Tensor fused = product(norm(norm1, eps1), qkv);
    rope_inplace(fused, fused.stride(0), T, s, pos0, heads + kv_heads, head_dim, cos, sin, 1);
    const at::Tensor view = fused.view({b, s, heads + 2 * kv_heads, head_dim});
    auto [att, lse] = attention_fwd_new(view.narrow(2, 0, heads), view.narrow(2, heads, kv_heads),
                                        view.narrow(2, heads + kv_heads, kv_heads), scale, true, 0, 0);
    launches += 2;
    branch = product(att.view({T, heads * head_dim}), out);
    auto [gu, act, n] = gemm_swiglu(norm(norm2, eps2), gate_up, false, -1);
    launches += n;
    branch = product(act, down);
  }
  at::Tensor logits = product(norm(final_norm, final_eps), head).view({b, s, head.size(0)});
  g_launches += launches;
  return logits;
}

void def_native_calls(pybind11::module_& m) {
  namespace py = pybind11;
  m.def("linear_node", [](const at::Tensor& x, const at::Tensor& w) { return LinearNode::apply(x, w); });
  m.def("attention_node", [](const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, bool causal,
                             double sm_scale) { return AttentionNode::apply(q, k, v, causal, sm_scale); });
  m.def("dense_forward", &dense_forward);
  m.def("native_launches", [] { return g_launches.load(); });
}

}  // namespace pico_torch
