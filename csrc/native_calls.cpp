// Host paths in native code: autograd nodes of the single operators that programs call by themselves, and the whole
// forward pass of a dense model where no gradient is recorded. The kernels are those of the Python operators, in the
// same order; with small tensors the Python between them takes longer than they do. Measured, us, through Python /
// here: forward of 4 layers of width 576 on 33 tokens 749 / 170 (153 of kernels; 329 with a tensor and its views per
// operator); forward and backward of attention, 256 tokens x 9 heads, 105 / 88; of a linear of 1999 x 960 x 2560, 96 /
// 74.
#include <ATen/core/grad_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>

#include <atomic>
#include <cmath>

#include "attention/attention.h"
#include "common/host.h"
#include "elementwise/elementwise.h"
#include "gemm/gemm.h"
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
    ctx->saved_data["w_learns"] = w.requires_grad();
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
    // needs_input_grad is about this backward, w_learns about the weight: a backward for x alone still accumulates into
    // main_grad or postpones, as the Python function (and those of the other projections) does
    if (ctx->saved_data["w_learns"].toBool() && !python_wgrad(w, dy2, x2, dw) && ctx->needs_input_grad(1)) {
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
                                          0, 0, c10::nullopt, c10::nullopt, 0, 0);
    g_launches += 3;
    return {dq, dk, dv, at::Tensor(), at::Tensor()};
  }
};

static void ok(int rc, const char* what) {
  TORCH_CHECK(rc == 0, what, " failed (", rc, "): ", pico_last_error());
}

// Logits [b, s, V] of a dense decoder without gradients; a layer is (norm, q | k | v, output projection, norm, gate |
// up, down projection, the two norms' eps). Each residual add rides in the norm that follows it (the sum is rounded to
// bf16 there as a separate add would round it). The activations live in one allocation, of a layer's size and not of
// the model's: what one layer is done with the next writes over, in stream order.
using LayerWeights = std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, at::Tensor, double, double>;

static at::Tensor dense_forward(const at::Tensor& ids_, const at::Tensor& embedding,
                                const std::vector<LayerWeights>& layers, const at::Tensor& final_norm,
                                double final_eps, const at::Tensor& head, int64_t heads, int64_t kv_heads,
                                int64_t head_dim, const at::Tensor& cos, const at::Tensor& sin, int64_t pos0) {
  at::NoGradGuard no_grad;
  const auto matrix = [&](const at::Tensor& w, int64_t rows, int64_t cols) {
    TORCH_CHECK(w.is_cuda() && w.device() == embedding.device() && w.scalar_type() == at::kBFloat16 && w.dim() == 2 &&
                    w.size(0) == rows && w.size(1) == cols && w.is_contiguous(),
                "dense_forward: a bf16 [", rows, ", ", cols, "] weight");
  };
  const auto vector = [&](const at::Tensor& w, int64_t n) {
    TORCH_CHECK(w.is_cuda() && w.device() == embedding.device() && w.scalar_type() == at::kBFloat16 &&
                    w.numel() == n && w.is_contiguous(), "dense_forward: a bf16 norm weight of the hidden size");
  };
  TORCH_CHECK(embedding.dim() == 2 && !layers.empty(), "dense_forward: an embedding and layers");
  const int64_t hidden = embedding.size(1), V = head.size(0);
  matrix(embedding, embedding.size(0), hidden);
  matrix(head, V, hidden);
  vector(final_norm, hidden);
  TORCH_CHECK(ids_.is_cuda() && ids_.device() == embedding.device() && ids_.scalar_type() == at::kLong &&
                  ids_.dim() == 2 && ids_.numel() > 0, "dense_forward: int64 ids [b, s]");
  const int64_t b = ids_.size(0), s = ids_.size(1), T = b * s, width = heads * head_dim;
  const int64_t fused = width + 2 * kv_heads * head_dim, inter = std::get<5>(layers[0]).size(1);
  TORCH_CHECK(T <= INT32_MAX, "dense_forward: too many tokens");
  TORCH_CHECK(cos.scalar_type() == at::kFloat && sin.scalar_type() == at::kFloat && cos.is_contiguous() &&
                  sin.is_contiguous() && cos.dim() == 2 && cos.size(1) == head_dim / 2 && cos.sizes() == sin.sizes() &&
                  cos.device() == embedding.device() && sin.device() == embedding.device(), "rope: fp32 tables");
  TORCH_CHECK(pos0 >= 0 && pos0 + s <= cos.size(0), "rope: position table too short");
  for (const auto& [norm1, qkv, out, norm2, gate_up, down, eps1, eps2] : layers) {
    vector(norm1, hidden);
    matrix(qkv, fused, hidden);
    matrix(out, hidden, width);
    vector(norm2, hidden);
    matrix(gate_up, 2 * inter, hidden);
    matrix(down, hidden, inter);
  }
  c10::cuda::CUDAGuard guard(embedding.device());
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream(embedding.device().index()).stream();
  const at::Tensor ids = ids_.is_contiguous() ? ids_ : ids_.contiguous();

  const bool in_epilogue = pico_gemm_swiglu_pays((int)T, (int)inter, (int)hidden, 0, 0);
  int64_t slab = 0;                                  // floats of the products that are summed in parts of K
  const auto parts_of = [&](int64_t N, int64_t K) { return pico_gemm_parts_of_k((int)T, (int)N, (int)K); };
  const int64_t shapes[][2] = {{fused, hidden}, {hidden, width}, {2 * inter, hidden}, {hidden, inter}, {V, hidden}};
  for (const auto& [N, K] : shapes) slab = std::max(slab, parts_of(N, K) * ((T + 127) / 128) * 128 * N);
  const auto room = [](int64_t bytes) { return (bytes + 255) & ~(int64_t)255; };
  const int64_t stream_bytes = room(T * hidden * 2);
  // attention's buffers and the MLP's are not in use at the same time
  const int64_t attn_bytes = room(T * fused * 2) + room(T * width * 2) + room(T * heads * 4);
  const int64_t mlp_bytes = (in_epilogue ? 0 : room(T * 2 * inter * 2)) + room(T * inter * 2);
  const at::Tensor work = at::empty({4 * stream_bytes + std::max(attn_bytes, mlp_bytes) + slab * 4},
                                    embedding.options().dtype(at::kByte));
  char* at_byte = (char*)work.data_ptr();
  const auto take = [&](int64_t bytes) {
    char* p = at_byte;
    at_byte += room(bytes);
    return p;
  };
  void* residual = take(stream_bytes);               // the residual stream, and where the next norm puts it
  void* residual_next = take(stream_bytes);
  void* normed = take(stream_bytes);
  void* branch = take(stream_bytes);                 // what is to be added to the stream
  float* slabs = (float*)take(slab * 4);
  char* shared = at_byte;
  void* qkv_rows = shared;
  void* att = shared + room(T * fused * 2);
  float* lse = (float*)(shared + room(T * fused * 2) + room(T * width * 2));
  void* gate_up_rows = shared;
  void* act = shared + (in_epilogue ? 0 : room(T * 2 * inter * 2));

  int64_t launches = 1;
  const auto product = [&](const void* x, const at::Tensor& w, void* y) {
    const int N = (int)w.size(0), K = (int)w.size(1), parts = parts_of(N, K);
    ok(parts > 0 ? pico_gemm_bf16_parts(x, w.data_ptr(), y, slabs, (int)T, N, K, K, K, N, 0, parts, stream)
                 : pico_gemm_bf16(x, w.data_ptr(), y, (int)T, N, K, K, K, N, 0, 0, 0, 0, nullptr, stream), "gemm");
    launches += parts > 0 ? 2 : 1;
  };
  bool pending = false;                              // `branch` waits to be added
  const auto norm = [&](const at::Tensor& w, double eps) {
    ok(pico_rmsnorm_fwd(pending ? branch : residual, pending ? residual : nullptr, w.data_ptr(), normed,
                        pending ? residual_next : nullptr, nullptr, (int)T, (int)hidden, (float)eps, stream),
       "rmsnorm_fwd");
    if (pending) std::swap(residual, residual_next);
    pending = true;
    ++launches;
  };
  PicoAttnParams p = {};
  p.batch = (int)b;
  p.seq_q = p.seq_k = (int)s;
  p.heads = (int)heads;
  p.kv_heads = (int)kv_heads;
  p.head_dim = (int)head_dim;
  p.q_row_stride = p.k_row_stride = p.v_row_stride = fused;
  p.q_batch_stride = p.k_batch_stride = p.v_batch_stride = s * fused;
  p.o_row_stride = width;
  p.o_batch_stride = s * width;
  p.sm_scale = (float)(1.0 / std::sqrt((double)head_dim));
  p.causal = 1;
  ok(pico_embedding_fwd(embedding.data_ptr(), ids.data_ptr<int64_t>(), residual, (int)T, (int)hidden,
                        (int)embedding.size(0), 0, stream), "embedding_fwd");
  for (const auto& [norm1, qkv, out, norm2, gate_up, down, eps1, eps2] : layers) {
    norm(norm1, eps1);
    product(normed, qkv, qkv_rows);
    ok(pico_rope_inplace(qkv_rows, fused, (int)T, (int)s, (int)pos0, (int)(heads + kv_heads), (int)head_dim,
                         cos.data_ptr<float>(), sin.data_ptr<float>(), 1, stream), "rope");
    ok(pico_attention_fwd(qkv_rows, (char*)qkv_rows + width * 2, (char*)qkv_rows + (width + kv_heads * head_dim) * 2,
                          att, lse, &p, stream), "attention_fwd");
    product(att, out, branch);
    norm(norm2, eps2);
    if (in_epilogue) {
      ok(pico_gemm_swiglu(normed, gate_up.data_ptr(), nullptr, act, (int)T, (int)inter, (int)hidden, (int)hidden,
                          (int)hidden, nullptr, 1, stream), "gemm_swiglu");
    } else {
      product(normed, gate_up, gate_up_rows);
      ok(pico_swiglu_fwd(gate_up_rows, 2 * inter, act, (int)T, (int)inter, nullptr, stream), "swiglu_fwd");
    }
    product(act, down, branch);
    launches += 3;
  }
  norm(final_norm, final_eps);
  at::Tensor logits = at::empty({b, s, V}, embedding.options());
  product(normed, head, logits.data_ptr());
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
