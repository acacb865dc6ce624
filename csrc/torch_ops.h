// Operators on torch tensors (bindings.cpp) that native code strings together (native_calls.cpp).
#pragma once
#include <torch/extension.h>

#include <tuple>

namespace pico_torch {

at::Tensor rows_of(const at::Tensor& x);
int64_t gemm(const at::Tensor& A, const at::Tensor& B, at::Tensor& D, int64_t M, int64_t N, int64_t K, int64_t lda,
             int64_t ldb, int64_t ldd, bool a_mn_major, bool b_mn_major, int64_t out_mode, int64_t max_ctas);
std::tuple<at::Tensor, int64_t> gemm_new(const at::Tensor& a, const at::Tensor& b, bool b_mn_major);
std::tuple<at::Tensor, at::Tensor, int64_t> linear_fwd(const at::Tensor& x, const at::Tensor& w);
std::tuple<at::Tensor, at::Tensor> attention_fwd_new(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                                                     double sm_scale, bool causal, int64_t q_pos0, int64_t k_pos0);
std::tuple<at::Tensor, at::Tensor, at::Tensor> attention_bwd_new(const at::Tensor& dout, const at::Tensor& q,
                                                                 const at::Tensor& k, const at::Tensor& v,
                                                                 const at::Tensor& out, const at::Tensor& lse,
                                                                 double sm_scale, bool causal, int64_t q_pos0,
                                                                 int64_t k_pos0, const c10::optional<at::Tensor>& cos,
                                                                 const c10::optional<at::Tensor>& sin,
                                                                 int64_t rope_pos0, int64_t splits);

void def_native_calls(pybind11::module_& m);

}  // namespace pico_torch
