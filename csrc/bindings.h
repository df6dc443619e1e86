// Functions of binding.cpp that the autograd nodes (native_autograd.cpp) call too.
#pragma once
#include <torch/extension.h>

#include <vector>

using at::Tensor;

std::vector<Tensor> rmsnorm_fwd(const Tensor& x, const Tensor& w, double eps);
std::vector<Tensor> rmsnorm_bwd(const Tensor& g, const Tensor& x, const Tensor& w, const Tensor& rstd);
std::vector<Tensor> add_rmsnorm_fwd(const Tensor& x, const Tensor& r, const Tensor& w, double eps);
std::vector<Tensor> add_rmsnorm_bwd(const Tensor& gy, const Tensor& gh, const Tensor& h, const Tensor& w, const Tensor& rstd);
Tensor swiglu_fwd(const Tensor& gu);
Tensor swiglu_bwd(const Tensor& go, const Tensor& gu);
std::vector<Tensor> rope_qkv_fwd(const Tensor& x, const Tensor& cos_t, const Tensor& sin_t, int64_t H, int64_t K);
Tensor rope_qkv_bwd(const Tensor& gq, const Tensor& gk, const Tensor& gv, const Tensor& cos_t, const Tensor& sin_t);
std::vector<Tensor> ce_loss(const Tensor& logits, const Tensor& target);
Tensor ce_backward(const Tensor& logits, const Tensor& target, const Tensor& lse, const Tensor& gout, int64_t vocab_start, double smoothing,
                   int64_t vocab);
std::vector<Tensor> flash_attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale, bool sbhd_out);
std::vector<Tensor> flash_attn_bwd(const Tensor& go, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                                   bool causal, double scale, bool sbhd_out, const c10::optional<Tensor>& dlse, int64_t parts);
void gemm_bf16(const Tensor& a, const Tensor& b, Tensor out, bool trans_a, bool trans_b, bool accumulate);
void gemm_bf16_2cta(const Tensor& a, const Tensor& b, Tensor out, bool trans_a, bool trans_b, bool accumulate);
Tensor gemm_few_rows(const Tensor& x, const Tensor& w, int64_t split);
void embedding_grad(const Tensor& ids, const Tensor& gy, Tensor out, bool zero_first);
c10::optional<Tensor> linear_swiglu(const Tensor& x, const Tensor& w, bool few, Tensor* keep);
Tensor gemv(const Tensor& x, const Tensor& w, const c10::optional<Tensor>& residual);

void bind_native_autograd(pybind11::module_& m);
