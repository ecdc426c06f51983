// The operators of bindings.cpp that other translation units of _C.so call directly.
#pragma once
#include <ATen/ATen.h>

#include <tuple>
#include <vector>

namespace lb_nodes {
void count(int64_t n);      // kernels launched from C++ (ops.launch_count())
}
namespace lb_ops {

using at::Tensor;

Tensor gemm(const Tensor& a, const Tensor& b, int64_t layout, const c10::optional<Tensor>& bias, const c10::optional<Tensor>& out_opt, bool accumulate,
            at::ScalarType out_dtype);
Tensor dgrad_actgrad(const Tensor& gy, const Tensor& w, const Tensor& pre, int64_t act, const c10::optional<Tensor>& bias_grad);
Tensor linear_bias_residual(const Tensor& x, const Tensor& w, const c10::optional<Tensor>& bias, const Tensor& residual);
std::tuple<Tensor, Tensor> linear_fwd(const Tensor& x, const Tensor& w, const c10::optional<Tensor>& bias, int64_t act, bool need_pre);
Tensor act_bwd(const Tensor& gy, const Tensor& pre, int64_t act);
Tensor colsum(const Tensor& x, const c10::optional<Tensor>& accum);
std::tuple<Tensor, Tensor, Tensor> norm_fwd(const Tensor& x, const Tensor& gamma, const c10::optional<Tensor>& beta, double eps, bool rms);
std::tuple<Tensor, Tensor, Tensor> norm_bwd(const Tensor& gy, const Tensor& x, const Tensor& gamma, const Tensor& mean, const Tensor& rstd, bool rms,
                                            bool has_bias, const c10::optional<Tensor>& dgamma_accum, const c10::optional<Tensor>& dbeta_accum,
                                            const c10::optional<Tensor>& gadd);
Tensor norm_bwd_sums(const Tensor& gy, const Tensor& x, const Tensor& gamma, const Tensor& mean, const Tensor& rstd, const Tensor& dgamma, const Tensor& dbeta,
                     const Tensor& gadd, const Tensor& sum_add, const Tensor& sum_out);
Tensor swiglu_packed_fwd(const Tensor& gu);
Tensor swiglu_packed_bwd(const Tensor& gy, const Tensor& gu);
Tensor rope_qkv(const Tensor& qkv, const Tensor& cosv, const Tensor& sinv, int64_t pos_offset, bool backward, bool inplace);
std::tuple<Tensor, Tensor, Tensor> ce_stats(const Tensor& logits, const Tensor& labels, int64_t vocab_start);
Tensor ce_bwd(const Tensor& logits, const Tensor& labels, const Tensor& lse, const Tensor& gloss, int64_t vocab_start);
std::tuple<Tensor, Tensor, Tensor> attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale, const c10::optional<Tensor>& kv_lens,
                                            const c10::optional<Tensor>& bias, const c10::optional<Tensor>& alibi_slopes, double p_drop, int64_t salt);
std::tuple<Tensor, Tensor, Tensor, Tensor> attn_bwd(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
                                                    bool causal, double scale, const c10::optional<Tensor>& kv_lens, const c10::optional<Tensor>& bias,
                                                    const c10::optional<Tensor>& alibi_slopes, c10::optional<Tensor> dbias, double p_drop,
                                                    const c10::optional<Tensor>& rng_state);
std::tuple<Tensor, Tensor> attn_mask_pack(const Tensor& mask, bool causal);
std::tuple<Tensor, Tensor, Tensor> attn_split_fwd(const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale,
                                                  const c10::optional<Tensor>& words, const c10::optional<Tensor>& fill, bool train);
void attn_split_bwd(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o32, const Tensor& lse, Tensor dq, Tensor dk,
                    Tensor dv, bool causal, double scale, const c10::optional<Tensor>& words, const c10::optional<Tensor>& fill);
// plain bf16 tensors of a block: contiguous, on 16 bytes, on x's device, of these sizes
bool block_tensor(const Tensor& t, const Tensor& x);
bool block_vector(const Tensor& t, const Tensor& x, int64_t n);
bool block_matrix(const Tensor& t, const Tensor& x, int64_t n, int64_t k);

}  // namespace lb_ops
