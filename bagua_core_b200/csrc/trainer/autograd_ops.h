// Autograd functions of the trainer's layers, without a Python frame in either direction.
//
// A training step of the benchmark models was paced by the launching threads: a Python autograd
// function costs 40-60 us per direction (argument packing, the GIL handed to the autograd thread and
// back, one Python call per tensor operation), against 10-15 us for the same operations from here.
#pragma once

#include <ATen/ATen.h>

#include <atomic>
#include <optional>
#include <vector>

namespace bagua {
namespace trainer {

// Weight gradients of linear layers that were added to an fp32 `.grad` by their GEMM / that took autograd's
// path although accumulation was asked for; kernels of this package launched by these functions.
struct OpStats {
  std::atomic<int64_t> accumulated{0}, declined{0}, launches{0};
  std::atomic<int> gemm_mode{0};  // 0 not decided, 1 one GEMM, 2 GEMM and an addition, 3 not available
  static OpStats& global();
};

// y = x Wᵀ + b in bf16.  `w_low`: W in bf16 when the caller has it, else it is cast here.  With `accumulate`, the
// backward adds the gradients of W and b to their fp32 `.grad` itself where nobody can tell the difference
// (autograd_ops.cc, `accumulates`), and hands autograd nothing for them.
// `activation`: applied to the result; its backward makes the bias gradient in the pass that applies the derivative
// (needs activation_fusable()).
enum Activation { kNone = 0, kGelu = 1, kRelu = 2 };
at::Tensor linear(const at::Tensor& x, const at::Tensor& weight, const std::optional<at::Tensor>& bias,
                  const std::optional<at::Tensor>& w_low, bool accumulate, int activation);
inline bool activation_fusable(const at::Tensor& x, int64_t out_features) {
  return x.is_cuda() && out_features % 8 == 0 && x.numel() > 0;
}

// layer_norm(x + r) of bf16 activations with fp32 parameters (r may be missing); CUDA.  The library's normalisation
// (its kernels run at the speed of their bytes) with the casts of the parameters as one launch.
at::Tensor add_layer_norm(const at::Tensor& x, const std::optional<at::Tensor>& r, const at::Tensor& gamma,
                          const at::Tensor& beta, double eps, bool accumulate);

// layer_norm(tok[ids] + pos[: seq] + typ[0]) in bf16 from fp32 tables; ids [batch, seq] of int64, at most
// `encoder_ops::kMaxTokens` of them.
at::Tensor embed_layer_norm(const at::Tensor& ids, const at::Tensor& tok, const at::Tensor& pos, const at::Tensor& typ,
                            const at::Tensor& gamma, const at::Tensor& beta, double eps, bool accumulate);

// (cross_entropy(logits[..., 0], start) + cross_entropy(logits[..., 1], end)) / 2 of bf16 logits [batch, seq, 2] with int64
// positions [batch]; rows with position -100 do not count.
at::Tensor span_loss(const at::Tensor& logits, const at::Tensor& start, const at::Tensor& end);

// Multi-head attention of a packed projection qkv [batch, seq, 3 * heads * dim] (bf16, CUDA): [batch, seq, heads * dim].
at::Tensor attention(const at::Tensor& qkv, int64_t heads, double dropout);

// max(conv(x, weight) + bias, 0), channels-last, followed by 2x2 pooling with `pool`.  Inside an autocast region
// x, weight and bias are taken in its type (the weight from `w_low` when given).
at::Tensor conv_bias_relu(const at::Tensor& x, const at::Tensor& weight, const at::Tensor& bias,
                          const std::vector<int64_t>& stride, const std::vector<int64_t>& padding,
                          const std::vector<int64_t>& dilation, int64_t groups, bool pool,
                          const std::optional<at::Tensor>& w_low, bool accumulate);

}  // namespace trainer
}  // namespace bagua
