// The three library GEMMs of a linear layer, with their set-up kept.
//
// The framework's matrix product spends 9-12 us of host time per call, most of it on describing the problem to
// the library and asking it for an algorithm, which for a given shape is the same every time.  Here both are
// kept per thread and shape, and a call is a look-up and a launch (4 us).  The products themselves are the
// library's (cuBLASLt), in bf16 with fp32 accumulation.
#pragma once

#include <ATen/ATen.h>

namespace bagua {
namespace trainer {
namespace gemm {

// All operands are 2-D, bf16, contiguous, of the sizes given here and on one CUDA device; false: not available for these,
// nothing was done.

// y [M, N] = x [M, K] w [N, K]ᵀ + b [N] (b may be undefined), at least 0 with `relu`
bool linear(const at::Tensor& x, const at::Tensor& w, const at::Tensor& b, bool relu, at::Tensor& y);
// dx [M, K] = dy [M, N] w [N, K]
bool input_grad(const at::Tensor& dy, const at::Tensor& w, at::Tensor& dx);
// g [N, K] (fp32) = dy [M, N]ᵀ x [M, K], added to what is there with `accumulate`
bool weight_grad(const at::Tensor& dy, const at::Tensor& x, at::Tensor& g, bool accumulate);

}  // namespace gemm
}  // namespace trainer
}  // namespace bagua
