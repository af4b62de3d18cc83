// The flat buffers an optimizer steps: laid out once, stepped and zeroed with one call each.
//
// From Python a step was one call per bucket (5-7 us each with its tensor checks); the buffers and their
// checks are the same at every step, only the hyperparameters may change.
#pragma once

#include <ATen/ATen.h>

#include <optional>
#include <vector>

#include "../kernels/kernels.h"

namespace bagua {
namespace trainer {

struct SgdGroup {
  float lr, momentum, dampening, weight_decay;
  bool nesterov;
};

class SgdPlan {
 public:
  // One buffer (or a slice of one) whose parameters all belong to parameter group `group`.
  void add(const at::Tensor& p, const at::Tensor& g, const at::Tensor& m, const std::optional<at::Tensor>& shadow,
           int group);
  // Steps every buffer with its group's hyperparameters; returns the number of kernels launched.
  int step(const std::vector<SgdGroup>& groups, uint64_t stream);
  void zero_grad(uint64_t stream);
  bool empty() const { return segs_.empty(); }

 private:
  int device_ = -1;
  std::vector<kernels::SgdSegment> segs_;
  std::vector<int> group_;
  std::vector<const void*> grad_buffer_;  // of each segment: the storage its gradient lies in
  std::vector<at::Tensor> keep_;
};

}  // namespace trainer
}  // namespace bagua
