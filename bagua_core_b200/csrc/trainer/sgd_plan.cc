#include "sgd_plan.h"

#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime.h>

#include <cstring>

namespace bagua {
namespace trainer {

void SgdPlan::add(const at::Tensor& p, const at::Tensor& g, const at::Tensor& m, const std::optional<at::Tensor>& shadow,
                  int group) {
  for (const at::Tensor* t : {&p, &g, &m})
    BAGUA_CHECK(t->scalar_type() == at::kFloat && t->is_contiguous() && t->numel() == p.numel() && t->device() == p.device(),
                Tensor, "fused SGD works on contiguous float32 buffers of one size on one device");
  if (shadow)
    BAGUA_CHECK(shadow->scalar_type() == at::kBFloat16 && shadow->is_contiguous() && shadow->numel() == p.numel() &&
                    shadow->device() == p.device(),
                Tensor, "the shadow must be a contiguous bf16 tensor of the parameters' size on their device");
  const int device = p.is_cuda() ? (int)p.device().index() : -1;
  BAGUA_CHECK(segs_.empty() || device == device_, Tensor, "the buffers of a plan live on one device");
  BAGUA_CHECK(group >= 0, Tensor, "negative parameter group");
  device_ = device;
  kernels::SgdSegment a{};
  a.p = (float*)p.data_ptr();
  a.g = (const float*)g.data_ptr();
  a.m = (float*)m.data_ptr();
  a.shadow = shadow ? shadow->data_ptr() : nullptr;
  a.n = p.numel();
  a.first = true;
  segs_.push_back(a);
  group_.push_back(group);
  grad_buffer_.push_back(g.storage().data());
  keep_.insert(keep_.end(), {p, g, m});
  if (shadow) keep_.push_back(*shadow);
}

int SgdPlan::step(const std::vector<SgdGroup>& groups, uint64_t stream) {
  for (size_t k = 0; k < segs_.size(); ++k) {
    BAGUA_CHECK((size_t)group_[k] < groups.size(), Tensor, "no hyperparameters for parameter group " << group_[k]);
    const SgdGroup& h = groups[(size_t)group_[k]];
    auto& a = segs_[k];
    a.lr = h.lr;
    a.momentum = h.momentum;
    a.dampening = h.dampening;
    a.weight_decay = h.weight_decay;
    a.nesterov = h.nesterov;
  }
  int launches = 0;
  if (device_ >= 0)
    launches = kernels::cuda::sgd_steps(segs_.data(), (int)segs_.size(), (cudaStream_t)stream);
  else
    for (const auto& a : segs_) {
      kernels::sgd_momentum_flat_shadow(a.p, a.g, a.m, a.shadow, a.n, a.lr, a.momentum, a.dampening, a.weight_decay,
                                        a.nesterov, a.first, kernels::Ctx{});
      ++launches;
    }
  for (auto& a : segs_) a.first = false;
  return launches;
}

void SgdPlan::zero_grad(uint64_t stream) {
  std::vector<kernels::cuda::FillSegment> fill;
  for (size_t k = 0; k < segs_.size();) {
    // slices of one buffer follow each other: one segment for all of them (never over two buffers, which may lie next
    // to each other in separate allocations)
    float* from = const_cast<float*>(segs_[k].g);
    const void* buffer = grad_buffer_[k];
    int64_t n = 0;
    for (; k < segs_.size() && grad_buffer_[k] == buffer && segs_[k].g == from + n; ++k) n += segs_[k].n;
    if (n) fill.push_back({from, n});
  }
  if (device_ >= 0) {
    const c10::cuda::CUDAGuard on((c10::DeviceIndex)device_);  // memory can be set from any device, a kernel not
    kernels::cuda::fill_zero(fill.data(), (int)fill.size(), (cudaStream_t)stream);
  } else {
    for (const auto& f : fill) std::memset(f.p, 0, (size_t)f.n * sizeof(float));
  }
}

}  // namespace trainer
}  // namespace bagua
