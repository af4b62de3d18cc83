#include "grad_hooks.h"

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/engine.h>
#include <torch/csrc/autograd/utils/lambda_post_hook.h>
#include <torch/csrc/autograd/variable.h>

#include <algorithm>

namespace bagua {
namespace trainer {

GradHooks::~GradHooks() {
  remove();
  for (auto& b : buckets_)
    if (b.event) cudaEventDestroy(b.event);
}

void GradHooks::add(const at::Tensor& param, const at::Tensor& grad, TensorPtr tensor, int bucket) {
  BAGUA_CHECK(bucket >= 0, Bucket, "negative bucket index");
  Entry e;
  e.param = param;
  e.grad = grad;
  e.tensor = std::move(tensor);
  e.bucket = bucket;
  entries_.push_back(std::move(e));
  if ((size_t)bucket >= buckets_.size()) buckets_.resize((size_t)bucket + 1);
  buckets_[(size_t)bucket].size++;
}

void GradHooks::install() {
  using torch::autograd::variable_list;
  std::weak_ptr<GradHooks> self = weak_from_this();
  for (size_t i = 0; i < entries_.size(); ++i) {
    Entry& e = entries_[i];
    // the node is kept alive here: the parameter itself only refers to it weakly
    e.accumulator = torch::autograd::impl::grad_accumulator(e.param);
    BAGUA_CHECK(e.accumulator != nullptr, Tensor, "only leaf parameters that require a gradient can be hooked");
    e.key = e.accumulator->add_post_hook(std::make_unique<torch::autograd::utils::LambdaPostHook>(
        [self, i](const variable_list& outputs, const variable_list&) {
          if (auto me = self.lock()) me->on_gradient(i);
          return outputs;
        }));
  }
  arm();
}

void GradHooks::remove() {
  for (auto& e : entries_)
    if (e.accumulator) {
      e.accumulator->del_post_hook(e.key);
      e.accumulator.reset();
    }
}

void GradHooks::arm() {
  for (auto& e : entries_) e.marked = false;
  for (auto& b : buckets_) {
    b.pending = b.size;
    b.streams.clear();
  }
}

void GradHooks::flush() {
  for (auto& e : entries_)
    if (!e.marked && buckets_[(size_t)e.bucket].pending > 0) mark(e);
}

void GradHooks::watch(const at::Tensor& output) {
  std::weak_ptr<GradHooks> self = weak_from_this();
  output.register_hook([self](const at::Tensor&) {
    auto me = self.lock();
    if (!me || !me->done_ || me->queued_.exchange(true)) return;
    // whichever output fires first: the loss may depend on any of them
    torch::autograd::Engine::get_default_engine().queue_callback([self]() {
      auto me2 = self.lock();
      if (!me2) return;
      me2->queued_ = false;
      me2->done_();
    });
  });
}

void GradHooks::on_gradient(size_t i) {
  if (!enabled_) return;
  Entry& e = entries_[i];
  const at::Tensor& now = e.param.grad();
  if (now.unsafeGetTensorImpl() != e.grad.unsafeGetTensorImpl()) {
    // .grad was replaced (e.g. zero_grad(set_to_none=True)): its value moves into the bucket, and the bucket's
    // view is the gradient again
    c10::NoGradGuard no_grad;
    if (now.defined())
      e.grad.copy_(now);
    else
      e.grad.zero_();
    e.param.mutable_grad() = e.grad;
  }
  mark(e);
}

void GradHooks::mark(Entry& e) {
  auto backend = backend_.lock();
  if (!backend) return;
  Bucket& b = buckets_[(size_t)e.bucket];
  e.marked = true;
  uint64_t event = 0;
  --b.pending;
  if (device_ >= 0) {
    const cudaStream_t now = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device_).stream();
    if (std::find(b.streams.begin(), b.streams.end(), now) == b.streams.end()) b.streams.push_back(now);
    if (b.pending == 0) {
      if (!b.event) BAGUA_CUDA_CHECK(cudaEventCreateWithFlags(&b.event, cudaEventDisableTiming));
      // gradients that were finished on other streams than the last one: the event stands for them too
      for (cudaStream_t s : b.streams)
        if (s != now) {
          BAGUA_CUDA_CHECK(cudaEventRecord(b.event, s));
          BAGUA_CUDA_CHECK(cudaStreamWaitEvent(now, b.event, 0));
        }
      BAGUA_CUDA_CHECK(cudaEventRecord(b.event, now));
      event = (uint64_t)(uintptr_t)b.event;
    }
  }
  backend->mark_communication_ready(e.tensor, event);
}

}  // namespace trainer
}  // namespace bagua
