// Gradient-ready hooks of a wrapped model: when autograd has finished with a parameter, its gradient
// is marked ready in the engine, without entering Python.
//
// One hook per parameter sits behind the node that accumulates its gradient.  It keeps the bucket's
// countdown, records the bucket's CUDA event with its last gradient (earlier ones are covered by it, being
// on the same stream or joined to it), and moves a gradient that was replaced from outside back into the bucket.  A Python
// hook with the same duties cost 6-8 us per parameter and step, and the GIL.
#pragma once

#include <ATen/ATen.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/function.h>

#include <atomic>
#include <functional>
#include <memory>
#include <vector>

#include "../runtime/backend.h"

namespace bagua {
namespace trainer {

class GradHooks : public std::enable_shared_from_this<GradHooks> {
 public:
  // device < 0: no events.  The hooks do nothing once the object or the backend is gone.
  GradHooks(std::weak_ptr<CommBackend> backend, int device) : backend_(std::move(backend)), device_(device) {}
  ~GradHooks();

  // `grad`: the tensor registered with the engine as `tensor`, which `param.grad` is expected to be.
  void add(const at::Tensor& param, const at::Tensor& grad, TensorPtr tensor, int bucket);
  void install();  // after the last add()
  void remove();
  void arm();              // before the next backward pass: nothing is marked
  void flush();            // marks what no hook has marked since arm(), in every bucket that is incomplete
  void set_enabled(bool on) { enabled_ = on; }
  // `done` runs once, when the backward pass that reaches any of the watched outputs ends.
  void set_callback(std::function<void()> done) { done_ = std::move(done); }
  void watch(const at::Tensor& output);

 private:
  struct Entry {
    at::Tensor param, grad;
    TensorPtr tensor;
    int bucket = 0;
    bool marked = false;
    std::shared_ptr<torch::autograd::Node> accumulator;
    uintptr_t key = 0;
  };
  struct Bucket {
    int size = 0, pending = 0;
    cudaEvent_t event = nullptr;
    std::vector<cudaStream_t> streams;  // on which gradients were finished since arm(): nearly always one
  };
  void on_gradient(size_t i);
  void mark(Entry& e);

  std::weak_ptr<CommBackend> backend_;
  const int device_;
  bool enabled_ = true;
  std::function<void()> done_;
  std::atomic<bool> queued_{false};
  std::vector<Entry> entries_;
  std::vector<Bucket> buckets_;
};

}  // namespace trainer
}  // namespace bagua
