#include "autograd_ops.h"

#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/autograd.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>

#include <array>
#include <functional>
#include <memory>
#include <mutex>
#include <unordered_map>

#include "../common.h"
#include "../kernels/encoder_ops.h"
#include "../kernels/kernels.h"
#include "../kernels/model_ops.h"
#include "../tensor/tensor.h"
#include "gemm.h"

namespace bagua {
namespace trainer {

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

OpStats& OpStats::global() {
  static OpStats s;
  return s;
}

namespace {

cudaStream_t stream_of(const at::Tensor& t) {
  return t.is_cuda() ? c10::cuda::getCurrentCUDAStream(t.device().index()).stream() : nullptr;
}
kernels::Ctx ctx_of(const at::Tensor& t) {
  return kernels::Ctx{t.is_cuda() ? (int)t.device().index() : -1, stream_of(t)};
}
void count_launches(int n) { OpStats::global().launches += n; }

// A contiguous tensor on `like`'s device.  Straight from the allocator: a step of a medium model makes a hundred, and
// the dispatcher costs as much as the allocation.
at::Tensor fresh(at::IntArrayRef sizes, at::ScalarType type, const at::Tensor& like) {
  if (like.is_cuda()) return at::detail::empty_cuda(sizes, type, like.device(), c10::nullopt);
  return at::empty(sizes, like.options().dtype(type));
}
at::Tensor fresh_like(const at::Tensor& t) {
  if (t.is_cuda() && t.is_contiguous()) return fresh(t.sizes(), t.scalar_type(), t);
  return at::empty_like(t);
}

// A gradient comes from whoever used the result, and may be a view that starts anywhere: these kernels, and the library's
// attention, read 16 bytes at a time without asking.
at::Tensor vector_aligned(const at::Tensor& t) { return (uintptr_t)t.data_ptr() % 16 == 0 ? t : t.clone(); }

// ---- uses of a weight in a graph ---------------------------------------------------------------
// Where a weight takes part in a graph more than once, autograd adds the uses' gradients first and
// accumulates once; accumulating each use by itself would round differently, so both uses of such a
// pair are marked and take autograd's path.  A use lives as long as its node.
struct Use {
  explicit Use(const c10::TensorImpl* key) : key(key) {}
  ~Use();
  const c10::TensorImpl* key;
  std::atomic<bool> shared{false}, done{false};
};
struct UseTable {
  std::mutex mu;
  std::unordered_map<const c10::TensorImpl*, std::weak_ptr<Use>> last;
  static UseTable& global() {
    static UseTable* t = new UseTable();  // nodes may outlive static destruction
    return *t;
  }
};
Use::~Use() {
  auto& t = UseTable::global();
  std::lock_guard<std::mutex> g(t.mu);
  auto it = t.last.find(key);
  if (it != t.last.end() && it->second.expired()) t.last.erase(it);
}
std::shared_ptr<Use> begin_use(const at::Tensor& param) {
  auto use = std::make_shared<Use>(param.unsafeGetTensorImpl());
  std::shared_ptr<Use> prev;  // released after the lock
  auto& t = UseTable::global();
  std::lock_guard<std::mutex> g(t.mu);
  auto& slot = t.last[use->key];
  prev = slot.lock();
  if (prev && !prev->done) {
    prev->shared = true;
    use->shared = true;
  }
  slot = use;
  return use;
}

// A bias of C values, one per column: any other shape that broadcasts is left to autograd, which folds its gradient.
bool per_column(const at::Tensor& bias, int64_t C) { return bias.dim() == 1 && bias.size(0) == C; }

// grad += aᵀ-shaped product a b of bf16 operands, accumulated in fp32.  False: not available, nothing changed.
bool gemm_into(at::Tensor grad, const at::Tensor& a, const at::Tensor& b) {
  if (!grad.is_cuda()) {  // host: no mixed-precision GEMM; widen the operands
    grad.addmm_(a.to(grad.scalar_type()), b.to(grad.scalar_type()));
    return true;
  }
  auto& mode = OpStats::global().gemm_mode;
  // A gradient that does not start on 16 bytes (it follows a tensor of odd size in its bucket) costs the library
  // its fast kernels: 82 us instead of 22 for 3072 x 1024 x 3072.  The product then goes to a buffer of its own and
  // is added from there, unless so few rows are summed that the second pass over the result costs more than the
  // slow kernel: device time apart / direct for 4096 x 4096 from 32, 128, 512 rows 76/54, 80/64, 95/118 us, for
  // 1024 x 1024 17.5/14.4, 17.5/16.4, 18.4/20.5 us, and a launch less.
  constexpr int64_t kFewRows = 256;
  const bool aligned = (uintptr_t)grad.data_ptr() % 16 == 0;
  const at::Tensor dy = a.t();
  if ((aligned || dy.size(0) <= kFewRows) && gemm::weight_grad(dy, b, grad, true)) {
    mode = 1;
    return true;
  }
  if (!aligned) {
    at::Tensor apart = fresh(grad.sizes(), grad.scalar_type(), grad);
    if (gemm::weight_grad(dy, b, apart, false)) {
      mode = mode == 0 ? 1 : mode.load();
      kernels::add_inplace(grad.data_ptr(), apart.data_ptr(), DType::F32, grad.numel(), ctx_of(grad));
      return true;
    }
  }
  if (mode <= 1 && (aligned || mode == 0)) {
    try {
      at::addmm_out(grad, grad, a, b, at::kFloat);
      mode = 1;
      return true;
    } catch (const c10::Error&) {
      if (mode == 1) throw;  // it worked before: a real error, not a missing overload
      mode = 2;
    }
  }
  if (mode == 3) return false;
  at::Tensor product;
  try {
    product = at::mm(a, b, at::kFloat);
  } catch (const c10::Error&) {
    mode = 3;
    return false;
  }
  kernels::add_inplace(grad.data_ptr(), product.data_ptr(), DType::F32, grad.numel(), ctx_of(grad));
  return true;
}

bool autocast_on(const at::Tensor& t) { return at::autocast::is_autocast_enabled(t.device().type()); }

// No autograd below this point, and no autocast.
struct PlainDispatch {
  at::AutoDispatchBelowADInplaceOrView below;
  c10::impl::ExcludeDispatchKeyGuard no_autocast{c10::autocast_dispatch_keyset};
};

// Rounds tensors to bf16, those that are fp32 on the first one's GPU in one launch together.  Undefined ones stay
// undefined.
template <size_t N>
void to_bf16(std::array<at::Tensor, N>& ts) {
  kernels::CastSegment segs[N];
  int n = 0;
  const at::Device device = ts[0].device();
  for (at::Tensor& t : ts) {
    if (!t.defined() || t.scalar_type() == at::kBFloat16) continue;
    if (!t.is_cuda() || t.device() != device || t.scalar_type() != at::kFloat || !t.is_non_overlapping_and_dense()) {
      t = t.to(at::kBFloat16);
      continue;
    }
    at::Tensor low = at::detail::empty_strided_cuda(t.sizes(), t.strides(), at::kBFloat16, t.device());
    segs[n++] = kernels::CastSegment{(const float*)t.data_ptr(), low.data_ptr(), t.numel()};
    // the source stays alive as the caller's tensor until the launch below
    t = low;
  }
  if (n) {
    kernels::cuda::cast_bf16(segs, n, stream_of(ts[0]));
    count_launches(1);
  }
}

// ---- gradients of gradients ----------------------------------------------------------------------
// The kernels leave no history.  Where a backward pass is itself to be differentiated (create_graph=True), a node makes
// its gradients from the plain composition of the framework's operations, evaluated again on the values that it saved.
using Composition = std::function<at::Tensor(const std::vector<at::Tensor>&)>;

// The same composition stands in for the kernels where they would pass somebody by who looks at the operations
// themselves: forward-mode differentiation, torch.func's transforms, tensor subclasses and dispatch modes (tracers, counters).
bool watched(std::initializer_list<const at::Tensor*> inputs) {
  static const c10::DispatchKeySet wrapped({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper});
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return true;
  for (const at::Tensor* t : inputs)
    if (t->defined() && (t->key_set().has_any(wrapped) || t->_fw_grad(/*level=*/0).defined())) return true;
  return false;
}

// Hands its gradient to each of its edges.
struct PassNode : public Node {
  std::string name() const override { return "BaguaSavedValueBackward"; }
  variable_list apply(variable_list&& grads) override { return variable_list(num_outputs(), grads[0]); }
};

// A saved value that stands for the node's inputs `inputs` (more than one: their sum), from which it may differ in type.
struct Saved {
  at::Tensor value;
  std::vector<uint32_t> inputs;
};

variable_list differentiable_gradients(const Node& self, const Composition& f, const std::vector<Saved>& saved, const at::Tensor& dy) {
  std::vector<at::Tensor> values;
  variable_list sources;
  std::vector<const Saved*> wanted;
  for (const Saved& s : saved) {
    values.push_back(s.value);
    if (!s.value.defined()) continue;
    torch::autograd::edge_list edges;
    bool want = false;
    for (uint32_t i : s.inputs) {
      if (self.next_edge(i).is_valid()) edges.push_back(self.next_edge(i));
      want = want || self.task_should_compute_output(i);
    }
    if (edges.empty()) continue;
    auto node = std::shared_ptr<PassNode>(new PassNode(), torch::autograd::deleteNode);
    node->set_next_edges(std::move(edges));
    values.back() = s.value.variable_data();
    torch::autograd::set_history(values.back(), node);
    if (!want) continue;
    sources.push_back(values.back());
    wanted.push_back(&s);
  }
  variable_list out(self.num_outputs());
  if (sources.empty()) return out;
  const variable_list got = torch::autograd::grad({f(values)}, sources, {dy}, /*retain_graph=*/true, /*create_graph=*/true, /*allow_unused=*/true);
  for (size_t k = 0; k < got.size(); ++k)
    for (uint32_t i : wanted[k]->inputs)
      if (self.task_should_compute_output(i)) out[i] = got[k];
  return out;
}

template <typename N>
std::shared_ptr<N> make_node(const at::Tensor& x, const at::Tensor& weight, const at::Tensor& bias) {
  auto node = std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(x, weight, bias));
  return node;
}

std::shared_ptr<PoolRawTensor> scratch_for(const at::Tensor& t, size_t bytes) {
  return PoolRawTensor::allocate((int)t.device().index(), DType::U8, (int64_t)bytes, (uint64_t)(uintptr_t)stream_of(t));
}

// A node that may add parameters' gradients to their `.grad` itself.
struct AccumulatingNode : public Node {
  // For a new node: every parameter that wants a gradient is counted as used.
  void accumulate_gradients(std::initializer_list<const at::Tensor*> params) {
    accumulate_ = true;
    size_t n = 0;
    for (const at::Tensor* p : params)
      if (p->defined() && p->requires_grad()) uses_[n++] = begin_use(*p);
  }

 protected:
  bool accumulates() const { return accumulate_; }
  void uses_done() {
    for (auto& u : uses_)
      if (u) u->done = true;
  }
  // Whether the gradient of input `i`, the parameter `param`, may be added to `param.grad` here: the node was asked to, none
  // of its parameters takes part in the graph elsewhere, the backward pass accumulates it (it is not one that returns the
  // gradient, as torch.autograd.grad does), an fp32 gradient of the parameter's shape and memory layout is there, and no
  // tensor hook wants to see it.
  bool adds(uint32_t i, const at::Tensor& param, const at::Tensor& like) const {
    if (!accumulate_ || !param.defined() || c10::GradMode::is_enabled() || !param.is_leaf() || !next_edge(i).is_valid()) return false;
    for (auto& u : uses_)
      if (u && u->shared) return false;
    const auto* info = torch::autograd::get_current_graph_task_exec_info();
    if (info && !info->empty()) {
      const auto it = info->find(next_edge(i).function.get());
      if (it == info->end() || !it->second.needed_ || it->second.captures_) return false;
    }
    const at::Tensor& grad = param.grad();
    return grad.defined() && grad.scalar_type() == at::kFloat && grad.sizes() == param.sizes() &&
           grad.strides() == param.strides() && grad.is_non_overlapping_and_dense() && grad.device() == like.device() &&
           torch::autograd::impl::hooks(param).empty();
  }
  // Has been done for input `i`.  Autograd orders the stream that a parameter's gradient is finished on (that of its
  // accumulation node, on which its hooks run) behind the stream that made it when it hands the gradient over.  It is
  // handed nothing here, so the order is made here; the streams differ when a model is trained on another stream than the
  // one it was wrapped on.
  void added(uint32_t i, const at::Tensor& on) const {
    if (!on.is_cuda() || !next_edge(i).is_valid()) return;
    const auto to = next_edge(i).function->stream();
    const auto from = c10::cuda::getCurrentCUDAStream(on.device().index());
    if (!to || *to == from.unwrap()) return;
    at::cuda::CUDAEvent done;
    done.record(from);
    done.block(c10::cuda::CUDAStream(*to));
  }

 private:
  bool accumulate_ = false;
  std::array<std::shared_ptr<Use>, 5> uses_;
};

// ---- linear ------------------------------------------------------------------------------------
at::Tensor linear_composition(const std::vector<at::Tensor>& in, int activation) {  // x, weight, bias in one type
  at::Tensor y = at::linear(in[0], in[1], in[2].defined() ? std::optional<at::Tensor>(in[2]) : std::nullopt);
  return activation == kGelu ? at::gelu(y) : activation == kRelu ? at::relu(y) : y;
}

struct LinearNode : public AccumulatingNode {
  SavedVariable x, w, z;  // z: what gelu was applied to, or the ReLU's result
  at::Tensor b;  // with an activation: the bias in bf16, for a second backward pass
  at::Tensor weight, bias;  // the parameters (bias may be undefined)
  int activation = kNone;

  std::string name() const override {
    return activation == kGelu ? "BaguaLinearGeluBackward" : activation == kRelu ? "BaguaLinearReLUBackward" : "BaguaLinearBackward";
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    x.reset_data();
    w.reset_data();
    z.reset_data();
    b = at::Tensor();
  }

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(3);
    uses_done();
    if (!grads[0].defined()) return out;
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    const at::Tensor dy = grads[0], xs = x.unpack(), ws = w.unpack();
    if (c10::GradMode::is_enabled()) {
      // (without an activation no gradient depends on the bias' value)
      const at::Tensor bs = b.defined() || !bias.defined() ? b : bias.detach().to(at::kBFloat16);
      return differentiable_gradients(*this, [this](const auto& in) { return linear_composition(in, activation); },
                                      {{xs, {0}}, {ws, {1}}, {bs, {2}}}, dy);
    }
    at::Tensor dy2 = vector_aligned(dy.dim() == 2 ? dy : dy.reshape({-1, dy.size(-1)}));
    if (activation) dy2 = through_activation(dy2.contiguous(), out);
    if (task_should_compute_output(0)) {
      at::Tensor dx = fresh({dy2.size(0), ws.size(1)}, dy2.scalar_type(), dy2);
      if (!gemm::input_grad(dy2, ws, dx)) dx = at::mm(dy2, ws);
      out[0] = dy.dim() == 2 ? dx : dx.view(xs.sizes());
    }
    if (task_should_compute_output(1)) {
      const at::Tensor x2 = xs.dim() == 2 ? xs : xs.reshape({-1, xs.size(-1)});
      bool done = false;
      if (accumulates()) {
        if (adds(1, weight, dy2) && weight.grad().is_contiguous()) {
          c10::NoGradGuard no_grad;
          done = gemm_into(weight.grad(), dy2.t(), x2);
          if (done) added(1, dy2);
        }
        auto& stats = OpStats::global();
        done ? ++stats.accumulated : ++stats.declined;
      }
      if (!done) out[1] = at::mm(dy2.t(), x2);  // autograd casts it to the parameter's type
    }
    if (!activation && bias.defined() && task_should_compute_output(2)) out[2] = bias_grad(dy2);
    return out;
  }

  // the activation's derivative applied to the incoming gradient, and the bias gradient of the result from the same pass
  at::Tensor through_activation(const at::Tensor& dy2, variable_list& out) {
    const at::Tensor zs = z.unpack(activation == kRelu ? shared_from_this() : std::shared_ptr<Node>());
    const int64_t rows = dy2.size(0);
    const int C = (int)dy2.size(1);
    const bool want = bias.defined() && task_should_compute_output(2);
    const bool add = want && per_column(bias, C) && adds(2, bias, dy2);
    at::Tensor db = add ? bias.grad() : fresh({C}, at::kFloat, dy2);
    at::Tensor dz = fresh_like(dy2);
    const size_t bytes = encoder_ops::activation_backward_scratch_bytes(rows, C);
    std::shared_ptr<PoolRawTensor> scratch = bytes ? scratch_for(dy2, bytes) : nullptr;
    encoder_ops::activation_backward(activation == kGelu, dy2.data_ptr(), zs.data_ptr(), dz.data_ptr(), db.data_ptr<float>(),
                                     add, scratch ? scratch->data_ptr() : nullptr, rows, C, stream_of(dy2));
    count_launches(bytes ? 2 : 1);
    if (add) added(2, dy2);
    if (want && !add) out[2] = db;
    return dz;
  }

  at::Tensor bias_grad(const at::Tensor& dy2) {
    const int64_t rows = dy2.size(0), C = dy2.size(1);
    if (!dy2.is_cuda() || dy2.scalar_type() != at::kBFloat16 || C > (1 << 24) ||
        !model_ops::column_sum_supported(rows, (int)C) || !dy2.is_contiguous() || (uintptr_t)dy2.data_ptr() % 16 != 0)
      return dy2.sum(at::IntArrayRef{0}, /*keepdim=*/false, at::kFloat);
    const bool add = per_column(bias, C) && adds(2, bias, dy2);
    at::Tensor db = add ? bias.grad() : fresh({C}, at::kFloat, dy2);
    const size_t bytes = model_ops::column_sum_scratch_bytes(rows, (int)C);
    std::shared_ptr<PoolRawTensor> scratch = bytes ? scratch_for(dy2, bytes) : nullptr;
    model_ops::column_sum_bf16(dy2.data_ptr(), db.data_ptr<float>(), rows, (int)C, scratch ? scratch->data_ptr() : nullptr,
                               stream_of(dy2), add);
    count_launches(bytes ? 2 : 1);
    if (add) added(2, dy2);
    return add ? at::Tensor() : db;
  }
};

// ---- convolution + bias + ReLU (+ pooling) -------------------------------------------------------
at::Tensor conv_composition(const std::vector<at::Tensor>& in, const std::vector<int64_t>& stride,  // x, weight, bias in one type
                            const std::vector<int64_t>& padding, const std::vector<int64_t>& dilation, int64_t groups, bool pool) {
  const std::vector<int64_t> zero{0, 0};
  const at::Tensor z = at::convolution(in[0], in[1], c10::nullopt, stride, padding, dilation, false, zero, groups);
  const at::Tensor y = at::relu(z + in[2].view({1, -1, 1, 1}));
  return pool ? at::max_pool2d(y, {2, 2}, {2, 2}) : y;
}

struct ConvNode : public AccumulatingNode {
  SavedVariable x, w, b, act;  // act: the activation, or with pooling the convolution's output (CPU)
  // CUDA: a bit per value of the activation, whether it is positive; with pooling four per pooled value, where it came from.
  // Not where first_layer() is expected to serve: that reads the activation.
  SavedVariable signs;
  at::Tensor weight, bias;
  std::vector<int64_t> stride, padding, dilation;
  int64_t groups = 1;
  bool pool = false;  // 2x2, behind the ReLU

  std::string name() const override { return pool ? "BaguaConvBiasReLUPoolBackward" : "BaguaConvBiasReLUBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    x.reset_data();
    w.reset_data();
    b.reset_data();
    act.reset_data();
    signs.reset_data();
  }

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(3);
    uses_done();
    if (!grads[0].defined()) return out;
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    const at::Tensor xs = x.unpack(), ws = w.unpack(), bits = signs.unpack();
    const at::Tensor a = pool && bits.defined() ? at::Tensor() : act.unpack(pool ? std::shared_ptr<Node>() : shared_from_this());
    if (c10::GradMode::is_enabled())
      return differentiable_gradients(*this, [this](const auto& in) { return conv_composition(in, stride, padding, dilation, groups, pool); },
                                      {{xs, {0}}, {ws, {1}}, {b.unpack(), {2}}}, grads[0]);
    const at::Tensor dy = vector_aligned(grads[0].contiguous(at::MemoryFormat::ChannelsLast));
    const int C = (int)ws.size(0);
    if (!pool && first_layer(xs, dy, a)) {
      first_layer_backward(xs, dy, a, out);
      return out;
    }
    at::Tensor dz = at::empty({dy.size(0), C, dy.size(2) * (pool ? 2 : 1), dy.size(3) * (pool ? 2 : 1)}, dy.options().dtype(at::kBFloat16),
                              at::MemoryFormat::ChannelsLast);
    // the bias gradient is added to `.grad` by the fold of its partial sums
    const bool add_bias = dy.is_cuda() && task_should_compute_output(2) && adds(2, bias, dy);
    at::Tensor db = add_bias ? bias.grad() : fresh({C}, at::kFloat, dz);
    backward_tail(dy, a, bits, dz, db, add_bias);
    if (add_bias) added(2, dy);
    if (task_should_compute_output(2) && !add_bias) out[2] = db;
    const bool need_x = task_should_compute_output(0), need_w = task_should_compute_output(1);
    const bool own = need_w && own_weight_gradient(xs, dz);
    if (need_x || (need_w && !own)) {
      const std::vector<int64_t> zero{0, 0};
      auto g = at::convolution_backward(dz, xs, ws, c10::nullopt, stride, padding, dilation, false, zero, groups,
                                        {need_x, need_w && !own, false});
      out[0] = std::get<0>(g);
      at::Tensor dw = std::get<1>(g);
      if (need_w && !own && dw.scalar_type() == at::kBFloat16 && adds(1, weight, dw) &&
          dw.strides() == weight.grad().strides()) {
        // the cast to fp32 and the addition in one pass; the same bits
        if (dw.is_cuda()) {
          kernels::cuda::accumulate_bf16((float*)weight.grad().data_ptr(), dw.data_ptr(), dw.numel(), stream_of(dw));
          count_launches(1);
        } else {
          c10::NoGradGuard no_grad;
          weight.grad().add_(dw);
        }
        added(1, dw);
      } else {
        out[1] = dw;
      }
    }
    if (own) out[1] = weight_gradient(xs, dz);
    return out;
  }

  bool is_plain3x3() const {
    const std::vector<int64_t> one{1, 1};
    return groups == 1 && weight.size(2) == 3 && weight.size(3) == 3 && stride == one && padding == one && dilation == one;
  }

  // The weight gradient of a 3 x 3 convolution of many channels, where this package's kernel is the faster one.  bf16 parameters
  // only: where they are fp32 (autocast) their gradients keep the bits of the library's.  This kernel's are the more exact ones (0.05-0.2 %
  // are not the exact sum's rounding, 0.35-1.4 % of the library's), but VGG-16 at batch 32, which would take 4185 us a step instead of 4521,
  // is chaotic: gradients 1e-4 apart (relative norm) in one step are 10 % apart in the next, as far as another choice of the
  // library's algorithms moves them (profiles/vgg16_weight_gradient_rounding.md).
  bool own_weight_gradient(const at::Tensor& xs, const at::Tensor& dz) const {
    return dz.is_cuda() && is_plain3x3() && weight.scalar_type() == at::kBFloat16 && xs.scalar_type() == at::kBFloat16 &&
           dz.scalar_type() == at::kBFloat16 && xs.is_contiguous(at::MemoryFormat::ChannelsLast) &&
           dz.is_contiguous(at::MemoryFormat::ChannelsLast) && (uintptr_t)xs.data_ptr() % 16 == 0 && (uintptr_t)dz.data_ptr() % 16 == 0 &&
           model_ops::conv_wgrad_preferred(dz.size(0), dz.size(2), dz.size(3), dz.size(1), xs.size(1));
  }
  static at::Tensor weight_gradient(const at::Tensor& xs, const at::Tensor& dz) {
    const int64_t N = dz.size(0), H = dz.size(2), W = dz.size(3), Co = dz.size(1), Ci = xs.size(1);
    const at::Tensor dw = at::empty({Co, Ci, 3, 3}, dz.options(), at::MemoryFormat::ChannelsLast);
    const int64_t strides[4] = {dw.stride(0), dw.stride(2), dw.stride(3), dw.stride(1)};
    const at::Tensor sums = fresh({(int64_t)model_ops::conv_wgrad_scratch_bytes(N, H, W, Co, Ci)}, at::kByte, dz);
    model_ops::conv_wgrad(dz.data_ptr(), xs.data_ptr(), dw.data_ptr(), strides, N, H, W, Co, Ci, sums.data_ptr(), stream_of(dz));
    count_launches(2);
    return dw;
  }

  // A 3 x 3 convolution of few channels whose input wants no gradient: both gradients come from one kernel.
  bool first_layer_shape(const at::Tensor& xs, const at::Tensor& a) const {
    return a.is_cuda() && is_plain3x3() && xs.scalar_type() == at::kBFloat16 && xs.is_contiguous(at::MemoryFormat::ChannelsLast) &&
           a.is_contiguous(at::MemoryFormat::ChannelsLast) && (uintptr_t)a.data_ptr() % 16 == 0 &&
           model_ops::first_conv_backward_supported(a.size(0), a.size(2), a.size(3), a.size(1), xs.size(1));
  }
  bool first_layer(const at::Tensor& xs, const at::Tensor& dy, const at::Tensor& a) {
    return !task_should_compute_output(0) && task_should_compute_output(1) && (uintptr_t)dy.data_ptr() % 16 == 0 &&
           first_layer_shape(xs, a);
  }
  void first_layer_backward(const at::Tensor& xs, const at::Tensor& dy, const at::Tensor& a, variable_list& out) {
    const int C = (int)a.size(1), Ci = (int)xs.size(1);
    const bool want_b = task_should_compute_output(2);
    const bool add_b = want_b && adds(2, bias, dy);
    const bool add_w = weight.is_contiguous(at::MemoryFormat::ChannelsLast) && adds(1, weight, dy);
    const auto f = a.options().dtype(at::kFloat);
    at::Tensor db = add_b ? bias.grad() : want_b ? at::empty({C}, f) : at::Tensor();
    at::Tensor dw = add_w ? weight.grad() : at::empty(weight.sizes(), f, at::MemoryFormat::ChannelsLast);
    auto scratch = scratch_for(a, model_ops::first_conv_backward_scratch_bytes(a.numel() / C, C, Ci));
    model_ops::first_conv_backward(dy.data_ptr(), a.data_ptr(), xs.data_ptr(), dw.data_ptr<float>(), add_w,
                                   db.defined() ? db.data_ptr<float>() : nullptr, add_b, a.size(0), a.size(2), a.size(3), C, Ci,
                                   scratch->data_ptr(), stream_of(a));
    count_launches(2);
    if (add_w)
      added(1, a);
    else
      out[1] = dw;
    if (add_b)
      added(2, a);
    else if (want_b)
      out[2] = db;
  }

  void backward_tail(const at::Tensor& dy, const at::Tensor& a, const at::Tensor& bits, at::Tensor& dz, at::Tensor& db, bool add) {
    const int64_t N = dz.size(0), H = dz.size(2), W = dz.size(3), rows = N * H * W;
    const int C = (int)dz.size(1);
    float* dbp = db.data_ptr<float>();
    if (!dz.is_cuda()) {
      if (pool) {
        at::Tensor y = a.clone();
        model_ops::bias_relu_inplace_bf16_host(y.data_ptr(), b.unpack().data_ptr(), rows, C);
        model_ops::bias_relu_pool_backward_bf16_host(dy.data_ptr(), y.data_ptr(), dz.data_ptr(), dbp, N, H, W, C);
      } else {
        model_ops::bias_relu_backward_bf16_host(dy.data_ptr(), a.data_ptr(), dz.data_ptr(), dbp, rows, C);
      }
      return;
    }
    auto scratch = scratch_for(dz, model_ops::bias_relu_backward_scratch_bytes(pool ? N * (H / 2) * (W / 2) : rows, C));
    if (pool)
      model_ops::bias_relu_pool_backward_codes_bf16(dy.data_ptr(), bits.data_ptr(), dz.data_ptr(), dbp, N, H, W, C, scratch->data_ptr(),
                                                    stream_of(dz), add);
    else
      model_ops::bias_relu_backward_bf16(dy.data_ptr(), a.data_ptr(), dz.data_ptr(), dbp, rows, C, scratch->data_ptr(),
                                         stream_of(dz), add, bits.defined() ? bits.data_ptr() : nullptr);
    count_launches(2);  // mask and partial sums, then their fold
  }
};

// ---- encoder layers ------------------------------------------------------------------------------
struct EncoderNode : public AccumulatingNode {
 protected:
  bool adds_contiguous(uint32_t i, const at::Tensor& param) const { return adds(i, param, param) && param.grad().is_contiguous(); }
  // Adds the gradient of input `i` to its place, or leaves it to autograd.
  void give(uint32_t i, const at::Tensor& param, const at::Tensor& g, variable_list& out) const {
    if (!g.defined()) return;
    if (!adds_contiguous(i, param)) {
      out[i] = g;  // autograd casts it to the parameter's type
      return;
    }
    if (g.scalar_type() == at::kBFloat16)
      kernels::cuda::accumulate_bf16((float*)param.grad().data_ptr(), g.data_ptr(), g.numel(), stream_of(g));
    else
      kernels::add_inplace(param.grad().data_ptr(), g.data_ptr(), DType::F32, g.numel(), ctx_of(g));
    count_launches(1);
    added(i, g);
  }
};

struct LayerNormNode : public EncoderNode {
  SavedVariable sum, mean, rstd, g, b;  // g, b: the parameters in bf16
  at::Tensor gamma, beta;
  bool residual = false;
  double eps = 0;

  std::string name() const override { return "BaguaAddLayerNormBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* v : {&sum, &mean, &rstd, &g, &b}) v->reset_data();
  }
  variable_list apply(variable_list&& grads) override {  // x, r, gamma, beta
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(4);
    uses_done();
    if (!grads[0].defined()) return out;
    const at::Tensor s = sum.unpack();
    if (c10::GradMode::is_enabled())
      return differentiable_gradients(
          *this, [this](const auto& in) { return at::layer_norm(in[0], {in[0].size(-1)}, in[1], in[2], eps); },
          {{s, {0, 1}}, {g.unpack(), {2}}, {b.unpack(), {3}}}, grads[0]);
    const auto d = at::native_layer_norm_backward(grads[0].contiguous(), s, {s.size(-1)}, mean.unpack(), rstd.unpack(),
                                                  g.unpack(), b.unpack(),
                                                  {true, task_should_compute_output(2), task_should_compute_output(3)});
    out[0] = std::get<0>(d);
    if (residual) out[1] = out[0];
    const at::Tensor &dg = std::get<1>(d), &db = std::get<2>(d);
    if (dg.defined() && db.defined() && adds_contiguous(2, gamma) && adds_contiguous(3, beta)) {
      kernels::cuda::accumulate_bf16_pair(gamma.grad().data_ptr<float>(), dg.data_ptr(), beta.grad().data_ptr<float>(),
                                          db.data_ptr(), dg.numel(), stream_of(s));
      count_launches(1);
      added(2, s);
      added(3, s);
      return out;
    }
    give(2, gamma, dg, out);
    give(3, beta, db, out);
    return out;
  }
};

at::Tensor embed_composition(const at::Tensor& ids, const std::vector<at::Tensor>& in, double eps) {  // tok, pos, typ, gamma, beta
  const at::Tensor x = at::embedding(in[0], ids) + in[1].narrow(0, 0, ids.size(1)).unsqueeze(0) + in[2].select(0, 0);
  return at::layer_norm(x, {x.size(-1)}, in[3], in[4], eps).to(at::kBFloat16);
}

struct EmbedNode : public EncoderNode {
  SavedVariable ids, sum, mean, rstd;
  at::Tensor param[5];  // tok, pos, typ, gamma, beta
  int64_t version[5];
  double eps = 0;

  std::string name() const override { return "BaguaEmbedLayerNormBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* v : {&ids, &sum, &mean, &rstd}) v->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(5);
    uses_done();
    if (!grads[0].defined()) return out;
    encoder_ops::check_indices();
    const at::Tensor id = ids.unpack(), s = sum.unpack();
    const int H = (int)param[0].size(1);
    const int64_t batch = id.size(0), seq = id.size(1);
    if (c10::GradMode::is_enabled()) {
      std::vector<Saved> saved;
      for (uint32_t k = 0; k < 5; ++k) {
        BAGUA_CHECK(param[k]._version() == version[k], Tensor,
                    "an embedding parameter needed for the gradient of a gradient was modified in place");
        saved.push_back({param[k].detach(), {k}});
      }
      return differentiable_gradients(*this, [&](const auto& in) { return embed_composition(id, in, eps); }, saved, grads[0]);
    }
    // only what is asked for: a frozen parameter has a gradient in its bucket all the same, which stays as it is
    bool want[5];
    for (uint32_t k = 0; k < 5; ++k) want[k] = task_should_compute_output(k);
    const auto d = at::native_layer_norm_backward(grads[0].to(at::kFloat).contiguous(), s, {H}, mean.unpack(), rstd.unpack(),
                                                  param[3], param[4], {want[0] || want[1] || want[2], want[3], want[4]});
    give(3, param[3], std::get<1>(d), out);
    give(4, param[4], std::get<2>(d), out);
    if (!want[0] && !want[1] && !want[2]) return out;
    bool add[3] = {false, false, false};
    float* grad[3] = {nullptr, nullptr, nullptr};
    for (uint32_t k = 0; k < 3; ++k) {
      if (!want[k]) continue;
      add[k] = adds_contiguous(k, param[k]);
      if (!add[k]) out[k] = at::zeros(param[k].sizes(), param[k].options());
      grad[k] = (add[k] ? param[k].grad() : out[k]).data_ptr<float>();
    }
    auto scratch = scratch_for(s, encoder_ops::embed_backward_scratch_bytes(batch * seq, H));
    count_launches(encoder_ops::embed_backward(std::get<0>(d).data_ptr<float>(), id.data_ptr<int64_t>(), param[0].size(0), grad[0],
                                               grad[1], grad[2], scratch->data_ptr(), batch, seq, H, stream_of(s)));
    for (uint32_t k = 0; k < 3; ++k)
      if (add[k]) added(k, s);
    return out;
  }
};

at::Tensor span_loss_composition(const at::Tensor& logits, const at::Tensor& start, const at::Tensor& end) {
  const at::Tensor f = logits.to(at::kFloat);
  return (at::cross_entropy_loss(f.select(2, 0), start) + at::cross_entropy_loss(f.select(2, 1), end)) / 2;
}

struct SpanLossNode : public Node {
  SavedVariable logits, start, end, stats;

  std::string name() const override { return "BaguaSpanLossBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* v : {&logits, &start, &end, &stats}) v->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(1);
    if (!grads[0].defined()) return out;
    const at::Tensor x = logits.unpack(), a = start.unpack(), b = end.unpack(), st = stats.unpack();
    if (c10::GradMode::is_enabled())
      return differentiable_gradients(*this, [&](const auto& in) { return span_loss_composition(in[0], a, b); }, {{x, {0}}}, grads[0]);
    at::Tensor dx = fresh_like(x);
    encoder_ops::span_loss_backward(x.data_ptr(), a.data_ptr<int64_t>(), b.data_ptr<int64_t>(), st.data_ptr<float>(),
                                    grads[0].data_ptr<float>(), dx.data_ptr(), x.size(0), x.size(1), stream_of(x));
    count_launches(1);
    out[0] = dx;
    return out;
  }
};

// q, k, v as views of the packed projection; backward writes their gradients into one packed tensor.
struct SplitHeadsNode : public Node {
  int64_t batch = 0, seq = 0, heads = 0, dim = 0;
  at::TensorOptions options;

  std::string name() const override { return "BaguaSplitHeadsBackward"; }
  variable_list apply(variable_list&& grads) override {
    variable_list out(1);
    if (c10::GradMode::is_enabled()) {
      for (at::Tensor& g : grads) g = (g.defined() ? g : at::zeros({batch, heads, seq, dim}, options)).transpose(1, 2);
      out[0] = at::stack({grads[0], grads[1], grads[2]}, 2).reshape({batch, seq, 3 * heads * dim});
      return out;
    }
    at::Tensor packed = at::empty({batch, seq, 3 * heads * dim}, options);
    const void* src[3];
    encoder_ops::HeadStrides st[3];
    at::Tensor keep[3];
    for (int q = 0; q < 3; ++q) {
      at::Tensor g = grads[(size_t)q].defined() ? grads[(size_t)q] : at::zeros({batch, heads, seq, dim}, options);
      const bool direct = g.stride(3) == 1 && g.stride(0) % 8 == 0 && g.stride(1) % 8 == 0 && g.stride(2) % 8 == 0 &&
                          (uintptr_t)g.data_ptr() % 16 == 0;
      keep[q] = direct ? g : vector_aligned(g.contiguous());
      src[q] = keep[q].data_ptr();
      st[q] = encoder_ops::HeadStrides{keep[q].stride(0), keep[q].stride(1), keep[q].stride(2)};
    }
    encoder_ops::merge_heads(src, st, packed.data_ptr(), batch, seq, (int)heads, (int)dim, stream_of(packed));
    count_launches(1);
    out[0] = packed;
    return out;
  }
};

bool fp32_param(const at::Tensor& p, int64_t H, const at::Tensor& like) {
  return p.scalar_type() == at::kFloat && p.is_contiguous() && p.size(-1) == H && p.device() == like.device();
}

}  // namespace

at::Tensor linear(const at::Tensor& x, const at::Tensor& weight, const std::optional<at::Tensor>& bias,
                  const std::optional<at::Tensor>& w_low, bool accumulate, int activation) {
  BAGUA_CHECK(activation == kNone || ((activation == kGelu || activation == kRelu) && activation_fusable(x, weight.size(0))), Tensor,
              "the activation cannot be fused with this layer");
  const at::Tensor b = bias.value_or(at::Tensor());
  if (watched({&x, &weight, &b})) {
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    return linear_composition({x.to(at::kBFloat16), weight.to(at::kBFloat16), b.defined() ? b.to(at::kBFloat16) : b}, activation);
  }
  std::shared_ptr<LinearNode> node;
  if (torch::autograd::compute_requires_grad(x, weight, b)) node = make_node<LinearNode>(x, weight, b);
  at::Tensor xs, ws, z, y;
  std::array<at::Tensor, 3> low{x, w_low ? *w_low : weight, b};
  {
    PlainDispatch plain;
    to_bf16(low);
    xs = low[0];
    ws = low[1];
    if (xs.is_cuda() && xs.is_contiguous() && xs.numel() > 0 && xs.dim() >= 2) {
      std::vector<int64_t> shape(xs.sizes().begin(), xs.sizes().end());
      shape.back() = ws.size(0);
      y = fresh(shape, xs.scalar_type(), xs);
      at::Tensor y2 = y.dim() == 2 ? y : y.view({-1, ws.size(0)});
      if (!gemm::linear(xs.dim() == 2 ? xs : xs.view({-1, xs.size(-1)}), ws, low[2], activation == kRelu, y2)) y = at::Tensor();
    }
    const bool product_only = !y.defined();
    if (!y.defined()) y = at::linear(xs, ws, b.defined() ? std::optional<at::Tensor>(low[2]) : std::nullopt);
    if (activation == kRelu) {
      if (product_only) y.relu_();
      y = y.contiguous();
    } else if (activation == kGelu) {
      z = y.contiguous();
      y = fresh_like(z);
      encoder_ops::gelu_forward(z.data_ptr(), y.data_ptr(), z.numel(), stream_of(z));
      count_launches(1);
    }
  }
  if (node) {
    node->x = SavedVariable(xs, false);
    node->w = SavedVariable(ws, false);
    if (activation) node->b = low[2];
    if (activation == kGelu) node->z = SavedVariable(z, false);
    node->activation = activation;
    node->weight = weight;
    node->bias = b;
    if (accumulate) node->accumulate_gradients({&weight, &b});
    torch::autograd::set_history(y, node);
    if (activation == kRelu) node->z = SavedVariable(y, /*is_output=*/true);
  }
  return y;
}

at::Tensor conv_bias_relu(const at::Tensor& x, const at::Tensor& weight, const at::Tensor& bias,
                          const std::vector<int64_t>& stride, const std::vector<int64_t>& padding,
                          const std::vector<int64_t>& dilation, int64_t groups, bool pool,
                          const std::optional<at::Tensor>& w_low, bool accumulate) {
  const bool cast = autocast_on(x);
  const at::ScalarType low = cast ? at::autocast::get_autocast_dtype(x.device().type()) : at::kBFloat16;
  if (watched({&x, &weight, &bias})) {
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    auto in = [&](const at::Tensor& t) { return cast ? t.to(low) : t; };
    return conv_composition({in(x), in(weight), in(bias)}, stride, padding, dilation, groups, pool);
  }
  std::shared_ptr<ConvNode> node;
  if (torch::autograd::compute_requires_grad(x, weight, bias)) {
    node = make_node<ConvNode>(x, weight, bias);
    node->weight = weight;
    node->bias = bias;
    node->stride = stride;
    node->padding = padding;
    node->dilation = dilation;
    node->groups = groups;
    node->pool = pool;
  }
  at::Tensor xs, ws, bs, z, out, signs;
  {
    PlainDispatch plain;
    std::array<at::Tensor, 3> ts{x, w_low ? *w_low : weight, bias};
    if (cast && low == at::kBFloat16)
      to_bf16(ts);
    else if (cast)
      for (at::Tensor& t : ts) t = t.to(low);
    xs = ts[0].contiguous(at::MemoryFormat::ChannelsLast);
    ws = ts[1];
    bs = ts[2].contiguous();
    const std::vector<int64_t> zero{0, 0};
    z = at::convolution(xs, ws, c10::nullopt, stride, padding, dilation, false, zero, groups)
            .contiguous(at::MemoryFormat::ChannelsLast);
    const int64_t N = z.size(0), H = z.size(2), W = z.size(3), rows = N * H * W;
    const int C = (int)z.size(1);
    BAGUA_CHECK(z.scalar_type() == at::kBFloat16 && bs.scalar_type() == at::kBFloat16, Tensor,
                "fused convolution blocks compute in bf16");
    BAGUA_CHECK(bs.dim() == 1 && bs.size(0) == C && bs.device() == z.device(), Tensor,
                "a convolution of " << C << " channels needs as many bias values on its device");
    if (pool) {
      out = at::empty({N, C, H / 2, W / 2}, z.options().memory_format(at::MemoryFormat::ChannelsLast));
      if (z.is_cuda()) {
        if (node) signs = fresh({out.numel() / 8}, at::kInt, z);
        model_ops::bias_relu_pool_only_bf16(z.data_ptr(), out.data_ptr(), bs.data_ptr(), N, H, W, C, stream_of(z),
                                            node ? signs.data_ptr() : nullptr);
      } else
        model_ops::bias_relu_pool_only_bf16_host(z.data_ptr(), out.data_ptr(), bs.data_ptr(), N, H, W, C);
    } else {
      out = z;
      if (z.is_cuda()) {
        if (node && (x.requires_grad() || !weight.requires_grad() || !node->first_layer_shape(xs, z)))
          signs = fresh({z.numel() / 8}, at::kByte, z);
        model_ops::bias_relu_inplace_bf16(z.data_ptr(), bs.data_ptr(), rows, C, stream_of(z), signs.defined() ? signs.data_ptr() : nullptr);
      } else
        model_ops::bias_relu_inplace_bf16_host(z.data_ptr(), bs.data_ptr(), rows, C);
    }
    if (z.is_cuda()) count_launches(1);
  }
  if (node) {
    node->x = SavedVariable(xs, false);
    node->w = SavedVariable(ws, false);
    if (accumulate) node->accumulate_gradients({&weight, &bias});
    torch::autograd::set_history(out, node);
    node->b = SavedVariable(bs, false);
    node->signs = SavedVariable(signs, false);
    if (!pool)
      node->act = SavedVariable(out, /*is_output=*/true);
    else if (!signs.defined())
      node->act = SavedVariable(z, false);
  }
  return out;
}

at::Tensor add_layer_norm(const at::Tensor& x, const std::optional<at::Tensor>& r, const at::Tensor& gamma,
                          const at::Tensor& beta, double eps, bool accumulate) {
  const int64_t H = x.size(-1);
  const at::Tensor res = r.value_or(at::Tensor());
  BAGUA_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.numel() > 0 && fp32_param(gamma, H, x) &&
                  fp32_param(beta, H, x) && gamma.dim() == 1 && beta.dim() == 1 &&
                  (!res.defined() || (res.sizes() == x.sizes() && res.scalar_type() == at::kBFloat16 && res.device() == x.device())),
              Tensor, "add_layer_norm needs bf16 CUDA activations of one shape and fp32 parameters");
  if (watched({&x, &res, &gamma, &beta})) {
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    return at::layer_norm(res.defined() ? x + res : x, {H}, gamma.to(x.scalar_type()), beta.to(x.scalar_type()), eps);
  }
  std::shared_ptr<LayerNormNode> node;
  if (torch::autograd::compute_requires_grad(x, res, gamma, beta)) {
    node = std::shared_ptr<LayerNormNode>(new LayerNormNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, res, gamma, beta));
  }
  at::Tensor sum, y, mean, rstd;
  std::array<at::Tensor, 2> low{gamma, beta};
  {
    PlainDispatch plain;
    sum = (res.defined() ? at::add(x, res) : x).contiguous();
    to_bf16(low);
    std::tie(y, mean, rstd) = at::native_layer_norm(sum, {H}, low[0], low[1], eps);
  }
  if (node) {
    node->sum = SavedVariable(sum, false);
    node->mean = SavedVariable(mean, false);
    node->rstd = SavedVariable(rstd, false);
    node->g = SavedVariable(low[0], false);
    node->b = SavedVariable(low[1], false);
    node->gamma = gamma;
    node->beta = beta;
    if (accumulate) node->accumulate_gradients({&gamma, &beta});
    node->residual = res.defined();
    node->eps = eps;
    torch::autograd::set_history(y, node);
  }
  return y;
}

at::Tensor embed_layer_norm(const at::Tensor& ids, const at::Tensor& tok, const at::Tensor& pos, const at::Tensor& typ,
                            const at::Tensor& gamma, const at::Tensor& beta, double eps, bool accumulate) {
  const int64_t H = tok.size(1);
  BAGUA_CHECK(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.dim() == 2 && ids.numel() > 0 &&
                  ids.numel() <= encoder_ops::kMaxTokens,
              Tensor, "embed_layer_norm: unsupported ids");
  for (const at::Tensor* p : {&tok, &pos, &typ, &gamma, &beta})
    BAGUA_CHECK(fp32_param(*p, H, ids), Tensor, "embed_layer_norm needs fp32 tables on the ids' device");
  BAGUA_CHECK(tok.dim() == 2 && pos.dim() == 2 && typ.dim() == 2 && tok.size(0) > 0 && typ.size(0) > 0 && gamma.dim() == 1 &&
                  beta.dim() == 1,
              Tensor, "embed_layer_norm needs tables with rows and parameters of one row");
  BAGUA_CHECK(ids.size(1) <= pos.size(0), Tensor, "sequence of " << ids.size(1) << " tokens, " << pos.size(0) << " positions");
  if (watched({&ids, &tok, &pos, &typ, &gamma, &beta})) {
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    return embed_composition(ids, {tok, pos, typ, gamma, beta}, eps);
  }
  std::shared_ptr<EmbedNode> node;
  if (torch::autograd::compute_requires_grad(tok, pos, typ, gamma, beta)) {
    node = std::shared_ptr<EmbedNode>(new EmbedNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(tok, pos, typ, gamma, beta));
  }
  encoder_ops::check_indices();
  at::Tensor idc, sum, mean, rstd;
  std::array<at::Tensor, 1> y;
  {
    PlainDispatch plain;
    idc = ids.contiguous();
    const int64_t batch = ids.size(0), seq = ids.size(1);
    sum = fresh({batch, seq, H}, at::kFloat, tok);
    encoder_ops::embed_sum(idc.data_ptr<int64_t>(), tok.size(0), tok.data_ptr<float>(), pos.data_ptr<float>(),
                           typ.data_ptr<float>(), sum.data_ptr<float>(), batch, seq, (int)H, stream_of(tok));
    count_launches(1);
    std::tie(y[0], mean, rstd) = at::native_layer_norm(sum, {H}, gamma, beta, eps);
    to_bf16(y);
  }
  if (node) {
    node->ids = SavedVariable(idc, false);
    node->sum = SavedVariable(sum, false);
    node->mean = SavedVariable(mean, false);
    node->rstd = SavedVariable(rstd, false);
    const at::Tensor* ps[5] = {&tok, &pos, &typ, &gamma, &beta};
    for (int k = 0; k < 5; ++k) {
      node->param[k] = *ps[k];
      node->version[k] = ps[k]->_version();
    }
    node->eps = eps;
    if (accumulate) node->accumulate_gradients({&tok, &pos, &typ, &gamma, &beta});
    torch::autograd::set_history(y[0], node);
  }
  return y[0];
}

at::Tensor span_loss(const at::Tensor& logits, const at::Tensor& start, const at::Tensor& end) {
  const int64_t B = logits.size(0);
  BAGUA_CHECK(logits.is_cuda() && logits.dim() == 3 && logits.size(2) == 2 && logits.scalar_type() == at::kBFloat16 &&
                  logits.numel() > 0 && logits.numel() < (1ll << 30),
              Tensor, "span_loss needs bf16 CUDA logits [batch, seq, 2]");
  for (const at::Tensor* t : {&start, &end})
    BAGUA_CHECK(t->device() == logits.device() && t->scalar_type() == at::kLong && t->dim() == 1 && t->size(0) == B, Tensor,
                "span_loss needs int64 positions [batch] on the logits' device");
  if (watched({&logits, &start, &end})) {
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::autocast_dispatch_keyset);
    return span_loss_composition(logits, start, end);
  }
  std::shared_ptr<SpanLossNode> node;
  if (torch::autograd::compute_requires_grad(logits)) {
    node = std::shared_ptr<SpanLossNode>(new SpanLossNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(logits));
  }
  encoder_ops::check_indices();
  at::Tensor x, a, b, loss, stats;
  {
    PlainDispatch plain;
    x = logits.contiguous();
    if ((uintptr_t)x.data_ptr() % 4 != 0) x = x.clone();
    a = start.contiguous();
    b = end.contiguous();
    loss = fresh({}, at::kFloat, x);
    stats = fresh({2 * B + 2}, at::kFloat, x);
    encoder_ops::span_loss_forward(x.data_ptr(), a.data_ptr<int64_t>(), b.data_ptr<int64_t>(), loss.data_ptr<float>(),
                                   stats.data_ptr<float>(), B, x.size(1), stream_of(x));
    count_launches(1);
  }
  if (node) {
    node->logits = SavedVariable(x, false);
    node->start = SavedVariable(a, false);
    node->end = SavedVariable(b, false);
    node->stats = SavedVariable(stats, false);
    torch::autograd::set_history(loss, node);
  }
  return loss;
}

at::Tensor attention(const at::Tensor& qkv, int64_t heads, double dropout) {
  BAGUA_CHECK(heads > 0 && qkv.is_cuda() && qkv.dim() == 3 && qkv.scalar_type() == at::kBFloat16 && qkv.size(2) % (3 * heads * 8) == 0,
              Tensor, "attention needs a packed bf16 projection [batch, seq, 3 * heads * dim] with dim a multiple of 8");
  const int64_t B = qkv.size(0), S = qkv.size(1), W = qkv.size(2), D = W / (3 * heads);
  variable_list parts;
  if (watched({&qkv})) {
    const at::Tensor p = qkv.view({B, S, 3, heads, D}).permute({2, 0, 3, 1, 4});
    const at::Tensor a = at::scaled_dot_product_attention(p.select(0, 0), p.select(0, 1), p.select(0, 2), c10::nullopt, dropout);
    return a.transpose(1, 2).reshape({B, S, heads * D});
  }
  std::shared_ptr<SplitHeadsNode> node;
  if (torch::autograd::compute_requires_grad(qkv)) {
    node = std::shared_ptr<SplitHeadsNode>(new SplitHeadsNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(qkv));
  }
  {
    PlainDispatch plain;
    const at::Tensor c = vector_aligned(qkv.contiguous());
    for (int64_t q = 0; q < 3; ++q)
      parts.push_back(c.detach().as_strided({B, heads, S, D}, {S * W, D, W, 1}, c.storage_offset() + q * heads * D));
  }
  if (node) {
    node->batch = B;
    node->seq = S;
    node->heads = heads;
    node->dim = D;
    node->options = qkv.options();
    for (at::Tensor& t : parts) torch::autograd::set_history(t, node);
  }
  const at::Tensor a = at::scaled_dot_product_attention(parts[0], parts[1], parts[2], c10::nullopt, dropout);
  if (node) a.register_hook([](const at::Tensor& g) { return vector_aligned(g); });
  return a.transpose(1, 2).reshape({B, S, heads * D});
}

}  // namespace trainer
}  // namespace bagua
