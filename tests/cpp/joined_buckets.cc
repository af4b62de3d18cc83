// Buckets that the engine hands to the GPU together (a communicator of one rank), without a GPU: the engine's own sources run
// over a stand-in for the CUDA runtime and for the kernels, in which device memory is host memory and a launch does its work
// at once.  The first bucket of a burst is held inside its launch until the others are scheduled, so that those are joined.
//
//   failing   a bucket that cannot be prepared fails alone
//   watchdog  a launch that does not return is reported under the names of all its buckets
//   locks     backends that hold the same buckets in opposite orders do not wait for each other
//   most      a launch has 16 buckets at most, none of them twice
//   staging   buckets that are staged together take one block from the pool, whichever of them meet
//   overlap   buckets that share memory, or whose tensors have moved to where they do, get what they get one after the other
#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <thread>

#include "comm/arena.h"
#include "comm/communicator.h"
#include "kernels/kernels_impl.h"
#include "ops/comm_op.h"
#include "pool/resource_pool.h"
#include "runtime/backend.h"

using namespace bagua;

namespace {
int failures = 0;
#define EXPECT(cond, ...)                             \
  do {                                                \
    if (!(cond)) {                                    \
      std::fprintf(stderr, "line %d: ", __LINE__);    \
      std::fprintf(stderr, __VA_ARGS__);              \
      std::fprintf(stderr, "\n");                     \
      ++failures;                                     \
    }                                                 \
  } while (0)

// ---- a launch that is held --------------------------------------------------------------------------
struct Gate {
  std::mutex mu;
  std::condition_variable cv;
  bool closed = false, reached = false, let_one = false;
  void close() {
    std::lock_guard<std::mutex> g(mu);
    closed = true;
    reached = false;
  }
  void pass() {
    std::unique_lock<std::mutex> lk(mu);
    reached = true;
    cv.notify_all();
    cv.wait(lk, [&] { return !closed || let_one; });
    if (let_one) reached = let_one = false;
  }
  void pass_one() {
    std::lock_guard<std::mutex> g(mu);
    let_one = true;
    reached = false;
    cv.notify_all();
  }
  void wait_reached() {
    std::unique_lock<std::mutex> lk(mu);
    cv.wait(lk, [&] { return reached; });
  }
  void open() {
    std::lock_guard<std::mutex> g(mu);
    closed = false;
    cv.notify_all();
  }
} gate;
std::mutex launches_mu;
std::vector<int> quantise_launches;  // buffers of each
}  // namespace

// ---- the stand-in for the CUDA runtime ----------------------------------------------------------------
extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
const cudaEvent_t kNoEvent = (cudaEvent_t)(uintptr_t)0xbad;
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t e, unsigned) { return e == kNoEvent ? cudaErrorInvalidResourceHandle : cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "no such event"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

// ---- a communicator of one rank, and the kernels -------------------------------------------------------
namespace bagua {
PeerArena::~PeerArena() {}
SingleCommunicator::SingleCommunicator(int rank, int nranks, int device_id, uint64_t stream, const std::string&)
    : rank_(rank), nranks_(nranks), device_id_(device_id), stream_(stream) {}
SingleCommunicator::~SingleCommunicator() {}
void SingleCommunicator::check_all_device_status() {}
std::shared_ptr<Communicator> Communicator::create(SingleCommPtr internode, SingleCommPtr, bool) {
  auto c = std::make_shared<Communicator>();
  c->internode_ = std::move(internode);
  return c;
}
uint64_t Communicator::stream() const { return internode_->stream(); }
void Communicator::execute_communication(RawTensor& t, bool, bool, bool, const std::function<void(SingleCommunicator&, RawTensor&)>& hook) {
  hook(*internode_, t);
}
namespace kernels {
namespace cuda {
void multi_copy_joined(const MultiCopyItem* items, int count, bool gather, cudaStream_t) {
  for (int k = 0; k < count; ++k)
    for (int s = 0; s < items[k].nseg; ++s) {
      const MultiCopySeg& sg = items[k].segs[s];
      char* flat = (char*)items[k].flat + sg.offset;
      std::memcpy(gather ? flat : (char*)sg.ptr, gather ? (char*)sg.ptr : flat, sg.bytes);
    }
}
void multi_copy(const MultiCopySeg* segs, int nseg, void* flat, size_t bytes, bool gather, cudaStream_t s) {
  const MultiCopyItem one{segs, nseg, flat, bytes};
  multi_copy_joined(&one, 1, gather, s);
}
size_t quantise_twice_scratch_bytes(const QuantiseItem*, int count, DType) { return 32 * (size_t)count; }
// x -> 2 x + 1 stands for the work: twice on the same values is not once.  All buffers of a launch are read before any is written.
void quantise_twice_minmax_u8(const QuantiseItem* items, int count, DType, void*, size_t, cudaStream_t) {
  gate.pass();
  {
    std::lock_guard<std::mutex> g(launches_mu);
    quantise_launches.push_back(count);
  }
  std::vector<std::vector<float>> read;
  for (int k = 0; k < count; ++k) read.emplace_back((float*)items[k].x, (float*)items[k].x + items[k].n);
  for (int k = 0; k < count; ++k)
    for (int64_t i = 0; i < items[k].n; ++i) ((float*)items[k].x)[i] = 2 * read[k][i] + 1;
}
}  // namespace cuda
}  // namespace kernels
}  // namespace bagua

namespace {
struct View : RawTensor {
  View(float* p, int64_t n) : p(p), n(n) {}
  void* data_ptr() const override { return p; }
  int64_t num_elements() const override { return n; }
  int64_t num_elements_allocated() const override { return n; }
  int device_id() const override { return 0; }
  DType dtype() const override { return DType::F32; }
  float* p;
  int64_t n;
};

std::shared_ptr<Communicator> one_rank(uint64_t stream) {
  return Communicator::create(std::make_shared<SingleCommunicator>(0, 1, 0, stream, "solo"), nullptr, false);
}

using Spans = std::vector<std::pair<float*, int64_t>>;
BucketPtr make_bucket(const std::string& name, const Spans& spans, const std::shared_ptr<CommOp>& op) {
  std::vector<TensorPtr> ts;
  for (auto& [p, n] : spans) ts.push_back(std::make_shared<BaguaTensor>(name + "_" + std::to_string(ts.size()), std::make_shared<View>(p, n)));
  auto b = std::make_shared<BaguaBucket>(name, ts);
  b->append_op(op);
  return b;
}
void mark(CommBackend& backend, const BucketPtr& b) {
  for (auto& t : b->tensors()) backend.mark_communication_ready(t, 0);
}
// The buckets in their order, the first held until the last is scheduled.
void burst(CommBackend& backend, const std::vector<BucketPtr>& buckets, const std::function<void()>& while_held = {},
           bool open = true) {
  gate.close();
  mark(backend, buckets[0]);
  gate.wait_reached();
  for (size_t k = 1; k < buckets.size(); ++k) mark(backend, buckets[k]);
  if (while_held) while_held();
  if (open) gate.open();
}

void overlap() {
  std::vector<float> x(1000), y(1000), first(16);
  auto op = make_centralized_low_precision_op(one_rank(1), true, "MinMaxUInt8");
  // b shares part of a's memory behind its first element, c none; d is staged, and one of its tensors lies in c's
  CommBackend backend(100, 0);
  const std::vector<BucketPtr> buckets = {make_bucket("first", {{first.data(), 16}}, op), make_bucket("a", {{x.data(), 600}}, op),
                                          make_bucket("b", {{x.data() + 400, 600}}, op), make_bucket("c", {{y.data(), 500}}, op),
                                          make_bucket("d", {{y.data() + 600, 100}, {y.data() + 450, 20}}, op)};
  backend.register_ordered_buckets(buckets);
  burst(backend, buckets);
  EXPECT(backend.wait_pending_comm_ops() == 5, "five buckets");
  for (int i = 0; i < 1000; ++i) {
    const float wx = i >= 400 && i < 600 ? 3 : 1, wy = i >= 450 && i < 470 ? 3 : i < 500 || (i >= 600 && i < 700) ? 1 : 0;
    if (x[i] != wx || y[i] != wy) {
      EXPECT(false, "value %d is %g / %g, not %g / %g", i, x[i], y[i], wx, wy);
      break;
    }
  }
  // c's tensor moves to where a is
  dynamic_cast<View&>(*buckets[3]->tensors()[0]->raw()).p = x.data();
  std::fill(x.begin(), x.end(), 0.f);
  burst(backend, buckets);
  backend.wait_pending_comm_ops();
  for (int i = 0; i < 1000; ++i) {
    const float want = i < 400 ? 3 : i < 500 ? 7 : i < 600 ? 3 : 1;
    if (x[i] != want) {
      EXPECT(false, "moved: value %d is %g, not %g", i, x[i], want);
      break;
    }
  }
}

// Two backends, the same buckets in opposite orders: a launch that waits for several buckets' locks takes them in one order.  (A deadlock
// shows as a test that does not end, and ThreadSanitizer reports two orders that only might have met.)
void locks() {
  std::vector<float> x(64), held(32);
  auto op = make_centralized_low_precision_op(one_rank(1), true, "MinMaxUInt8");
  std::vector<BucketPtr> buckets;
  for (int k = 0; k < 4; ++k) buckets.push_back(make_bucket("b" + std::to_string(k), {{x.data() + 16 * k, 16}}, op));
  for (int turn = 0; turn < 2; ++turn) {
    CommBackend backend(100, 0);
    std::vector<BucketPtr> order = buckets;
    if (turn) std::reverse(order.begin(), order.end());
    order.insert(order.begin(), make_bucket("held", {{held.data() + 16 * turn, 16}}, op));
    backend.register_ordered_buckets(order);
    burst(backend, order);
    EXPECT(backend.wait_pending_comm_ops() == 5, "five buckets");
  }
  EXPECT(quantise_launches == (std::vector<int>{1, 4, 1, 4}), "the four were not joined");
  for (float v : x) EXPECT(v == 3, "%g", v);
}

std::string error_of_wait(CommBackend& backend) {
  try {
    backend.wait_pending_comm_ops();
  } catch (const std::exception& e) {
    return e.what();
  }
  return "";
}

void failing() {
  for (const bool staged : {false, true}) {
    std::vector<float> x(6 * 16), held(16);
    auto op = make_centralized_low_precision_op(one_rank(1), true, "MinMaxUInt8");
    CommBackend backend(100, 0);
    std::vector<BucketPtr> buckets = {make_bucket("held", {{held.data(), 16}}, op)};
    for (int k = 0; k < 6; ++k) {
      float* at = x.data() + 16 * k;
      buckets.push_back(make_bucket("b" + std::to_string(k), staged ? Spans{{at, 4}, {at + 8, 8}} : Spans{{at, 16}}, op));
    }
    backend.register_ordered_buckets(buckets);
    quantise_launches.clear();
    gate.close();
    mark(backend, buckets[0]);
    gate.wait_reached();
    for (size_t k = 1; k < buckets.size(); ++k)
      for (auto& t : buckets[k]->tensors()) backend.mark_communication_ready(t, k == 3 ? (uint64_t)(uintptr_t)kNoEvent : 0);
    gate.open();
    const std::string error = error_of_wait(backend);
    EXPECT(error.find("no such event") != std::string::npos, "the error was: %s", error.c_str());
    EXPECT(quantise_launches == (std::vector<int>{1, 5}), "the other five were not worked on together");
    for (int i = 0; i < 96; ++i) {
      const float want = i / 16 == 2 || (staged && i % 16 >= 4 && i % 16 < 8) ? 0 : 1;
      if (x[(size_t)i] != want) {
        EXPECT(false, "value %d is %g", i, x[(size_t)i]);
        break;
      }
    }
    // and the next time it is a bucket like the others
    burst(backend, buckets);
    EXPECT(error_of_wait(backend).empty(), "the second burst failed");
    EXPECT(x[32] == 1 && x[0] == 3, "%g %g", x[32], x[0]);
  }
}

void watchdog() {
  std::vector<float> x(64);
  auto op = make_centralized_low_precision_op(one_rank(1), true, "MinMaxUInt8");
  CommBackend backend(100, 0);
  std::vector<BucketPtr> buckets;
  for (int k = 0; k < 4; ++k) buckets.push_back(make_bucket("b" + std::to_string(k), {{x.data() + 16 * k, 16}}, op));
  backend.register_ordered_buckets(buckets);
  burst(backend, buckets, [] {
    gate.pass_one();
    gate.wait_reached();
  }, /*open=*/false);
  backend.set_watchdog_timeout(0.05);
  const std::string error = error_of_wait(backend);
  EXPECT(error.find("buckets `b1`, `b2`, `b3` comm op has not finished") != std::string::npos, "the report was: %s", error.c_str());
  backend.set_watchdog_timeout(0);
  gate.open();
  error_of_wait(backend);
  for (float v : x) EXPECT(v == 1, "%g", v);
}

// Twelve staged buckets of 6 MB: executed one by one, then in bursts of any length.
void staging() {
  constexpr int64_t kHalf = 3 << 18;  // floats
  constexpr int kBuckets = 12;
  std::vector<float> x((size_t)kBuckets * 2 * (kHalf + 16));
  auto op = make_centralized_low_precision_op(one_rank(1), true, "MinMaxUInt8");
  CommBackend backend(100, 0);
  std::vector<BucketPtr> buckets;
  for (int k = 0; k < kBuckets; ++k) {
    float* at = x.data() + (size_t)k * 2 * (kHalf + 16);
    buckets.push_back(make_bucket("b" + std::to_string(k), {{at, kHalf}, {at + kHalf + 16, kHalf}}, op));
  }
  backend.register_ordered_buckets(buckets);
  const MemoryPool& pool = MemoryPool::for_device(0);
  for (auto& b : buckets) {
    mark(backend, b);
    backend.wait_pending_comm_ops();
  }
  const PoolStats first = pool.stats();
  EXPECT(first.bytes_reserved <= (32 << 20) + kBuckets * 4096, "%llu bytes reserved", (unsigned long long)first.bytes_reserved);
  quantise_launches.clear();
  burst(backend, buckets);
  backend.wait_pending_comm_ops();
  EXPECT(quantise_launches == (std::vector<int>{1, 5, 5, 1}), "five buckets at a time stay below 32 MB");
  for (size_t many = 1; many <= kBuckets; ++many)
    for (size_t from = 0; from < kBuckets; from += many) {
      burst(backend, {buckets.begin() + from, buckets.begin() + std::min<size_t>(from + many, kBuckets)});
      backend.wait_pending_comm_ops();
    }
  EXPECT(pool.stats().device_allocs == first.device_allocs, "%llu allocations, %llu before",
         (unsigned long long)pool.stats().device_allocs, (unsigned long long)first.device_allocs);
  const float want = (float)((1 << (kBuckets + 2)) - 1);
  for (int k = 0; k < kBuckets; ++k)
    for (int64_t i = 0; i < 2 * kHalf + 32; ++i) {
      const bool mine = i < kHalf || (i >= kHalf + 16 && i < 2 * kHalf + 16);
      const float v = x[(size_t)k * 2 * (kHalf + 16) + (size_t)i];
      if (v != (mine ? want : 0.f)) {
        EXPECT(false, "bucket %d, value %lld: %g", k, (long long)i, v);
        return;
      }
    }
}

void most() {
  std::vector<float> x(21 * 16), y(16);
  auto op = make_centralized_low_precision_op(one_rank(1), true, "MinMaxUInt8");
  {
    CommBackend backend(100, 0);
    std::vector<BucketPtr> buckets;
    for (int k = 0; k < 21; ++k) buckets.push_back(make_bucket("b" + std::to_string(k), {{x.data() + 16 * k, 16}}, op));
    backend.register_ordered_buckets(buckets);
    burst(backend, buckets);
    EXPECT(backend.wait_pending_comm_ops() == 21, "21 buckets");
    EXPECT(quantise_launches == (std::vector<int>{1, 16, 4}), "not 16 at a time");
    for (float v : x) EXPECT(v == 1, "%g", v);
  }
  CommBackend backend(100, 0);
  const BucketPtr one = make_bucket("one", {{y.data(), 16}}, op);
  backend.register_ordered_buckets({one});
  quantise_launches.clear();
  burst(backend, {one, one, one});
  EXPECT(backend.wait_pending_comm_ops() == 3, "three times");
  EXPECT(quantise_launches == (std::vector<int>{1, 1, 1}), "joined with itself");
  for (float v : y) EXPECT(v == 7, "%g", v);
}

const std::map<std::string, void (*)()> kCases = {
    {"failing", failing}, {"locks", locks}, {"most", most}, {"overlap", overlap}, {"staging", staging}, {"watchdog", watchdog}};
}  // namespace

int main(int argc, char** argv) {
  if (argc != 2 || !kCases.count(argv[1])) return 2;
  kCases.at(argv[1])();
  std::printf("%s: %d failures\n", argv[1], failures);
  return failures ? 1 : 0;
}
