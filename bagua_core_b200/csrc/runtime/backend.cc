#include "backend.h"

#include <algorithm>

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include "../telemetry/telemetry.h"

namespace bagua {

CommBackend::CommBackend(size_t cap, int device_id)
    : device_id_(device_id), schedule_(cap == 0 ? 1 : cap), not_waited_(0),
      watchdog_s_(env_double("BAGUA_B200_WATCHDOG_S", 300.0)) {
  if (device_id_ >= 0) BAGUA_CUDA_CHECK(cudaSetDevice(device_id_));
  Telemetry::instance().init_from_env_once();
  worker_ = std::thread([this] { worker_loop(); });
  monitor_thread_ = std::thread([this] { monitor_loop(); });
}

CommBackend::~CommBackend() {
  schedule_.close();
  {
    std::lock_guard<std::mutex> g(current_.mu);
    current_.stop = true;
  }
  current_.stop_cv.notify_all();
  if (worker_.joinable()) worker_.join();
  if (monitor_thread_.joinable()) monitor_thread_.join();
}

void CommBackend::worker_loop() {
  if (device_id_ >= 0) {
    cudaError_t e = cudaSetDevice(device_id_);
    if (e != cudaSuccess) BAGUA_LOG(Error, "comm worker cannot select device " << device_id_);
  }
  std::vector<std::shared_ptr<ScheduledCommOp>> batch;
  for (;;) {
    batch.clear();
    if (next_) {
      batch.push_back(std::move(next_));
      next_.reset();
    } else {
      auto item = schedule_.recv(kSpinUs);
      if (!item) return;
      batch.push_back(std::move(*item));
    }
    const bool joinable = batch[0]->joins();
    if (joinable) join_followers(batch);
    execute(batch, joinable);
    if (!joinable) continue;
    int64_t bytes = 0;
    for (auto& item : batch) bytes += item->layout->bytes;
    busy_until_ = std::max(busy_until_, std::chrono::steady_clock::now()) +
                  std::chrono::microseconds(batch[0]->ops[0]->joined_base_us() + bytes / kJoinBytesPerUs);
  }
}

void CommBackend::join_followers(std::vector<std::shared_ptr<ScheduledCommOp>>& batch) {
  const auto now = std::chrono::steady_clock::now();
  const auto until = std::min(busy_until_ - std::chrono::microseconds(kJoinAheadUs), now + std::chrono::microseconds(kJoinMostUs));
  int64_t staged = batch[0]->layout->staged_bytes();
  while (batch.size() < (size_t)kernels::kMaxJoined) {
    std::optional<std::shared_ptr<ScheduledCommOp>> item;
    spin_until(
        [&] {
          return (item = schedule_.try_recv()) || waiters_.load(std::memory_order_acquire) > 0 ||
                 std::chrono::steady_clock::now() >= until;
        },
        (int)kJoinMostUs);
    if (!item && !(item = schedule_.try_recv())) break;  // (what was sent before the waiter came)
    const ScheduledCommOp& op = **item;
    bool joins = op.joins() && batch[0]->ops[0]->joins_with(*op.ops[0]) && op.bucket->dtype() == batch[0]->bucket->dtype();
    for (auto& b : batch) joins = joins && b->bucket != op.bucket;  // twice in a row is one after the other
    if (joins) joins = (staged += op.layout->staged_bytes()) <= batch[0]->staging_bytes;
    if (!joins) {
      next_ = std::move(*item);
      break;
    }
    batch.push_back(std::move(*item));
  }
}

namespace {
std::string names_of(const std::vector<BucketPtr>& buckets) {
  std::string s = buckets.size() > 1 ? "buckets " : "bucket ";
  for (size_t k = 0; k < buckets.size(); ++k) s += (k ? ", `" : "`") + buckets[k]->name() + "`";
  return s;
}
}  // namespace

void CommBackend::execute(const std::vector<std::shared_ptr<ScheduledCommOp>>& batch, bool joined) {
  for (auto& item : batch) {
    BAGUA_LOG(Debug, "worker received scheduled communication operation " << item->name);
    if (log_enabled(LogLevel::Debug)) {
      std::string names;
      for (auto& t : item->bucket->tensors()) names += (names.empty() ? "" : ",") + t->name();
      BAGUA_LOG(Debug, "executing communication op `" << item->name << "` on bucket `" << item->bucket->name()
                                                      << "`, tensors [" << names << "]");
    }
  }
  const ScheduledCommOp& op = *batch[0];
  const std::vector<BucketPtr>& buckets = current_.buckets;  // which only this thread writes
  {
    std::lock_guard<std::mutex> g(current_.mu);
    for (auto& item : batch) current_.buckets.push_back(item->bucket);
    current_.since = std::chrono::steady_clock::now();
    current_.reported = false;
  }
  const uint64_t t0 = Telemetry::instance().now();
  std::string err;
  JoinedFailures failed;
  // Optional NVTX range per bucket or joined batch (BAGUA_B200_NVTX=1) so that profiler timelines line up
  // with bucket names; a no-op when no tool is attached.
  static const bool nvtx = env_long("BAGUA_B200_NVTX", 0) != 0;
  if (nvtx) nvtxRangePushA(batch.size() > 1 ? names_of(buckets).c_str() : op.bucket->name().c_str());
  try {
    if (joined) {
      failed = op.ops[0]->execute_joined(buckets, op.staging_bytes);
      EngineStats::global().ops_executed += batch.size() - failed.size();
      for (auto& [k, why] : failed)
        BAGUA_LOG(Error, "communication op on bucket `" << buckets[k]->name() << "` failed: " << why);
    } else {
      for (auto& o : op.ops) {
        o->execute_background_communication(op.bucket);
        EngineStats::global().ops_executed++;
      }
    }
  } catch (const std::exception& e) {
    err = e.what();
    BAGUA_LOG(Error, "communication op on " << names_of(buckets) << " failed: " << err);
  }
  if (nvtx) nvtxRangePop();
  for (auto& item : batch) Telemetry::instance().record("bucket_executed", item->bucket->name(), t0);
  {
    std::lock_guard<std::mutex> g(current_.mu);
    current_.buckets.clear();
  }
  for (size_t k = 0; k < batch.size(); ++k) {
    const std::string* why = err.empty() ? nullptr : &err;
    for (auto& f : failed)
      if (f.first == k) why = &f.second;
    if (!why)
      batch[k]->event.finish();
    else
      batch[k]->event.fail(*why);
    BAGUA_LOG(Debug, "comm op executed: " << batch[k]->name);
  }
}

void CommBackend::monitor_loop() {
  std::unique_lock<std::mutex> lk(current_.mu);
  while (!current_.stop) {
    const double limit = watchdog_s_.load();
    // often enough to report within a tenth of the limit, at most ten times a second
    const double look = limit <= 0 ? 0.1 : std::min(0.1, std::max(0.005, limit / 10));
    current_.stop_cv.wait_for(lk, std::chrono::duration<double>(look), [&] { return current_.stop; });
    if (current_.stop || current_.buckets.empty() || current_.reported || limit <= 0) continue;
    const std::chrono::duration<double> running = std::chrono::steady_clock::now() - current_.since;
    if (running.count() < limit) continue;
    // reported once; the op may still complete, the error goes to the next waiter
    current_.reported = true;
    const std::string what = names_of(current_.buckets) + " comm op has not finished for " + fmt_double(limit) + " s";
    BAGUA_LOG(Error, what);
    std::lock_guard<std::mutex> g(err_mu_);
    if (watchdog_error_.empty()) watchdog_error_ = what;
  }
}

void CommBackend::register_ordered_buckets(const std::vector<BucketPtr>& buckets) {
  wait_pending_comm_ops();
  std::lock_guard<std::mutex> g(mu_);
  ordered_buckets_.clear();
  layouts_.clear();
  std::unordered_set<std::string> names;
  std::unordered_set<uint64_t> ptrs;
  for (auto& b : buckets) {
    BAGUA_CHECK(!b->all_padding(), Bucket,
                "bucket `" << b->name() << "` contains only padding tensors and would always be ready");
    for (auto& t : b->tensors()) {
      const uint64_t p = t->data_ptr();
      if (names.count(t->name()) || ptrs.count(p)) {
        ordered_buckets_.clear();
        throw BaguaError(ErrorKind::Tensor,
                         "duplicated tensor detected, name " + t->name() + ", ptr " + std::to_string(p));
      }
      names.insert(t->name());
      ptrs.insert(p);
    }
    ordered_buckets_.push_back(b);
  }
  // Tensors may overlap without starting at one address (views).  By their starts, one that overlaps any in front of it overlaps the
  // one of them that ends last.
  struct Span {
    uint64_t from, to;
    const BaguaBucket* bucket;
  };
  std::vector<Span> spans;
  for (auto& b : buckets) {
    auto layout = std::make_shared<const BucketLayout>(b->layout());
    for (auto& [from, to] : layout->spans)
      if (from < to) spans.push_back({from, to, b.get()});
    layouts_[b.get()] = std::move(layout);
  }
  std::sort(spans.begin(), spans.end(), [](const Span& a, const Span& b) { return a.from < b.from; });
  for (size_t k = 1, last = 0; k < spans.size(); ++k) {
    if (spans[k].from < spans[last].to && spans[k].bucket != spans[last].bucket) {
      layouts_.erase(spans[k].bucket);
      layouts_.erase(spans[last].bucket);
    }
    if (spans[k].to > spans[last].to) last = k;
  }
  staging_bytes_ = 0;
  for (auto& [bucket, layout] : layouts_)
    if (layout->bytes <= kJoinedBytes) staging_bytes_ += layout->staged_bytes();
  staging_bytes_ = std::min(staging_bytes_, kJoinedBytes);
}

bool CommBackend::should_schedule() const {
  if (ordered_buckets_.empty()) throw BaguaError(ErrorKind::Backend, "ordered buckets not yet set in comm backend");
  return ordered_buckets_.front()->ready_for_comm();
}

void CommBackend::schedule_comm(const BucketPtr& bucket) {
  auto op = std::make_shared<ScheduledCommOp>();
  op->name = bucket->name();
  op->bucket = bucket;
  op->ops = bucket->ops_snapshot();
  if (auto it = layouts_.find(bucket.get()); it != layouts_.end()) op->layout = it->second;
  op->staging_bytes = staging_bytes_;
  EventChannel ev = op->event;
  const uint64_t t0 = Telemetry::instance().now();
  if (!schedule_.send(std::move(op))) throw BaguaError(ErrorKind::InternalChannel, "schedule channel is closed");
  not_waited_.send(ev);
  EngineStats::global().buckets_scheduled++;
  Telemetry::instance().record("bucket_scheduled", bucket->name(), t0);
}

void CommBackend::mark_communication_ready(const TensorPtr& tensor, uint64_t ready_cuda_event) {
  const uint64_t t0 = Telemetry::instance().now();
  tensor->mark_comm_ready(ready_cuda_event);
  schedule_ready();
  Telemetry::instance().record("tensor_ready", tensor->name(), t0);
}

bool CommBackend::try_mark_ready(const TensorPtr& tensor, uint64_t ready_cuda_event) {
  const uint64_t t0 = Telemetry::instance().now();
  tensor->mark_comm_ready(ready_cuda_event);
  Telemetry::instance().record("tensor_ready", tensor->name(), t0);
  std::unique_lock<std::mutex> g(mu_, std::try_to_lock);
  return g.owns_lock() && !should_schedule();
}

void CommBackend::schedule_ready() {
  std::lock_guard<std::mutex> g(mu_);
  while (should_schedule()) {
    BucketPtr bucket = ordered_buckets_.front();
    ordered_buckets_.pop_front();
    BAGUA_LOG(Debug, "bucket " << bucket->name() << " ready for communication");
    bucket->reset_comm_ready();
    ordered_buckets_.push_back(bucket);
    schedule_comm(bucket);
  }
}

size_t CommBackend::wait_pending_comm_ops() {
  size_t n = 0;
  std::string first_error;
  struct Waiting {
    std::atomic<int>& n;
    explicit Waiting(std::atomic<int>& n) : n(n) { ++n; }
    ~Waiting() { --n; }
  } waiting(waiters_);
  for (;;) {
    auto ev = not_waited_.try_recv();
    if (!ev) break;
    // Poll so that a watchdog report reaches the caller even if the op never returns.
    while (!ev->wait_for(std::chrono::milliseconds(200))) {
      std::lock_guard<std::mutex> g(err_mu_);
      if (!watchdog_error_.empty()) {
        std::string w = watchdog_error_;
        watchdog_error_.clear();
        // the op is still running: a later wait must still see how it ended
        not_waited_.send(*ev);
        throw BaguaError(ErrorKind::Backend, "watchdog: " + w);
      }
    }
    std::string err = ev->wait();
    if (!err.empty() && first_error.empty()) first_error = err;
    ++n;
  }
  {
    std::lock_guard<std::mutex> g(err_mu_);
    if (first_error.empty() && !watchdog_error_.empty()) first_error = "watchdog: " + watchdog_error_;
    watchdog_error_.clear();
  }
  if (!first_error.empty()) throw BaguaError(ErrorKind::Backend, "communication failed: " + first_error);
  // Every bucket has been queued; kernels of earlier buckets (or steps) may have given up on a
  // peer in the meantime.  Their status records are host-mapped, so looking costs a few loads.
  if (device_id_ >= 0) SingleCommunicator::check_all_device_status();
  return n;
}

}  // namespace bagua
