// The communication backend: ordered-bucket scheduler, worker thread and watchdog.
//
// Reference: BaguaCommBackend (bagua-core-internal/src/lib.rs:125-337).
//   * `register_ordered_buckets` fixes the order in which buckets are communicated.
//   * `mark_communication_ready(tensor, event)` marks a tensor; while the FRONT bucket
//     of the queue is fully ready it is rotated to the back and scheduled.  Only the
//     front is ever tested, so every rank issues buckets in the registered order no
//     matter in which order gradients arrive.
//   * scheduling = pushing {bucket, snapshot of its ops, completion event} into a
//     bounded channel (back-pressure) consumed by ONE worker thread, which runs the ops.
//   * `wait_pending_comm_ops` blocks until every scheduled bucket has been executed by
//     the worker and returns how many there were.
//   * a watchdog thread reports a bucket whose ops do not finish within the timeout
//     (reference: 300 s, then panic).  Here the timeout is configurable and the failure
//     is delivered as an exception from `wait_pending_comm_ops` rather than by exiting.
//
// Differences on purpose: a bucket whose tensors are all padding is rejected at
// registration (the reference would spin forever on it); op errors are caught on the
// worker and re-raised to the caller of `wait_pending_comm_ops`.
#pragma once

#include <deque>
#include <thread>
#include <unordered_map>
#include <unordered_set>

#include "../ops/comm_op.h"
#include "../tensor/tensor.h"
#include "channel.h"

namespace bagua {

struct ScheduledCommOp {
  std::string name;
  BucketPtr bucket;
  std::vector<std::shared_ptr<CommOp>> ops;
  EventChannel event{"comm_op"};
  // How the bucket's tensors lay when it was registered; null: it shared memory with another.
  std::shared_ptr<const BucketLayout> layout;
  int64_t staging_bytes = 0;  // of a batch that it is executed in
  // Whether it may be executed together with others.
  // (asked for every bucket on the worker, so with one pass over its tensors)
  bool joins() const { return layout && ops.size() == 1 && ops[0]->joins(*bucket, *layout) && bucket->lies_as(*layout); }
};

class CommBackend {
 public:
  // device_id < 0: host-only backend (no CUDA calls).
  CommBackend(size_t schedule_channel_cap, int device_id);
  ~CommBackend();
  CommBackend(const CommBackend&) = delete;

  void register_ordered_buckets(const std::vector<BucketPtr>& buckets);
  void mark_communication_ready(const TensorPtr& tensor, uint64_t ready_cuda_event);
  // The same without ever blocking: false when there is a bucket to schedule (or another thread holds the
  // scheduler), and schedule_ready() is still to be called.
  bool try_mark_ready(const TensorPtr& tensor, uint64_t ready_cuda_event);
  void schedule_ready();
  size_t wait_pending_comm_ops();

  // seconds; <= 0 disables the watchdog.  Default: BAGUA_B200_WATCHDOG_S or 300.
  void set_watchdog_timeout(double seconds) { watchdog_s_.store(seconds); }
  double watchdog_timeout() const { return watchdog_s_.load(); }
  int device_id() const { return device_id_; }
  size_t pending() const { return not_waited_.size(); }

 private:
  bool should_schedule() const;
  void schedule_comm(const BucketPtr& bucket);
  void worker_loop();
  // Runs the ops of `batch`, of one bucket or of several that are executed together (`joined`: as such, also if there is one).
  void execute(const std::vector<std::shared_ptr<ScheduledCommOp>>& batch, bool joined);
  // Adds to `batch` what is scheduled behind it and can be executed with it; what was received and cannot stays in `next_`.
  void join_followers(std::vector<std::shared_ptr<ScheduledCommOp>>& batch);
  void monitor_loop();

  const int device_id_;
  std::deque<BucketPtr> ordered_buckets_;
  std::unordered_map<const BaguaBucket*, std::shared_ptr<const BucketLayout>> layouts_;  // of those that share no memory with others
  int64_t staging_bytes_ = 0;  // what those of them that are staged take, at most kJoinedBytes
  std::mutex mu_;  // guards ordered_buckets_ and registration state

  Channel<std::shared_ptr<ScheduledCommOp>> schedule_;
  Channel<EventChannel> not_waited_;
  // Buckets that become ready faster than the GPU takes them one by one are handed over together: one that finds the GPU busy with
  // earlier ones for longer than a launch takes to reach it (kJoinAheadUs) waits for more, unless somebody waits for the buckets.  How
  // long the GPU is busy is reckoned: 8 us for what is quantised, 6 for what is copied, and 4 us for every 10 MB (quantised twice: 12.3 us
  // for one bucket of 10 MB, 16.4 for two, 24.5 for four).  Bursts over one rank, us, alone / together: 13 fp32 buckets of 8 MB quantised 164 / 125, 7 staged bf16
  // ones of 7 MB quantised 186 / 124, 7 staged fp16 ones copied 102 / 89, 3 staged fp32 ones of 8 MB, which come too slowly, 54-66 both.
  // Ahead by 12 us: 126, 141, 98; waiting until the GPU is done: 13 buckets 122, but 3 quantised ones 50 / 55.  Ahead by 8 us and with 8 us
  // for copies too, as it was while the worker took longer to hand over, / as here: 13 buckets 127 / 121, 7 staged bf16 ones 134 / 115, 22
  // staged fp16 ones of 2 MB 249 / 243, 3 staged fp32 ones of 8 MB 46 / 47; with 8 us for copies 52.
  // A joined launch waits for the youngest of its buckets' gradients.  Training steps over one rank, quantised, us, alone / together, in
  // two runs each: VGG-16 at batch 32 4609-4642 / 4585-4613, at batch 8 with buckets of 5 MB 2508-2543 / 2488-2490, MLPs of 6 layers
  // of width 4096 1584-1594 / 1582-1590, of 2048 870-880 / 830-881: buckets that come 40 us apart are not joined.
  static constexpr int64_t kJoinBytesPerUs = 2500000, kJoinAheadUs = 6, kJoinMostUs = 40;
  std::shared_ptr<ScheduledCommOp> next_;                // worker only
  std::chrono::steady_clock::time_point busy_until_{};   // worker only: the GPU, as reckoned
  std::atomic<int> waiters_{0};                                 // threads in wait_pending_comm_ops()
  // What the worker is executing, for the watchdog, which looks at it now and then: a message per bucket would
  // wake it twice for each.
  struct Current {
    std::mutex mu;
    std::condition_variable stop_cv;
    std::vector<BucketPtr> buckets;  // empty: nothing
    std::chrono::steady_clock::time_point since;
    bool reported = false, stop = false;
  } current_;
  std::atomic<double> watchdog_s_;
  std::mutex err_mu_;
  std::string watchdog_error_;
  std::thread worker_, monitor_thread_;
};

}  // namespace bagua
