// Thread-safe channels used by the scheduler.
//
//  * `EventChannel` — one-shot completion flag handed out per scheduled bucket
//    (reference: bagua-core-internal/src/events.rs:5-31).  The wait loops on a
//    predicate, so a spurious wake-up cannot release a waiter early (the reference
//    tests the flag with a single `if`).
//  * `Channel<T>`   — MPMC queue, optionally bounded.  A bounded channel blocks the
//    sender when full, which is how back-pressure reaches `mark_communication_ready`
//    (reference: flume::bounded in bagua-core-internal/src/lib.rs:84-100).
#pragma once

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <optional>

#include "../common.h"

namespace bagua {

// Looks at `pred` for up to `us` microseconds before the caller goes to sleep on a condition variable.  Waking a
// sleeping thread costs both sides a system call and the sleeper a scheduling delay (10-50 us on the virtual
// machines this runs on); the buckets of a backward pass follow each other faster than that.
template <typename P>
inline bool spin_until(P pred, int us) {
  if (pred()) return true;
  const auto end = std::chrono::steady_clock::now() + std::chrono::microseconds(us);
  do {
    for (int i = 0; i < 32; ++i) {
      if (pred()) return true;
#if defined(__x86_64__)
      __builtin_ia32_pause();
#endif
    }
  } while (std::chrono::steady_clock::now() < end);
  return pred();
}
constexpr int kSpinUs = 50;

class EventChannel {
 public:
  explicit EventChannel(std::string name) : state_(std::make_shared<State>()) { state_->name = std::move(name); }

  void finish() const {
    {
      std::lock_guard<std::mutex> g(state_->mu);
      state_->finished = true;
      state_->seen.store(true, std::memory_order_release);
    }
    state_->cv.notify_all();
  }
  void fail(const std::string& err) const {
    {
      std::lock_guard<std::mutex> g(state_->mu);
      state_->error = err;
      state_->finished = true;
      state_->seen.store(true, std::memory_order_release);
    }
    state_->cv.notify_all();
  }
  // Blocks until finish()/fail(); returns the error text ("" when none).
  std::string wait() const {
    spin_until([this] { return state_->seen.load(std::memory_order_acquire); }, kSpinUs);
    std::unique_lock<std::mutex> lk(state_->mu);
    state_->cv.wait(lk, [&] { return state_->finished; });
    return state_->error;
  }
  // Returns false on timeout.
  bool wait_for(std::chrono::milliseconds d) const {
    spin_until([this] { return state_->seen.load(std::memory_order_acquire); }, kSpinUs);
    std::unique_lock<std::mutex> lk(state_->mu);
    return state_->cv.wait_for(lk, d, [&] { return state_->finished; });
  }
  bool finished() const {
    std::lock_guard<std::mutex> g(state_->mu);
    return state_->finished;
  }
  const std::string& name() const { return state_->name; }

 private:
  struct State {
    std::string name;
    std::mutex mu;
    std::condition_variable cv;
    bool finished = false;
    std::atomic<bool> seen{false};  // finished, for those who look without the lock
    std::string error;
  };
  std::shared_ptr<State> state_;
};

template <typename T>
class Channel {
 public:
  // cap == 0 → unbounded
  explicit Channel(size_t cap = 0) : cap_(cap) {}

  // Blocks while full.  Returns false if the channel was closed.
  bool send(T v) {
    std::unique_lock<std::mutex> lk(mu_);
    not_full_.wait(lk, [&] { return closed_ || cap_ == 0 || q_.size() < cap_; });
    if (closed_) return false;
    q_.push_back(std::move(v));
    size_.store(q_.size(), std::memory_order_release);
    lk.unlock();
    not_empty_.notify_one();
    return true;
  }
  // Blocks while empty, after looking for `spin_us` without sleeping.  nullopt once closed and drained.
  std::optional<T> recv(int spin_us = 0) {
    if (spin_us > 0) spin_until([this] { return size_.load(std::memory_order_acquire) > 0; }, spin_us);
    std::unique_lock<std::mutex> lk(mu_);
    not_empty_.wait(lk, [&] { return closed_ || !q_.empty(); });
    if (q_.empty()) return std::nullopt;
    T v = std::move(q_.front());
    q_.pop_front();
    size_.store(q_.size(), std::memory_order_release);
    lk.unlock();
    not_full_.notify_one();
    return v;
  }
  std::optional<T> try_recv() {
    if (size_.load(std::memory_order_acquire) == 0) return std::nullopt;  // without the lock, for those who poll
    std::unique_lock<std::mutex> lk(mu_);
    if (q_.empty()) return std::nullopt;
    T v = std::move(q_.front());
    q_.pop_front();
    size_.store(q_.size(), std::memory_order_release);
    lk.unlock();
    not_full_.notify_one();
    return v;
  }
  void close() {
    {
      std::lock_guard<std::mutex> g(mu_);
      closed_ = true;
    }
    not_empty_.notify_all();
    not_full_.notify_all();
  }
  size_t size() const {
    std::lock_guard<std::mutex> g(mu_);
    return q_.size();
  }
  size_t capacity() const { return cap_; }

 private:
  const size_t cap_;
  mutable std::mutex mu_;
  std::condition_variable not_empty_, not_full_;
  std::deque<T> q_;
  std::atomic<size_t> size_{0};
  bool closed_ = false;
};

}  // namespace bagua
