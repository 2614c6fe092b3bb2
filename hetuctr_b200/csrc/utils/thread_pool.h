// Single-queue worker pool behind async_preprocess / async_push_pull: tasks run in submission order
// on `n` threads (the table uses n = 1, so asynchronous calls keep program order).
// Same role as the reference's ThreadPool (csrc/utils/thread_pool.h:16-50).
#pragma once
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <functional>
#include <future>
#include <mutex>
#include <thread>
#include <vector>

#include "utils/spin.h"

namespace hetuCTR {

// Waits for the result of a queued call, awake for the time a step takes; rethrows a failure of the call.
inline void wait_awake(std::future<void> &f) {
  spin_for(1000, queue_workers() + 1, [&] { return f.wait_for(std::chrono::seconds(0)) == std::future_status::ready; });
  f.get();
}

class ThreadPool {
 public:
  explicit ThreadPool(size_t n) {
    queue_workers() += (int)n;
    for (size_t i = 0; i < n; i++) workers_.emplace_back([this] { run(); });
  }
  ~ThreadPool() {
    {
      std::lock_guard<std::mutex> g(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto &t : workers_) t.join();
    queue_workers() -= (int)workers_.size();
  }
  std::future<void> Enqueue(std::function<void()> fn) {
    std::packaged_task<void()> task(std::move(fn));
    std::future<void> f = task.get_future();
    {
      std::lock_guard<std::mutex> g(mu_);
      if (stop_) throw std::runtime_error("enqueue on stopped ThreadPool");
      queue_.emplace_back(std::move(task));
      queued_.store(queue_.size(), std::memory_order_release);
    }
    cv_.notify_one();
    return f;
  }

 private:
  void run() {
    for (;;) {
      std::packaged_task<void()> task;
      // a step's calls follow each other within tens of microseconds
      spin_for(100, queue_workers() + 1, [&] { return queued_.load(std::memory_order_acquire) != 0; });
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [this] { return stop_ || !queue_.empty(); });
        if (queue_.empty()) return;
        task = std::move(queue_.front());
        queue_.pop_front();
        queued_.store(queue_.size(), std::memory_order_release);
      }
      task();
    }
  }
  std::mutex mu_;
  std::condition_variable cv_;
  std::deque<std::packaged_task<void()>> queue_;
  std::vector<std::thread> workers_;
  std::atomic<size_t> queued_{0};  // size of queue_, readable without the lock
  bool stop_ = false;
};

}  // namespace hetuCTR
