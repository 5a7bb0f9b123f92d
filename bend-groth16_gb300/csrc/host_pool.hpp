// A process-wide pool of host worker threads for the serial host steps of an MSM that split
// into independent pieces (the per-window part sums of msm_finish).  parallel_for runs
// f(0..n-1) on the pool's idle workers and on the calling thread, so it completes even when
// every worker is busy with another caller's work; calls from several threads (batch lanes,
// the serving loop) interleave freely.
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <deque>
#include <exception>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace bg {

class HostPool {
 public:
  // the shared pool: min(hardware threads - 1, 7) workers, created on first use
  static HostPool& get() {
    static HostPool pool(std::min(7u, std::max(1u, std::thread::hardware_concurrency()) - 1u));
    return pool;
  }

  unsigned workers() const { return (unsigned)threads_.size(); }

  // f(0..n-1), begun on idle workers while the caller goes on; wait() runs what no worker has taken
  // and returns when all are done.  The handle waits when it goes out of scope.
  class Task;
  Task start(int n, std::function<void(int)> f);

  void parallel_for(int n, const std::function<void(int)>& f) {
    if (n <= 0) return;
    if (n == 1 || workers() == 0) {
      for (int i = 0; i < n; i++) f(i);
      return;
    }
    auto job = std::make_shared<Job>();
    job->n = n;
    job->f = f;
    submit(job, std::min<unsigned>(workers(), (unsigned)n - 1u));
    job->finish();
  }

  ~HostPool() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : threads_) t.join();
  }

 private:
  struct Job {
    int n = 0;
    std::function<void(int)> f;
    std::atomic<int> next{0};
    int done = 0;  // indices finished (guarded by mu)
    std::exception_ptr error;
    std::mutex mu;
    std::condition_variable cv;
    void run() {
      int mine = 0;
      std::exception_ptr err;
      for (int i; (i = next.fetch_add(1)) < n; mine++) {
        try {
          if (!err) f(i);
        } catch (...) {
          err = std::current_exception();
        }
      }
      if (mine == 0) return;
      std::lock_guard<std::mutex> lk(mu);
      if (err && !error) error = err;
      done += mine;
      if (done == n) cv.notify_all();
    }
    // Waits for the indices that helpers took, not for the helpers: one that wakes after the last
    // index is taken (tens of microseconds later, longer than a small MSM's whole window sum) finds
    // none left.
    void finish() {
      run();
      std::unique_lock<std::mutex> lk(mu);
      cv.wait(lk, [&] { return done == n; });
      if (error) std::rethrow_exception(error);
    }
  };
  void submit(const std::shared_ptr<Job>& job, unsigned helpers) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      for (unsigned h = 0; h < helpers; h++) queue_.push_back(job);
    }
    if (helpers == 1) cv_.notify_one();
    else cv_.notify_all();
  }

  explicit HostPool(unsigned n) {
    for (unsigned i = 0; i < n; i++) threads_.emplace_back([this] { loop(); });
  }

  void loop() {
    for (;;) {
      std::shared_ptr<Job> job;
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return stop_ || !queue_.empty(); });
        if (stop_ && queue_.empty()) return;
        job = queue_.front();
        queue_.pop_front();
      }
      job->run();
    }
  }

  std::vector<std::thread> threads_;
  std::deque<std::shared_ptr<Job>> queue_;
  std::mutex mu_;
  std::condition_variable cv_;
  bool stop_ = false;
};

class HostPool::Task {
 public:
  Task() = default;
  explicit Task(std::shared_ptr<Job> j) : job_(std::move(j)) {}
  Task(Task&&) = default;
  Task& operator=(Task&&) = default;
  void wait() {
    if (!job_) return;
    const std::shared_ptr<Job> j = std::move(job_);
    j->finish();
  }
  ~Task() {
    try {
      wait();  // what it runs refers to the caller's frame
    } catch (...) {
    }
  }

 private:
  std::shared_ptr<Job> job_;
};

inline HostPool::Task HostPool::start(int n, std::function<void(int)> f) {
  auto job = std::make_shared<Job>();
  job->n = n;
  job->f = std::move(f);
  submit(job, std::min<unsigned>(workers(), (unsigned)n));
  return Task(job);
}

}  // namespace bg
