// gtk_crew.hpp -- a few helper threads for host work that one core is slow at: gathering strings that lie all over
// the heap (one core copies them at 9 GB/s, the host link carries 55), and decoding.
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace gtk {

// Belongs to one handle: started at the first large job, joined with the handle.  One job at a time; whoever finds the
// crew busy (decoding may run on several threads) does the work alone.
class Crew {
 public:
  static constexpr int kHelpers = 3;

  ~Crew()
  {
    {
      std::lock_guard<std::mutex> lock(mu_);
      stop_ = true;
    }
    wake_.notify_all();
    for (std::thread& t : threads_) t.join();
  }

  // Blocks 0 .. n-1 of a job, handed out in order to the helpers and to whoever waits for one.
  class Job {
   public:
    Job(Crew& crew, int64_t n, std::function<void(int64_t)> work) : crew_(crew), n_(n), work_(std::move(work)), done_(new std::atomic<bool>[size_t(n)])
    {
      for (int64_t i = 0; i < n; ++i) done_[size_t(i)].store(false, std::memory_order_relaxed);
      helped_ = n > 1 && crew_.begin(this);
    }
    ~Job()
    {
      if (helped_) crew_.end();
    }
    Job(const Job&) = delete;
    Job& operator=(const Job&) = delete;

    // returns when blocks 0 .. i are done
    void wait(int64_t i)
    {
      for (; seen_ <= i; ++seen_)
        while (!done_[size_t(seen_)].load(std::memory_order_acquire))
          if (!step()) std::this_thread::yield();  // a helper is at it
    }
    void finish() { wait(n_ - 1); }

   private:
    friend class Crew;
    bool step()  // false: nothing left to take
    {
      const int64_t i = next_.fetch_add(1, std::memory_order_relaxed);
      if (i >= n_) return false;
      work_(i);
      done_[size_t(i)].store(true, std::memory_order_release);
      return true;
    }
    Crew& crew_;
    const int64_t n_;
    std::function<void(int64_t)> work_;
    std::unique_ptr<std::atomic<bool>[]> done_;
    std::atomic<int64_t> next_{0};
    int64_t seen_ = 0;
    bool helped_  = false;
  };

 private:
  bool begin(Job* job)
  {
    if (!turn_.try_lock()) return false;
    std::lock_guard<std::mutex> lock(mu_);
    const int want = std::min<int>(kHelpers, int(std::thread::hardware_concurrency()) - 1);
    try {
      while (int(threads_.size()) < want) threads_.emplace_back([this] { serve(); });
    } catch (const std::system_error&) {  // fewer helpers, or none
    }
    job_ = job;
    ++number_;
    wake_.notify_all();
    return true;
  }
  void end()  // no helper touches the job behind this
  {
    {
      std::unique_lock<std::mutex> lock(mu_);
      job_ = nullptr;
      idle_.wait(lock, [this] { return active_ == 0; });
    }
    turn_.unlock();
  }
  void serve()
  {
    uint64_t seen = 0;
    std::unique_lock<std::mutex> lock(mu_);
    for (;;) {
      wake_.wait(lock, [&] { return stop_ || (job_ != nullptr && number_ != seen); });
      if (stop_) return;
      seen     = number_;
      Job* job = job_;
      ++active_;
      lock.unlock();
      while (job->step()) {
      }
      lock.lock();
      if (--active_ == 0) idle_.notify_all();
    }
  }

  std::mutex turn_;  // one job at a time
  std::mutex mu_;
  std::condition_variable wake_, idle_;
  std::vector<std::thread> threads_;
  Job* job_        = nullptr;
  uint64_t number_ = 0;
  int active_      = 0;
  bool stop_       = false;
};

}  // namespace gtk
