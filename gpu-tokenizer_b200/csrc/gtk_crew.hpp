// gtk_crew.hpp -- a few helper threads for host work that one core is slow at: gathering strings that lie all over
// the heap (one core copies them at 9 GB/s, the host link carries 55), and decoding.
#pragma once
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace gtk {

// Belongs to one handle: started at the first large job, joined with the handle.  One job at a time; whoever finds the
// crew busy (decoding may run on several threads) does the work alone.
//
// A forked child has the memory of the helpers but not the threads, and whatever lock was held at the fork stays held: it
// neither joins nor touches the team that it has inherited (which is never freed there), and starts one of its own for its first job.
class Crew {
 public:
  static constexpr int kHelpers = 3;

  ~Crew()
  {
    Team* team = team_.load(std::memory_order_acquire);
    if (!team || team->pid != getpid()) return;
    {
      std::lock_guard<std::mutex> lock(team->mu);
      team->stop = true;
    }
    team->wake.notify_all();
    for (std::thread& t : team->threads) t.join();
    delete team;
  }

 private:
  struct Team;

 public:
  // Blocks 0 .. n-1 of a job, handed out in order to the helpers and to whoever waits for one.  The work must not throw (it may
  // run on a helper, where nobody catches): it works in memory that it is given.
  class Job {
   public:
    Job(Crew& crew, int64_t n, std::function<void(int64_t)> work) : n_(n), work_(std::move(work)), done_(new std::atomic<bool>[size_t(n)])
    {
      for (int64_t i = 0; i < n; ++i) done_[size_t(i)].store(false, std::memory_order_relaxed);
      if (n > 1) team_ = crew.begin(this);
    }
    ~Job()
    {
      if (team_) end(*team_);
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
    const int64_t n_;
    std::function<void(int64_t)> work_;
    std::unique_ptr<std::atomic<bool>[]> done_;
    std::atomic<int64_t> next_{0};
    int64_t seen_ = 0;
    Team* team_   = nullptr;  // that helps
  };

 private:
  struct Team {
    const pid_t pid = getpid();  // of the process whose threads they are
    std::mutex turn;             // one job at a time
    std::mutex mu;
    std::condition_variable wake, idle;
    std::vector<std::thread> threads;
    Job* job        = nullptr;
    uint64_t number = 0;
    int active      = 0;
    bool stop       = false;
  };

  Team* team()
  {
    Team* t = team_.load(std::memory_order_acquire);
    while (!t || t->pid != getpid()) {
      std::unique_ptr<Team> fresh(new Team);
      if (team_.compare_exchange_strong(t, fresh.get(), std::memory_order_acq_rel)) return fresh.release();
    }
    return t;
  }
  Team* begin(Job* job)  // nullptr: busy
  {
    Team* const t = team();
    if (!t->turn.try_lock()) return nullptr;
    std::lock_guard<std::mutex> lock(t->mu);
    const int want = std::min<int>(kHelpers, int(std::thread::hardware_concurrency()) - 1);
    try {
      while (int(t->threads.size()) < want) t->threads.emplace_back([t] { serve(*t); });
    } catch (...) {  // no thread or no memory for one: fewer helpers, or none
    }
    t->job = job;
    ++t->number;
    t->wake.notify_all();
    return t;
  }
  static void end(Team& t)  // no helper touches the job behind this
  {
    {
      std::unique_lock<std::mutex> lock(t.mu);
      t.job = nullptr;
      t.idle.wait(lock, [&t] { return t.active == 0; });
    }
    t.turn.unlock();
  }
  static void serve(Team& t)
  {
    uint64_t seen = 0;
    std::unique_lock<std::mutex> lock(t.mu);
    for (;;) {
      t.wake.wait(lock, [&] { return t.stop || (t.job != nullptr && t.number != seen); });
      if (t.stop) return;
      seen     = t.number;
      Job* job = t.job;
      ++t.active;
      lock.unlock();
      while (job->step()) {
      }
      lock.lock();
      if (--t.active == 0) t.idle.notify_all();
    }
  }

  std::atomic<Team*> team_{nullptr};
};

}  // namespace gtk
