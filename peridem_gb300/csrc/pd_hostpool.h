// pd_hostpool.h -- host threads shared by all handles for the engine's parallel host loops. Starting
// a thread costs ~30 us on the GPU machine's Arm cores, a dozen loops of a small handle's creation or
// of a state read start up to 15 each; the pool's threads sleep between loops and end after two idle
// seconds.
#ifndef PD_HOSTPOOL_H
#define PD_HOSTPOOL_H

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <exception>
#include <functional>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace pdg {

class HostPool {
 public:
  static constexpr unsigned kMax = 31;  // threads beside the callers

  // The process's pool: never destroyed (its threads may outlive static destruction), and another one
  // in a forked child, which has none of the parent's threads and must not touch locks they may hold.
  static HostPool &get() {
    static std::atomic<HostPool *> pool(nullptr);
    HostPool *p = pool.load();
    while (!p || p->pid_ != getpid()) {
      HostPool *fresh = new HostPool;
      if (pool.compare_exchange_strong(p, fresh)) return *fresh;
      delete fresh;  // another thread made it; p is its pool now
    }
    return *p;
  }

  // Calls work(0) here and work(1) .. work(helpers) on pool threads as far as they are free, and
  // returns when every call that began has returned (work shares its items out itself, so it does
  // not matter how many helpers come). Several threads may call at once. The first exception of
  // a call is rethrown here.
  void run(unsigned helpers, const std::function<void(unsigned)> &work) {
    Job job{&work, std::min(helpers, kMax)};
    bool posted = false;
    if (job.wanted) {
      std::unique_lock<std::mutex> lk(mu_);
      jobs_.push_back(&job);
      posted = true;
      for (unsigned need = job.wanted; need > idle_ && threads_ < kMax; --need) {
        try {
          std::thread([this] { loop(); }).detach();
        } catch (const std::system_error &) {
          break;  // no more threads: the callers do the work
        }
        ++threads_;
      }
      wake_.notify_all();
    }
    std::exception_ptr first;
    try {
      work(0);
    } catch (...) {
      first = std::current_exception();
    }
    if (posted) {
      std::unique_lock<std::mutex> lk(mu_);
      jobs_.erase(std::find(jobs_.begin(), jobs_.end(), &job));
      done_.wait(lk, [&] { return job.running == 0; });
      if (!first) first = job.error;
    }
    if (first) std::rethrow_exception(first);
  }

 private:
  struct Job {
    const std::function<void(unsigned)> *work;
    unsigned wanted, entered = 0, running = 0;
    std::exception_ptr error;
  };

  void loop() {
    std::unique_lock<std::mutex> lk(mu_);
    for (;;) {
      Job *job = nullptr;
      for (Job *j : jobs_)
        if (j->entered < j->wanted) {
          job = j;
          break;
        }
      if (!job) {
        ++idle_;
        const bool woken = wake_.wait_for(lk, std::chrono::seconds(2)) == std::cv_status::no_timeout;
        --idle_;
        if (woken || !jobs_.empty()) continue;
        --threads_;
        return;
      }
      const unsigned slot = ++job->entered;
      ++job->running;
      lk.unlock();
      std::exception_ptr e;
      try {
        (*job->work)(slot);
      } catch (...) {
        e = std::current_exception();
      }
      lk.lock();
      if (e && !job->error) job->error = e;
      if (--job->running == 0) done_.notify_all();
    }
  }

  std::mutex mu_;
  std::condition_variable wake_, done_;
  std::vector<Job *> jobs_;
  unsigned threads_ = 0, idle_ = 0;
  const pid_t pid_ = getpid();
};

// Threads a loop of n items is spread over (the caller among them).
inline unsigned host_width(uint64_t n) {
  const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
  return (unsigned)std::min<uint64_t>(std::min(hw, HostPool::kMax + 1), n);
}

// Runs f(i, slot) for i in [0, n) on up to `width` threads, work handed out one index at a time; slot <
// max(width, 1) tells the threads apart. (The width is the caller's: the number of online cores, and
// with it host_width, may change from one call to the next.)
template <class F>
void parallel_slots(uint64_t n, unsigned width, F f) {
  const unsigned T = (unsigned)std::min<uint64_t>(std::min(width, HostPool::kMax + 1), n);
  if (T <= 1) {
    for (uint64_t i = 0; i < n; ++i) f(i, 0u);
    return;
  }
  std::atomic<uint64_t> next(0);
  HostPool::get().run(T - 1, [&](unsigned slot) {
    for (uint64_t i = next++; i < n; i = next++) f(i, slot);
  });
}

// Runs f(i) for i in [0, n) on the host's cores.
template <class F>
void parallel_items(uint64_t n, F f) {
  parallel_slots(n, host_width(n), [&](uint64_t i, unsigned) { f(i); });
}

}  // namespace pdg
#endif
