// A few host threads that copy memory: one thread moves 13 GB/s from pageable to pinned memory on
// the machines measured, eight reach 100 GB/s, twice what the link to the GPU takes.
//
// The threads are started on first use and stay: starting eight threads per call cost 150 us.
// Between jobs they spin for a moment (a prediction comes with a job every few hundred
// microseconds) and then sleep.  One job runs at a time; a caller that finds the pool busy, or that
// is a forked child (which has no such threads), does its job alone.
#pragma once

#include <pthread.h>
#include <signal.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstddef>
#include <mutex>
#include <thread>
#include <vector>

namespace b2fil {

// Size of a pinned buffer for `bytes`: the next power of two up to a megabyte, then the next of four steps
// to the next power of two.
inline size_t pinned_size(size_t bytes)
{
  size_t power = size_t(64) << 10;
  while (power < bytes) power *= 2;
  if (power <= (size_t(1) << 20)) return power;
  const size_t step = power / 8;  // a quarter of the power of two below
  return (bytes + step - 1) / step * step;
}

class CopyPool {
 public:
  // The process-wide pool with `threads` threads, the caller's included (first call decides).
  static CopyPool& get(int threads)
  {
    static CopyPool* pool = new CopyPool(threads);  // its threads end with the process
    return *pool;
  }

  // fn(i) for every i in [0, n), on the pool's threads and the caller's; returns when all are done.
  template <typename F>
  void run(size_t n, F&& fn)
  {
    run(n, fn, [] { return true; });
  }
  // The same, and the caller calls watch() after each of its items and, when no item is left, until
  // it returns true: it can act on what the others have finished.
  template <typename F, typename W>
  void run(size_t n, F&& fn, W&& watch)
  {
    std::unique_lock<std::mutex> job(job_mu_, std::try_to_lock);
    if (n <= 1 || !job.owns_lock() || workers_ == 0 || forked()) {
      for (size_t i = 0; i < n; ++i) {
        fn(i);
        watch();
      }
      while (!watch()) relax();
      return;
    }
    call_ = [](void* f, size_t i) { (*static_cast<std::remove_reference_t<F>*>(f))(i); };
    arg_  = const_cast<void*>(static_cast<const void*>(&fn));
    n_    = n;
    next_.store(0);
    open_.store(true);
    generation_.fetch_add(1);
    // (a short job is done before a sleeping thread would be there)
    if (n > 8 && sleepers_.load() > 0) {
      std::lock_guard<std::mutex> lock(sleep_mu_);
      wake_.notify_all();
    }
    for (size_t i; (i = next_.fetch_add(1)) < n_;) {
      fn(i);
      watch();
    }
    while (!watch()) relax();
    // a worker that enters from here on finds the job closed; those inside are finishing
    open_.store(false);
    while (inside_.load() != 0) relax();
  }

 private:
  explicit CopyPool(int threads)
  {
    pthread_atfork(nullptr, nullptr, [] { forked_flag().store(true); });
    // signals are for the threads of the program
    sigset_t all, before;
    sigfillset(&all);
    pthread_sigmask(SIG_SETMASK, &all, &before);
    try {
      for (int i = 1; i < threads; ++i) {
        std::thread(&CopyPool::work, this).detach();
        ++workers_;
      }
    } catch (const std::exception&) {
      // fewer threads then
    }
    pthread_sigmask(SIG_SETMASK, &before, nullptr);
  }
  static std::atomic<bool>& forked_flag()
  {
    static std::atomic<bool> flag{false};
    return flag;
  }
  static bool forked() { return forked_flag().load(std::memory_order_relaxed); }
  static void relax()
  {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
  }
  void take_items()
  {
    for (size_t i; (i = next_.fetch_add(1)) < n_;) call_(arg_, i);
  }
  void work()
  {
    using clock   = std::chrono::steady_clock;
    uint64_t seen = 0;
    for (;;) {
      const auto until = clock::now() + std::chrono::microseconds(200);
      while (generation_.load() == seen) {
        for (int i = 0; i < 32 && generation_.load() == seen; ++i) relax();
        if (clock::now() < until) continue;
        std::unique_lock<std::mutex> lock(sleep_mu_);
        sleepers_.fetch_add(1);
        wake_.wait(lock, [&] { return generation_.load() != seen; });
        sleepers_.fetch_sub(1);
      }
      seen = generation_.load();
      inside_.fetch_add(1);
      if (open_.load()) take_items();
      inside_.fetch_sub(1);
    }
  }

  int workers_ = 0;
  std::mutex job_mu_, sleep_mu_;
  std::condition_variable wake_;
  std::atomic<uint64_t> generation_{0};
  std::atomic<size_t> next_{0};
  std::atomic<int> inside_{0}, sleepers_{0};
  std::atomic<bool> open_{false};
  // the job: written while no worker is inside, read by workers that found it open
  void (*call_)(void*, size_t) = nullptr;
  void* arg_                   = nullptr;
  size_t n_                    = 0;
};

}  // namespace b2fil
