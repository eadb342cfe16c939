// Host worker threads for the library's FP64 set-up loops (model
// coefficients, validity checks, copies).
//
// Starting a std::thread costs tens of microseconds on the Grace host, so a
// parallel loop that spawned 16 threads spent about 1 ms on that alone; the
// set-up of a 1040 x 540 electromag2 model runs five such loops.  The pool
// starts its workers once per process and wakes them per loop.
//
// One loop runs at a time (callers from several host threads take turns);
// a task must not start a loop of its own.  A process forked after the
// workers started gets a fresh pool on its first loop.
#pragma once

#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

namespace sfd {

class HostPool {
 public:
  static constexpr unsigned kMaxThreads = 16;

  // The process's pool (created on first use, or anew in a forked child).
  static HostPool& get() {
    static std::mutex create_m;
    static HostPool* pool = nullptr;
    std::lock_guard<std::mutex> g(create_m);
    if (!pool || pool->pid_ != getpid()) pool = new HostPool();  // a forked child's copy is left unused
    return *pool;
  }

  // Threads that run(): the workers plus the caller.
  unsigned size() const { return (unsigned)workers_.size() + 1; }

  // task(0) .. task(ntasks - 1), on the workers and the calling thread.
  void run(int ntasks, const std::function<void(int)>& task) {
    std::lock_guard<std::mutex> one_at_a_time(run_m_);
    {
      std::lock_guard<std::mutex> lk(m_);
      task_ = &task;
      ntasks_ = ntasks;
      next_.store(0);
      ++gen_;
    }
    cv_work_.notify_all();
    for (int i; (i = next_.fetch_add(1)) < ntasks;) task(i);
    std::unique_lock<std::mutex> lk(m_);
    cv_done_.wait(lk, [&] { return active_ == 0; });
    task_ = nullptr;  // a worker that wakes later finds no loop to join
  }

 private:
  HostPool() : pid_(getpid()) {
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    const unsigned n = std::min(kMaxThreads, hw) - 1;
    for (unsigned t = 0; t < n; ++t) workers_.emplace_back([this] { work(); });
    for (auto& w : workers_) w.detach();  // the pool lives until the process exits
  }

  void work() {
    uint64_t seen = 0;
    std::unique_lock<std::mutex> lk(m_);
    for (;;) {
      cv_work_.wait(lk, [&] { return gen_ != seen; });
      seen = gen_;
      if (!task_) continue;
      const std::function<void(int)>* task = task_;
      const int n = ntasks_;
      ++active_;
      lk.unlock();
      for (int i; (i = next_.fetch_add(1)) < n;) (*task)(i);
      lk.lock();
      if (--active_ == 0) cv_done_.notify_all();
    }
  }

  const pid_t pid_;
  std::vector<std::thread> workers_;
  std::mutex run_m_, m_;
  std::condition_variable cv_work_, cv_done_;
  const std::function<void(int)>* task_ = nullptr;
  int ntasks_ = 0;
  std::atomic<int> next_{0};
  int active_ = 0;
  uint64_t gen_ = 0;
};

// f(begin, end) over [0, n) in contiguous chunks on the host pool, each
// with at least `grain` items (the calling thread alone for small n).  The
// model set-up's FP64 loops and copies run this way: a 1040 x 540
// electromag2 model is 27 MB of input planes.  Chunks of 8192 cells: of 32768,
// a 440 x 240 model ran on three threads (its set-up 1.1 against 0.66 ms, the
// gradient's chain rule 1.5 against 0.45 ms; of 2048 0.62 and 0.38).
constexpr size_t kHostGrain = 1u << 13;
// Values that are only copied or looked at: a 120 x 90 model's six planes (64,800
// values) took 70 us longer on seven threads than on one.
constexpr size_t kCopyGrain = 1u << 15;
template <class F>
void parallel_for(size_t n, const F& f, size_t grain = kCopyGrain) {
  const size_t want = std::max<size_t>(1, n / std::max<size_t>(1, grain));
  if (want <= 1) {
    f((size_t)0, n);
    return;
  }
  HostPool& pool = HostPool::get();
  const size_t nt = std::min<size_t>(pool.size(), want);
  const size_t chunk = (n + nt - 1) / nt;
  pool.run((int)nt, [&](int t) {
    const size_t b = std::min(n, (size_t)t * chunk), e = std::min(n, b + chunk);
    if (b < e) f(b, e);
  });
}

// rows [0, nrows) of `ncols` values each, split between threads by whole rows
template <class F>
void parallel_rows(int nrows, int ncols, const F& row) {
  parallel_for((size_t)nrows, [&](size_t b, size_t e) {
    for (size_t k = b; k < e; ++k) row((int)k);
  }, std::max<size_t>(1, kHostGrain / (size_t)std::max(1, ncols)));
}

}  // namespace sfd
