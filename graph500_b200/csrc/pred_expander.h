// Host threads that expand packed pred entries into int64 ones while they are
// still arriving.  Plain C++: what marks the chunks is known by the marks and by
// a callback that tells its state.
#pragma once

#include <stdint.h>
#ifdef __linux__
#include <sys/prctl.h>
#endif

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "packed_entry.h"

namespace g500 {

// What is known of the work that marks the chunks.
enum class WorkState { running, complete, refused };

inline void cpu_pause() {
#if defined(__x86_64__) || defined(__i386__)
  __builtin_ia32_pause();
#endif
}

// Host threads that expand the chunks: each waits for a chunk's mark and
// expands its slice of it, so one wake-up per run serves every chunk.
class PredExpander {
 public:
  explicit PredExpander(int nthreads, std::chrono::steady_clock::duration give_up = std::chrono::seconds(5))
      : give_up_(give_up) {
    th_.reserve((size_t)nthreads);
    try {
      for (int t = 1; t < nthreads; ++t) th_.emplace_back([this, t] { loop(t); });
    } catch (const std::system_error&) {  // no more threads to be had: those there are do the work
    }
    n_ = (int)th_.size() + 1;  // read by them in a run only
  }
  ~PredExpander() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : th_) t.join();
  }

  // Expand src[0, n) into dst, nchunks chunks of equal length, as run `run` marks
  // them (ready[c] >> 1); state() tells about the work that does.  A mark's low
  // bit says that an entry up to there did not fit: nothing more is expanded, for
  // the caller copies the whole array another way.  False if the work ended
  // without marking them all (nothing is waited for any more then).
  bool run(const uint32_t* src, int64_t* dst, int64_t n, int nchunks, const volatile uint32_t* ready, uint32_t run,
           const std::function<WorkState()>& state) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      src_ = src;
      dst_ = dst;
      nchunks_ = nchunks;
      len_ = n / nchunks_;
      ready_ = ready;
      run_ = run;
      gave_up_.store(false);
      pending_ = n_ - 1;
      ++gen_;
    }
    cv_.notify_all();
    failing_ = false;  // what an earlier run saw says nothing about this one
    work(0, &state);
    std::unique_lock<std::mutex> lk(mu_);
    cv_done_.wait(lk, [&] { return pending_ == 0; });
    return !gave_up_.load();
  }

 private:
  void loop(int t) {
#ifdef __linux__
    prctl(PR_SET_TIMERSLACK, 1000);  // naps of a few microseconds: the default rounds them up by 50
#endif
    uint64_t seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return stop_ || gen_ != seen; });
        if (stop_) return;
        seen = gen_;
      }
      work(t, nullptr);
      {
        std::lock_guard<std::mutex> lk(mu_);
        --pending_;
      }
      cv_done_.notify_one();
    }
  }

  // Thread 0 watches the work: once it has ended, in whatever way, a chunk that
  // is not marked never will be, and every thread gives up.
  // The others poll for SPIN, then give their processor to whoever wants it
  // between looks, and after AWAKE sleep an eighth of what they have waited (at
  // most NAP), so that a long search keeps one processor busy instead of all of
  // the threads'.  Sleeping from the start cost the next chunks' expansion up to
  // a tenth (4 processors, SCALE 22: 1050 -> 1200 us a call); with yields alone the
  // call takes what it took without them, and three processes on 16 processors
  // stand less in each other's way (SCALE 16: 891 -> 884 us, SCALE 20: 1280 -> 1211).
  bool wait_for(int c, const std::function<WorkState()>* state) {
    using clock = std::chrono::steady_clock;
    clock::time_point t0;
    for (uint32_t spins = 1;; ++spins) {
      if ((ready_[c] >> 1) == run_) break;
      if (gave_up_.load(std::memory_order_relaxed)) return false;
      if (state) {
        if ((spins & 0xFFF) == 0 && ended((*state)()) && (ready_[c] >> 1) != run_) {
          gave_up_.store(true);
          return false;
        }
      } else if ((spins & 0x1F) == 0) {
        const auto now = clock::now();
        if (spins == 0x20) t0 = now;
        if (now - t0 > AWAKE) std::this_thread::sleep_for(std::min<clock::duration>((now - t0) / 8, NAP));
        else if (now - t0 > SPIN) std::this_thread::yield();
        if (now - t0 > SPIN) spins = 0x3F;  // look at the mark and the time after each
      }
      cpu_pause();
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return true;
  }

  // The work is over: complete, or its state refused for some seconds (a query
  // may also be refused for a while, as during another thread's capture).
  bool ended(WorkState w) {
    if (w == WorkState::complete) return true;
    if (w == WorkState::running) {
      failing_ = false;
      return false;
    }
    const auto now = std::chrono::steady_clock::now();
    if (!failing_) since_ = now;
    failing_ = true;
    return now - since_ > give_up_;
  }

  void work(int t, const std::function<WorkState()>* state) {
    for (int k = 0; k < nchunks_; ++k) {
      const int64_t b = len_ * k;
      const int64_t lo = b + len_ * t / n_, hi = b + len_ * (t + 1) / n_;
      if (!wait_for(k, state)) return;
      if (ready_[k] & 1u) return;
      const uint32_t* src = src_;
      int64_t* d = dst_;
      for (int64_t i = lo; i < hi; ++i) {
        const uint32_t e = src[i];
        d[i] = e == PACK_NONE ? -1 : (int64_t)(e & PACK_ID) | ((int64_t)(e >> PACK_BITS) << 48);
      }
    }
  }

  static constexpr std::chrono::microseconds SPIN{20}, AWAKE{500}, NAP{200};

  int n_ = 1;
  const std::chrono::steady_clock::duration give_up_;
  bool failing_ = false;  // thread 0 only
  std::chrono::steady_clock::time_point since_;
  std::vector<std::thread> th_;
  std::mutex mu_;
  std::condition_variable cv_, cv_done_;
  std::atomic<bool> gave_up_{false};
  bool stop_ = false;
  uint64_t gen_ = 0;
  int pending_ = 0;
  const uint32_t* src_ = nullptr;
  int64_t* dst_ = nullptr;
  int64_t len_ = 0;
  int nchunks_ = 1;
  const volatile uint32_t* ready_ = nullptr;
  uint32_t run_ = 0;
};

}  // namespace g500
